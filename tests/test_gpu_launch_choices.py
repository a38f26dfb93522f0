"""The choices that a plan makes by batch: narrower tiles for few signals, one thread per 32-point line, launches that
overlap the drain of the one before, host calls cut in chunks; and the native call path against the general one."""
import numpy as np
import pytest

from oracle import fft_oracle as orc
from turbofft_b200 import planner

pytestmark = pytest.mark.gpu

CD = {0: np.complex64, 1: np.complex128}


def _same(torch, a, b):
    return torch.equal(torch.view_as_real(a), torch.view_as_real(b))


# every size with narrower kernels: two launches, and three (complex128 2^20); batches around the 128 and 512 tile limits; the
# next sizes, where one signal has tiles enough
@pytest.mark.parametrize("dtype,logn", [(0, n) for n in range(15, 22)] + [(1, n) for n in range(13, 22)])
@pytest.mark.parametrize("batch", [1, 2, 5, 16, 33])
def test_narrow_tiles_give_the_bits_of_wide_ones(torch_cuda, dtype, logn, batch):
    import turbofft_b200 as tf

    torch = torch_cuda
    if batch << logn > 1 << 22:
        batch = max(1, (1 << 22) >> logn) + 1  # largest batch worth its time, odd
    x = torch.from_numpy(orc.make_input(batch, 1 << logn, CD[dtype], seed=logn + batch)).cuda()
    small = tf.Plan(logn, batch, dtype)
    y = small(x)
    wide = max(batch, min(600, (1 << 25) >> logn))  # enough tiles for the row's own tiles in every launch
    xw = torch.zeros(wide, 1 << logn, dtype=x.dtype, device="cuda")
    xw[:batch] = x
    large = tf.Plan(logn, wide, dtype)
    yw = large(xw)
    assert _same(torch, y, yw[:batch])
    # the plans did run different kernels: the row's own tiles, and in some launch narrower ones
    own = [1 << l.logc for l in planner.launches_of_row(planner.load_params(("float2", "double2")[dtype], "B200")[logn])]
    few, many = ([l["lines_per_tile"] for l in p.info()] for p in (small, large))
    assert many == own
    assert all(f <= o for f, o in zip(few, own)) and (batch > 1 or (few == own) == (logn >= 20 + dtype))
    assert orc.rel_l2(y[-1:].cpu().numpy(), orc.fft_forward(x[-1:].cpu().numpy())) <= orc.tolerance(CD[dtype], logn)


@pytest.mark.parametrize("if_ft", [0, 1])
@pytest.mark.parametrize("batch", [1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 4097])
def test_32_point_lines_at_the_edges_of_a_tile(torch_cuda, batch, if_ft):
    import turbofft_b200 as tf

    torch = torch_cuda
    x_np = orc.make_input(batch, 32, np.complex64, seed=batch)
    x = torch.from_numpy(x_np).cuda()
    guard = torch.full((batch + 2, 32), 7 + 7j, dtype=torch.complex64, device="cuda")
    plan = tf.Plan(5, batch, 0, if_ft=if_ft, thread_bs=2)
    plan(x, guard[1:-1])
    assert orc.rel_l2(guard[1:-1].cpu().numpy(), orc.fft_forward(x_np)) <= orc.tolerance(np.complex64, 5)
    assert bool((guard[[0, -1]] == 7 + 7j).all())  # nothing stored beside the batch
    if if_ft:
        assert plan.ft_status()[0] == 0


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("logn,batch", [(2, 5000), (5, 700), (12, 3), (16, 2), (16, 600), (22, 1)])
def test_a_chain_of_launches_reads_what_the_one_before_wrote(torch_cuda, logn, batch, dtype):
    """Forward and back, in place and out of place, twenty times without a wait in between."""
    import turbofft_b200 as tf

    torch = torch_cuda
    x = torch.from_numpy(orc.make_input(batch, 1 << logn, CD[dtype], seed=3)).cuda()
    fwd, bwd = tf.Plan(logn, batch, dtype), tf.Plan(logn, batch, dtype)
    bwd.set_direction(True, 1.0 / (1 << logn))
    y, z = x.clone(), torch.empty_like(x)
    for _ in range(10):
        fwd(y, z)
        bwd(z, z)
        y.copy_(z)  # a launch of another library between two of ours
    z = y
    for _ in range(10):
        a = fwd(z)
        z = bwd(a)
        del a       # its memory is free for the next call's output
    # forty transforms, each within the tolerance of one
    assert float(torch.linalg.vector_norm(z - x) / torch.linalg.vector_norm(x)) <= 40 * orc.tolerance(CD[dtype], logn)
    # the same steps with a wait after each give the same bits
    y = x.clone()
    for _ in range(20):
        y = fwd(y)
        torch.cuda.synchronize()
        y = bwd(y)
        torch.cuda.synchronize()
    assert _same(torch, y, z)


# 2 MiB chunks: just under and over three of them, a ragged last one, and a call of more than sixteen
@pytest.mark.parametrize("logn,batch", [(10, 767), (10, 768), (10, 769), (12, 1000), (12, 4099), (18, 5)])
def test_host_calls_of_a_few_chunks(torch_cuda, logn, batch):
    import turbofft_b200 as tf

    torch = torch_cuda
    x = torch.from_numpy(orc.make_input(batch, 1 << logn, np.complex64, seed=9)).pin_memory()
    plan = tf.Plan(logn, batch, 0)
    for _ in range(2):
        assert _same(torch, plan.exec_host(x), plan(x.cuda()).cpu())


def test_native_call_path_and_general_one_agree(torch_cuda):
    """Calls that the native path takes, and near ones that it leaves to the general path."""
    import turbofft_b200 as tf

    torch = torch_cuda

    class Sub(torch.Tensor):
        pass

    x = torch.from_numpy(orc.make_input(12, 256, np.complex64, seed=1)).cuda()
    want = torch.fft.fft(x.to(torch.complex128))

    def close(y, w):
        return float(torch.linalg.vector_norm(y.as_subclass(torch.Tensor) - w) / torch.linalg.vector_norm(w)) <= orc.tolerance(np.complex64, 8)

    for _ in range(2):  # the first call makes the plan, the second finds it
        assert close(tf.fft(x), want) and close(tf.fft(x.as_subclass(Sub)), want)
        assert close(tf.fft(x.view(3, 4, 256)), want.view(3, 4, 256))
        assert close(tf.fft(x.t().contiguous().t()), want)           # strided view: copied first
        assert close(tf.fft(x.view(3, 4, 256), dim=1), torch.fft.fft(x.view(3, 4, 256).to(torch.complex128), dim=1))
        assert close(tf.fft(x[0]), want[0]) and close(tf.ifft(tf.fft(x)), x)
        out = torch.empty_like(x)
        assert close(tf.fft(x, out=out), want) and close(out, want)
        odd = torch.empty(12 * 256 + 1, dtype=torch.complex64, device="cuda")[1:].view(12, 256)  # 8 bytes off a 16-byte boundary
        odd.copy_(x)
        assert close(tf.fft(odd), want)
        for norm in ("ortho", "forward"):
            assert close(tf.fft(x, norm=norm), torch.fft.fft(x.to(torch.complex128), norm=norm))
    for bad in (x[:, :255].contiguous(), x.cpu(), x.real.contiguous()):
        with pytest.raises(Exception):
            tf.fft(bad)
    plan = tf.Plan(8, 12, 0)
    for args in ((x[:11].contiguous(),), (x.to(torch.complex128),), (x.cpu(),), (x, torch.empty(3, 256, dtype=x.dtype, device="cuda"))):
        with pytest.raises(ValueError):
            plan(*args)
    assert close(plan(x), want)


@pytest.mark.parametrize("dtype", [0, 1])
def test_status_counts_come_from_the_last_exec(torch_cuda, dtype):
    import turbofft_b200 as tf

    torch = torch_cuda
    x = torch.from_numpy(orc.make_input(96, 4096, CD[dtype], seed=2)).cuda()
    plan = tf.Plan(12, 96, dtype, if_ft=1, if_err=1, thread_bs=4)
    assert plan.ft_status()[:2] == (0, 0)          # before the first exec
    plan.set_ft_params(1e5, 1000.0, 1e-3)
    for _ in range(3):
        plan(x)
        nd, nc, located = plan.ft_status()
        assert nd == nc == sum(k != -1 for k in located) == len(located) > 0
    plan.set_injection(False)
    plan(x)
    assert plan.ft_status()[:2] == (0, 0)


# small tiles (1 to 2 KB, a tile per block): the last count that overlaps the launch before and the first that does not
@pytest.mark.parametrize("dtype,logn,inner", [(0, 3, 32), (0, 4, 4), (0, 6, 4), (0, 8, 1), (1, 4, 4), (1, 5, 1)])
def test_many_small_tiles_along_a_strided_axis(torch_cuda, dtype, logn, inner):
    import turbofft_b200 as tf

    torch = torch_cuda
    n = 1 << logn
    x = torch.from_numpy(orc.make_input(4097 * inner, n, CD[dtype], seed=logn)).cuda().view(4097, n, inner)
    want = torch.fft.fft(x.to(torch.complex128), dim=1)
    few, many = tf.fft(x[:4096], dim=1), tf.fft(x, dim=1)
    assert _same(torch, few, many[:4096])
    assert float(torch.linalg.vector_norm(many - want) / torch.linalg.vector_norm(want)) <= orc.tolerance(CD[dtype], logn)
    # launches of either kind, and of the kernels between, read what the one before wrote
    def step(v):
        v = tf.ifft(tf.fft(v, dim=1), dim=1)
        return tf.fft(v, dim=2, norm="ortho") if inner > 1 else v

    y = z = x
    for _ in range(6):
        y = step(y)
        torch.cuda.synchronize()
    for _ in range(6):
        z = step(z)
    assert _same(torch, y, z)


def _located(batch, lines, tbs, n_blocks):
    """Which tile of each block carries the injected fault, -1 where that tile is beyond the batch."""
    n_tiles = -(-batch // lines)
    return [k if (k := orc.injected_tile_iteration(b, tbs)) <= len(orc.b200_block_tiles(b, n_blocks, n_tiles, tbs)) else -1
            for b in range(n_blocks)]


def _check_32_point_plan(torch, plan, batch, if_err, csum):
    """Output and, with a fault of 1000 in every block, what was located and repaired."""
    x = orc.make_input(batch, 32, np.complex64, seed=batch)
    plan.set_ft_params(1000.0, 1000.0, 1e-3)
    if csum:
        plan.set_correction(True)
    y, ref = plan(torch.from_numpy(x).cuda()).cpu().numpy(), orc.fft_forward(x)
    if csum:
        # y_bad - (sum of y - F(sum of x)): five stages, the sums over two tiles and the subtraction, each rounded at the
        # size of the fault, of which a line of the sum holds the results of two
        assert np.abs(y - ref).max() <= 16 * 2.0**-24 * (1000 + 2 * np.abs(ref).max())
    else:
        assert orc.rel_l2(y, ref) <= orc.tolerance(np.complex64, 5)
    if if_err:
        nd, nc, located = plan.ft_status()
        want = _located(batch, plan.info()[0]["lines_per_tile"], 2, len(located))
        assert located == want and nd == nc == sum(k > 0 for k in want)


FT_MODES = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (1, 1, 1)]


@pytest.mark.parametrize("if_ft,if_err,csum", FT_MODES)
@pytest.mark.parametrize("batch", [1, 33, 200])
def test_a_parameter_file_with_the_row_that_another_replaced(torch_cuda, tmp_path, batch, if_ft, if_err, csum):
    """32-point complex64 lines as four threads of 8 points, the shipped row until one thread took a whole line."""
    import turbofft_b200 as tf

    rows = ["0, " * 10 + "0"] + [f"{n}, 1, {n}, 0, 0, 64, 0, 0, {min(1 << n, 16)}, 0, 0" for n in range(1, 5)]
    path = tmp_path / "param.csv"
    path.write_text("\n".join(rows + ["5, 1, 5, 0, 0, 32, 0, 0, 8, 0, 0"]) + "\n")
    plan = tf.Plan(5, batch, 0, if_ft=if_ft, if_err=if_err, thread_bs=2, param_csv=str(path))
    assert plan.info()[0]["points_per_thread"] == 8 and plan.info()[0]["lines_per_tile"] == 32
    _check_32_point_plan(torch_cuda, plan, batch, if_err, csum)


@pytest.mark.parametrize("if_ft,if_err,csum", FT_MODES)
@pytest.mark.parametrize("batch", [1, 64, 65, 128, 129, 1000])
def test_faults_in_staged_32_point_lines(torch_cuda, batch, if_ft, if_err, csum):
    """The shipped row, one thread per line staged through shared memory: location, repair by recomputing and from the
    checksums."""
    import turbofft_b200 as tf

    plan = tf.Plan(5, batch, 0, if_ft=if_ft, if_err=if_err, thread_bs=2)
    assert plan.info()[0]["points_per_thread"] == 32
    _check_32_point_plan(torch_cuda, plan, batch, if_err, csum)


# lengths with a kernel of half the columns per tile
@pytest.mark.parametrize("dtype,logn", [(0, 8), (0, 9), (0, 10), (1, 6), (1, 7), (1, 8), (1, 9)])
def test_narrow_strided_tiles_give_the_bits_of_wide_ones(torch_cuda, dtype, logn):
    import turbofft_b200 as tf

    torch = torch_cuda
    outer = 1 << 14 >> logn  # 512 tiles and more of 4 columns
    x = torch.from_numpy(orc.make_input(outer * 128, 1 << logn, CD[dtype], seed=logn)).cuda().view(outer, 1 << logn, 128)
    y, y1 = tf.fft(x, dim=1), tf.fft(x[:1], dim=1)
    lines = [tf._plan_cache[("strided", 0, logn, 128, o, dtype, False, 0.0)].info()[0]["lines_per_tile"] for o in (outer, 1)]
    assert lines[1] < lines[0]
    assert _same(torch, y1, y[:1])
    want = torch.fft.fft(x.to(torch.complex128), dim=1)
    assert float(torch.linalg.vector_norm(y - want) / torch.linalg.vector_norm(want)) <= orc.tolerance(CD[dtype], logn)


CHAIN = [(2, 5000), (5, 700), (12, 3), (16, 2), (16, 600), (22, 1)]


def _round_trips(torch, tf, logn, batch, dtype):
    """Plans and a step of launches that each read what the one before wrote, in place and out of place, with another
    library's kernel among them."""
    fwd, bwd = tf.Plan(logn, batch, dtype), tf.Plan(logn, batch, dtype)
    bwd.set_direction(True, 1.0 / (1 << logn))

    def step(y, z):
        fwd(y, z)
        bwd(z, z)
        fwd(z, y)
        z.copy_(y)
        bwd(z, y)

    x = torch.from_numpy(orc.make_input(batch, 1 << logn, CD[dtype], seed=6)).cuda()
    want, z = x.clone(), torch.empty_like(x)
    for _ in range(4):
        step(want, z)
        torch.cuda.synchronize()
    return fwd, bwd, step, x, want


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("logn,batch", CHAIN)
def test_a_captured_chain_of_launches(torch_cuda, logn, batch, dtype):
    """Overlapped launches become programmatic edges of a graph; replayed twice on the same buffers."""
    import turbofft_b200 as tf

    torch = torch_cuda
    _, _, step, x, want = _round_trips(torch, tf, logn, batch, dtype)
    y, z = x.clone(), torch.empty_like(x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step(y, z)
        step(y, z)
    y.copy_(x)
    graph.replay()
    graph.replay()
    assert _same(torch, y, want)


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("logn,batch", CHAIN)
def test_a_chain_of_launches_across_two_streams(torch_cuda, logn, batch, dtype):
    """An event between two streams orders the whole of what an exec wrote, not only the blocks that had started."""
    import turbofft_b200 as tf

    torch = torch_cuda
    _, _, step, x, want = _round_trips(torch, tf, logn, batch, dtype)
    streams = [torch.cuda.Stream() for _ in range(2)]
    y, z = x.clone(), torch.empty_like(x)
    streams[0].wait_stream(torch.cuda.current_stream())
    for i in range(4):
        with torch.cuda.stream(streams[i % 2]):
            step(y, z)
        streams[1 - i % 2].wait_stream(streams[i % 2])
    torch.cuda.synchronize()
    assert _same(torch, y, want)
