"""What the Python entry points owe their callers whatever the tensor, stream or thread: lazily conjugated inputs,
calls of one shape from several streams and threads, errors of the kind torch raises."""
import numpy as np
import pytest

from oracle import fft_oracle as orc

pytestmark = pytest.mark.gpu

CD = {0: np.complex64, 1: np.complex128}


def _same(torch, a, b):
    return torch.equal(torch.view_as_real(a), torch.view_as_real(b))


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("lazy", ["conj", "neg"])
def test_lazy_conjugate_and_negative_bits_are_applied(torch_cuda, dtype, lazy):
    """x.conj() is a contiguous view of x's own memory: every entry point has to transform its value, not its memory."""
    import turbofft_b200 as tf
    from turbofft_b200.multi_gpu import DeviceBackend, SingleProcessFourStep

    torch = torch_cuda
    x = torch.from_numpy(orc.make_input(16, 256, CD[dtype], seed=5)).cuda()
    view = x.conj() if lazy == "conj" else torch._neg_view(x)
    value = view.clone().resolve_conj().resolve_neg()
    assert (view.is_conj() or view.is_neg()) and view.data_ptr() == x.data_ptr()
    plan = tf.Plan(8, 16, dtype)
    for _ in range(2):  # the first call of a shape makes its plan, the second finds it
        assert _same(torch, tf.fft(view), tf.fft(value))
        assert _same(torch, tf.ifft(view), tf.ifft(value))
        assert _same(torch, tf.fft(view, dim=0), tf.fft(value, dim=0))
        assert _same(torch, tf.fft2(view), tf.fft2(value))
        assert _same(torch, plan(view), plan(value))
    host, host_view = value.cpu(), (x.cpu().conj() if lazy == "conj" else torch._neg_view(x.cpu()))
    assert _same(torch, plan.exec_host(host_view), plan.exec_host(host))
    # a result cannot be stored through such a view, and a call that returns early cannot make a copy of its input
    out = torch.empty_like(value)
    make = torch.Tensor.conj if lazy == "conj" else torch._neg_view
    bad, bad_host = make(out), make(torch.empty_like(host))
    for call in (lambda: tf.fft(value, out=bad), lambda: plan(value, bad), lambda: plan.exec_host(host, bad_host),
                 lambda: plan.exec_host_async(host_view, torch.empty_like(host))):
        with pytest.raises(ValueError):
            call()
    be = DeviceBackend(dtype, 0)
    assert _same(torch, be.permute102(view.reshape(-1), 4, 4, 256), be.permute102(value.reshape(-1), 4, 4, 256))
    two = SingleProcessFourStep(12, dtype, [0, 0])  # one device twice
    got, want = two(list(view.reshape(2, -1))), two(list(value.reshape(2, -1)))
    assert all(_same(torch, a, b) for a, b in zip(got, want))
    two.close()


# two launches, three launches (complex128 2^20), with and without FT; kernels long enough to overlap
SHARED = [(0, 16, 64, False, False), (1, 17, 32, False, False), (0, 22, 4, False, False), (0, 18, 32, True, False),
          (1, 20, 4, True, True)]


def _shared_plans(tf, logn):
    return [p for k, p in tf._plan_cache.items() if k[0] != "strided" and k[1] == logn]


@pytest.mark.parametrize("dtype,logn,batch,ft,err", SHARED)
def test_calls_of_one_shape_share_nothing(torch_cuda, dtype, logn, batch, ft, err):
    """Calls of one shape on several streams and from several threads overlap; the cached plan they share has no
    buffer of its own that they could overwrite for each other."""
    import threading

    import turbofft_b200 as tf

    torch = torch_cuda
    xs = [torch.from_numpy(orc.make_input(batch, 1 << logn, CD[dtype], seed=s)).cuda() for s in range(3)]
    call = lambda x: tf.fft(x, ft=ft, err=err)  # noqa: E731
    call(xs[0])
    size = (batch << logn) * (8 << dtype)
    assert all(p.workspace_bytes < size for p in _shared_plans(tf, logn))
    want = []
    for x in xs:
        want.append(call(x))
        torch.cuda.synchronize()
    # one thread, a stream per input
    streams = [torch.cuda.Stream() for _ in xs]
    got = [[] for _ in xs]
    for _ in range(6):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(call(xs[i]))
    torch.cuda.synchronize()
    assert all(_same(torch, y, want[i]) for i in range(3) for y in got[i])
    # a thread per input, all on one stream and then each on its own
    for own_stream in (False, True):
        got = [[] for _ in xs]

        def work(i):
            with torch.cuda.stream(streams[i if own_stream else 0]):
                for _ in range(10):
                    got[i].append(call(xs[i]))

        threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
        [t.start() for t in threads]
        [t.join() for t in threads]
        torch.cuda.synchronize()
        assert all(len(got[i]) == 10 and all(_same(torch, y, want[i]) for y in got[i]) for i in range(3))


@pytest.mark.parametrize("dtype,logn,batch,ft,err", SHARED)
def test_captured_calls_beside_ordinary_ones(torch_cuda, dtype, logn, batch, ft, err):
    """A captured call keeps its intermediate buffer in the graph's own pool: it can be replayed while the same shape
    runs on another stream."""
    import turbofft_b200 as tf

    torch = torch_cuda
    x, z = (torch.from_numpy(orc.make_input(batch, 1 << logn, CD[dtype], seed=s)).cuda() for s in (7, 8))
    want_x, want_z = tf.fft(x, ft=ft, err=err), tf.fft(z, ft=ft, err=err)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = tf.fft(x, ft=ft, err=err)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    got = []
    for _ in range(5):
        graph.replay()
        with torch.cuda.stream(side):
            got.append(tf.fft(z, ft=ft, err=err))
    torch.cuda.synchronize()
    assert _same(torch, y, want_x) and all(_same(torch, g, want_z) for g in got)


def test_plans_without_scratch_refuse_what_needs_it(torch_cuda):
    import turbofft_b200 as tf

    torch = torch_cuda
    lib = tf.lib()
    x = torch.from_numpy(orc.make_input(2, 1 << 16, np.complex64, seed=1)).cuda()
    y = torch.empty_like(x)
    plan = tf.Plan(16, 2, 0, own_scratch=False)
    assert lib.tfft_exec(plan._h, x.data_ptr(), y.data_ptr(), 0) == -2
    assert lib.tfft_exec_ws(plan._h, x.data_ptr(), y.data_ptr(), None, 0) == -1
    assert lib.tfft_exec_host(plan._h, x.data_ptr(), y.data_ptr(), 0) == -2
    assert lib.tfft_plan_fuse_launches(plan._h, 2, 1) == -2
    assert _same(torch, plan(x), tf.Plan(16, 2, 0)(x))
    # the second buffer of three launches that repair by recomputing
    both = [tf.Plan(22, 1, 0, if_ft=1, if_err=1, own_scratch=own) for own in (True, False)]
    assert [lib.tfft_scratch_bytes(p._h) for p in both] == [1 << 25, 2 << 25]
    # one launch that repairs its output from its input cannot run in place, with either plan
    one = tf.Plan(10, 4, 0, if_ft=1, if_err=1, own_scratch=False)
    assert lib.tfft_exec_ws(one._h, x.data_ptr(), x.data_ptr(), None, 0) == -2


@pytest.mark.parametrize("logn", [10, 18])
def test_no_memory_is_reported_as_torch_reports_it(torch_cuda, logn):
    """Programs catch torch.OutOfMemoryError to try a smaller batch; a call that ends so keeps no hold of its plan."""
    import sys

    import turbofft_b200 as tf

    torch = torch_cuda
    x = torch.zeros((1 << 23) >> logn, 1 << logn, dtype=torch.complex64, device="cuda")  # 64 MiB
    plan = tf.Plan(logn, x.shape[0], 0)
    tf.fft(x), plan(x)
    cached = next(p for k, p in tf._plan_cache.items() if k[:4] == (0, logn, x.shape[0], 0))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    refs = sys.getrefcount(cached), sys.getrefcount(plan)
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (8 << 20)) / total)
    held = []
    try:
        with pytest.raises(torch.OutOfMemoryError):  # what the allocator still has free in its segments
            while True:
                held.append(torch.empty(8 << 20, dtype=torch.uint8, device="cuda"))
        for call in (lambda: tf.fft(x), lambda: plan(x)):
            for _ in range(3):
                with pytest.raises(torch.OutOfMemoryError):
                    call()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        del held
    assert (sys.getrefcount(cached), sys.getrefcount(plan)) == refs
    assert _same(torch, tf.fft(x), plan(x))


def test_whole_numbers_beyond_a_machine_word(torch_cuda):
    """An axis is taken modulo the rank, a launch number modulo 2^32, whatever their size."""
    import turbofft_b200 as tf

    torch = torch_cuda
    x = torch.from_numpy(orc.make_input(16, 256, np.complex64, seed=4)).cuda()
    for _ in range(2):
        for dim in (-1, 0):
            y = tf.fft(x, dim=dim)
            assert all(_same(torch, tf.fft(x, dim=dim + k), y) for k in (1 << 40, 1 << 70, -(1 << 70)))
    plan = tf.Plan(8, 16, 0, if_ft=1)
    plan(x)
    assert plan.ft_status(1 << 70) == plan.ft_status(0) == plan.ft_status()
    assert plan.ft_status((1 << 70) - 1) == plan.ft_status(-1)


@pytest.mark.parametrize("make", ["plain", "multi", "ft", "strided", "single_pass"])
def test_making_a_plan_waits_for_nothing_the_caller_has_queued(torch_cuda, make):
    import turbofft_b200 as tf

    torch = torch_cuda
    x = torch.zeros(64, 8, 16, dtype=torch.complex64, device="cuda")

    def new(batch):
        if make == "strided":
            return tf.fft(torch.zeros(batch, 8, 16, dtype=torch.complex64, device="cuda"), dim=1)
        if make == "single_pass":
            return tf.Plan(15, batch, 0, single_pass=-1)
        return tf.Plan(18 if make == "multi" else 10, batch, 0, if_ft=int(make == "ft"))

    kept = [new(61)]  # the first of its kind loads its kernels, which may wait
    torch.cuda.synchronize()
    x.add_(1)
    torch.cuda._sleep(400_000_000)  # a fifth of a second on the default stream
    kept.append(new(62))
    assert not torch.cuda.default_stream().query()
    torch.cuda.synchronize()
