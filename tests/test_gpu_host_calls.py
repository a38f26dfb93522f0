"""Host-buffer calls whose batch is cut into chunks: first calls of one plan from several threads, buffers that share
memory, buffers that are not page locked."""
import threading

import numpy as np
import pytest

from oracle import fft_oracle as orc

pytestmark = pytest.mark.gpu


def _same(torch, a, b):
    return torch.equal(torch.view_as_real(a), torch.view_as_real(b))


@pytest.mark.parametrize("logn,batch", [(10, 1001), (16, 40)])  # whole chunks and a ragged one
def test_first_calls_of_one_plan_from_several_threads(torch_cuda, logn, batch):
    """exec_host serialises its callers: the plans for one chunk are made under the same lock."""
    import turbofft_b200 as tf

    torch = torch_cuda
    xs = [torch.from_numpy(orc.make_input(batch, 1 << logn, np.complex64, seed=s)).pin_memory() for s in range(4)]
    want = [tf.Plan(logn, batch, 0)(x.cuda()).cpu() for x in xs]
    for _ in range(10):
        plan = tf.Plan(logn, batch, 0)
        got = [None] * len(xs)
        start = threading.Barrier(len(xs))

        def work(i):
            start.wait()
            got[i] = plan.exec_host(xs[i])

        threads = [threading.Thread(target=work, args=(i,)) for i in range(len(xs))]
        [t.start() for t in threads]
        [t.join() for t in threads]
        assert all(_same(torch, g, w) for g, w in zip(got, want))


@pytest.mark.parametrize("logn,batch", [(10, 1001), (16, 40)])
@pytest.mark.parametrize("shift", [0, 1, -1, 5, -5])
@pytest.mark.parametrize("asynchronous", [False, True])
def test_buffers_that_share_memory(torch_cuda, logn, batch, shift, asynchronous):
    """The input is read before the output lands on it, wherever the two lie in one array (shift in signals)."""
    import turbofft_b200 as tf

    torch = torch_cuda
    x = torch.from_numpy(orc.make_input(batch, 1 << logn, np.complex64, seed=logn))
    plan = tf.Plan(logn, batch, 0)
    want = plan(x.cuda()).cpu()
    both = torch.zeros(batch + abs(shift), 1 << logn, dtype=x.dtype).pin_memory()
    src = both[max(0, -shift):][:batch]
    dst = both[max(0, shift):][:batch]
    for _ in range(2):
        src.copy_(x)
        if asynchronous:
            plan.exec_host_async(src, dst)
            tf.host_sync()
        else:
            plan.exec_host(src, dst)
        assert _same(torch, dst, want)


@pytest.mark.parametrize("logn,batch", [(12, 1000), (12, 6500), (18, 100)])  # 31 and 203 MiB, 200 MiB of longer signals
def test_page_locked_and_ordinary_buffers_alternate_on_one_plan(torch_cuda, logn, batch):
    """They are cut differently (ordinary buffers not at all below three chunks of 64 MiB), each with plans of its own
    that follow a change of direction."""
    import turbofft_b200 as tf

    torch = torch_cuda
    x = torch.from_numpy(orc.make_input(batch, 1 << logn, np.complex64, seed=logn))
    locked, plan = x.pin_memory(), tf.Plan(logn, batch, 0)
    for inverse in (False, True, False):
        plan.set_direction(inverse, 0.5)
        want = plan(x.cuda()).cpu()
        for src, dst in ((x, torch.empty_like(x)), (locked, torch.empty_like(x).pin_memory()), (locked, torch.empty_like(x)), (x, None)):
            assert _same(torch, plan.exec_host(src, dst), want)
