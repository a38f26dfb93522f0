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
