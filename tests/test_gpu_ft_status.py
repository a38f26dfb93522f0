"""tfft_ft_status against what may lie between the exec and the read: replayed graphs, totals over several execs, other
plans and threads that wait, buffers that the call did not ask for."""
import ctypes as C

import numpy as np
import pytest

from oracle import fft_oracle as orc

pytestmark = pytest.mark.gpu


def _plan(tf, logn=12, batch=64, tbs=4, err=1):
    plan = tf.Plan(logn, batch, 0, if_ft=1, if_err=err, thread_bs=tbs)
    plan.set_ft_params(1e5, 1000.0, 1e-3)
    return plan


def _input(torch, logn=12, batch=64):
    return torch.from_numpy(orc.make_input(batch, 1 << logn, np.complex64, seed=logn + batch)).cuda()


def _captured(torch, plan, x, inject):
    plan.set_injection(inject)
    y = torch.empty_like(x)
    plan(x, y)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan(x, y)
    torch.cuda.synchronize()
    return graph


def test_status_is_read_behind_replays_on_the_default_stream(torch_cuda):
    """An exec captured on one stream and replayed on the default one, where it waits behind other work when the status is
    asked for."""
    import turbofft_b200 as tf

    torch = torch_cuda
    plan, x = _plan(tf), _input(torch)
    faulty, clean = _captured(torch, plan, x, True), _captured(torch, plan, x, False)
    blocks = plan.info()[0]["grid"]
    for graph, counts in ((faulty, (blocks, blocks)), (clean, (0, 0))) * 3:
        torch.cuda._sleep(20_000_000)  # ten milliseconds on the default stream
        graph.replay()
        assert plan.ft_status()[:2] == counts


@pytest.mark.parametrize("logn,batch", [(12, 64), (18, 8)])
def test_totals_over_replays_of_an_exec_captured_before(torch_cuda, logn, batch):
    """set_ft_accumulate after the capture: the replays add up, and again from zero after each read."""
    import turbofft_b200 as tf

    torch = torch_cuda
    plan, x = _plan(tf, logn, batch), _input(torch, logn, batch)
    graph = _captured(torch, plan, x, True)
    graph.replay()
    nd, nc = plan.ft_status()[:2]
    assert nd == nc > 0
    plan.set_ft_accumulate(True)
    for n in (1, 3, 2):
        for _ in range(n):
            graph.replay()
        assert plan.ft_status()[:2] == (n * nd, n * nc)
    plan.set_ft_accumulate(False)
    for _ in range(2):
        graph.replay()
    assert plan.ft_status()[:2] == (nd, nc)


def test_a_status_read_that_waits_holds_up_no_other_plan(torch_cuda):
    """One thread waits for a long queue on its stream; another plan's status is read meanwhile."""
    import threading
    import time

    import turbofft_b200 as tf

    torch = torch_cuda
    slow, quick, x = _plan(tf), _plan(tf), _input(torch)
    busy, idle = torch.cuda.Stream(), torch.cuda.Stream()
    blocks = quick.info()[0]["grid"]
    for plan, stream in ((slow, busy), (quick, idle)):  # first reads, outside of what is timed
        with torch.cuda.stream(stream):
            plan(x)
        plan.ft_status()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(1_500_000_000)  # most of a second
        slow(x)
    ended = []
    waiter = threading.Thread(target=lambda: ended.append((slow.ft_status()[0], time.monotonic())))
    waiter.start()
    time.sleep(0.1)                       # the waiter is inside its call
    with torch.cuda.stream(idle):
        quick(x)
    assert quick.ft_status()[0] == blocks
    read = time.monotonic()
    waiter.join()
    assert ended[0][0] == blocks and read < ended[0][1] - 0.1


@pytest.mark.parametrize("logn,batch,tbs,total", [(12, 64, 4, False), (12, 64, 4, True), (7, 1 << 18, 1, False), (7, 1 << 18, 1, True),
                                                  (18, 40, 2, False), (18, 40, 2, True), (22, 3, 2, True)])
def test_every_form_of_the_call_gives_the_same_answer(torch_cuda, logn, batch, tbs, total):
    """Counts alone, counts with the blocks of one launch, a buffer that is too short, nothing at all; results on both
    sides of the size that is read through pinned memory; totals are cleared by each read."""
    import turbofft_b200 as tf

    torch = torch_cuda
    plan, x = _plan(tf, logn, batch, tbs), _input(torch, logn, batch)
    lib, info = tf.lib(), plan.info()
    stream = torch.cuda.Stream()  # not ordered with the default stream by itself
    stream.wait_stream(torch.cuda.current_stream())
    plan.set_injection(True, launch=0)
    plan.set_ft_accumulate(total)

    def status(launch, cap, counts=True, blocks=True):
        with torch.cuda.stream(stream):
            for _ in range(2):
                plan(x)
        nd, nc, nb = C.c_int(-7), C.c_int(-7), C.c_int(-7)
        loc = (C.c_int * max(cap, 1))(*[-7] * max(cap, 1))
        rc = lib.tfft_ft_status(plan._h, C.byref(nd) if counts else None, C.byref(nc) if counts else None, launch,
                                loc if cap else None, cap, C.byref(nb) if blocks else None)
        assert rc == 0
        return nd.value, nc.value, nb.value, list(loc)[:cap]

    grids = [l["grid"] for l in info]
    runs = 2 if total else 1
    want = (runs * grids[0], runs * grids[0])
    for launch in range(len(info)):
        nd, nc, nb, loc = status(launch, grids[launch])
        assert (nd, nc, nb) == (*want, grids[launch])
        assert all((k != -1) == (launch == 0) for k in loc)
        short = max(1, grids[launch] // 3)
        assert status(launch, short)[3] == loc[:short]
        assert status(launch, 0)[:3] == (*want, grids[launch])
        assert status(launch, grids[launch], counts=False, blocks=False)[3] == loc
    assert status(-1, 0, counts=False, blocks=False)[:3] == (-7, -7, -7)
    plan.set_injection(False)
    assert status(0, grids[0])[:2] == (0, 0)
    assert lib.tfft_ft_status(plan._h, None, None, len(info), None, 0, None) == -1
