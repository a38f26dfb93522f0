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
