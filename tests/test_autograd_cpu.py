"""What the C++ host path (``flash_attn_v100_cuda.attention``) refuses where it passes autograd by.  Needs no
GPU: the two ops get stand-in kernels for CPU tensors."""
import pytest
import torch


@pytest.fixture
def ops_on_cpu(built_library):
    from flash_attn_v100 import flash_attn_interface  # noqa: F401 (defines the ops)

    def fwd(q, k, v, scale, causal, seqused_q=None, seqused_k=None):
        s = torch.einsum("znhd,zmhd->zhnm", q, k) * scale
        return torch.einsum("zhnm,zmhd->znhd", s.softmax(-1), v), s.logsumexp(-1)

    lib = torch.library.Library("flash_attn_v100", "IMPL")
    lib.impl("fwd", fwd, "CPU")
    yield
    lib._destroy()


def _qkv():
    g = torch.Generator().manual_seed(3)
    return [torch.randn(2, 32, 2, 64, generator=g) for _ in range(3)]


def _calls():
    from flash_attn_v100.flash_attn_interface import flash_attn_func, flash_attn_padded_func

    return flash_attn_func, flash_attn_padded_func


@pytest.mark.parametrize("which", range(3))
@pytest.mark.parametrize("no_grad,requires_grad", [(False, False), (True, False), (False, True)])
def test_a_forward_mode_tangent_is_refused(ops_on_cpu, which, no_grad, requires_grad):
    """An output without a tangent would say that the derivative is zero."""
    import torch.autograd.forward_ad as fw

    for call in _calls():
        inputs = [t.requires_grad_(requires_grad) for t in _qkv()]
        call(*inputs)
        with fw.dual_level(), torch.set_grad_enabled(not no_grad):
            inputs[which] = fw.make_dual(inputs[which], torch.ones_like(inputs[which]))
            with pytest.raises(NotImplementedError, match="forward-mode"):
                call(*inputs)
            with fw._set_fwd_grad_enabled(False):
                call(*inputs)


@pytest.mark.parametrize("no_grad", [False, True])
def test_function_transforms_are_refused(ops_on_cpu, no_grad):
    """vmap, grad and jvp, with and without gradients to record: the autograd function has no rules for them
    (vmap would run the op in a loop over the batch)."""
    for call in _calls():
        q, k, v = _qkv()
        with torch.set_grad_enabled(not no_grad):
            with pytest.raises(RuntimeError, match="functorch"):
                torch.vmap(lambda a: call(a, k, v))(torch.stack([q, q]))
            with pytest.raises(RuntimeError, match="functorch"):
                torch.func.grad(lambda a: call(a, k, v).sum())(q)
            with pytest.raises(RuntimeError, match="functorch"):
                torch.func.jvp(lambda a: call(a, k, v), (q,), (torch.ones_like(q),))
            call(q, k, v)
