"""GPU tests of the backward where dP and D are large (loss-scaled training): dS = P o (dP - D) is finite where P and
the result are, whatever the size of the difference."""
import pytest
import torch

pytestmark = pytest.mark.gpu

U = 2.0 ** -11     # rounding to fp16, relative
TINY = 2.0 ** -25  # ... and below its normal range, absolute


def _inputs(N, H, D, v_size, dout_size):
    """Keys in two halves: those with sign + get nearly all of P, those with sign - a few thousandths.  v is +- v_size
    by the sign and dout is dout_size over 64 columns, so dP = +-64 * v_size * dout_size and D is near the upper one."""
    g = torch.Generator().manual_seed(17)
    sign = torch.where(torch.arange(N) % 2 == 0, 1.0, -1.0).view(1, N, 1, 1)
    q, k = (0.5 * torch.randn((1, N, H, D), generator=g) for _ in range(2))
    q[..., 0] = 3.0
    k[..., 0] = (sign * D ** 0.5).expand(1, N, H, 1)[..., 0]
    v = 0.01 * torch.randn((1, N, H, D), generator=g) + sign * v_size
    dout = torch.zeros((1, N, H, D))
    dout[..., :64] = dout_size
    return tuple(t.half().cuda() for t in (q, k, v, dout))


def _exact(q, k, v, dout, scale, causal):
    """Gradients in 64 bits, and for each element a bound of what an implementation that rounds O, P, dS and the
    results to fp16 may be off by."""
    q, k, v, do = (t.double().transpose(1, 2) for t in (q, k, v, dout))
    s = q @ k.transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], device=s.device).triu(1).bool(), float("-inf"))
    p = s.softmax(-1)
    o, dp = p @ v, do @ v.transpose(-1, -2)
    delta = (do * o).sum(-1, keepdim=True)
    diff = dp - delta
    ds = p * diff
    # P is rounded to fp16 (and comes of fp32 arguments: 2^-18); D is formed from the rounded O; dP and D
    # are fp32 sums of up to 128 products (2^-17 of their sizes), rounded to fp16, and so is P D; dS, too
    e_p = p * (U + 2.0 ** -18) + TINY
    e_diff = U * ((do * o).abs().sum(-1, keepdim=True) + dp.abs() + 2 * delta.abs())
    e_diff = e_diff + 2.0 ** -17 * (do.abs() @ v.abs().transpose(-1, -2) + delta.abs())
    e_ds = e_p * diff.abs() + p * e_diff + U * ds.abs() + 2 * TINY
    grads = scale * ds @ k, scale * ds.transpose(-1, -2) @ q, p.transpose(-1, -2) @ do
    sums = scale * e_ds @ k.abs(), scale * e_ds.transpose(-1, -2) @ q.abs(), e_p.transpose(-1, -2) @ do.abs()
    bounds = [1.01 * (e + U * g.abs() + TINY) for e, g in zip(sums, grads)]
    return [t.transpose(1, 2) for t in grads], [t.transpose(1, 2) for t in bounds], (dp, delta, diff, ds)


@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("deterministic", [False, True])
def test_difference_beyond_fp16(D, causal, deterministic):
    from flash_attn_v100 import cabi

    N, H, scale = 320, 3, D ** -0.5
    q, k, v, dout = _inputs(N, H, D, 20.0, 40.0)
    grads, bounds, (dp, delta, diff, ds) = _exact(q, k, v, dout, scale, causal)
    # each of the two fits fp16, their difference does not; every result does
    assert max(dp.abs().max(), delta.abs().max()) < 65504 < 9e4 < diff.abs().max()
    assert max(t.abs().max() for t in (ds, *grads)) < 6e4
    out, lse = cabi.fwd(q, k, v, scale, causal)
    got = cabi.bwd(q, k, v, out, dout, lse, scale, causal, flags=cabi.FMHA_BWD_DETERMINISTIC if deterministic else 0)
    for name, a, ref, bound in zip(("dq", "dk", "dv"), got, grads, bounds):
        assert torch.isfinite(a).all(), name
        worst = ((a.double() - ref).abs() / bound).max().item()
        print(f"{name} D{D} causal={causal}: error / bound {worst:.2f}")
        assert worst <= 1.0, name
