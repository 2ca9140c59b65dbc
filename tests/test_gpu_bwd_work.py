"""GPU parity tests of how the backward kernel's work is taken: more items (KV tiles) than SMs, so that
a CTA runs several and hands its tiles and accumulators over from one to the next."""
import pytest
import torch

from oracle import attention_oracle as oracle
from tests import helpers
from tests.test_gpu_padded import _oracle_padded

pytestmark = pytest.mark.gpu


def _tols(dtype):
    if dtype == torch.float16:
        return helpers.TOL_O_MAX_ABS, helpers.TOL_GRAD_REL_L2
    return helpers.TOL_O_MAX_ABS_BF16, helpers.TOL_GRAD_REL_L2_BF16


# H chosen so that Z * H * KV tiles is 2 to 4 times the 148 SMs
@pytest.mark.parametrize("H,n_q,n_k,causal,shift", [
    (100, 288, 288, False, 0),   # three KV tiles of three query tiles, ragged
    (100, 320, 320, True, 0),    # items of 3, 2 and 1 query tiles
    (25, 32, 2016, False, 0),    # one query tile per item, ragged last KV tile
    (300, 640, 96, False, 0),    # one KV tile per head
    (50, 256, 1152, True, 128),  # KV tiles that no query sees: runs of items without work
])
@pytest.mark.parametrize("D,dtype", [(64, torch.float16), (64, torch.bfloat16), (96, torch.float16),
                                     (128, torch.float16), (128, torch.bfloat16)])
def test_more_items_than_sms(H, n_q, n_k, causal, shift, D, dtype):
    q, _, _, dout = oracle.make_inputs(1, n_q, H, D, seed=71)
    _, k, v, _ = oracle.make_inputs(1, n_k, H, D, seed=72)
    q, k, v, dout = (t.to(dtype) for t in (q, k, v, dout))
    scale = oracle.default_scale(D)
    got = helpers.gpu_fwd_bwd(q, k, v, dout, scale, causal, shift)
    ref = oracle.attention_fwd_bwd(q, k, v, dout, scale, causal, shift)
    helpers.check_against_oracle(got, ref, f"H{H} {n_q}x{n_k} D{D}", *_tols(dtype))
    if causal:  # keys beyond the last one that is seen: exact zeros
        assert not got[3][:, n_q + shift:].any() and not got[4][:, n_q + shift:].any()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("overwrite", [False, True])
def test_fp32_accumulation_over_many_items(D, overwrite):
    """dK and dV added into (or in place of) fp32 buffers, with KV tiles that no query sees."""
    from flash_attn_v100 import cabi

    H, n_q, n_k, shift = 50, 256, 1152, 128
    q, _, _, dout = oracle.make_inputs(1, n_q, H, D, seed=73)
    _, k, v, _ = oracle.make_inputs(1, n_k, H, D, seed=74)
    scale = oracle.default_scale(D)
    ref = oracle.attention_fwd_bwd(q, k, v, dout, scale, True, shift)
    q, k, v, dout = (t.cuda() for t in (q, k, v, dout))
    out, lse = cabi.fwd(q, k, v, scale, True, shift)
    acc = [torch.full((1, n_k, H, D), 3.0, device="cuda") for _ in range(2)]
    cabi.bwd(q, k, v, out, dout, lse, scale, True, shift, dk_accum=acc[0], dv_accum=acc[1],
             flags=cabi.FMHA_BWD_ACCUM_OVERWRITE if overwrite else 0)
    for a, r in zip(acc, ref[3:]):
        assert oracle.rel_l2(a.cpu() - (0.0 if overwrite else 3.0), r) <= helpers.TOL_GRAD_REL_L2
        assert (a[:, n_q + shift:] == (0.0 if overwrite else 3.0)).all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_runs_of_padding_between_items(D, causal):
    """A padded batch whose short entries leave runs of far more empty items than are published ahead."""
    from flash_attn_v100 import cabi

    Z, H, N = 4, 24, 1024
    lens = [1024, 33, 130, 700]
    q, k, v, dout = oracle.make_inputs(Z, N, H, D, seed=75)
    lens_d = torch.tensor(lens, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    scale = oracle.default_scale(D)
    qd, kd, vd, dod = (t.cuda() for t in (q, k, v, dout))
    out, lse = cabi.fwd(qd, kd, vd, scale, causal, status=status, seqused_q=lens_d, seqused_k=lens_d)
    grads = cabi.bwd(qd, kd, vd, out, dod, lse, scale, causal, status=status, seqused_q=lens_d, seqused_k=lens_d)
    assert int(status.item()) == 0
    ref = _oracle_padded(q, k, v, dout, scale, causal, lens, lens)
    helpers.check_against_oracle((out.cpu(), lse.cpu(), *(t.cpu() for t in grads)), ref, f"padding runs D{D}")


@pytest.mark.parametrize("D,dtype", [(64, torch.float16), (96, torch.float16), (96, torch.bfloat16), (128, torch.bfloat16)])
@pytest.mark.parametrize("wide", ["dk", "dv"])
def test_one_of_dk_and_dv_in_fp32(D, dtype, wide):
    """One of them goes through the staging buffers that dQ uses in turn (an odd number of chunks per tile at 96), the
    other does not; more items than SMs, of one, two and three query tiles, the last rows of a tile missing."""
    from flash_attn_v100 import cabi

    H, N = 100, 352
    q, k, v, dout = (t.to(dtype) for t in oracle.make_inputs(1, N, H, D, seed=76))
    scale = oracle.default_scale(D)
    ref = oracle.attention_fwd_bwd(q, k, v, dout, scale, True, 0)
    q, k, v, dout = (t.cuda() for t in (q, k, v, dout))
    out, lse = cabi.fwd(q, k, v, scale, True)
    acc = torch.full((1, N, H, D), 3.0, device="cuda")
    guard = torch.full((1, N + 32, H, D), 7.0, dtype=dtype, device="cuda")
    kw = {"dk_accum": acc, "dv": guard[:, :N]} if wide == "dk" else {"dv_accum": acc, "dk": guard[:, :N]}
    dq, _, _ = cabi.bwd(q, k, v, out, dout, lse, scale, True, flags=cabi.FMHA_BWD_ACCUM_OVERWRITE, **kw)
    tol = _tols(dtype)[1]
    assert oracle.rel_l2(dq.float().cpu(), ref[2]) <= tol
    assert oracle.rel_l2(acc.cpu(), ref[3] if wide == "dk" else ref[4]) <= tol
    assert oracle.rel_l2(guard[:, :N].float().cpu(), ref[4] if wide == "dk" else ref[3]) <= tol
    assert (guard[:, N:] == 7.0).all()


@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("wide", ["both", "dk", "dv"])
def test_fp32_dk_dv_are_added_and_replaced_alike(D, wide):
    """What is added is what would replace: bit for bit, and nothing to rows of padding keys, behind the last key or
    between batch entries.  More items than SMs, the last KV tile not full, KV tiles that no query sees."""
    from flash_attn_v100 import cabi

    Z, H, n_q, n_k, gap = 3, 40, 200, 500, 24
    g = torch.Generator(device="cuda").manual_seed(97)
    q, dout = (torch.randn((Z, n_q, H, D), generator=g, device="cuda", dtype=torch.float16) for _ in range(2))
    k, v = (torch.randn((Z, n_k, H, D), generator=g, device="cuda", dtype=torch.float16) for _ in range(2))
    used = torch.tensor([500, 130, 0], dtype=torch.int32, device="cuda")
    start = [torch.randn((Z, n_k + gap, H, D), generator=g, device="cuda") for _ in range(2)]
    out, lse = cabi.fwd(q, k, v, 0.1, True, 100, seqused_k=used)
    names = {"both": ["dk", "dv"], "dk": ["dk"], "dv": ["dv"]}[wide]

    def run(flags):
        acc = dict(zip(("dk", "dv"), (t.clone() for t in start)))
        kw = {name + "_accum": acc[name][:, :n_k] for name in names}
        kw |= {name: torch.full_like(k, float("nan")) for name in ("dk", "dv") if name not in names}
        _, dk, dv = cabi.bwd(q, k, v, out, dout, lse, 0.1, True, 100, flags=flags, seqused_k=used, **kw)
        return acc, {"dk": dk, "dv": dv}

    added, narrow = run(0)
    replaced, again = run(cabi.FMHA_BWD_ACCUM_OVERWRITE)
    plain = dict(zip(("dq", "dk", "dv"), cabi.bwd(q, k, v, out, dout, lse, 0.1, True, 100, seqused_k=used)))
    for name, before in zip(("dk", "dv"), start):
        if name not in names:
            assert torch.equal(narrow[name], plain[name]) and torch.equal(again[name], plain[name])
            assert torch.equal(added[name], before)
            continue
        new = replaced[name][:, :n_k]
        assert torch.equal(new.half(), plain[name])
        assert torch.equal(replaced[name][:, n_k:], before[:, n_k:])
        assert torch.equal(added[name][:, :n_k], before[:, :n_k] + new)
        assert torch.equal(added[name][:, n_k:], before[:, n_k:])
        for z, n in enumerate(used.tolist()):
            assert torch.equal(added[name][z, n:], before[z, n:]) and not new[z, n:].any()
