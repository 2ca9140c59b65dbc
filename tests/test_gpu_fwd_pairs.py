"""GPU parity tests of the forward for few queries over many keys, where an item is two chunks of the keys for the
same query rows."""
import pytest
import torch

from oracle import attention_oracle as oracle
from tests import helpers
from tests.test_gpu_padded import _oracle_padded

pytestmark = pytest.mark.gpu


def _run(q, k, v, scale, causal, shift=0, **kw):
    import ctypes

    from flash_attn_v100 import cabi

    q, k, v = q.cuda(), k.cuda(), v.cuda()
    out, lse = torch.full_like(q, float("nan")), torch.empty((q.shape[0], q.shape[2], q.shape[1]), device="cuda")
    p = cabi.fwd_params(q, k, v, out, lse, scale, causal, shift, **kw)
    ws = torch.full((cabi.load_library().fmha_fwd_workspace_bytes(ctypes.byref(p)),), 255, dtype=torch.uint8, device="cuda")
    assert ws.numel() > 0  # the keys are cut
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    cabi.fwd(q, k, v, scale, causal, shift, out=out, lse=lse, status=status, workspace=ws, **kw)
    assert int(status.item()) == 0
    return out.cpu(), lse.cpu()


# an even and an odd number of KV tiles, ragged ones, one row and full tiles, more items than SMs (128 rows are
# not cut for 2048 keys, where whole items are faster: tests/test_fwd_plan_cpu.py)
@pytest.mark.parametrize("H,n_q,n_k,causal,shift", [
    (130, 128, 6144, False, 0), (130, 33, 2500, False, 0), (130, 1, 2305, False, 0), (300, 64, 2176, False, 0),
    (130, 64, 2500, True, 2300),  # the diagonal is in the last chunks
    (130, 64, 3000, True, 2100),  # keys that no row sees
])
@pytest.mark.parametrize("D,dtype", [(64, torch.float16), (64, torch.bfloat16)])
def test_pairs_of_chunks(H, n_q, n_k, causal, shift, D, dtype):
    q, _, _, dout = oracle.make_inputs(1, n_q, H, D, seed=61)
    _, k, v, _ = oracle.make_inputs(1, n_k, H, D, seed=62)
    q, k, v, dout = (t.to(dtype) for t in (q, k, v, dout))
    scale = oracle.default_scale(D)
    out, lse = _run(q, k, v, scale, causal, shift)
    ref = oracle.attention_fwd_bwd(q, k, v, dout, scale, causal, shift)
    tol = helpers.TOL_O_MAX_ABS if dtype == torch.float16 else helpers.TOL_O_MAX_ABS_BF16
    assert oracle.max_abs(out.float(), ref[0]) <= tol
    assert oracle.max_abs(lse, ref[1]) <= helpers.TOL_LSE_MAX_ABS


@pytest.mark.parametrize("D", [96, 128])
def test_pairs_of_chunks_wide_heads(D):
    q, _, _, dout = oracle.make_inputs(1, 64, 72, D, seed=63)
    _, k, v, _ = oracle.make_inputs(1, 8160, 72, D, seed=64)
    scale = oracle.default_scale(D)
    out, lse = _run(q, k, v, scale, False)
    s = torch.einsum("qhd,khd->hqk", q[0].float(), k[0].float()) * scale
    ref = torch.einsum("hqk,khd->qhd", s.softmax(-1), v[0].float())
    assert oracle.max_abs(out[0].float(), ref) <= helpers.TOL_O_MAX_ABS
    assert oracle.max_abs(lse[0], s.logsumexp(-1)) <= helpers.TOL_LSE_MAX_ABS


def test_pairs_of_chunks_in_a_padded_batch():
    Z, n_q, n_k, H, D = 5, 64, 2304, 30, 64
    sq, sk = [64, 17, 0, 64, 1], [2304, 1000, 500, 0, 1]
    q, _, _, dout = oracle.make_inputs(Z, n_q, H, D, seed=65)
    _, k, v, _ = oracle.make_inputs(Z, n_k, H, D, seed=66)
    scale = oracle.default_scale(D)
    out, lse = _run(q, k, v, scale, False, seqused_q=torch.tensor(sq, dtype=torch.int32, device="cuda"),
                    seqused_k=torch.tensor(sk, dtype=torch.int32, device="cuda"))
    ref = _oracle_padded(q, k, v, dout, scale, False, sq, sk)
    assert oracle.max_abs(out.float(), ref[0]) <= helpers.TOL_O_MAX_ABS
    assert torch.equal(torch.isfinite(lse), torch.isfinite(ref[1]))
    finite = torch.isfinite(lse)
    assert oracle.max_abs(lse[finite], ref[1][finite]) <= helpers.TOL_LSE_MAX_ABS
