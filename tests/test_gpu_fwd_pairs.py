"""GPU parity tests of the forward for few queries over many keys, where an item is two chunks of the keys for the
same query rows."""
import pytest
import torch

from oracle import attention_oracle as oracle
from tests import helpers
from tests.test_gpu_fwd_scores import _check
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


# ------------------------------------------------------------------------------------------
# More than eight items per SM, where nothing but pairs asks for a workspace: items follow one another on
# their SM, through rings of two slots at D = 96 and 128.
# ------------------------------------------------------------------------------------------
Z, H = 5, 266  # nine waves of 148, the last one full


def _many(n_q, n_k, D, dtype, seed):
    assert Z * H > 8 * torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(seed)
    return tuple(torch.randn((Z, n, H, D), generator=g, device="cuda", dtype=dtype) for n in (n_q, n_k, n_k))


def _reference(q, k, v, scale, causal=False, shift=0, sq=None, sk=None):
    """fp32 softmax on the GPU; rows that see nothing: O = 0, LSE = -inf."""
    out, lse = torch.empty(q.shape, device="cuda"), torch.empty((q.shape[0], q.shape[2], q.shape[1]), device="cuda")
    row, key = (torch.arange(t.shape[1], device="cuda") for t in (q, k))
    for z in range(q.shape[0]):
        qz, kz, vz = (t[z].float().transpose(0, 1) for t in (q, k, v))
        s = qz @ kz.transpose(1, 2) * scale
        hidden = (key >= (len(key) if sk is None else sk[z]))[None, :] | (row >= (len(row) if sq is None else sq[z]))[:, None]
        if causal:
            hidden = hidden | (key[None, :] > row[:, None] + shift)
        s = s.masked_fill(hidden, float("-inf"))
        p = s.softmax(-1).masked_fill(hidden.all(-1)[:, None], 0.0)
        out[z], lse[z] = (p @ vz).transpose(0, 1), s.logsumexp(-1)
    return out, lse


def _tol(dtype):
    return helpers.TOL_O_MAX_ABS if dtype == torch.float16 else helpers.TOL_O_MAX_ABS_BF16


def _run_pairs(q, k, v, scale, causal=False, shift=0, **kw):
    out, lse = _run(q, k, v, scale, causal, shift, **kw)
    return out.cuda(), lse.cuda()


@pytest.mark.parametrize("n_q,n_k,causal,shift", [
    (16, 3200, False, 0), (16, 3150, False, 0),  # 25 tiles: the second chunk is a tile shorter
    (1, 3072, False, 0), (64, 6100, False, 0),
    (16, 3300, True, 3000),  # the diagonal and keys that no row sees in the second chunk
    (16, 3300, True, 3064),  # ... the diagonal crosses tiles
])
@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_pairs_one_after_the_other(n_q, n_k, causal, shift, D, dtype):
    q, k, v = _many(n_q, n_k, D, dtype, seed=67)
    scale = oracle.default_scale(D)
    out, lse = _run_pairs(q, k, v, scale, causal, shift)
    r_out, r_lse = _reference(q, k, v, scale, causal, shift)
    assert oracle.max_abs(out.float(), r_out) <= _tol(dtype)
    assert oracle.max_abs(lse, r_lse) <= helpers.TOL_LSE_MAX_ABS


@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_pairs_one_after_the_other_in_a_padded_batch(D, dtype):
    # 25 tiles; in chunks of 13 and 12, which the next test has, too, entries with one tile in the second chunk and with none
    n_q, n_k, sq, sk = 16, 3200, [16, 1, 16, 0, 9], [3200, 1665, 1664, 77, 0]
    q, k, v = _many(n_q, n_k, D, dtype, seed=68)
    scale = oracle.default_scale(D)
    lens = {"seqused_q": sq, "seqused_k": sk}
    out, lse = _run_pairs(q, k, v, scale, **{n: torch.tensor(x, dtype=torch.int32, device="cuda") for n, x in lens.items()})
    r_out, r_lse = _reference(q, k, v, scale, sq=sq, sk=sk)
    assert oracle.max_abs(out.float(), r_out) <= _tol(dtype)
    seen = torch.isfinite(r_lse)
    assert torch.equal(torch.isfinite(lse), seen)
    assert oracle.max_abs(lse[seen], r_lse[seen]) <= helpers.TOL_LSE_MAX_ABS
    assert not out[~seen.transpose(1, 2)].any()


@pytest.mark.parametrize("heads,chunks,sk", [
    (266, 4, [2689, 1793, 897, 1, 0]),  # 25 tiles in chunks of 7, 7, 7, 4: one tile in the fourth, third, second, first
    (66, 2, [3200, 1665, 1664, 77, 0]),  # in chunks of 13 and 12: a full second chunk, one tile in it, none
])
@pytest.mark.parametrize("D", [64, 96, 128])
def test_pairs_once_and_twice_per_head_in_a_padded_batch(D, heads, chunks, sk):
    import ctypes

    from flash_attn_v100 import cabi

    n_q, n_k, sq = 16, 3200, [16, 1, 16, 7, 9]
    q, k, v = (t[:, :, :heads].contiguous() for t in _many(n_q, n_k, D, torch.bfloat16, seed=70))
    lens = {n: torch.tensor(x, dtype=torch.int32, device="cuda") for n, x in (("seqused_q", sq), ("seqused_k", sk))}
    p = cabi.fwd_params(q, k, v, q, torch.empty(1, device="cuda"), 1.0, False, **lens)
    assert cabi.load_library().fmha_fwd_workspace_bytes(ctypes.byref(p)) == chunks * Z * heads * n_q * (D + 1) * 4
    scale = oracle.default_scale(D)
    out, lse = _run_pairs(q, k, v, scale, **lens)
    r_out, r_lse = _reference(q, k, v, scale, sq=sq, sk=sk)
    assert oracle.max_abs(out.float(), r_out) <= _tol(torch.bfloat16)
    seen = torch.isfinite(r_lse)
    assert torch.equal(torch.isfinite(lse), seen)
    assert oracle.max_abs(lse[seen], r_lse[seen]) <= helpers.TOL_LSE_MAX_ABS
    assert not out[~seen.transpose(1, 2)].any()


@pytest.mark.parametrize("what", ["query rows", "keys of the first chunk", "keys of the second chunk"])
@pytest.mark.parametrize("D", [64, 96, 128])
def test_pairs_with_rows_that_are_not_finite(D, what):
    """Every row that sees one is not finite, the rows of other heads are right."""
    q, k, v = _many(16, 3200, D, torch.float16, seed=69)
    scale = oracle.default_scale(D)
    for h in range(0, H, 3):
        for z in range(Z):
            if what == "query rows":
                q[z, h % 16, h, 3] = float("nan") if h % 2 else float("inf")
            else:  # in either half of a round and in every column that may take a path of its own
                k[z, (0 if "first" in what else 1664) + 128 * z + h % 128, h, 7] = float("nan")
    _check(_run_pairs(q, k, v, scale), _reference(q, k, v, scale), helpers.TOL_O_MAX_ABS)


@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_pairs_with_leaping_scores(D, dtype):
    """One key far above all others, in either half of the first, a middle and the last round of either chunk."""
    q, k, v = _many(16, 3200, D, dtype, seed=70)
    scale = oracle.default_scale(D)
    q[:, ::2, :, 0], q[:, 1::2, :, 0], k[..., 0] = 20.0, -20.0, 0.0
    for z, leap in enumerate((95.0, 130.0, 180.0, 256.0, 400.0)):
        for h in range(H):
            tile = (0, 6, 12, 13, 19, 24)[h % 6]
            k[z, tile * 128 + (h // 6 * 16 + h // 48) % 128, h, 0] = leap / (20.0 * scale)
    ref = _reference(q, k, v, scale)
    # weights on a key or two, each rounded to the 16-bit type, and so is O
    bound = (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8) * (v.abs().max().item() + ref[0].abs().max().item())
    _check(_run_pairs(q, k, v, scale), ref, bound)


@pytest.mark.parametrize("D", [64, 96, 128])
def test_pairs_with_sms_left_free(D):
    """Items dealt out over eight SMs, nine to each."""
    q, k, v = (t[:1, :, :72].contiguous() for t in _many(16, 3200, D, torch.bfloat16, seed=71))
    scale = oracle.default_scale(D)
    margin = torch.cuda.get_device_properties(0).multi_processor_count - 8
    out, lse = _run_pairs(q, k, v, scale, sm_margin=margin)
    r_out, r_lse = _reference(q, k, v, scale)
    assert oracle.max_abs(out.float(), r_out) <= _tol(torch.bfloat16)
    assert oracle.max_abs(lse, r_lse) <= helpers.TOL_LSE_MAX_ABS


# chunks of 4 to 17 tiles through a ring of three (six at D = 64) slots each, full tiles of 128 rows
@pytest.mark.parametrize("n_k", [2500, 4100, 8200])
@pytest.mark.parametrize("n_q", [1, 128])
@pytest.mark.parametrize("D,dtype", [(64, torch.bfloat16), (96, torch.float16), (128, torch.float16), (128, torch.bfloat16)])
def test_pairs_of_short_chunks(n_q, n_k, D, dtype):
    g = torch.Generator(device="cuda").manual_seed(72)
    q, k, v = (torch.randn((1, n, 32, D), generator=g, device="cuda", dtype=dtype) for n in (n_q, n_k, n_k))
    scale = oracle.default_scale(D)
    out, lse = _run_pairs(q, k, v, scale)
    r_out, r_lse = _reference(q, k, v, scale)
    assert oracle.max_abs(out.float(), r_out) <= _tol(dtype)
    assert oracle.max_abs(lse, r_lse) <= helpers.TOL_LSE_MAX_ABS
