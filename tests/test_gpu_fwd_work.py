"""GPU parity tests of how the forward kernel's work is cut and taken: query blocks whose KV range is
cut into chunks (partial results joined by a second kernel), items taken over through cluster
launch control, runs of items with nothing to do, and a new softmax reference in mid-round."""
import pytest
import torch

from oracle import attention_oracle as oracle
from tests import helpers

pytestmark = pytest.mark.gpu


def _fwd(q, k, v, scale, causal, sq=None, sk=None):
    """Through the extension, which hands the kernel a workspace for cut query blocks."""
    import flash_attn_v100_cuda as ext

    lens = [None if x is None else torch.tensor(x, dtype=torch.int32, device="cuda") for x in (sq, sk)]
    out, lse = ext.fwd_lse(q.cuda(), k.cuda(), v.cuda(), None, scale, causal, *lens)
    return out.cpu(), lse.cpu()


def _check(got, ref, dtype=torch.float16):
    tol = helpers.TOL_O_MAX_ABS if dtype == torch.float16 else helpers.TOL_O_MAX_ABS_BF16
    finite = torch.isfinite(ref[1])
    assert torch.equal(torch.isfinite(got[1]), finite)
    assert oracle.max_abs(got[0].float(), ref[0]) <= tol
    assert oracle.max_abs(got[1][finite], ref[1][finite]) <= helpers.TOL_LSE_MAX_ABS


@pytest.mark.parametrize("Z,H,n_q,n_k,D,causal,dtype", [
    (1, 1, 32, 8192, 128, False, torch.float16),   # one block in 32 chunks
    (1, 3, 64, 2080, 64, False, torch.bfloat16),   # ragged last tile
    (2, 5, 288, 1056, 96, False, torch.float16),   # two blocks, the second one ragged
    (1, 1, 4096, 4096, 128, True, torch.float16),  # causal: long blocks cut, short ones not
    (1, 2, 2080, 2080, 64, True, torch.bfloat16),
])
def test_cut_query_blocks(Z, H, n_q, n_k, D, causal, dtype):
    q, _, _, _ = oracle.make_inputs(Z, n_q, H, D, seed=61)
    _, k, v, _ = oracle.make_inputs(Z, n_k, H, D, seed=62)
    q, k, v = (t.to(dtype) for t in (q, k, v))
    scale = oracle.default_scale(D)
    _check(_fwd(q, k, v, scale, causal), oracle.attention_forward(q, k, v, scale, causal), dtype)


def test_cut_query_blocks_of_a_padded_batch():
    """Chunks that lie wholly in the padding of the keys, a query tile that is all padding, an entry
    without keys."""
    Z, H, N, D = 3, 1, 1024, 128
    sq, sk = [1024, 100, 640], [1000, 130, 0]
    q, k, v, _ = oracle.make_inputs(Z, N, H, D, seed=63)
    scale = oracle.default_scale(D)
    out, lse = _fwd(q, k, v, scale, False, sq, sk)
    ref_o, ref_l = torch.zeros((Z, N, H, D)), torch.full((Z, H, N), float("-inf"))
    for z in range(2):
        r = oracle.attention_forward(q[z:z + 1, :sq[z]], k[z:z + 1, :sk[z]], v[z:z + 1, :sk[z]], scale, False)
        ref_o[z, :sq[z]], ref_l[z, :, :sq[z]] = r[0][0], r[1][0]
    _check((out, lse), (ref_o, ref_l))


def test_no_memory_for_the_workspace():
    """A call that would be cut runs uncut where the workspace cannot be had (here 97 MiB), as it did before
    there was one."""
    Z, H, N, D = 1, 1, 32768, 128
    q, k, v, _ = oracle.make_inputs(Z, N, H, D, seed=66)
    q, k, v = q.cuda(), k.cuda(), v.cuda()
    scale = oracle.default_scale(D)
    want = _fwd(q, k, v, scale, True)
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (60 << 20)) / total)
    try:
        with pytest.raises(torch.cuda.OutOfMemoryError):
            torch.empty(90 << 20, dtype=torch.uint8, device="cuda")
        got = _fwd(q, k, v, scale, True)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert oracle.max_abs(got[0].float(), want[0].float()) <= 2 * helpers.TOL_O_MAX_ABS
    assert oracle.max_abs(got[1], want[1]) <= 2 * helpers.TOL_LSE_MAX_ABS


@pytest.mark.parametrize("D", [64, 128])
def test_runs_of_items_without_work(D):
    """Far more items than SMs, most of them of entries without a single row, in runs longer than the
    kernel publishes items ahead."""
    Z, H, N = 24, 16, 512
    lens = [0] * Z
    lens[0], lens[5], lens[6], lens[17], lens[23] = 512, 1, 300, 129, 64
    q, k, v, _ = oracle.make_inputs(Z, N, H, D, seed=64)
    scale = oracle.default_scale(D)
    out, lse = _fwd(q, k, v, scale, True, lens, lens)
    for z in range(Z):
        a = lens[z]
        assert not out[z, a:].any() and torch.isinf(lse[z, :, a:]).all()
        if a:
            ref = oracle.attention_forward(q[z:z + 1, :a], k[z:z + 1, :a], v[z:z + 1, :a], scale, True)
            _check((out[z:z + 1, :a], lse[z:z + 1, :, :a]), ref)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("first_large", [0, 64, 128, 192, 448])
def test_new_reference_in_mid_round(first_large, D):
    """Scores that leap by far more than 2^10 at a key in the first or second half of a 128-key round, in
    the first, a middle and the last round: the reference found before it must be replaced, the
    accumulator and the row sum rescaled, whichever half of a round notices it."""
    Z, N, H = 1, 512, 2
    q, k, v, _ = oracle.make_inputs(Z, N, H, D, seed=65)
    k = k.float()
    k[:, first_large:] *= 6.0
    k = k.half()
    scale = oracle.default_scale(D)
    (out, lse), (r_out, r_lse) = _fwd(q, k, v, scale, False), oracle.attention_forward(q, k, v, scale, False)
    # these rows see one or two keys, so O is as large as V: every weight is rounded to fp16 (relative
    # 2^-11, the row sum is not), and so is O
    bound = 2.0 ** -11 * (v.float().abs().max().item() + r_out.abs().max().item())
    assert oracle.max_abs(out.float(), r_out) <= bound
    assert oracle.max_abs(lse, r_lse) <= helpers.TOL_LSE_MAX_ABS
