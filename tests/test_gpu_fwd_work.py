"""GPU parity tests of how the forward kernel's work is cut and taken: query blocks whose KV range is
cut into chunks (partial results joined by a second kernel), items taken over through cluster
launch control, runs of items with nothing to do, and a new softmax reference in mid-round."""
import ctypes
import random

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


# seeds whose sizes make a call that is cut
@pytest.mark.parametrize("seed", [1, 4, 8, 12, 15, 19, 21, 25, 29, 30, 44, 52, 64, 71, 72, 76])
def test_cut_and_uncut_calls_agree(seed):
    """The same call with and without a workspace, over what the C ABI takes: odd lengths, shifted masks,
    per-batch lengths (zero among them), packed and transposed tensors, all head dims and types, SMs
    left free; a workspace one byte short is as good as none."""
    from flash_attn_v100 import cabi

    rng = random.Random(seed)
    Z, H, D = rng.choice([1, 2]), rng.choice([1, 3]), (64, 96, 128)[seed % 3]
    n_q, n_k = rng.choice([1, 33, 200, 513]), rng.choice([1025, 1999, 4000])
    if seed % 4 == 1:
        n_q = n_k = rng.choice([1025, 1999])
    dtype = rng.choice([torch.float16, torch.bfloat16])
    causal = seed % 4 == 1 or rng.random() < 0.4
    shift = 0 if not causal else rng.choice([0, n_k - n_q, 700, -150 if n_q > 150 else 0])
    layout = rng.choice(["dense", "packed", "heads first"])
    g = torch.Generator(device="cuda").manual_seed(seed)

    def tensor(n):
        x = torch.randn((Z, n, H, D), generator=g, device="cuda").to(dtype)
        if layout == "packed":
            return x.unsqueeze(2).expand(Z, n, 3, H, D).contiguous()[:, :, 1]
        return x.transpose(1, 2).contiguous().transpose(1, 2) if layout == "heads first" else x

    q, k, v, out = tensor(n_q), tensor(n_k), tensor(n_k), tensor(n_q)
    lens = [None, None]
    if rng.random() < 0.5:
        lens = [torch.tensor([rng.choice([n, n // 2 + 1] + [0] * z) for z in range(Z)], dtype=torch.int32, device="cuda")
                for n in (n_q, n_k)]
    kw = dict(sm_margin=rng.choice([0, 0, 20]), seqused_q=lens[0], seqused_k=lens[1])
    scale = rng.choice([1, -1]) * D ** -0.5
    want = cabi.fwd(q, k, v, scale, causal, shift, **kw)
    lse = torch.empty((Z, H, n_q), device="cuda")
    p = cabi.fwd_params(q, k, v, out, lse, scale, causal, shift, **kw)
    nbytes = cabi.load_library().fmha_fwd_workspace_bytes(ctypes.byref(p))
    assert nbytes > 0, "not a call that is cut"
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    guard = torch.full((nbytes + 256,), 0xFF, dtype=torch.uint8, device="cuda")  # NaN
    cabi.fwd(q, k, v, scale, causal, shift, out=out, lse=lse, status=status, workspace=guard[:nbytes], **kw)
    assert int(status.item()) == 0 and bool((guard[nbytes:] == 0xFF).all())
    _check((out.cpu(), lse.cpu()), (want[0].float().cpu(), want[1].cpu()), dtype)
    short = cabi.fwd(q, k, v, scale, causal, shift, workspace=guard[:nbytes - 1], **kw)
    assert torch.equal(short[0], want[0]) and torch.equal(short[1], want[1])


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
