"""GPU tests of the forward kernel on scores that N(0, 1) inputs never have: not finite, or far above
everything that their row has seen before.  Each runs with several work items per SM (the epilogue
of an item waits behind the first round of the next) and, through the extension, with query blocks
cut into chunks.  The expected values are torch's own softmax in fp32."""
import pytest
import torch

from oracle import attention_oracle as oracle
from tests import helpers

pytestmark = pytest.mark.gpu

MANY = (30, 16, 256)  # 480 items of 256 query rows: more than three per SM
FEW = (1, 2, 1024)    # 8 items: cut into chunks of the KV range where a workspace is given


def _reference(q, k, v, scale, causal):
    q, k, v = (t.float().transpose(1, 2) for t in (q, k, v))
    s = q @ k.transpose(2, 3) * scale
    if causal:
        s = s.masked_fill(~torch.ones(s.shape[2:], dtype=torch.bool).tril(), float("-inf"))
    return (s.softmax(-1) @ v).transpose(1, 2), s.logsumexp(-1)


def _run(q, k, v, scale, causal):
    """(out, lse) through the C ABI (uncut; the status word has to stay 0) and through the extension (cut
    where that pays)."""
    import flash_attn_v100_cuda as ext
    from flash_attn_v100 import cabi

    q, k, v = q.cuda(), k.cuda(), v.cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, lse = cabi.fwd(q, k, v, scale, causal, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0, f"a wait gave up: {int(status.item()):#x}"
    yield out.cpu(), lse.cpu()
    out, lse = ext.fwd_lse(q, k, v, None, scale, causal, None, None)
    yield out.cpu(), lse.cpu()


def _check(got, ref, tol_o):
    """Rows whose LSE is not finite have no finite output, all others are right."""
    (out, lse), (r_out, r_lse) = got, ref
    good = torch.isfinite(r_lse)
    assert torch.equal(torch.isfinite(lse), good)
    rows = good.transpose(1, 2)  # (Z, N, H) like the rows of out
    assert not torch.isfinite(out[~rows]).any()
    assert oracle.max_abs(out[rows].float(), r_out[rows]) <= tol_o
    # fp32 on both sides: a few roundings of numbers as large as the LSE
    bound = helpers.TOL_LSE_MAX_ABS + 2.0 ** -21 * r_lse[good].abs().max().item()
    assert oracle.max_abs(lse[good], r_lse[good]) <= bound


@pytest.mark.parametrize("shape", [MANY])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [64, 96, 128])
def test_query_rows_that_are_not_finite(D, causal, shape):
    """NaN and inf in single rows of Q: in the first round of an item nothing may wait for the first
    O += of that item, which itself waits for the epilogue of the item before."""
    Z, H, N = shape
    q, k, v, _ = oracle.make_inputs(Z, N, H, D, seed=70)
    scale = oracle.default_scale(D)
    for z in range(Z):
        for h in range(z % 2, H, 2):
            q[z, 100 + h, h, 3] = float("nan")
            q[z, N - 100 + h, h, 1] = float("inf") if z % 3 else float("-inf")
    ref = _reference(q, k, v, scale, causal)
    for got in _run(q, k, v, scale, causal):
        _check(got, ref, helpers.TOL_O_MAX_ABS)


@pytest.mark.parametrize("shape", [MANY, FEW])
@pytest.mark.parametrize("D", [64, 128])
def test_rows_whose_first_keys_are_all_minus_inf(D, shape):
    """bf16 scores that overflow to -inf for the 128 keys of an item's first round: such a row has no
    reference until the second round and is an ordinary row from there on."""
    Z, H, N = shape
    q, k, v, _ = oracle.make_inputs(Z, N, H, D, seed=71, dtype=torch.bfloat16)
    q[..., 0], k[..., 0] = 0.0, 0.0
    k[:, :128, :, 0] = 1e38
    q[:, 5::16, :, 0] = -1e38
    scale = oracle.default_scale(D)
    ref = _reference(q, k, v, scale, False)
    assert torch.isfinite(ref[1]).all()
    for got in _run(q, k, v, scale, False):
        _check(got, ref, helpers.TOL_O_MAX_ABS_BF16)


@pytest.mark.parametrize("shape", [MANY, FEW])
@pytest.mark.parametrize("D", [64, 128])
def test_leap_in_the_second_half_of_the_first_round(D, shape):
    """Keys 64-127 score far above keys 0-63 (by more than 2^10 in P, which asks for a new reference), in
    items that follow others on their SM."""
    Z, H, N = shape
    q, k, v, _ = oracle.make_inputs(Z, N, H, D, seed=72)
    k[:, 64:128] *= 8.0
    k[:, 128:] *= 0.5
    scale = oracle.default_scale(D)
    ref = _reference(q, k, v, scale, False)
    # rows with all their weight on a key or two: P is rounded to fp16 (2^-11, the row sum is not), so is O
    bound = 2.0 ** -11 * (v.float().abs().max().item() + ref[0].abs().max().item())
    for got in _run(q, k, v, scale, False):
        _check(got, ref, bound)
