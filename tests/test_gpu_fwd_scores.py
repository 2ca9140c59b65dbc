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
FEW = (1, 2, 1024)    # 8 items: cut into chunks of the KV range where the extension gives a workspace


def _reference(q, k, v, scale, causal):
    out, lse = torch.empty(q.shape), torch.empty((q.shape[0], q.shape[2], q.shape[1]))
    for z in range(q.shape[0]):
        qz, kz, vz = (t[z].float().transpose(0, 1) for t in (q, k, v))
        s = qz @ kz.transpose(1, 2) * scale
        if causal:
            s = s.masked_fill(~torch.ones(s.shape[1:], dtype=torch.bool).tril(), float("-inf"))
        out[z], lse[z] = (s.softmax(-1) @ vz).transpose(0, 1), s.logsumexp(-1)
    return out, lse


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


def _bound_few_keys(v, ref):
    """Max-abs error of rows with all their weight on a key or two, where O is as large as V: every
    weight is rounded to fp16 (relative 2^-11, the row sum is not), and so is O."""
    return 2.0 ** -11 * (v.float().abs().max().item() + ref[0].abs().max().item())


@pytest.mark.parametrize("shape", [MANY, FEW])
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


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [64, 96, 128])
def test_a_key_row_that_is_nan(D, causal):
    """NaN in one row of K, in another of 31 neighbouring columns from head to head: every row that sees
    the key is NaN, whichever unit its exponential comes from, and no other (the last head has none)."""
    Z, H, N = 8, 32, 512
    q, k, v, _ = oracle.make_inputs(Z, N, H, D, seed=75)
    scale = oracle.default_scale(D)
    for z in range(Z):
        for h in range(H - 1):
            k[z, 64 * z + h, h, 7] = float("nan")
    ref = _reference(q, k, v, scale, causal)
    for got in _run(q, k, v, scale, causal):
        _check(got, ref, helpers.TOL_O_MAX_ABS)


@pytest.mark.parametrize("key", [0, 8, 700])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [64, 96, 128])
def test_a_key_row_that_is_nan_in_one_of_several_chunks(D, causal, key):
    """The chunk that holds the key is NaN for the rows that see it, the others are not: so is the result."""
    Z, H, N = FEW
    q, k, v, _ = oracle.make_inputs(Z, N, H, D, seed=77)
    k[0, key, 0, 7] = float("nan")
    scale = oracle.default_scale(D)
    ref = _reference(q, k, v, scale, causal)
    for got in _run(q, k, v, scale, causal):
        _check(got, ref, helpers.TOL_O_MAX_ABS)


@pytest.mark.parametrize("D", [64, 96, 128])
def test_merged_partial_results_that_are_nan(D):
    """Both merges of ring attention: a row that is NaN in any of its parts, or in all of them, is NaN."""
    from flash_attn_v100 import cabi

    Z, H, N = 1, 2, 128
    q, k, v, _ = oracle.make_inputs(Z, N, H, D, seed=78, n_k=384)
    k[0, 130, 0, 3] = float("nan")  # head 0: the second part of three
    q[0, 5, 1, 3] = float("nan")    # head 1: row 5 of every part
    r_out, r_lse = _reference(q, k, v, 0.1, False)
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    o_acc = torch.empty((Z, N, H, D), device="cuda")
    l_acc = torch.full((Z, H, N), float("-inf"), device="cuda")
    parts = [cabi.fwd(qd, kd[:, lo:lo + 128], vd[:, lo:lo + 128], 0.1, False) for lo in (0, 128, 256)]
    for o, l in parts:
        cabi.merge(o_acc, l_acc, o, l)
    out, lse = torch.empty((Z, N, H, D), dtype=torch.float16, device="cuda"), torch.empty((Z, H, N), device="cuda")
    cabi.merge_parts([o for o, _ in parts], [l for _, l in parts], [0, 0, 0], out, lse)
    for got in ((o_acc.cpu(), l_acc.cpu()), (out.cpu(), lse.cpu())):
        _check(got, (r_out, r_lse), helpers.TOL_O_MAX_ABS)


@pytest.mark.parametrize("D", [64, 128])
def test_a_value_row_that_is_not_finite(D):
    """NaN and inf in V reach the column they are in, of every row."""
    Z, H, N = 8, 32, 512
    q, k, v, _ = oracle.make_inputs(Z, N, H, D, seed=76)
    scale = oracle.default_scale(D)
    for z in range(Z):
        for h in range(H):
            v[z, 64 * z + h, h, h] = float("nan") if h % 2 else float("inf")
    r_out, r_lse = _reference(q, k, v, scale, False)
    good = torch.isfinite(r_out)
    for out, lse in _run(q, k, v, scale, False):
        assert torch.equal(torch.isfinite(out), good)
        assert oracle.max_abs(out[good].float(), r_out[good]) <= helpers.TOL_O_MAX_ABS
        assert oracle.max_abs(lse, r_lse) <= helpers.TOL_LSE_MAX_ABS


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
    for got in _run(q, k, v, scale, False):
        _check(got, ref, _bound_few_keys(v, ref))


@pytest.mark.parametrize("D", [64, 96, 128])
def test_one_key_far_above_the_rest(D):
    """A single key above all others by 95 to 400, once in each of 16 neighbouring columns (some of whose
    exponentials are a polynomial), in either half of the first, a middle and the last round.  Only
    every second row sees it so; the others are ordinary rows of the same warps."""
    Z, H, N = 5, 96, 512
    q, k, v, _ = oracle.make_inputs(Z, N, H, D, seed=73)
    scale = oracle.default_scale(D)
    q[:, ::2, :, 0], q[:, 1::2, :, 0], k[..., 0] = 20.0, -20.0, 0.0
    for z, leap in enumerate((95.0, 130.0, 180.0, 256.0, 400.0)):
        for h in range(H):
            column, half, rnd = h % 16, (h // 16) % 2, (0, 1, 3)[h // 32]
            k[z, rnd * 128 + half * 64 + 16 * (h % 4) + column, h, 0] = leap / (20.0 * scale)
    ref = _reference(q, k, v, scale, False)
    for got in _run(q, k, v, scale, False):
        _check(got, ref, _bound_few_keys(v, ref))


@pytest.mark.parametrize("D", [64, 128])
def test_scores_of_large_standard_deviation(D):
    """q and k ten times as large as usual: nearly all the weight of a row is on one key, and every row
    meets its maximum somewhere in the middle.  Forward and gradients."""
    from flash_attn_v100 import flash_attn_func

    Z, H, N = 2, 4, 2048
    q, k, v, dout = oracle.make_inputs(Z, N, H, D, seed=74)
    q, k = q * 10, k * 10
    scale = oracle.default_scale(D)
    ref = _reference(q, k, v, scale, False)
    for got in _run(q, k, v, scale, False):
        _check(got, ref, _bound_few_keys(v, ref))
    leaves = [t.cuda().requires_grad_() for t in (q, k, v)]
    grads = torch.autograd.grad(flash_attn_func(*leaves), leaves, dout.cuda())
    for z in range(Z):
        qz, kz, vz, doz, oz = (t[z].float().transpose(0, 1) for t in (q, k, v, dout, ref[0]))
        x = (qz @ kz.transpose(1, 2) * scale - ref[1][z][..., None])
        p, dp = x.exp(), doz @ vz.transpose(1, 2)
        delta = (doz * oz).sum(-1, keepdim=True)
        ds = p * (dp - delta) * scale
        # relative error of P: its fp16 argument (x / ln 2 in base 2), the fp16 exponential (2^-9.9) and
        # its rounding; of dP, O (in delta), delta, P delta and dS: one fp16 rounding each
        e_p = p * (x.abs() * 2.0 ** -11 + 2.0 ** -9.9 + 2.0 ** -11)
        e_ds = scale * (e_p + p * 5 * 2.0 ** -11) * (dp.abs() + (doz * oz).abs().sum(-1, keepdim=True))
        for got, want, bound in ((grads[0], ds @ kz, e_ds @ kz.abs()),
                                 (grads[1], ds.transpose(1, 2) @ qz, e_ds.transpose(1, 2) @ qz.abs()),
                                 (grads[2], p.transpose(1, 2) @ doz, e_p.transpose(1, 2) @ doz.abs())):
            got = got[z].float().cpu().transpose(0, 1)
            # ... and the result itself; 1e-4: weights below the fp16 range (6e-8 each, 2048 of them)
            worst = ((got - want).abs() / (bound + want.abs() * 2.0 ** -11 + 1e-4 * 50)).max().item()
            assert worst <= 1.0, worst


@pytest.mark.parametrize("D", [64, 128])
def test_row_sum_where_the_polynomial_makes_up_most_of_it(D):
    """LSE of rows with one key of score 0 and two of score -r / 1024 in columns whose exponential is a
    polynomial, all else being far below; inputs and products are exact.  The exponential has to be
    as good as the hardware's (2 ulp)."""
    from flash_attn_v100 import cabi

    n_q, n_k = 1024, 128
    q, k = torch.zeros(1, n_q, 1, D), torch.zeros(1, n_k, 1, D)
    q[0, :, 0, 0], q[0, :, 0, 1] = -torch.arange(n_q) / 1024, 1.0
    k[0, :, 0, 1] = -1000.0
    k[0, 8, 0] = 0.0
    k[0, :2, 0, 0], k[0, :2, 0, 1] = 1.0, 0.0
    v = torch.zeros(1, n_k, 1, D).half()
    _, lse = cabi.fwd(q.half().cuda(), k.half().cuda(), v.cuda(), 1.0, False)
    want = torch.log1p(2 * torch.exp(-torch.arange(n_q).double() / 1024))
    # exponentials 2 ulp (2^-22) times their share of the sum (2/3); their arguments (up to 1.44 in base
    # 2) two roundings; the sum two; the logarithm 1 ulp of up to 1.6, its product with ln 2 one
    u = 2.0 ** -24
    bound = 4 * u * 2 / 3 + 2 * u * 1.44 * 0.7 * 2 / 3 + 2 * u + 2 * u * 1.1 + u * 1.1
    assert oracle.max_abs(lse[0, 0].cpu(), want) <= bound
