"""GPU tests of the order in which deterministic dQ is added: under a causal mask from the diagonal
downwards, where the diagonal depends on the shift and on the lengths of a padded batch."""
import pytest
import torch

from oracle import attention_oracle as oracle
from tests import helpers
from tests.test_gpu_padded import _oracle_padded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,n_q,n_k,causal,shift", [
    (40, 640, 640, True, 0),      # more items than SMs, several head groups, the last one not full
    (3, 640, 640, True, 37),      # the diagonal crosses tiles
    (3, 640, 640, True, -200),    # query rows that see nothing
    (3, 256, 1000, True, 300),    # KV tiles that no query sees
    (3, 1000, 256, True, 0),      # more query tiles than KV tiles
    (3, 300, 300, True, 100000),  # every key seen
    (40, 640, 384, False, 0),
])
@pytest.mark.parametrize("D", [64, 96, 128])
def test_order_of_dq(H, n_q, n_k, causal, shift, D):
    from flash_attn_v100 import cabi

    q, _, _, dout = oracle.make_inputs(1, n_q, H, D, seed=91)
    _, k, v, _ = oracle.make_inputs(1, n_k, H, D, seed=92)
    scale = oracle.default_scale(D)
    qd, kd, vd, dod = (t.cuda() for t in (q, k, v, dout))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, lse = cabi.fwd(qd, kd, vd, scale, causal, shift)
    runs = [cabi.bwd(qd, kd, vd, out, dod, lse, scale, causal, shift, flags=cabi.FMHA_BWD_DETERMINISTIC, status=status)
            for _ in range(2)]
    assert int(status.item()) == 0
    assert all(torch.equal(a, b) for a, b in zip(*runs))
    ref = oracle.attention_fwd_bwd(q, k, v, dout, scale, causal, shift)
    helpers.check_against_oracle((out.cpu(), lse.cpu(), *(t.cpu() for t in runs[0])), ref, f"order D{D}")


@pytest.mark.parametrize("H", [4, 24])  # 100 items; 600: most of them wait for blocks that are dispatched later
@pytest.mark.parametrize("q_row_begin", [0, 256])
def test_order_of_dq_in_a_padded_batch(q_row_begin, H):
    from flash_attn_v100 import cabi

    Z, N, D = 5, 640, 128
    sq, sk = [640, 130, 0, 513, 300], [640, 640, 128, 1, 0]
    q, k, v, dout = oracle.make_inputs(Z, N, H, D, seed=93)
    qd, kd, vd, dod = (t.cuda() for t in (q, k, v, dout))
    sqd, skd = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in (sq, sk))
    scale = oracle.default_scale(D)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, lse = cabi.fwd(qd, kd, vd, scale, True, seqused_q=sqd, seqused_k=skd)
    runs = [cabi.bwd(qd, kd, vd, out, dod, lse, scale, True, flags=cabi.FMHA_BWD_DETERMINISTIC, status=status,
                     seqused_q=sqd, seqused_k=skd, q_row_begin=q_row_begin) for _ in range(2)]
    assert int(status.item()) == 0
    assert all(torch.equal(a, b) for a, b in zip(*runs))
    # rows before q_row_begin take no part: their dQ is zero, and dK and dV are those of a dout that is zero there
    dout[:, :q_row_begin] = 0
    ref = _oracle_padded(q, k, v, dout, scale, True, sq, sk)
    assert not runs[0][0][:, :q_row_begin].any()
    helpers.check_against_oracle((out.cpu(), lse.cpu(), *(t.cpu() for t in runs[0])), ref, "order, padded")


@pytest.mark.parametrize("D,dtype", [(64, torch.bfloat16), (96, torch.float16), (128, torch.float16)])
@pytest.mark.parametrize("causal", [False, True])
def test_order_of_dq_over_many_items(D, dtype, causal):
    """Six times as many items as SMs, of one to three query tiles: a CTA has the next one while the one in work waits
    for its turns."""
    from flash_attn_v100 import cabi

    H, N = 300, 352
    g = torch.Generator(device="cuda").manual_seed(94)
    q, k, v, dout = (torch.randn((1, N, H, D), generator=g, device="cuda", dtype=dtype) for _ in range(4))
    scale = oracle.default_scale(D)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, lse = cabi.fwd(q, k, v, scale, causal)
    a, b, c = (cabi.bwd(q, k, v, out, dout, lse, scale, causal, flags=f, status=status)
               for f in (cabi.FMHA_BWD_DETERMINISTIC, cabi.FMHA_BWD_DETERMINISTIC, 0))
    assert int(status.item()) == 0
    for x, y, z in zip(a, b, c):
        assert torch.equal(x, y)
        # the other mode adds the same terms in another order and rounds once (2^-9 for bf16)
        assert oracle.rel_l2(x.float().cpu(), z.float().cpu()) < 2e-3
