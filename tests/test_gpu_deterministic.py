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


@pytest.mark.parametrize("H", [4, 24])  # 100 items; 600: most of them are drawn by CTAs that have done others
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


@pytest.mark.parametrize("Z,H,N,D,causal", [
    (1, 3, 256, 64, False),   # fewer items than SMs
    (1, 37, 512, 128, True),  # as many
    (2, 40, 640, 96, False),  # more
    (2, 16, 512, 64, True),   # order words that fill their last 256 bytes
    (1, 1, 128, 128, False),  # one item, one query tile
    (1, 2, 128, 64, True),
])
def test_every_item_is_drawn_from_the_counter(Z, H, N, D, causal):
    """No item may be handed out before one that it waits for.  A counter among the order words of the workspace
    says so: it has counted every item, and one draw of every CTA that found none left."""
    from flash_attn_v100 import cabi

    q, k, v, dout = (t.cuda() for t in oracle.make_inputs(Z, N, H, D, seed=95))
    scale = oracle.default_scale(D)
    out, lse = cabi.fwd(q, k, v, scale, causal)
    tiles = N // 128
    at = Z * H * (N * D + 2 * tiles * 128)  # behind the dQ accumulator and two statistics of every row
    workspace = torch.full((cabi.bwd_workspace_bytes(Z, N, H, D) // 4,), 0x7f7f7f7f, dtype=torch.int32, device="cuda")
    for _ in range(2):
        cabi.bwd(q, k, v, out, dout, lse, scale, causal, workspace=workspace, flags=cabi.FMHA_BWD_DETERMINISTIC)
        items = Z * H * tiles
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        first, drawn, *words = workspace[at:at + max(2, items)].tolist()
        assert drawn == items + min(items, sms)
        # every KV tile has had its turn at every query tile that sees it
        words = ([first & 0xffff, first >> 16] + words)[:items]
        assert words == [t + 1 if causal else tiles for _ in range(Z * H) for t in range(tiles)]


def test_more_turns_than_half_a_word_holds():
    """65538 KV tiles: the first two query tiles of the call share one word, 16 bits each."""
    from flash_attn_v100 import cabi

    n_q, n_k, D = 256, 65538 * 128, 64
    g = torch.Generator(device="cuda").manual_seed(96)
    q, dout = (torch.randn((1, n_q, 1, D), generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    k, v = (torch.randn((1, n_k, 1, D), generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    scale = oracle.default_scale(D)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, lse = cabi.fwd(q, k, v, scale)
    a, b, c = (cabi.bwd(q, k, v, out, dout, lse, scale, flags=f, status=status)
               for f in (cabi.FMHA_BWD_DETERMINISTIC, cabi.FMHA_BWD_DETERMINISTIC, 0))
    assert int(status.item()) == 0
    for x, y, z in zip(a, b, c):
        assert torch.equal(x, y)
        # the other mode adds the same 65538 fp32 terms in another order (sqrt(65538) 2^-24 of their size, which is less
        # than ten times that of the sum) and rounds once (2^-9)
        assert float((x.float() - z.float()).norm() / z.float().norm()) < 2e-3
