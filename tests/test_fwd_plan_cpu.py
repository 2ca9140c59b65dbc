"""CPU tests of how the forward's work is cut for few queries: the workspace that a call asks for (one plane of fp32 rows and
LSE per chunk) tells the number of chunks.  Without a device the plan is that for 148 SMs."""
import ctypes

import pytest

from flash_attn_v100 import cabi


def _chunks(heads, n_q, n_k, D, causal=0, shift=0, padded=False):
    p = cabi.FmhaFwdParams()
    p.seqused_k = 16 if padded else None  # an address that a plan does not follow
    p.batch, p.heads, p.seqlen_q, p.seqlen_k, p.head_dim = 1, heads, n_q, n_k, D
    p.scale, p.causal, p.causal_shift = D ** -0.5, causal, shift
    plane = heads * n_q * (D + 1) * 4
    nbytes = cabi.load_library().fmha_fwd_workspace_bytes(ctypes.byref(p))
    assert nbytes % plane == 0
    return nbytes // plane


# pairs of chunks against whole items, us, bf16, where the partial rows weigh more than the idle half of the SM costs
@pytest.mark.parametrize("heads,n_q,n_k,D", [
    (1200, 128, 2048, 64),  # 246 / 192
    (296, 128, 2048, 64),   # 66 / 53
    (128, 128, 2048, 64),   # 35 / 30
    (148, 112, 2048, 64),   # 39 / 34
    (1200, 128, 2500, 64),  # 275 / 239
    (148, 127, 2500, 64),   # 45 / 41
])
def test_not_cut_where_that_is_slower(built_library, heads, n_q, n_k, D):
    assert _chunks(heads, n_q, n_k, D) == 0


# more than eight items per SM are cut in pairs of chunks only
@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("n_q", [1, 16, 64, 80])
def test_pairs_however_many_items(built_library, n_q, D):
    assert _chunks(1200, n_q, 8192, D) % 2 == 0
    assert _chunks(1200, n_q, 8192, D) >= 2
    assert _chunks(1200, n_q, 512, D) == 0  # chunks of less than 8 tiles


@pytest.mark.parametrize("D", [64, 96, 128])
def test_more_query_rows_are_not_cut_sooner(built_library, D):
    """Partial rows cost and nothing else depends on their number, up to full tiles."""
    for n_k in (2048, 2500, 3000, 4096, 8192):
        for heads in (64, 148, 296, 600, 1200):
            cut = [_chunks(heads, n_q, n_k, D) > 0 for n_q in (1, 32, 64, 96, 112, 127)]
            assert cut == sorted(cut, reverse=True), (heads, n_k, cut)


@pytest.mark.parametrize("heads,n_q,n_k,D", [(160, 64, 8192, 64), (600, 64, 3000, 64), (160, 96, 8192, 64), (64, 32, 8192, 128)])
def test_a_mask_that_hides_nothing_changes_no_plan(built_library, heads, n_q, n_k, D):
    """(two waves of 160 whole items under a causal mask 199 us, in pairs 108)"""
    assert _chunks(heads, n_q, n_k, D, 1, n_k) == _chunks(heads, n_q, n_k, D) >= 2


# 8 entries of n_k / 8 to n_k keys, pairs against whole items, us
@pytest.mark.parametrize("heads,n_q,n_k,D", [
    (600, 96, 2048, 64),   # 101 / 77
    (600, 128, 4096, 64),  # 152 / 119
    (296, 64, 2048, 64),   # 52 / 45
    (600, 64, 4096, 128),  # 179 / 159
])
def test_a_padded_batch_is_not_cut_where_that_is_slower(built_library, heads, n_q, n_k, D):
    assert _chunks(heads, n_q, n_k, D, padded=True) == 0


# ... 43 / 35 where the alternative is cut, too, and 105 / 76 for many keys
@pytest.mark.parametrize("heads,n_q,n_k,D", [(64, 64, 4096, 128), (128, 64, 8192, 64), (1200, 16, 8192, 128)])
def test_a_padded_batch_is_cut_in_pairs(built_library, heads, n_q, n_k, D):
    assert _chunks(heads, n_q, n_k, D, padded=True) >= 2


# one or two whole waves of items, us, whole items / pairs: full waves leave little idle, and many rows many partial results
@pytest.mark.parametrize("heads,n_q,n_k,D", [
    (148, 128, 4096, 128),  # 59 / 73
    (148, 128, 2500, 96),   # 38 / 47
    (296, 128, 3000, 96),   # 82 / 99
    (148, 127, 2048, 96),   # 35 / 43
    (296, 112, 4096, 128),  # 122 / 137
    (200, 128, 3000, 128),  # 80 / 91
])
def test_full_waves_are_not_cut_in_pairs(built_library, heads, n_q, n_k, D):
    assert _chunks(heads, n_q, n_k, D) == 0


# 8 entries of n_k / 8 to n_k keys, us: two items per head / one, where one is a little more than an SM
@pytest.mark.parametrize("heads,n_q,n_k,D", [(200, 128, 8192, 64), (200, 127, 6144, 64), (200, 96, 8192, 128)])
def test_a_padded_batch_is_cut_twice_where_once_is_slower(built_library, heads, n_q, n_k, D):
    """(83 / 110, 77 / 101, 107 / 140)"""
    assert _chunks(heads, n_q, n_k, D, padded=True) == 4


@pytest.mark.parametrize("padded", [False, True])
@pytest.mark.parametrize("D", [64, 96, 128])
def test_bytes_of_the_workspace_are_bounded(built_library, D, padded):
    """The bounds that include/fmha_b200.h states, for those who size scratch without asking."""
    worst = [0.0, 0.0]
    for n_q in (128,):
        for tiles in [*range(1, 50), 65, 128]:
            for n_k in (128 * (tiles - 1) + 1, 128 * tiles):
                for heads in (1, 27, 28, 40):
                    share = _chunks(heads, n_q, n_k, D, padded=padded) * n_q * (D + 1) / (n_k * D)
                    few = heads < 28 or n_k < 1921
                    worst[few] = max(worst[few], share)
    assert 0.25 < worst[False] <= 0.34
    assert 0.34 < worst[True] <= 0.62
