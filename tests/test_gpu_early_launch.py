"""GPU tests of a kernel that is set up while the one before it is still in work (the join of a cut forward): in a
captured graph, and call after call on two streams, it sees what the kernel before it wrote, and the backward what it
wrote."""
import pytest
import torch

from oracle import attention_oracle as oracle

pytestmark = pytest.mark.gpu

SHAPES = [  # Z, H, n_q, n_k, D, deterministic
    (1, 32, 64, 8192, 128, False),  # pairs of chunks
    (1, 300, 32, 4096, 64, False),  # ... more items than SMs
    (1, 2, 512, 4096, 128, True),   # an ordinary cut
    (2, 40, 384, 384, 96, False),   # none
]


def _calls(shape, seed, dtype):
    from flash_attn_v100 import cabi, flash_attn_interface  # noqa: F401 (registers the ops)

    Z, H, n_q, n_k, D, det = shape
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v, dout = (torch.randn((Z, n, H, D), generator=g, device="cuda", dtype=dtype) for n in (n_q, n_k, n_k, n_q))
    scale = oracle.default_scale(D)
    flags = cabi.FMHA_BWD_DETERMINISTIC if det else 0

    def run():
        out, lse = torch.ops.flash_attn_v100.fwd(q, k, v, scale, False)  # (takes the workspace that a cut needs)
        return (out, lse, *cabi.bwd(q, k, v, out, dout, lse, scale, flags=flags))

    return run, (q, k, v, dout)


def _close(got, want):
    for a, b in zip(got, want):
        assert torch.isfinite(a).all()
        # dQ: another order of fp32 additions, rounded once
        assert oracle.rel_l2(a.float().cpu(), b.float().cpu()) < 2e-3


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_captured(shape, dtype):
    run, inputs = _calls(shape, 1, dtype)
    run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run()
    for seed in (2, 3):
        other, values = _calls(shape, seed, dtype)
        want = [t.clone() for t in other()]
        for t, x in zip(inputs, values):
            t.copy_(x)
        for t in got:
            t.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        _close(got, want)


@pytest.mark.parametrize("shape", SHAPES)
def test_call_after_call_on_two_streams(shape):
    runs = [_calls(shape, seed, torch.float16)[0] for seed in (4, 5)]
    want = [[t.clone() for t in r()] for r in runs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in runs]
    got = [[], []]
    for _ in range(6):
        for i, (r, s) in enumerate(zip(runs, streams)):
            with torch.cuda.stream(s):
                got[i].append(r())
    torch.cuda.synchronize()
    for results, w in zip(got, want):
        for x in results:
            _close(x, w)
