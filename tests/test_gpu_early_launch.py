"""GPU tests of a kernel that is launched before the writes of the one before it are visible, and waits for them itself
(the join of a cut forward): in a captured graph, and call after call on two streams, it sees what the kernel before it
wrote, and the backward what it wrote."""
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


@pytest.mark.parametrize("shape", SHAPES[:3])
@pytest.mark.parametrize("poison", [False, True])
def test_join_sees_the_chunks_of_its_own_call(shape, poison):
    """A workspace holds the partial results of the call before, on other inputs, or NaN: a join that did not wait would
    read them.  Against the uncut forward."""
    import ctypes

    from flash_attn_v100 import cabi

    Z, H, n_q, n_k, D, _ = shape
    scale = oracle.default_scale(D)
    streams = [torch.cuda.Stream() for _ in range(2)]
    jobs = []
    for i, s in enumerate(streams):
        data = [_calls(shape, 10 + 2 * i + k, torch.float16)[1][:3] for k in range(2)]
        out, lse = (torch.empty((8, Z, n_q, H, D), dtype=torch.float16, device="cuda"),
                    torch.empty((8, Z, H, n_q), device="cuda"))
        p = cabi.fwd_params(*data[0], out[0], lse[0], scale, False)
        nbytes = cabi.load_library().fmha_fwd_workspace_bytes(ctypes.byref(p))
        assert nbytes > 0
        jobs.append((s, data, out, lse, torch.full((nbytes,), 255, dtype=torch.uint8, device="cuda")))
    torch.cuda.synchronize()
    for n in range(8):
        for s, data, out, lse, workspace in jobs:
            with torch.cuda.stream(s):
                if poison:
                    workspace.fill_(255)
                cabi.fwd(*data[n % 2], scale, out=out[n], lse=lse[n], workspace=workspace)
    torch.cuda.synchronize()
    for _, data, out, lse, _ in jobs:
        for k in range(2):
            want, want_lse = cabi.fwd(*data[k], scale)
            for n in range(k, 8, 2):
                # (the probabilities, at most 1, are rounded to fp16, 2^-11, relative to other references)
                assert oracle.max_abs(out[n].float(), want.float()) <= 2e-3
                assert oracle.max_abs(lse[n], want_lse) <= 1e-4
