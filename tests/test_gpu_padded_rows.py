"""GPU tests of what the helper kernels of the backward do with padding rows: dQ is zero there, whatever the
workspace held before and whichever call converts it."""
import pytest
import torch

from oracle import attention_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,dtype", [(64, torch.float16), (96, torch.bfloat16), (128, torch.float16)])
@pytest.mark.parametrize("in_steps", [False, True])
def test_padding_rows_of_dq(D, dtype, in_steps):
    from flash_attn_v100 import cabi

    Z, N, H = 5, 320, 3
    lens = [320, 129, 128, 1, 0]
    q, k, v, dout = (t.to(dtype).cuda() for t in oracle.make_inputs(Z, N, H, D, seed=95))
    lens_d = torch.tensor(lens, dtype=torch.int32, device="cuda")
    scale = oracle.default_scale(D)
    out, lse = cabi.fwd(q, k, v, scale, True, seqused_q=lens_d, seqused_k=lens_d)

    def run(fill, out, dout):
        ws = torch.full((cabi.bwd_workspace_bytes(Z, N, H, D),), fill, dtype=torch.uint8, device="cuda")
        dq = torch.full_like(q, float("nan"))
        kw = dict(workspace=ws, seqused_q=lens_d, seqused_k=lens_d)
        if not in_steps:
            return cabi.bwd(q, k, v, out, dout, lse, scale, True, dq=dq, **kw)
        cabi.bwd(q, k, v, out, dout, lse, scale, True, flags=cabi.FMHA_BWD_PREPROCESS_ONLY, **kw)
        _, dk, dv = cabi.bwd(q, k, v, None, dout, lse, scale, True, **kw,
                             flags=cabi.FMHA_BWD_KEEP_WORKSPACE | cabi.FMHA_BWD_SKIP_DQ_CONVERT)
        return cabi.bwd_convert_dq(ws, dq, scale), dk, dv

    clean = run(0, out, dout)
    junk_out, junk_dout = out.clone(), dout.clone()
    for z in range(Z):
        junk_out[z, lens[z]:] = 9.0
        junk_dout[z, lens[z]:] = 9.0
    dirty = run(255, junk_out, junk_dout)  # bytes of 255 are NaN in fp32
    for a, b in zip(clean, dirty):
        assert torch.isfinite(b).all()
        assert oracle.rel_l2(a.float().cpu(), b.float().cpu()) < 1e-3  # dQ: the order of its additions varies
    for z in range(Z):
        assert not dirty[0][z, lens[z]:].any()


# a backward continued on the workspace of one that was complete in itself: the accumulator carries over, its padding
# rows as zeros
@pytest.mark.parametrize("D,dtype", [(64, torch.float16), (96, torch.bfloat16), (128, torch.float16)])
@pytest.mark.parametrize("then", ["nothing", "convert", "keep", "keep, convert"])
def test_padding_rows_of_dq_on_a_kept_workspace(D, dtype, then):
    from flash_attn_v100 import cabi

    Z, N, H = 5, 320, 3
    lens = [320, 129, 128, 1, 0]
    q, k, v, dout = (t.to(dtype).cuda() for t in oracle.make_inputs(Z, N, H, D, seed=96))
    lens_d = torch.tensor(lens, dtype=torch.int32, device="cuda")
    scale = oracle.default_scale(D)
    out, lse = cabi.fwd(q, k, v, scale, True, seqused_q=lens_d, seqused_k=lens_d)
    ws = torch.full((cabi.bwd_workspace_bytes(Z, N, H, D),), 255, dtype=torch.uint8, device="cuda")  # NaN in fp32
    kw = dict(workspace=ws, seqused_q=lens_d, seqused_k=lens_d)
    first, _, _ = cabi.bwd(q, k, v, out, dout, lse, scale, True, **kw)
    dq = torch.full_like(q, float("nan"))
    if then == "nothing":  # the workspace is given up: the same result on another one full of NaN
        ws.fill_(255)
        cabi.bwd(q, k, v, out, dout, lse, scale, True, dq=dq, flags=cabi.FMHA_BWD_DROP_WORKSPACE, **kw)
    elif then == "keep":
        cabi.bwd(q, k, v, None, dout, lse, scale, True, dq=dq, flags=cabi.FMHA_BWD_KEEP_WORKSPACE, **kw)
    else:
        if then == "keep, convert":
            cabi.bwd(q, k, v, None, dout, lse, scale, True, **kw,
                     flags=cabi.FMHA_BWD_KEEP_WORKSPACE | cabi.FMHA_BWD_SKIP_DQ_CONVERT)
        cabi.bwd_convert_dq(ws, dq, scale)
    assert torch.isfinite(dq).all()
    for z in range(Z):
        assert not dq[z, lens[z]:].any()
    # two calls add the same dQ twice; each result is rounded to the 16-bit type on its own (2^-8 for bf16)
    times = 2 if "keep" in then else 1
    assert oracle.rel_l2(dq.float().cpu(), times * first.float().cpu()) < 5e-3
