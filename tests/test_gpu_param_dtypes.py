"""Gates, betas and parameters are read (and their gradients written) in the caller's element type by the kernels
themselves: the same results as with the tensors widened to fp32 first, gradients rounded once."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DTYPES = [torch.bfloat16, torch.float16]


@pytest.mark.parametrize('dtype', DTYPES)
@pytest.mark.parametrize('mixed', [False, True])
def test_gate_and_beta_dtype(dtype, mixed):
    from b200gdn import chunk_gated_delta_rule, fused_recurrent_gated_delta_rule
    gen = torch.Generator(device='cuda').manual_seed(3)
    rn = lambda *s: torch.randn(*s, device='cuda', generator=gen)
    B, T, H, HV, K = 2, 77, 2, 4, 64
    q, k, v = (rn(B, T, h, K).to(torch.bfloat16) for h in (H, H, HV))
    g, beta = rn(B, T, HV).to(dtype), rn(B, T, HV).to(torch.float32 if mixed else dtype)
    A_log, dt_bias, do = rn(HV) * 0.3, rn(HV) * 0.3, rn(B, T, HV, K).to(torch.bfloat16)
    opts = dict(use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True)

    def run(g_, b_):
        leaves = [x.detach().requires_grad_(True) for x in (q, k, v, g_, b_, A_log, dt_bias)]
        o, _ = chunk_gated_delta_rule(*leaves[:5], A_log=leaves[5], dt_bias=leaves[6], **opts)
        return [o] + list(torch.autograd.grad(o, leaves, do))
    narrow, wide = run(g, beta), run(g.float(), beta.float())
    for i, (a, b) in enumerate(zip(narrow, wide)):
        assert torch.equal(a, b.to(a.dtype)), i
    assert narrow[4].dtype == dtype and narrow[5].dtype == beta.dtype
    with torch.no_grad():
        for t in (1, T):
            a = fused_recurrent_gated_delta_rule(q[:, :t], k[:, :t], v[:, :t], g[:, :t], beta=beta[:, :t], A_log=A_log, dt_bias=dt_bias,
                                                 output_final_state=True, **opts)
            b = fused_recurrent_gated_delta_rule(q[:, :t], k[:, :t], v[:, :t], g[:, :t].float(), beta=beta[:, :t].float(), A_log=A_log,
                                                 dt_bias=dt_bias, output_final_state=True, **opts)
            assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


@pytest.mark.parametrize('dtype', DTYPES)
def test_parameter_dtype_of_the_modules(dtype):
    from b200gdn import causal_conv1d, rms_norm_gated
    gen = torch.Generator(device='cuda').manual_seed(4)
    rn = lambda *s: torch.randn(*s, device='cuda', generator=gen)
    x, dy = rn(2, 75, 128).to(dtype), rn(2, 75, 128).to(dtype)
    w, b, gate, nw = rn(128, 1, 4).to(dtype), rn(128).to(dtype), rn(2, 75, 128).to(dtype), rn(128).to(dtype)

    def run(w_, b_, nw_):
        leaves = [t.detach().requires_grad_(True) for t in (x, gate, w_, b_, nw_)]
        y, _ = causal_conv1d(leaves[0], leaves[2], leaves[3], activation='silu')
        z = rms_norm_gated(y, leaves[1], leaves[4])
        return [y, z] + list(torch.autograd.grad(z, leaves, dy))
    narrow, wide = run(w, b, nw), run(w.float().squeeze(1), b.float(), nw.float())
    for i, (a, c) in enumerate(zip(narrow, wide)):
        assert torch.equal(a, c.to(a.dtype).view_as(a)), i
    assert narrow[4].shape == w.shape and narrow[4].dtype == dtype
