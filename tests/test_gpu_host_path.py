"""What the operators keep of torch's own machinery below the native host path."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operators():
    """name: (call on a list of tensors, the list for a number of tokens and a seed)"""
    from b200gdn import FusedRMSNormGated, ShortConvolution, chunk_gated_delta_rule, fused_recurrent_gated_delta_rule
    torch.manual_seed(0)
    conv, norm = ShortConvolution(64, 4, bias=True, device='cuda'), FusedRMSNormGated(64, device='cuda')

    def rn(seed, *shapes):
        gen = torch.Generator(device='cuda').manual_seed(seed)
        return [torch.randn(*s, device='cuda', generator=gen) for s in shapes]

    def mixer(tokens, seed):
        q, k, v, g, beta = rn(seed, *[(1, tokens, 2, 64)] * 3, *[(1, tokens, 2)] * 2)
        q, k = (torch.nn.functional.normalize(x, dim=-1) for x in (q, k))
        return [x.to(torch.bfloat16) for x in (q, k, v)] + [torch.nn.functional.logsigmoid(g), beta.sigmoid()]
    return {
        'recurrent': (lambda q, k, v, g, b: fused_recurrent_gated_delta_rule(q, k, v, g, beta=b, output_final_state=True), mixer),
        'chunk': (lambda *a: chunk_gated_delta_rule(*a, output_final_state=True), mixer),
        'conv': (lambda x: conv(x, output_final_state=True), lambda t, s: rn(s, (1, t, 64))),
        'conv_step': (lambda x, c: conv(x, cache=c, output_final_state=True), lambda t, s: rn(s, (t, 1, 64), (t, 64, 4))),
        'norm': (lambda x, g: norm(x, g), lambda t, s: rn(s, (t, 64), (t, 64))),
    }


NAMES = ['recurrent', 'chunk', 'conv', 'conv_step', 'norm']


@pytest.mark.parametrize('grad', [False, True])
@pytest.mark.parametrize('name', NAMES)
def test_forward_mode_tangents_are_refused(name, grad):
    """No operator has a forward-mode derivative: a tangent raises and is not dropped."""
    import torch.autograd.forward_ad as fw
    call, inputs = _operators()[name]
    with torch.set_grad_enabled(grad), fw.dual_level():
        first, *rest = inputs(5, 0)
        with pytest.raises((NotImplementedError, RuntimeError), match='jvp'):
            call(fw.make_dual(first, torch.ones_like(first)), *rest)
        call(first, *rest)
