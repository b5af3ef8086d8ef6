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


@pytest.mark.parametrize('grad', [False, True])
@pytest.mark.parametrize('name', [n for n in NAMES if n != 'conv_step'])
def test_a_trace_replays_the_operator(name, grad):
    """torch.jit.trace keeps a call as an operation: other inputs, of another length too, give what the call gives."""
    call, inputs = _operators()[name]

    class Call(torch.nn.Module):   # the modules' weights belong to the traced module
        def __init__(self):
            super().__init__()
            self.op = next((c.cell_contents for c in call.__closure__ or () if isinstance(c.cell_contents, torch.nn.Module)), None)

        def forward(self, *args):
            return call(*args)
    with torch.set_grad_enabled(grad):
        traced = torch.jit.trace(Call(), tuple(x.requires_grad_(grad) for x in inputs(70, 0)), check_trace=False)
        for tokens in (70, 90):
            args = [x.requires_grad_(grad) for x in inputs(tokens, 1)]
            want, got = ([y] if torch.is_tensor(y) else list(y) for y in (call(*args), traced(*args)))
            assert all(torch.equal(a, b) for a, b in zip(want, got)) and len(want) == len(got)
            if grad and name != 'recurrent':
                dy = torch.ones_like(want[0])
                for a, b in zip(torch.autograd.grad(want[0], args, dy), torch.autograd.grad(got[0], args, dy)):
                    assert torch.equal(a, b)


def test_a_state_updated_in_place_is_not_recorded():
    from b200gdn.modules import causal_conv1d
    x, w, cache = (torch.ones(*s, device='cuda') for s in ((3, 1, 64), (64, 4), (3, 64, 4)))
    with pytest.raises(RuntimeError, match='cannot be recorded'):
        torch.jit.trace(lambda *a: causal_conv1d(*a, initial_state=cache, output_final_state=True, inplace_state=True), (x, w))


def test_sizes_of_zero_and_unclear_switches_raise():
    """Mistakes that native code would end the process for, or notice too late."""
    from b200gdn import B200GDNError
    from b200gdn.modules import causal_conv1d, rms_norm_gated
    with pytest.raises(B200GDNError, match='without elements'):
        rms_norm_gated(torch.zeros(4, 0, device='cuda'), torch.zeros(4, 0, device='cuda'), None)
    x, w = torch.zeros(1, 4, 64, device='cuda'), torch.zeros(64, 4, device='cuda')
    with pytest.raises(RuntimeError, match='ambiguous'):
        causal_conv1d(x, w, output_final_state=torch.ones(2))


def _forget_tables():
    """Everything that the package keeps about sequences is dropped and the memory it was in is written over."""
    import gc
    from b200gdn import index
    index._cache.clear()
    index._split_cache.clear()
    gc.collect()
    return [torch.zeros(128, dtype=torch.int32, device='cuda') for _ in range(4096)]


@pytest.mark.parametrize('name', ['chunk', 'conv'])
@pytest.mark.parametrize('pieces', [None, 3])
def test_a_captured_graph_keeps_its_tables(name, pieces):
    """A graph is replayed after the tables of its sequences have left the cache; its end gives them back."""
    from b200gdn import _lib, index
    call, inputs = _operators()[name]
    args = [x.requires_grad_(True) for x in inputs(200, 0)]

    def step():
        out = call(*args)[0]
        return (out.detach(), *torch.autograd.grad(out, args, torch.ones_like(out)))
    index.FORCE_PIECES = pieces
    try:
        _forget_tables()
        before = _lib.host().plans_alive()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = step()
        graph.replay()
        want = [x.clone() for x in got]
        torch.cuda.synchronize()
        kept = _forget_tables()
        assert _lib.host().plans_alive() > before
        for x in got:
            x.fill_(float('nan'))
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(want, got))
        del graph, kept
        torch.cuda.synchronize()
        _forget_tables()
        call(*inputs(7, 0))   # makes a plan, which drops what ended graphs held
        _forget_tables()
        assert _lib.host().plans_alive() == before
    finally:
        index.FORCE_PIECES = None


@pytest.mark.parametrize('name', ['chunk', 'conv'])
def test_tables_outlast_their_use_on_another_stream(name):
    """The tables leave the cache while a stream other than the one they were made on has yet to read them."""
    call, inputs = _operators()[name]
    args = inputs(200, 0)
    with torch.no_grad():
        want = call(*args)
        _forget_tables()
        call(*args)              # the tables are made here
        torch.cuda.synchronize()
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            torch.cuda._sleep(20_000_000)
            got = call(*args)
        kept = _forget_tables()
        side.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(want, got)) and len(kept)


def test_tensors_too_short_or_elsewhere_are_refused():
    """The kernels take their sizes from q and v (x): another tensor that is shorter, or not on the device, is refused before
    anything is launched."""
    from b200gdn import B200GDNError, chunk_gated_delta_rule, fused_recurrent_gated_delta_rule
    from b200gdn.modules import causal_conv1d, rms_norm_gated
    z = lambda *s, **kw: torch.zeros(*s, device='cuda', **kw)   # noqa: E731
    q, v, g, state = z(2, 65, 2, 64), z(2, 65, 4, 64), z(2, 65, 4), z(2, 4, 64, 64)
    good = dict(k=q, v=v, g=g, beta=g, initial_state=state, A_log=z(4), dt_bias=z(4))
    gate = dict(use_gate_in_kernel=True, output_final_state=True)

    def variants(args, **short):
        for name, x in short.items():
            for bad in (x, args[name].cpu()):
                yield name, {**args, name: bad}
    for op in (chunk_gated_delta_rule, fused_recurrent_gated_delta_rule):
        op(q, **good, **gate)
        for name, args in variants(good, k=q[:1], v=v[:1], g=g[:, :64], beta=g[:1], initial_state=state[:1], dt_bias=z(3)):
            with pytest.raises(B200GDNError, match='expected'):
                op(q, **args, **gate)
    x = z(2, 65, 64)
    conv = dict(weight=z(64, 4), bias=z(64), residual=x, initial_state=z(2, 64, 4))
    causal_conv1d(x, **conv)
    for name, args in variants(conv, weight=z(32, 4), bias=z(63), residual=x[:, :64], initial_state=z(1, 64, 4)):
        with pytest.raises(B200GDNError, match=f'{name} .* expected'):
            causal_conv1d(x, **args)
    norm = dict(g=x, weight=z(64), bias=z(64))
    rms_norm_gated(x, **norm)
    for name, args in variants(norm, g=x[:1], weight=z(63), bias=z(1)):
        with pytest.raises(B200GDNError, match=f'{name} .* expected'):
            rms_norm_gated(x, **args)
