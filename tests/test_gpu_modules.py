"""GPU parity of the two steps either side of the mixer (short causal convolution, gated RMS norm) against their
oracles and the reference fixtures; tolerances as in the reference's tests (tests/modules/test_conv.py: 1e-3 err-ratio
in fp32, 5e-3 in half precision; tests/modules/test_layernorm_gated.py: 1e-3)."""
import os

import numpy as np
import pytest
import torch

from oracle import gdn_oracle as O
from tests.golden.make_modules_golden import CONV_CASES

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), 'golden')


@pytest.mark.parametrize('name', list(CONV_CASES))
def test_conv_against_reference_fixture(name):
    from b200gdn.modules import causal_conv1d
    B, T, D, W, act, has_bias, has_cache = CONV_CASES[name]
    gold = {k: torch.from_numpy(v).float() for k, v in np.load(os.path.join(GOLD, name + '.npz')).items()}
    dev = 'cuda'
    x = gold['x'].to(dev).requires_grad_(True)
    w = gold['w'].to(dev).requires_grad_(True)
    b = gold['b'].to(dev).requires_grad_(True) if has_bias else None
    cache = None
    if has_cache:
        c = gold['cache'].to(dev).requires_grad_(True)
        cache = torch.cat([torch.zeros(B, D, 1, device=dev), c], dim=-1)
    y, final = causal_conv1d(x, w, b, initial_state=cache, output_final_state=True, activation=act)
    (y * gold['dy'].to(dev)).sum().backward()
    O.assert_close('y', gold['y'], y.detach().cpu(), 1e-4)
    assert torch.allclose(final[..., 1:].cpu(), gold['final'], atol=1e-6)
    O.assert_close('dx', gold['dx'], x.grad.cpu(), 1e-4)
    O.assert_close('dw', gold['dw'], w.grad.cpu(), 1e-4)
    if has_bias:
        O.assert_close('db', gold['db'], b.grad.cpu(), 1e-4)
    if has_cache:
        O.assert_close('dcache', gold['dcache'], c.grad.cpu(), 1e-4)


@pytest.mark.parametrize('dtype,tol', [(torch.float32, 1e-4), (torch.bfloat16, 5e-3), (torch.float16, 2e-3)])
@pytest.mark.parametrize('W', [2, 3, 4])
def test_conv_packed_sequences_with_cache_and_residual(dtype, tol, W):
    """Packed ragged sequences (one shorter than the kernel, one spanning several 64-token tiles), cache, bias, residual."""
    from b200gdn.modules import causal_conv1d
    dev = 'cuda'
    cu = [0, 2, 3, 140, 204, 333]
    T, D, N = 333, 2048 + 64, 5
    gen = torch.Generator().manual_seed(11)
    x = torch.randn(1, T, D, generator=gen).to(dtype)
    w = (torch.randn(D, W, generator=gen) * 0.5)
    b = torch.randn(D, generator=gen)
    res = torch.randn(1, T, D, generator=gen).to(dtype)
    cache = torch.randn(N, D, W, generator=gen).to(dtype)
    dy = torch.randn(1, T, D, generator=gen).to(dtype)
    leaves = [t.float().double().requires_grad_(True) for t in (x, w, b, res, cache)]
    ry, rfinal = O.causal_conv1d_ref(*leaves[:4], leaves[4], 'silu', cu, True)
    (ry * dy.double()).sum().backward()
    g = [t.to(dev).requires_grad_(True) for t in (x, w, b, res, cache)]
    y, final = causal_conv1d(g[0], g[1], g[2], residual=g[3], initial_state=g[4], output_final_state=True, activation='silu',
                             cu_seqlens=torch.tensor(cu, device=dev))
    y.backward(dy.to(dev))
    assert y.dtype == dtype and final.dtype == dtype and final.shape == (N, D, W)
    O.assert_close('y', ry.float(), y.float().cpu(), tol)
    O.assert_close('final', rfinal.float(), final.float().cpu(), tol)
    for nme, a, r in zip(('dx', 'dw', 'db', 'dres', 'dcache'), g, leaves):
        got, want = a.grad.float().cpu(), r.grad.float()
        if nme == 'dcache':   # the oldest cache entry never enters the convolution
            assert torch.count_nonzero(got[..., 0]) == 0
        O.assert_close(nme, want, got, tol * (4 if nme in ('dw', 'db') and dtype != torch.float32 else 1))


def test_short_convolution_module_prefill_then_decode():
    """The layer object: a prefill with final state, then single-token steps that update the cache in place, against one
    pass over the whole sequence (tests/modules/test_conv.py:365-437, 560-640 of the reference test this contract)."""
    from b200gdn.modules import ShortConvolution
    dev = 'cuda'
    B, T, D, W = 3, 70, 256, 4
    torch.manual_seed(0)
    conv = ShortConvolution(D, W, bias=True, activation='silu', device=dev, dtype=torch.float32)
    x = torch.randn(B, T + 3, D, device=dev)
    full, _ = conv(x)
    y0, cache = conv(x[:, :T], output_final_state=True)
    assert torch.allclose(y0, full[:, :T], atol=1e-5)
    ptr = cache.data_ptr()
    for t in range(T, T + 3):
        yt, cache = conv(x[:, t:t + 1], cache=cache, output_final_state=True)
        assert cache.data_ptr() == ptr
        assert torch.allclose(yt[:, 0], full[:, t], atol=1e-5)
    want = O.causal_conv1d_ref(x.cpu().double(), conv.weight.squeeze(1).cpu().double(), conv.bias.cpu().double(), None, None, 'silu')[0]
    O.assert_close('module vs oracle', want.float(), full.cpu(), 1e-4)
    with pytest.raises(ValueError):
        conv(x, mask=torch.ones(B, T + 3, device=dev), cu_seqlens=torch.tensor([0, 1], device=dev))


@pytest.mark.parametrize('dtype,tol', [(torch.float32, 1e-4), (torch.bfloat16, 5e-3), (torch.float16, 2e-3)])
@pytest.mark.parametrize('D,act,affine', [(128, 'swish', True), (64, 'sigmoid', False), (256, 'silu', True), (512, 'swish', True)])
def test_rms_norm_gated(dtype, tol, D, act, affine):
    from b200gdn.modules import FusedRMSNormGated
    dev = 'cuda'
    B, T, H = 2, 300, 3
    gen = torch.Generator().manual_seed(7)
    x = torch.randn(B, T, H, D, generator=gen).to(dtype)
    g = torch.randn(B, T, H, D, generator=gen).to(dtype)
    dy = torch.randn(B, T, H, D, generator=gen).to(dtype)
    w = torch.randn(D, generator=gen) if affine else None
    norm = FusedRMSNormGated(D, elementwise_affine=affine, eps=1e-5, activation=act, device=dev)
    if affine:
        norm.weight.data.copy_(w)
    xr, gr = x.double().requires_grad_(True), g.double().requires_grad_(True)
    wr = w.double().requires_grad_(True) if affine else None
    ry = O.rms_norm_gated_ref(xr, gr, wr, None, act, 1e-5)
    (ry * dy.double()).sum().backward()
    xg, gg = x.to(dev).requires_grad_(True), g.to(dev).requires_grad_(True)
    y = norm(xg, gg)
    y.backward(dy.to(dev))
    assert y.dtype == dtype and y.shape == x.shape
    O.assert_close('y', ry.float(), y.float().cpu(), tol)
    O.assert_close('dx', xr.grad.float(), xg.grad.float().cpu(), tol)
    O.assert_close('dg', gr.grad.float(), gg.grad.float().cpu(), tol)
    if affine:
        O.assert_close('dw', wr.grad.float(), norm.weight.grad.float().cpu(), tol * 2)


def test_module_errors():
    from b200gdn import B200GDNError
    from b200gdn.modules import causal_conv1d, rms_norm_gated
    x = torch.zeros(1, 8, 16, device='cuda')
    with pytest.raises(ValueError, match='not supported'):
        causal_conv1d(x, torch.zeros(16, 4, device='cuda'), activation='gelu')
    with pytest.raises(B200GDNError, match='kernel size'):
        causal_conv1d(x, torch.zeros(16, 5, device='cuda'))
    with pytest.raises(NotImplementedError):
        rms_norm_gated(x, x, None, residual=x)
    with pytest.raises(B200GDNError, match='are built'):
        rms_norm_gated(torch.zeros(4, 96, device='cuda'), torch.zeros(4, 96, device='cuda'), None)


@pytest.mark.parametrize('W', [2, 3, 4])
@pytest.mark.parametrize('misaligned', [False, True])
def test_conv_single_token_step(W, misaligned):
    """One token per sequence: the same output and shifted cache as the general walk, in place, also for a cache that does
    not start on a 16-byte boundary."""
    from b200gdn.modules import causal_conv1d
    gen = torch.Generator(device='cuda').manual_seed(W)
    rn = lambda *s: torch.randn(*s, device='cuda', generator=gen).to(torch.bfloat16)
    N, D = 5, 520
    x, w, b, r, c = rn(N, 1, D), rn(D, W), rn(D), rn(N, 1, D), rn(N, D, W)
    want = (c[..., 1:].float() * w[:, :-1].float()).sum(-1) + x[:, 0].float() * w[:, -1].float() + b.float()
    want = want * torch.sigmoid(want) + r[:, 0].float()
    cache = torch.cat([c.new_zeros(1), c.flatten()])[1:].view(c.shape) if misaligned else c.clone()
    with torch.no_grad():
        y, new = causal_conv1d(x, w, b, r, cache, True, 'silu', inplace_state=True)
    assert new.data_ptr() == cache.data_ptr()
    O.assert_close('y', want.cpu(), y[:, 0].float().cpu(), 4e-3)
    assert torch.equal(new, torch.cat([c[..., 1:], x[:, 0, :, None]], -1))


@pytest.mark.parametrize('rows,D', [(1, 128), (14209, 128), (2 * 444 * 32 - 3, 64), (9473, 256), (2369, 512)])
@pytest.mark.parametrize('bias', [False, True])
def test_rms_norm_gated_rows_around_a_wave(rows, D, bias):
    """A single row and row counts at and past what one wave of CTAs takes per turn, with and without a bias."""
    from b200gdn.modules import rms_norm_gated
    gen = torch.Generator(device='cuda').manual_seed(rows)
    x, g, dy = (torch.randn(1, rows, 1, D, device='cuda', generator=gen).to(torch.bfloat16) for _ in range(3))
    leaves = [x, g, torch.randn(D, device='cuda', generator=gen)] + ([torch.randn(D, device='cuda', generator=gen)] if bias else [])
    leaves = [t.requires_grad_(True) for t in leaves]
    wide = [t.detach().double().requires_grad_(True) for t in leaves]
    ry = O.rms_norm_gated_ref(wide[0], wide[1], wide[2], wide[3] if bias else None)
    y = rms_norm_gated(*leaves[:3], leaves[3] if bias else None)
    O.assert_close('y', ry, y.double(), 5e-3)
    for n, w, t in zip(('dx', 'dg', 'dweight', 'dbias'), torch.autograd.grad(ry, wide, dy.double()), torch.autograd.grad(y, leaves, dy)):
        O.assert_close(n, w, t.double(), 1e-2)


@pytest.mark.parametrize('act', [None, 'silu'])
@pytest.mark.parametrize('with_residual', [False, True])
@pytest.mark.parametrize('with_bias', [False, True])
def test_conv_forms_at_group_and_share_edges(act, with_residual, with_bias):
    """Every compiled form (activation, residual, bias) on sequences of 1 .. 131 tokens: either side of the groups of four
    tokens, of the shares and of the tiles."""
    from b200gdn.modules import causal_conv1d
    lens, D = [1, 3, 4, 5, 8, 31, 33, 63, 64, 65, 131], 72
    cu = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32, device='cuda')
    gen = torch.Generator(device='cuda').manual_seed(5)
    mk = lambda *s: torch.randn(*s, device='cuda', generator=gen)   # noqa: E731
    x, w, dy = mk(1, sum(lens), D).requires_grad_(True), mk(D, 4).requires_grad_(True), mk(1, sum(lens), D)
    b = mk(D).requires_grad_(True) if with_bias else None
    res = mk(1, sum(lens), D).requires_grad_(True) if with_residual else None
    leaves = [t for t in (x, w, b, res) if t is not None]
    y, _ = causal_conv1d(x, w, b, residual=res, activation=act, cu_seqlens=cu)
    got = torch.autograd.grad(y, leaves, dy)
    parts = []
    for s, e in zip(cu.tolist()[:-1], cu.tolist()[1:]):
        z = torch.nn.functional.conv1d(torch.nn.functional.pad(x[:, s:e].double().transpose(1, 2), (3, 0)), w.double()[:, None],
                                       None if b is None else b.double(), groups=D).transpose(1, 2)
        parts.append(torch.nn.functional.silu(z) if act else z)
    ref = torch.cat(parts, 1) + (0 if res is None else res.double())
    O.assert_close('y', ref, y.double(), 1e-5)
    for i, (r, t) in enumerate(zip(torch.autograd.grad(ref, leaves, dy.double()), got)):
        O.assert_close(f'grad {i}', r.double(), t.double(), 1e-5)


@pytest.mark.parametrize('W', [2, 3, 4])
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float32])
def test_conv_cache_updated_in_place(W, dtype):
    """Several tokens per sequence with the final state written over the cache: bit for bit what separate tensors give, for
    sequences shorter than the kernel, of one share and of several shares and tiles."""
    from b200gdn.modules import causal_conv1d
    lens, D = [1, 2, 3, 5, 15, 16, 17, 31, 32, 33, 64, 65, 200], 520
    cu = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32, device='cuda')
    gen = torch.Generator(device='cuda').manual_seed(W)
    rn = lambda *s: torch.randn(*s, device='cuda', generator=gen).to(dtype)   # noqa: E731
    x, w, cache = rn(1, sum(lens), D), rn(D, W), rn(len(lens), D, W)
    y, new = causal_conv1d(x, w, initial_state=cache, output_final_state=True, activation='silu', cu_seqlens=cu)
    want = O.causal_conv1d_ref(x.double().cpu(), w.double().cpu(), None, None, cache.double().cpu(), 'silu', cu.tolist(), True)[1]
    assert torch.equal(new.double().cpu(), want)   # inputs and cache entries, moved only
    for _ in range(20):
        own = cache.clone()
        y2, new2 = causal_conv1d(x, w, initial_state=own, output_final_state=True, activation='silu', cu_seqlens=cu,
                                 inplace_state=True)
        assert new2.data_ptr() == own.data_ptr() and torch.equal(y2, y) and torch.equal(own, new)


@pytest.mark.parametrize('with_cache', [False, True])
def test_conv_sequences_without_tokens(with_cache):
    """An empty sequence of a packed batch keeps its cache (zeros without one) as its final state and takes no gradient; the
    memory that the results come from is filled with NaN first."""
    from b200gdn.modules import causal_conv1d
    cu, D, W = [0, 0, 5, 5, 70, 70], 64, 4
    gen = torch.Generator(device='cuda').manual_seed(3)
    x, w, c = (torch.randn(*s, device='cuda', generator=gen) for s in ((1, 70, D), (D, W), (5, D, W)))
    c = c.requires_grad_(True) if with_cache else None
    want = O.causal_conv1d_ref(x.cpu(), w.cpu(), None, None, c.detach().cpu() if with_cache else None, None, cu, True)[1]
    torch.cuda.synchronize()

    def poison():
        del (junk := [torch.full((5, D, W), float('nan'), device='cuda') for _ in range(64)])[:]
    poison()
    y, new = causal_conv1d(x, w, initial_state=c, output_final_state=True, cu_seqlens=torch.tensor(cu, device='cuda'))
    assert torch.equal(new.cpu(), want)
    if with_cache:
        poison()
        dc, = torch.autograd.grad(y.sum(), c)
        assert torch.isfinite(dc).all() and torch.count_nonzero(dc[[0, 2, 4]]) == 0


@pytest.mark.parametrize('lens', [[1, 1, 1], [1, 2, 20]])
def test_conv_gradients_with_the_cache_updated_in_place(lens):
    """The backward pass of a call that overwrote its cache uses the cache that the forward pass read."""
    from b200gdn.modules import causal_conv1d
    cu = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32, device='cuda')
    gen = torch.Generator(device='cuda').manual_seed(8)
    rn = lambda *s: torch.randn(*s, device='cuda', generator=gen)   # noqa: E731
    x, w, c, dy = rn(1, sum(lens), 64).requires_grad_(True), rn(64, 4).requires_grad_(True), rn(3, 64, 4), rn(1, sum(lens), 64)
    want = torch.autograd.grad(causal_conv1d(x, w, initial_state=c, output_final_state=True, activation='silu', cu_seqlens=cu)[0],
                               (x, w), dy)
    y, _ = causal_conv1d(x, w, initial_state=c.clone(), output_final_state=True, activation='silu', cu_seqlens=cu,
                         inplace_state=True)
    assert all(torch.equal(a, b) for a, b in zip(want, torch.autograd.grad(y, (x, w), dy)))
