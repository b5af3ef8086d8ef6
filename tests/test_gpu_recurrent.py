"""GPU parity of the decode path against the oracle recurrence (reference tolerance 0.002,
tests/ops/test_gdn.py:48-105; fp32 inputs are held to 1e-5)."""
import pytest
import torch

from oracle import gdn_oracle as O

pytestmark = pytest.mark.gpu


def _inputs(B, T, H, HV, K, V, seed, dtype):
    gen = torch.Generator().manual_seed(seed)
    q = torch.randn(B, T, H, K, generator=gen).to(dtype)
    k = torch.randn(B, T, H, K, generator=gen).to(dtype)
    v = torch.randn(B, T, HV, V, generator=gen).to(dtype)
    graw = torch.randn(B, T, HV, generator=gen)
    braw = torch.randn(B, T, HV, generator=gen)
    A_log = torch.randn(HV, generator=gen) * 0.3
    dt_bias = torch.randn(HV, generator=gen) * 0.3
    return q, k, v, graw, braw, A_log, dt_bias, gen


@pytest.mark.parametrize('K,V', [(128, 128), (64, 64), (32, 64), (256, 128)])
@pytest.mark.parametrize('v_first', [False, True])
@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
def test_recurrent_options(K, V, v_first, dtype):
    from b200gdn import fused_recurrent_gated_delta_rule
    B, T, H, HV = 2, 9, 2, 4
    q, k, v, graw, braw, A_log, dt_bias, gen = _inputs(B, T, H, HV, K, V, 1, dtype)
    h0 = torch.randn(B, HV, *((V, K) if v_first else (K, V)), generator=gen) * 0.5
    ref_o, ref_ht = O.recurrent_step_options(
        q.float(), k.float(), v.float(), graw, braw, None, h0, True, True, True, A_log, dt_bias, True, True, v_first)
    dev = 'cuda'
    o, ht = fused_recurrent_gated_delta_rule(
        q.to(dev), k.to(dev), v.to(dev), graw.to(dev), beta=braw.to(dev), initial_state=h0.to(dev),
        output_final_state=True, use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, A_log=A_log.to(dev),
        dt_bias=dt_bias.to(dev), use_beta_sigmoid_in_kernel=True, allow_neg_eigval=True, state_v_first=v_first)
    assert o.dtype == dtype and ht.dtype == torch.float32
    tol = 1e-5 if dtype == torch.float32 else 0.004
    O.assert_close('o', ref_o, o.float().cpu(), tol)
    O.assert_close('ht', ref_ht, ht.cpu(), 1e-5)


def test_recurrent_plain_varlen_and_inplace():
    from b200gdn import fused_recurrent_gated_delta_rule
    H, HV, K, V = 2, 2, 128, 128
    cu = [0, 3, 4, 20, 31]
    T = cu[-1]
    d = O.make_inputs(1, T, H, HV, K, V, seed=2, cu_seqlens=cu, h0_std=0.5)
    ref_o, ref_ht = O.naive_recurrent(d['q'], d['k'], d['v'], d['g'], d['beta'], None, d['h0'], True, cu)
    dev = 'cuda'
    state = d['h0'].to(dev).clone()
    o, ht = fused_recurrent_gated_delta_rule(
        d['q'].to(dev), d['k'].to(dev), d['v'].to(dev), d['g'].to(dev), beta=d['beta'].to(dev), initial_state=state,
        output_final_state=True, cu_seqlens=torch.tensor(cu, device=dev), inplace_state=True)
    assert ht.data_ptr() == state.data_ptr()
    O.assert_close('o', ref_o, o.cpu(), 1e-5)
    O.assert_close('ht', ref_ht, ht.cpu(), 1e-5)
    # no initial state, no final state, beta defaults to ones
    o2, none = fused_recurrent_gated_delta_rule(d['q'].to(dev), d['k'].to(dev), d['v'].to(dev), d['g'].to(dev))
    ref_o2, _ = O.naive_recurrent(d['q'], d['k'], d['v'], d['g'], torch.ones_like(d['beta']), None, None, False)
    assert none is None
    O.assert_close('o2', ref_o2, o2.cpu(), 1e-5)


def test_recurrent_matches_config1_fixture():
    """BASELINE config 1 (B1 T1024 H4 K=V=64 fp32) against the reference's own output."""
    import os
    import numpy as np
    from b200gdn import fused_recurrent_gated_delta_rule
    gold = np.load(os.path.join(os.path.dirname(__file__), 'golden', 'config1_naive_cpu.npz'))
    d = O.make_inputs(1, 1024, 4, 4, 64, 64, seed=0)
    dev = 'cuda'
    o, ht = fused_recurrent_gated_delta_rule(d['q'].to(dev), d['k'].to(dev), d['v'].to(dev), d['g'].to(dev),
                                             beta=d['beta'].to(dev), initial_state=d['h0'].to(dev),
                                             output_final_state=True)
    O.assert_close('o', torch.from_numpy(gold['o']), o.cpu()[:, ::8], 1e-5)
    O.assert_close('ht', torch.from_numpy(gold['ht']), ht.cpu(), 1e-5)


def test_recurrent_errors():
    from b200gdn import fused_recurrent_gated_delta_rule
    dev = 'cuda'
    q = torch.zeros(1, 4, 2, 64, device=dev)
    g = torch.zeros(1, 4, 2, device=dev)
    with pytest.raises(NotImplementedError):
        fused_recurrent_gated_delta_rule(q, q, q, g, gk=q)
    with pytest.raises(ValueError, match='A_log'):
        fused_recurrent_gated_delta_rule(q, q, q, g, use_gate_in_kernel=True)
    o, _ = fused_recurrent_gated_delta_rule(q.requires_grad_(True), q, q, g)
    with pytest.raises(NotImplementedError):
        o.sum().backward()


@pytest.mark.parametrize('B', [1, 16, 256])
def test_decode_sweep_single_token_steps(B):
    """Decode sweep of the long-context configuration: single-token steps at batch 1..256 with a
    [B,16,128,128] fp32 state, three consecutive steps with the state carried in place; checked against
    the delta-rule update written out in plain fp32 torch on the same device."""
    from b200gdn import fused_recurrent_gated_delta_rule
    dev = 'cuda'
    H, K, V = 16, 128, 128
    gen = torch.Generator(device=dev).manual_seed(B)
    state = torch.randn(B, H, K, V, device=dev, generator=gen) * 0.1
    ref = state.clone()
    scale = K ** -0.5
    for step in range(3):
        q = torch.nn.functional.normalize(torch.randn(B, 1, H, K, device=dev, generator=gen), dim=-1)
        k = torch.nn.functional.normalize(torch.randn(B, 1, H, K, device=dev, generator=gen), dim=-1)
        v = torch.randn(B, 1, H, V, device=dev, generator=gen)
        g = torch.nn.functional.logsigmoid(torch.randn(B, 1, H, device=dev, generator=gen))
        beta = torch.sigmoid(torch.randn(B, 1, H, device=dev, generator=gen))
        o, ht = fused_recurrent_gated_delta_rule(q, k, v, g, beta=beta, initial_state=state, output_final_state=True,
                                                 inplace_state=True)
        assert ht.data_ptr() == state.data_ptr()
        # S <- S e^g ; u = beta (v - S^T k) ; S <- S + k u^T ; o = scale S^T q      (fla/ops/gated_delta_rule/naive.py:41-60)
        ref = ref * g[:, 0, :, None, None].exp()
        u = (v[:, 0] - torch.einsum('bhkv,bhk->bhv', ref, k[:, 0])) * beta[:, 0, :, None]
        ref = ref + torch.einsum('bhk,bhv->bhkv', k[:, 0], u)
        o_ref = torch.einsum('bhkv,bhk->bhv', ref, q[:, 0]) * scale
        O.assert_close(f'o step {step}', o_ref.cpu(), o[:, 0].cpu(), 1e-5)
        O.assert_close(f'state step {step}', ref.cpu(), state.cpu(), 1e-5)


def test_decode_step_in_cuda_graph():
    """The decode step only enqueues work on the caller's stream, so a serving loop can capture it in a CUDA graph
    (static input buffers, state updated in place) and replay it; replays must reproduce the eager steps."""
    from b200gdn import fused_recurrent_gated_delta_rule
    dev = 'cuda'
    B, H, K, V = 8, 16, 128, 128
    gen = torch.Generator(device=dev).manual_seed(5)
    mk = lambda *s: torch.randn(*s, device=dev, generator=gen)
    steps = [dict(q=torch.nn.functional.normalize(mk(B, 1, H, K), dim=-1), k=torch.nn.functional.normalize(mk(B, 1, H, K), dim=-1),
                  v=mk(B, 1, H, V), g=torch.nn.functional.logsigmoid(mk(B, 1, H)), beta=torch.sigmoid(mk(B, 1, H)))
             for _ in range(4)]
    state0 = mk(B, H, K, V) * 0.1
    # eager
    s_e = state0.clone()
    outs_e = []
    for st in steps:
        o, _ = fused_recurrent_gated_delta_rule(st['q'], st['k'], st['v'], st['g'], beta=st['beta'], initial_state=s_e,
                                                output_final_state=True, inplace_state=True)
        outs_e.append(o.clone())
    # captured once, replayed per step
    buf = {n: torch.empty_like(x) for n, x in steps[0].items()}
    s_g = state0.clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):   # warm-up outside the capture (library load, first launch)
        for n in buf:
            buf[n].copy_(steps[0][n])
        fused_recurrent_gated_delta_rule(buf['q'], buf['k'], buf['v'], buf['g'], beta=buf['beta'], initial_state=s_g.clone(),
                                         output_final_state=True, inplace_state=True)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        o_g, _ = fused_recurrent_gated_delta_rule(buf['q'], buf['k'], buf['v'], buf['g'], beta=buf['beta'], initial_state=s_g,
                                                  output_final_state=True, inplace_state=True)
    s_g.copy_(state0)
    for i, st in enumerate(steps):
        for n in buf:
            buf[n].copy_(st[n])
        graph.replay()
        assert torch.equal(o_g, outs_e[i]), f'step {i}'
    assert torch.equal(s_g, s_e)


@pytest.mark.parametrize('K', [128, 64])
@pytest.mark.parametrize('T', [1, 3])
@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16, torch.float16])
def test_large_batch_kernels_with_options(K, T, dtype):
    """Enough (sequence, head) pairs for the large-batch kernels: T = 1 takes the streaming kernel (bulk-copy ring,
    persistent CTAs), T = 3 the whole-state kernel; both with every in-kernel option on, grouped value heads, and the
    state out of place, against the oracle recurrence."""
    from b200gdn import fused_recurrent_gated_delta_rule
    B, H, HV, V = 40, 4, 8, 128     # 320 (sequence, head) pairs
    q, k, v, graw, braw, A_log, dt_bias, gen = _inputs(B, T, H, HV, K, V, 3, dtype)
    h0 = torch.randn(B, HV, K, V, generator=gen) * 0.5
    ref_o, ref_ht = O.recurrent_step_options(
        q.float(), k.float(), v.float(), graw, braw, None, h0, True, True, True, A_log, dt_bias, True, True, False)
    dev = 'cuda'
    o, ht = fused_recurrent_gated_delta_rule(
        q.to(dev), k.to(dev), v.to(dev), graw.to(dev), beta=braw.to(dev), initial_state=h0.to(dev),
        output_final_state=True, use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, A_log=A_log.to(dev),
        dt_bias=dt_bias.to(dev), use_beta_sigmoid_in_kernel=True, allow_neg_eigval=True)
    assert o.dtype == dtype and ht.dtype == torch.float32
    tol = 1e-5 if dtype == torch.float32 else 0.004
    O.assert_close('o', ref_o, o.float().cpu(), tol)
    O.assert_close('ht', ref_ht, ht.cpu(), 1e-5)
    import b200gdn
    b200gdn.device_status()


@pytest.mark.parametrize('B,T', [(40, 1), (40, 2), (6, 1)])
def test_state_pool_addressed_by_indices(B, T):
    """`state_indices`: the state lives in a pool of slots (a serving engine's cache); each sequence reads and
    updates its slot in place.  Must equal gather -> plain call -> scatter, bit for bit, and leave other slots alone.
    (B = 40 exercises the streaming and the whole-state kernels, B = 6 the sliced kernel.)"""
    from b200gdn import fused_recurrent_gated_delta_rule
    dev = 'cuda'
    H, HV, K, V, P = 4, 8, 128, 128, 64
    gen = torch.Generator(device=dev).manual_seed(B * 10 + T)
    mk = lambda *s: torch.randn(*s, device=dev, generator=gen)
    q, k = torch.nn.functional.normalize(mk(B, T, H, K), dim=-1), torch.nn.functional.normalize(mk(B, T, H, K), dim=-1)
    v, g, beta = mk(B, T, HV, V), torch.nn.functional.logsigmoid(mk(B, T, HV)), torch.sigmoid(mk(B, T, HV))
    pool = mk(P, HV, K, V) * 0.3
    idx = torch.randperm(P, device=dev, generator=gen)[:B]
    o_ref, ht_ref = fused_recurrent_gated_delta_rule(q, k, v, g, beta=beta, initial_state=pool[idx].contiguous(),
                                                     output_final_state=True)
    want = pool.clone()
    want[idx] = ht_ref
    o, out_pool = fused_recurrent_gated_delta_rule(q, k, v, g, beta=beta, initial_state=pool, state_indices=idx)
    assert out_pool.data_ptr() == pool.data_ptr()
    assert torch.equal(o, o_ref)
    assert torch.equal(pool, want)


@pytest.mark.parametrize('K,V', [(128, 128), (64, 64), (32, 32), (256, 64)])
@pytest.mark.parametrize('T', [1, 2, 16, 33, 65])
@pytest.mark.parametrize('misaligned', [False, True])
def test_token_blocks_and_unaligned_rows(K, V, T, misaligned):
    """The token walk at the edges of its blocks (8 to 32 tokens by K), the single-token step, and q / k / v that do not
    start on a 16-byte boundary (read element by element)."""
    from b200gdn import fused_recurrent_gated_delta_rule
    dev, H, HV = 'cuda', 2, 4
    q, k, v, graw, braw, A_log, dt_bias, gen = _inputs(2, T, H, HV, K, V, 5, torch.bfloat16)
    h0 = torch.randn(2, HV, K, V, generator=gen) * 0.5
    ref_o, ref_ht = O.recurrent_step_options(q.float(), k.float(), v.float(), graw, braw, None, h0, True, True, True, A_log, dt_bias,
                                             True, True, False)

    def place(x):
        x = x.to(dev)
        return torch.cat([x.new_zeros(1), x.flatten()])[1:].view(x.shape) if misaligned else x
    o, ht = fused_recurrent_gated_delta_rule(
        place(q), place(k), place(v), graw.to(dev), beta=braw.to(dev), initial_state=h0.to(dev), output_final_state=True,
        use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, A_log=A_log.to(dev), dt_bias=dt_bias.to(dev),
        use_beta_sigmoid_in_kernel=True, allow_neg_eigval=True)
    O.assert_close('o', ref_o, o.float().cpu(), 0.004)
    O.assert_close('ht', ref_ht, ht.cpu(), 1e-5)


@pytest.mark.parametrize('K,V,N,HV', [(128, 128, 32, 8), (128, 128, 31, 8), (64, 64, 65, 16), (64, 64, 305, 16), (128, 64, 43, 12), (64, 128, 150, 4)])
def test_single_token_steps_around_the_streaming_size(K, V, N, HV):
    """One token per sequence on a pool of states, either side of the size from which the states are streamed, with a
    sequence that is padding (index -1); the largest case gives every CTA more than 32 states."""
    from b200gdn import fused_recurrent_gated_delta_rule
    H, slots = HV // 2, N + 3
    gen = torch.Generator(device='cuda').manual_seed(N)
    mk = lambda *s: torch.randn(*s, device='cuda', generator=gen)   # noqa: E731
    q, k, v = (mk(N, 1, h, d).to(torch.bfloat16) for h, d in ((H, K), (H, K), (HV, V)))
    g, beta, pool = mk(N, 1, HV), mk(N, 1, HV), mk(slots, HV, K, V) * 0.1
    a_log, dt_bias = mk(HV) * 0.3, mk(HV) * 0.3
    at = torch.randperm(slots, device='cuda', generator=gen)[:N].to(torch.int32)
    at[N // 2] = -1
    before = pool.clone()
    o, _ = fused_recurrent_gated_delta_rule(q, k, v, g, beta=beta, initial_state=pool, output_final_state=True, state_indices=at,
                                            inplace_state=True, use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True,
                                            A_log=a_log, dt_bias=dt_bias, use_beta_sigmoid_in_kernel=True)
    used = at >= 0
    qf, kf = (torch.nn.functional.normalize(x[:, 0].double(), dim=-1).repeat_interleave(2, 1)[used] for x in (q, k))
    dec = (-a_log.double().exp() * torch.nn.functional.softplus(g[used, 0].double() + dt_bias)).exp()
    S = before[at[used].long()].double() * dec[..., None, None]
    r = (v[used, 0].double() - torch.einsum('nhkv,nhk->nhv', S, kf)) * torch.sigmoid(beta[used, 0].double())[..., None]
    S = S + torch.einsum('nhk,nhv->nhkv', kf, r)
    O.assert_close('o', torch.einsum('nhkv,nhk->nhv', S, qf) * K ** -0.5, o[used, 0].double(), 0.004)
    O.assert_close('states', S, pool[at[used].long()].double(), 1e-5)
    rest = torch.ones(slots, dtype=torch.bool, device='cuda')
    rest[at[used].long()] = False
    assert torch.equal(pool[rest], before[rest]), 'a slot that no sequence uses was written'


@pytest.mark.parametrize('K,V', [(32, 32), (64, 64), (128, 128), (256, 64)])
@pytest.mark.parametrize('lens,v_first', [([12], False), ([13, 12], True), ([16, 17, 7, 33], False), ([64, 0, 31, 1], True), ([65, 32], False)])
def test_tokens_in_pairs(K, V, lens, v_first):
    """Enough tokens to be taken in pairs: odd and even lengths, blocks that are full, nearly full and just exceeded, a sequence of one
    token and one of none beside longer ones; fp32, where the recurrence's own tolerance (1e-5) holds."""
    from b200gdn import fused_recurrent_gated_delta_rule
    H, HV, dev, T, N = 2, 4, 'cuda', sum(lens), len(lens)
    cu = torch.tensor([0] + lens).cumsum(0)
    q, k, v, graw, braw, A_log, dt_bias, gen = _inputs(1, T, H, HV, K, V, 31, torch.float32)
    h0 = torch.randn(N, HV, *((V, K) if v_first else (K, V)), generator=gen) * 0.5
    ref_o, ref_ht = [], []
    for i in range(N):
        rows = slice(int(cu[i]), int(cu[i + 1]))
        if lens[i] == 0:
            ref_ht.append(h0[i:i + 1])
            continue
        ro, rs = O.recurrent_step_options(q[:, rows], k[:, rows], v[:, rows], graw[:, rows], braw[:, rows], None, h0[i:i + 1], True, True, True,
                                          A_log, dt_bias, True, True, v_first)
        ref_o.append(ro)
        ref_ht.append(rs)
    o, ht = fused_recurrent_gated_delta_rule(
        *(x.to(dev) for x in (q, k, v, graw)), beta=braw.to(dev), initial_state=h0.to(dev), output_final_state=True,
        use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, A_log=A_log.to(dev), dt_bias=dt_bias.to(dev),
        use_beta_sigmoid_in_kernel=True, allow_neg_eigval=True, state_v_first=v_first, cu_seqlens=cu.to(dev))
    O.assert_close('o', torch.cat(ref_o, 1), o.cpu(), 1e-5)
    O.assert_close('ht', torch.cat(ref_ht, 0), ht.cpu(), 1e-5)


@pytest.mark.parametrize('K', [32, 64])
def test_pairs_of_a_block_are_prepared_in_two_passes(K):
    """Blocks of 32 tokens, of which a warp prepares four at a time in two passes over the same scratch row: against the fp32
    recurrence for every length from a first pass alone to several blocks, and the same bits every time."""
    from b200gdn import fused_recurrent_gated_delta_rule
    H, HV, N, dev = 2, 4, 48, 'cuda'
    for T in (15, 17, 31, 32, 33, 64):
        q, k, v, graw, braw, A_log, dt_bias, gen = _inputs(N, T, H, HV, K, K, 53, torch.float32)
        h0 = torch.randn(N, HV, K, K, generator=gen) * 0.5
        options = (True, True, True, A_log, dt_bias, True, True, False)
        ref_o, ref_ht = O.recurrent_step_options(q, k, v, graw, braw, None, h0, *options)
        args = [x.to(dev) for x in (q, k, v, graw)]
        runs = [fused_recurrent_gated_delta_rule(
            *args, beta=braw.to(dev), initial_state=h0.to(dev), output_final_state=True, use_qk_l2norm_in_kernel=True,
            use_gate_in_kernel=True, A_log=A_log.to(dev), dt_bias=dt_bias.to(dev), use_beta_sigmoid_in_kernel=True,
            allow_neg_eigval=True) for _ in range(8)]
        for o, ht in runs[1:]:
            assert torch.equal(o, runs[0][0]) and torch.equal(ht, runs[0][1])
        O.assert_close(f'o T={T}', ref_o, runs[0][0].cpu(), 1e-5)
        O.assert_close(f'ht T={T}', ref_ht, runs[0][1].cpu(), 1e-5)


@pytest.mark.parametrize('K,v_first', [(64, False), (128, False), (128, True)])
@pytest.mark.parametrize('start', ['nothing', 'large'])
def test_gates_of_a_pair_whose_product_leaves_fp32(K, v_first, start):
    """Two gates of a pair that fp32 holds one by one but not as a product: e^50 twice on a state of zeros, which stays zero until the
    first token has written, and e^-60 twice on a state of 1e30, which keeps 1e-22 (and comes back by e^45, the only token written out
    then).  The second tokens of the pairs, and the pair that an odd length leaves, take part.  Tolerance of the fp32 recurrence."""
    from b200gdn import fused_recurrent_gated_delta_rule
    T, H, dev = 13, 2, 'cuda'
    d = O.make_inputs(1, T, H, H, K, K, seed=7, h0_std=1.)
    g, beta, h0 = d['g'], d['beta'], None
    if start == 'nothing':
        g[:, :2], g[:, 6:8] = 50., -50.
    else:
        g.zero_(), beta.zero_()
        g[:, 2:4], g[:, 8], h0 = -60., 45., d['h0'] * 1e30
    ref_o, ref_ht = O.naive_recurrent(d['q'], d['k'], d['v'], g, beta, None, h0, True, dtype=torch.float64)
    flip = (lambda x: x.transpose(-1, -2).contiguous()) if v_first else (lambda x: x)
    o, ht = fused_recurrent_gated_delta_rule(*(d[n].to(dev) for n in 'qkv'), g.to(dev), beta=beta.to(dev),
                                             initial_state=None if h0 is None else flip(h0).to(dev), output_final_state=True,
                                             state_v_first=v_first)
    assert torch.isfinite(o).all() and torch.isfinite(ht).all()
    for t in range(T):   # magnitudes differ by forty decades: token by token
        O.assert_close(f'o {t}', ref_o[:, t], o[:, t].double().cpu(), 1e-5)
    O.assert_close('ht', ref_ht, flip(ht).double().cpu(), 1e-5)
