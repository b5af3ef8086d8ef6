"""GPU parity of the chunk path: every stage through the C ABI against the oracle's stage, then the
public API against the naive recurrence with the reference's own tolerances
(tests/ops/test_gdn.py:108-200: o/ht 0.005, dq/dk/dv/dh0 0.008, dbeta/dg 0.02)."""
import ctypes
import os

import numpy as np
import pytest
import torch

from oracle import gdn_oracle as O
from tests.golden.make_golden import CASES
from tests.gpu_util import flat, make_case, oracle_chain, run_abi

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), 'golden')

STAGE_CASES = {
    'd64_dense': dict(B=2, T=128, H=2, HV=2, K=64, V=64),
    'd128_dense': dict(B=2, T=256, H=2, HV=2, K=128, V=128),
    'd128_gva': dict(B=1, T=192, H=2, HV=4, K=128, V=128),
    'd128_ragged': dict(B=1, T=333, H=1, HV=2, K=128, V=128, cu=[0, 1, 16, 80, 143, 270, 333]),
    'd64_ragged_gva': dict(B=1, T=300, H=2, HV=4, K=64, V=64, cu=[0, 37, 101, 165, 300]),
    'd128_nh0': dict(B=1, T=100, H=2, HV=2, K=128, V=128, with_h0=False),
    'd128_group4': dict(B=2, T=130, H=1, HV=4, K=128, V=128),
}

# err-ratio bounds per tensor (bf16 storage: eps = 2^-8 = 0.0039 per rounding)
FWD_TOL = dict(gamma=1e-5, A=0.005, qk=0.005, w=0.005, u=0.005, h=0.005, v_new=0.005, ht=0.005, o=0.005)
BWD_TOL = dict(dh=0.008, dh0=0.008, dv2=0.008, dq=0.008, dk=0.008, dv=0.008, dbeta=0.02, dg=0.02)


@pytest.mark.parametrize('name', list(STAGE_CASES))
def test_stages_against_oracle(name):
    d = make_case(seed=3, **STAGE_CASES[name])
    fwd, bwd = oracle_chain(d)
    out = run_abi(d)
    for n, tol in FWD_TOL.items():
        O.assert_close(f'{name}:{n}', fwd[n], out[n], tol)
    if d['h0'] is None:
        BWD = {k: v for k, v in BWD_TOL.items() if k != 'dh0'}
    else:
        BWD = BWD_TOL
    for n, tol in BWD.items():
        O.assert_close(f'{name}:{n}', bwd[n], out[n], tol)


@pytest.mark.parametrize('name', ['d128_dense', 'd64_ragged_gva'])
def test_backward_stages_isolated(name):
    """Each backward kernel alone, fed with the oracle's inputs for that stage."""
    from b200gdn import _lib
    d = make_case(seed=5, **STAGE_CASES[name])
    fwd, bwd = oracle_chain(d)
    saved = {n: fwd[n] for n in ('gamma', 'A', 'qk', 'w', 'h', 'v_new')}
    o1 = run_abi(d, fwd_mask=-1, bwd_mask=_lib.BWD_DVLOCAL, overrides=dict(saved))
    O.assert_close('dv_local', bwd['dv_local'], o1['dv2'], 0.005)
    o2 = run_abi(d, fwd_mask=-1, bwd_mask=_lib.BWD_SCAN, overrides=dict(saved, dv2=bwd['dv_local']))
    for n in ('dh', 'dh0', 'dv2'):
        O.assert_close(n, bwd[n], o2[n], 0.005)
    # the same two stages in one kernel (dv_local formed inside the reverse scan from the forward pass's qk tile)
    o2f = run_abi(d, fwd_mask=-1, bwd_mask=_lib.BWD_DVLOCAL | _lib.BWD_SCAN, overrides=dict(saved))
    for n in ('dh', 'dh0', 'dv2'):
        O.assert_close(n + ' (fused scan)', bwd[n], o2f[n], 0.005)
    o3 = run_abi(d, fwd_mask=-1, bwd_mask=_lib.BWD_DQKWG, overrides=dict(saved, dv2=bwd['dv2'], dh=bwd['dh']))
    # after this stage the dk buffer holds the chunk-local part of dk (bf16), to which the WY stage adds in place
    for n, m in (('dq', 'dq'), ('dk', 'dk_part'), ('dG', 'dG')):
        O.assert_close(n, bwd[m], o3[n], 0.005)
    o4 = run_abi(d, fwd_mask=-1, bwd_mask=_lib.BWD_WY,
                 overrides=dict(saved, dv2=bwd['dv2'], dk=bwd['dk_part'], dG=bwd['dG']))
    for n in ('dk', 'dv', 'dbeta', 'dg'):
        O.assert_close(n, bwd[n], o4[n], 0.005)


@pytest.mark.parametrize('name', [n for n in CASES if CASES[n][-1]])
def test_public_api_against_reference_fixture(name):
    """chunk_gated_delta_rule + autograd against the reference's own outputs and gradients."""
    from b200gdn import chunk_gated_delta_rule
    B, T, H, HV, K, V, cu, seed, _ = CASES[name]
    gold = {k: torch.from_numpy(v) for k, v in np.load(os.path.join(GOLD, name + '.npz')).items()}
    d = O.make_inputs(B, T, H, HV, K, V, seed=seed, cu_seqlens=cu)
    dev = 'cuda'
    q, k, v = (d[n].to(dev).to(torch.bfloat16).requires_grad_(True) for n in ('q', 'k', 'v'))
    g, beta, h0 = (d[n].to(dev).requires_grad_(True) for n in ('g', 'beta', 'h0'))
    cu_t = None if cu is None else torch.tensor(cu, dtype=torch.long, device=dev)
    o, ht = chunk_gated_delta_rule(q, k, v, g, beta, initial_state=h0, output_final_state=True, cu_seqlens=cu_t)
    ((o.float() * d['do'].to(dev)).sum() + (ht * d['dht'].to(dev)).sum()).backward()
    assert o.dtype == torch.bfloat16 and ht.dtype == torch.float32
    O.assert_close('o', gold['o'], o.float().cpu(), 0.005)
    O.assert_close('ht', gold['ht'], ht.cpu(), 0.005)
    O.assert_close('dq', gold['dq'], q.grad.float().cpu(), 0.008)
    O.assert_close('dk', gold['dk'], k.grad.float().cpu(), 0.008)
    O.assert_close('dv', gold['dv'], v.grad.float().cpu(), 0.008)
    O.assert_close('dh0', gold['dh0'], h0.grad.cpu(), 0.008)
    O.assert_close('dbeta', gold['dbeta'], beta.grad.cpu(), 0.02)
    O.assert_close('dg', gold['dg'], g.grad.cpu(), 0.02)


@pytest.mark.parametrize('HV', [4, 2])
def test_options_equal_preprocessing(HV):
    """In-kernel options == the op on pre-processed inputs (tests/ops/test_gdn.py:281-448, 881-1190); grouped value
    heads (HV = 4 over H = 2) and one value head per q/k head: the L2 norm's backward is applied where dq and dk are
    completed, which the two cases do in different code paths."""
    from b200gdn import chunk_gated_delta_rule
    dev = 'cuda'
    B, T, H, K, V = 2, 150, 2, 128, 128
    gen = torch.Generator().manual_seed(9)
    q = torch.randn(B, T, H, K, generator=gen).to(dev).to(torch.bfloat16)
    k = torch.randn(B, T, H, K, generator=gen).to(dev).to(torch.bfloat16)
    v = torch.randn(B, T, HV, V, generator=gen).to(dev).to(torch.bfloat16)
    graw = torch.randn(B, T, HV, generator=gen).to(dev)
    braw = torch.randn(B, T, HV, generator=gen).to(dev)
    A_log = (torch.randn(HV, generator=gen) * 0.3).to(dev)
    dt_bias = (torch.randn(HV, generator=gen) * 0.3).to(dev)
    h0 = (torch.randn(B, HV, V, K, generator=gen) * 0.1).to(dev)

    def run(in_kernel):
        leaves = [x.clone().requires_grad_(True) for x in (q, k, v, graw, braw, A_log, dt_bias, h0)]
        q_, k_, v_, g_, b_, A_, dt_, h0_ = leaves
        if in_kernel:
            o, ht = chunk_gated_delta_rule(q_, k_, v_, g_, b_, initial_state=h0_, output_final_state=True,
                                           use_qk_l2norm_in_kernel=True, use_beta_sigmoid_in_kernel=True,
                                           allow_neg_eigval=True, state_v_first=True, use_gate_in_kernel=True,
                                           A_log=A_, dt_bias=dt_, chunk_size=32)
        else:
            qn = O.l2norm(q_.float()).to(torch.bfloat16)
            kn = O.l2norm(k_.float()).to(torch.bfloat16)
            o, ht = chunk_gated_delta_rule(qn, kn, v_, O.gdn_gate(g_, A_, dt_), 2 * torch.sigmoid(b_),
                                           initial_state=h0_.transpose(-1, -2), output_final_state=True)
            ht = ht.transpose(-1, -2)
        (o.float().square().sum() + ht.square().sum()).backward()
        return [o.float(), ht] + [x.grad.float() for x in leaves]
    a, b = run(True), run(False)
    # the two sides round the normalised q / k to bf16 from fp32 values that differ in the last bit here and there
    # (1/sqrt in the kernel as in the reference's l2norm kernel, rsqrt in torch): a flipped bf16 ulp is 4e-3 relative.
    for i, (x, y) in enumerate(zip(a, b)):
        if i not in (2, 3):
            O.assert_close(f'option-equivalence[{i}]', y.cpu(), x.cpu(), 1e-3)
    # dq / dk (results 2, 3).  The kernels apply the norm's backward (dy - y <dy,y>) rstd from the fp32 dy with y the
    # bf16-normalised tensor; the route above does it in torch from the bf16-rounded dy with y in fp32.  With this loss
    # the final-state gradient makes dk of the last rows almost parallel to k (component along k 40 times the rest), the
    # projection cancels it, and what is left is dominated by bf16 rounding on either route: both are held to the fp64
    # recurrence with the options inside the graph, and the kernels' route must be at least as close to it as torch's
    # (or within the tolerance the reference holds this option to, tests/ops/test_gdn.py:225-280)
    G = HV // H
    q64, k64 = q.cpu().double().requires_grad_(True), k.cpu().double().requires_grad_(True)
    o64, ht64 = O.naive_recurrent(O.l2norm(q64).repeat_interleave(G, 2), O.l2norm(k64).repeat_interleave(G, 2), v.cpu().double(),
                                  O.gdn_gate(graw.cpu().double(), A_log.cpu().double(), dt_bias.cpu().double()),
                                  2 * torch.sigmoid(braw.cpu().double()), scale=K ** -0.5,
                                  initial_state=h0.cpu().double().transpose(-1, -2), output_final_state=True, dtype=torch.float64)
    (o64.square().sum() + ht64.square().sum()).backward()
    for i, ref in ((2, q64.grad), (3, k64.grad)):
        e_kernel, e_torch = O.err_ratio(ref.float(), a[i].cpu()), O.err_ratio(ref.float(), b[i].cpu())
        assert e_kernel <= max(0.005, 1.1 * e_torch), f'option-equivalence[{i}]: {e_kernel} vs oracle, torch route {e_torch}'


@pytest.mark.parametrize('HV,dht_scale', [(2, 0.1), (2, 30.0), (4, 30.0)])
def test_l2norm_option_against_the_oracle(HV, dht_scale):
    """use_qk_l2norm_in_kernel: dq and dk (the norm's backward is applied where the kernels complete them) against the
    fp64 recurrence with the norm inside the graph, with one value head per q/k head and with grouped heads, and with a
    final-state gradient large enough to dominate the last rows (where dk is nearly parallel to k and the projection
    cancels most of it).  The north star's tolerance for dq / dk; the route through pre-normalised inputs is held to
    the same, as a yardstick."""
    from b200gdn import chunk_gated_delta_rule
    dev = 'cuda'
    B, T, H, K, V = 2, 150, 2, 128, 128
    gen = torch.Generator().manual_seed(9)
    q = torch.randn(B, T, H, K, generator=gen).to(torch.bfloat16)
    k = torch.randn(B, T, H, K, generator=gen).to(torch.bfloat16)
    v = torch.randn(B, T, HV, V, generator=gen).to(torch.bfloat16)
    g = torch.nn.functional.logsigmoid(torch.randn(B, T, HV, generator=gen))
    b = torch.sigmoid(torch.randn(B, T, HV, generator=gen))
    do = torch.randn(B, T, HV, V, generator=gen).to(torch.bfloat16)
    dht = torch.randn(B, HV, K, V, generator=gen) * dht_scale

    def run(in_kernel):
        q_, k_ = (x.to(dev).clone().requires_grad_(True) for x in (q, k))
        if in_kernel:
            o, ht = chunk_gated_delta_rule(q_, k_, v.to(dev), g.to(dev), b.to(dev), output_final_state=True,
                                           use_qk_l2norm_in_kernel=True)
        else:
            o, ht = chunk_gated_delta_rule(O.l2norm(q_.float()).to(torch.bfloat16), O.l2norm(k_.float()).to(torch.bfloat16),
                                           v.to(dev), g.to(dev), b.to(dev), output_final_state=True)
        torch.autograd.backward([o, ht], [do.to(dev), dht.to(dev)])
        return q_.grad.float().cpu(), k_.grad.float().cpu()
    fused, pre = run(True), run(False)
    q64, k64 = q.double().requires_grad_(True), k.double().requires_grad_(True)
    G = HV // H
    o, ht = O.naive_recurrent(O.l2norm(q64).repeat_interleave(G, 2), O.l2norm(k64).repeat_interleave(G, 2), v.double(),
                              g.double(), b.double(), scale=K ** -0.5, initial_state=None, output_final_state=True,
                              dtype=torch.float64)
    ((o * do.double()).sum() + (ht * dht.double()).sum()).backward()
    for name, ref, got, yard in (('dq', q64.grad, fused[0], pre[0]), ('dk', k64.grad, fused[1], pre[1])):
        O.assert_close(f'{name} fused norm backward vs oracle', ref.float(), got, 0.008)
        O.assert_close(f'{name} pre-normalised route vs oracle', ref.float(), yard, 0.008)
        O.assert_close(f'{name} last rows, fused vs oracle', ref[:, -3:].float(), got[:, -3:], 0.008)


def test_api_errors():
    from b200gdn import chunk_gated_delta_rule
    dev = 'cuda'
    q = torch.zeros(2, 64, 2, 128, device=dev, dtype=torch.bfloat16)
    v = torch.zeros(2, 64, 3, 128, device=dev, dtype=torch.bfloat16)
    g = torch.zeros(2, 64, 3, device=dev)
    with pytest.raises(ValueError, match='evenly divisible'):
        chunk_gated_delta_rule(q, q, v, g, g)
    v = torch.zeros(2, 64, 2, 128, device=dev, dtype=torch.bfloat16)
    g = torch.zeros(2, 64, 2, device=dev)
    with pytest.raises(ValueError, match='batch size is expected to be 1'):
        chunk_gated_delta_rule(q, q, v, g, g, cu_seqlens=torch.tensor([0, 64, 128], device=dev))
    with pytest.raises(DeprecationWarning):
        chunk_gated_delta_rule(q, q, v, g, g, head_first=True)
    with pytest.raises(ValueError, match='chunk_size'):
        chunk_gated_delta_rule(q, q, v, g, g, chunk_size=128)
    with pytest.raises(ValueError, match='allow_neg_eigval'):
        chunk_gated_delta_rule(q, q, v, g, g, allow_neg_eigval=True)


def test_determinism_and_no_uninitialised_reads():
    """Two runs are bit-identical (no atomics anywhere), and outputs never contain the NaN the buffers
    were poisoned with (the reference's NaN-poison fixture, tests/conftest.py:135-148)."""
    d = make_case(seed=7, **STAGE_CASES['d128_ragged'])
    a = run_abi(d)
    b = run_abi(d)
    for n in ('o', 'ht', 'dq', 'dk', 'dv', 'dg', 'dbeta', 'dh0'):
        assert not torch.isnan(a[n]).any(), n
        assert torch.equal(a[n], b[n]), n
    # none of the bounded device waits (mbarriers of TMA copies and tensor-core commits) expired
    import b200gdn
    b200gdn.device_status()


def test_full_size_properties():
    """Headline shape (B4 T4096 H16 K=V=128): the oracle is too slow here, so check properties:
    chunk path == token-by-token kernel (an independent implementation), and linearity in v."""
    from b200gdn import chunk_gated_delta_rule, fused_recurrent_gated_delta_rule
    dev = 'cuda'
    B, T, H, K = 4, 4096, 16, 128
    gen = torch.Generator(device=dev).manual_seed(0)
    q = torch.nn.functional.normalize(torch.randn(B, T, H, K, device=dev, generator=gen), dim=-1).to(torch.bfloat16)
    k = torch.nn.functional.normalize(torch.randn(B, T, H, K, device=dev, generator=gen), dim=-1).to(torch.bfloat16)
    v1 = torch.randn(B, T, H, K, device=dev, generator=gen).to(torch.bfloat16)
    v2 = torch.randn(B, T, H, K, device=dev, generator=gen).to(torch.bfloat16)
    g = torch.nn.functional.logsigmoid(torch.randn(B, T, H, device=dev, generator=gen))
    beta = torch.sigmoid(torch.randn(B, T, H, device=dev, generator=gen))
    h0 = torch.randn(B, H, K, K, device=dev, generator=gen) * 0.1
    o_c, ht_c = chunk_gated_delta_rule(q, k, v1, g, beta, initial_state=h0, output_final_state=True)
    o_r, ht_r = fused_recurrent_gated_delta_rule(q, k, v1, g, beta=beta, initial_state=h0, output_final_state=True)
    O.assert_close('o chunk vs recurrent', o_r.float().cpu(), o_c.float().cpu(), 0.005)
    O.assert_close('ht chunk vs recurrent', ht_r.cpu(), ht_c.cpu(), 0.005)
    o1, _ = chunk_gated_delta_rule(q, k, v1, g, beta)
    o2, _ = chunk_gated_delta_rule(q, k, v2, g, beta)
    o12, _ = chunk_gated_delta_rule(q, k, (v1.float() + v2.float()).to(torch.bfloat16), g, beta)
    O.assert_close('linearity in v', (o1.float() + o2.float()).cpu(), o12.float().cpu(), 0.01)


def _inputs(B, T, H, HV, K, V, seed, dev='cuda'):
    gen = torch.Generator(device=dev).manual_seed(seed)
    q = torch.nn.functional.normalize(torch.randn(B, T, H, K, device=dev, generator=gen), dim=-1).to(torch.bfloat16)
    k = torch.nn.functional.normalize(torch.randn(B, T, H, K, device=dev, generator=gen), dim=-1).to(torch.bfloat16)
    v = torch.randn(B, T, HV, V, device=dev, generator=gen).to(torch.bfloat16)
    g = torch.nn.functional.logsigmoid(torch.randn(B, T, HV, device=dev, generator=gen))
    beta = torch.sigmoid(torch.randn(B, T, HV, device=dev, generator=gen))
    do = torch.randn(B, T, HV, V, device=dev, generator=gen).to(torch.bfloat16)
    return q, k, v, g, beta, do


def _fwd_bwd(q, k, v, g, beta, do, **kw):
    from b200gdn import chunk_gated_delta_rule
    leaves = [x.detach().clone().requires_grad_(True) for x in (q, k, v, g, beta)]
    o, ht = chunk_gated_delta_rule(*leaves, output_final_state=True, **kw)
    o.backward(do)
    return [o, ht] + [x.grad for x in leaves]


def test_full_size_varlen_gva_equals_per_sequence_runs():
    """Packed GVA configuration at full size (16 q/k heads, 32 value heads, K=V=128, 16 sequences with lengths
    in [256, 8192] summing to 65536 tokens): the packed run must reproduce, sequence by sequence, the runs of
    each sequence on its own (outputs, final states and all gradients), and the chunk forward must agree with the
    token-by-token kernel."""
    from b200gdn import fused_recurrent_gated_delta_rule
    rng = np.random.default_rng(0)
    n, total = 16, 65536
    lens = rng.integers(256, 8193, size=n).astype(np.int64)
    lens = np.maximum(256, (lens * (total / lens.sum())).astype(np.int64))
    lens[-1] += total - lens.sum()
    assert lens.min() >= 256 and lens.sum() == total
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device='cuda')
    q, k, v, g, beta, do = _inputs(1, total, 16, 32, 128, 128, seed=3)
    packed = _fwd_bwd(q, k, v, g, beta, do, cu_seqlens=cu)
    o_r, ht_r = fused_recurrent_gated_delta_rule(q, k, v, g, beta=beta, output_final_state=True, cu_seqlens=cu)
    O.assert_close('o chunk vs recurrent', o_r.float().cpu(), packed[0].float().cpu(), 0.005)
    O.assert_close('ht chunk vs recurrent', ht_r.cpu(), packed[1].cpu(), 0.005)
    names = ('o', 'ht', 'dq', 'dk', 'dv', 'dg', 'dbeta')
    for i in (0, 7, 15):   # first, a middle and the last sequence (the others take the same code path)
        s, e = int(cu[i]), int(cu[i + 1])
        alone = _fwd_bwd(q[:, s:e], k[:, s:e], v[:, s:e], g[:, s:e], beta[:, s:e], do[:, s:e])
        for nme, a, p in zip(names, alone, packed):
            ref = p[i:i + 1] if nme == 'ht' else p[:, s:e]
            assert torch.equal(a, ref), f'sequence {i}: {nme} differs between the packed and the single run'


def test_full_size_head_and_batch_shards_are_independent():
    """Training shape B8 T8192 H32 K=V=128: a head shard and a batch shard computed on their own are bit-identical
    to the corresponding slices of the full computation (what lets heads / batch be split over GPUs with no
    communication), and the forward agrees with the token-by-token kernel on a slice."""
    from b200gdn import fused_recurrent_gated_delta_rule
    q, k, v, g, beta, do = _inputs(8, 8192, 32, 32, 128, 128, seed=4)
    full = _fwd_bwd(q, k, v, g, beta, do)
    hs = slice(8, 16)
    part = _fwd_bwd(q[:, :, hs], k[:, :, hs], v[:, :, hs], g[:, :, hs], beta[:, :, hs], do[:, :, hs])
    for nme, a, f in zip(('o', 'ht', 'dq', 'dk', 'dv', 'dg', 'dbeta'), part, full):
        ref = f[:, hs] if nme == 'ht' else f[:, :, hs]
        assert torch.equal(a, ref), f'head shard: {nme}'
    part = _fwd_bwd(q[2:4], k[2:4], v[2:4], g[2:4], beta[2:4], do[2:4])
    for nme, a, f in zip(('o', 'ht', 'dq', 'dk', 'dv', 'dg', 'dbeta'), part, full):
        assert torch.equal(a, f[2:4]), f'batch shard: {nme}'
    o_r, ht_r = fused_recurrent_gated_delta_rule(q[:1, :, :4], k[:1, :, :4], v[:1, :, :4], g[:1, :, :4], beta=beta[:1, :, :4],
                                                 output_final_state=True)
    O.assert_close('o chunk vs recurrent', o_r.float().cpu(), full[0][:1, :, :4].float().cpu(), 0.005)
    O.assert_close('ht chunk vs recurrent', ht_r.cpu(), full[1][:1, :4].cpu(), 0.005)


@pytest.mark.parametrize('qk_dtype,gb_dtype', [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16),
                                               (torch.float16, torch.float32)])
def test_layer_option_kernels_against_torch(qk_dtype, gb_dtype):
    """The pre/post pass of the library (L2 norm, gate, beta sigmoid; forward and backward) against the same
    formulas in plain fp32 torch with autograd (fla/modules/l2norm.py:84-144, fla/ops/gated_delta_rule/gate.py:21-46,
    fla/ops/common/gate.py:18-50).  Tolerances: fp32 results 1e-5; results stored in bf16 / fp16 2e-3."""
    from b200gdn import _lib
    from b200gdn.chunk import LayerOptionsFunction
    dev = 'cuda'
    B, T, H, HV, K = 2, 300, 3, 6, 128
    gen = torch.Generator(device=dev).manual_seed(11)
    q = (torch.randn(B, T, H, K, device=dev, generator=gen) * 2).to(qk_dtype)
    k = (torch.randn(B, T, H, K, device=dev, generator=gen) * 0.5).to(qk_dtype)
    g = (torch.randn(B, T, HV, device=dev, generator=gen) * 3).to(gb_dtype)     # both softplus branches
    g[0, 0, 0] = 25.0
    beta = torch.randn(B, T, HV, device=dev, generator=gen).to(gb_dtype)
    A_log = torch.randn(HV, device=dev, generator=gen) * 0.3
    dt_bias = torch.randn(HV, device=dev, generator=gen) * 0.3
    grads = [torch.randn(B, T, H, K, device=dev, generator=gen).to(torch.bfloat16) for _ in range(2)]
    grads += [torch.randn(B, T, HV, device=dev, generator=gen) for _ in range(2)]
    flags = _lib.PREP_L2NORM | _lib.PREP_GATE | _lib.PREP_BETA_SIGMOID | _lib.PREP_NEG_EIGVAL

    leaves = [x.clone().requires_grad_(True) for x in (q, k, g, beta, A_log, dt_bias)]
    outs = LayerOptionsFunction.apply(*leaves, flags)
    torch.autograd.backward(outs, grads)

    ref = [x.clone().float().requires_grad_(True) for x in (q, k, g, beta, A_log, dt_bias)]
    rq, rk, rg, rb, rA, rdt = ref
    r_outs = [rq * torch.rsqrt(rq.square().sum(-1, keepdim=True) + 1e-6),
              rk * torch.rsqrt(rk.square().sum(-1, keepdim=True) + 1e-6),
              -rA.exp() * torch.nn.functional.softplus(rg + rdt), 2 * torch.sigmoid(rb)]
    torch.autograd.backward(r_outs, [x.float() for x in grads])

    assert outs[0].dtype == torch.bfloat16 and outs[2].dtype == torch.float32 and outs[3].dtype == torch.float32
    O.assert_close('qn', r_outs[0].cpu(), outs[0].float().cpu(), 2e-3)
    O.assert_close('kn', r_outs[1].cpu(), outs[1].float().cpu(), 2e-3)
    O.assert_close('g', r_outs[2].cpu(), outs[2].cpu(), 1e-5)
    O.assert_close('beta', r_outs[3].cpu(), outs[3].cpu(), 1e-5)
    lo_qk = 1e-5 if qk_dtype == torch.float32 else 2e-3
    lo_gb = 1e-5 if gb_dtype == torch.float32 else 3e-3
    for name, a, b, tol in (('dq', leaves[0], ref[0], lo_qk), ('dk', leaves[1], ref[1], lo_qk), ('dg', leaves[2], ref[2], lo_gb),
                            ('dbeta', leaves[3], ref[3], lo_gb), ('dA_log', leaves[4], ref[4], 1e-5),
                            ('ddt_bias', leaves[5], ref[5], 1e-5)):
        assert a.grad.dtype == a.dtype, name
        O.assert_close(name, b.grad.cpu(), a.grad.float().cpu(), tol)


def test_chunk_forward_in_cuda_graph():
    """A prefill step (forward only, static buffers) captured in a CUDA graph replays to the eager result: the library
    only enqueues kernels on the caller's stream, and the tensor maps it builds on the host are kernel parameters."""
    from b200gdn import chunk_gated_delta_rule
    q, k, v, g, beta, _ = _inputs(2, 512, 4, 4, 128, 128, seed=6)
    with torch.no_grad():
        o_e, ht_e = chunk_gated_delta_rule(q, k, v, g, beta, output_final_state=True)   # also warms the chunk tables
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            chunk_gated_delta_rule(q, k, v, g, beta, output_final_state=True)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            o_g, ht_g = chunk_gated_delta_rule(q, k, v, g, beta, output_final_state=True)
        v2 = torch.randn_like(v.float()).to(torch.bfloat16)
        o_e2, ht_e2 = chunk_gated_delta_rule(q, k, v2, g, beta, output_final_state=True)
        graph.replay()
        assert torch.equal(o_g, o_e) and torch.equal(ht_g, ht_e)
        v.copy_(v2)
        graph.replay()
        assert torch.equal(o_g, o_e2) and torch.equal(ht_g, ht_e2)


@pytest.mark.parametrize('name', ['triton_d128_dense', 'triton_d128_varlen_gva', 'triton_d64_dense'])
def test_public_api_against_reference_triton_path(name):
    """Outputs and gradients of the reference's own Triton chunk path on a B200 (tests/golden/make_triton_golden.py)
    on identical seeded inputs; tolerances of the reference's tests (tests/ops/test_gdn.py:203-278: o, ht 0.005;
    dq, dk, dv, dh0 0.008; dbeta, dg 0.02)."""
    from b200gdn import chunk_gated_delta_rule
    from tests.golden.make_triton_golden import TRITON_CASES
    B, T, H, HV, K, V, cu, seed = TRITON_CASES[name]
    gold = np.load(os.path.join(os.path.dirname(__file__), 'golden', name + '.npz'))
    d = O.make_inputs(B, T, H, HV, K, V, seed=seed, cu_seqlens=cu)
    dev = 'cuda'
    leaves = {n: d[n].to(torch.bfloat16).to(dev).requires_grad_(True) for n in ('q', 'k', 'v')}
    leaves.update({n: d[n].float().to(dev).requires_grad_(True) for n in ('g', 'beta', 'h0')})
    cu_t = None if cu is None else torch.tensor(cu, dtype=torch.long, device=dev)
    o, ht = chunk_gated_delta_rule(leaves['q'], leaves['k'], leaves['v'], leaves['g'], leaves['beta'], scale=K ** -0.5,
                                   initial_state=leaves['h0'], output_final_state=True, cu_seqlens=cu_t)
    ((o.float() * d['do'].to(torch.bfloat16).float().to(dev)).sum() + (ht * d['dht'].to(dev)).sum()).backward()
    O.assert_close('o', torch.from_numpy(gold['o']), o.float().cpu(), 0.005)
    O.assert_close('ht', torch.from_numpy(gold['ht']), ht.cpu(), 0.005)
    for n, tol in (('q', 0.008), ('k', 0.008), ('v', 0.008), ('h0', 0.008), ('beta', 0.02), ('g', 0.02)):
        O.assert_close('d' + n, torch.from_numpy(gold['d' + n]), leaves[n].grad.float().cpu(), tol)


def test_wait_expiry_is_reported_and_context_survives():
    """Failure detection without a GPU fault: a kernel whose wait can never complete gives up after its (short)
    limit, the host reads B200GDN_ERR_TIMEOUT, the flag clears, and the context keeps working."""
    import b200gdn
    from b200gdn import _lib
    lib = _lib.load()
    b200gdn.device_status()                                     # clean before
    st = torch.cuda.current_stream().cuda_stream
    assert lib.b200gdn_selftest_wait_expiry(ctypes.c_void_p(st)) == 0
    with pytest.raises(b200gdn.B200GDNError, match='selftest'):
        b200gdn.device_status()
    b200gdn.device_status()                                     # flag was cleared by the read
    d = make_case(seed=1, **STAGE_CASES['d128_dense'])          # and real work still runs and is right
    fwd, _ = oracle_chain(d)
    out = run_abi(d, do_bwd=False)
    O.assert_close('o after expiry', fwd['o'], out['o'], 0.005)


@pytest.mark.parametrize('gscale', [0.02, 12.0])
def test_extreme_gates(gscale):
    """Nearly no decay (g ~ -0.01) and very strong decay (g down to -100 per token: 2^gamma underflows inside a
    chunk): every factor the kernels form is 2^(non-positive), so nothing overflows and results stay finite and
    within tolerance of the fp64 oracle chain."""
    d = make_case(seed=13, **STAGE_CASES['d128_ragged'])
    d['g'] = d['g'] * gscale
    fwd, bwd = oracle_chain(d, dtype=torch.float64)
    out = run_abi(d)
    for n in ('o', 'ht', 'dq', 'dk', 'dv', 'dg', 'dbeta', 'dh0'):
        assert torch.isfinite(out[n]).all(), n
    for n, tol in FWD_TOL.items():
        if n != 'gamma':
            O.assert_close(f'{n}', fwd[n].float(), out[n], tol)
    for n, tol in BWD_TOL.items():
        O.assert_close(f'{n}', bwd[n].float(), out[n], tol)


def test_fused_gate_and_beta_equal_the_separate_passes():
    """The gate / beta activations fused into the first forward and the last backward kernel against the same
    activations run as separate passes (LayerOptionsFunction) around the plain op: identical outputs, gradients
    equal to fp32 rounding (the two evaluate sigmoid in a different order)."""
    from b200gdn import _lib, chunk_gated_delta_rule
    from b200gdn.chunk import LayerOptionsFunction
    dev = 'cuda'
    B, T, H, HV, K, V = 2, 200, 2, 4, 128, 128
    q, k, v, _, _, do = _inputs(B, T, H, HV, K, V, seed=21)
    gen = torch.Generator(device=dev).manual_seed(22)
    graw = torch.randn(B, T, HV, device=dev, generator=gen) * 2
    braw = torch.randn(B, T, HV, device=dev, generator=gen)
    A_log = torch.randn(HV, device=dev, generator=gen) * 0.3
    dt_bias = torch.randn(HV, device=dev, generator=gen) * 0.3

    def run(fused):
        leaves = [x.clone().requires_grad_(True) for x in (q, k, v, graw, braw, A_log, dt_bias)]
        q_, k_, v_, g_, b_, A_, dt_ = leaves
        if fused:
            o, _ = chunk_gated_delta_rule(q_, k_, v_, g_, b_, use_gate_in_kernel=True, A_log=A_, dt_bias=dt_,
                                          use_beta_sigmoid_in_kernel=True, allow_neg_eigval=True)
        else:
            flags = _lib.PREP_GATE | _lib.PREP_BETA_SIGMOID | _lib.PREP_NEG_EIGVAL
            _, _, g2, b2 = LayerOptionsFunction.apply(q_, k_, g_, b_, A_, dt_, flags)
            o, _ = chunk_gated_delta_rule(q_, k_, v_, g2, b2)
        o.backward(do)
        return [o] + [x.grad for x in leaves]
    a, b = run(True), run(False)
    assert torch.equal(a[0], b[0])
    for i in (1, 2, 3):
        assert torch.equal(a[i], b[i]), i            # dq, dk, dv do not pass through the activations
    for i, name in ((4, 'dg'), (5, 'dbeta'), (6, 'dA_log'), (7, 'ddt_bias')):
        O.assert_close(name, b[i].float().cpu(), a[i].float().cpu(), 1e-5)


def _record(name, ratios):
    """Keep the measured err-ratios of the full-size checks in the folder B200GDN_TEST_ARTIFACTS names (when it is
    set and exists); the assertions themselves do not depend on it."""
    import json
    out = os.environ.get('B200GDN_TEST_ARTIFACTS', '')
    if out and os.path.isdir(out):
        with open(os.path.join(out, f'parity_{name}.json'), 'w') as f:
            json.dump({k: float(v) for k, v in ratios.items()}, f, indent=1)


# err-ratio bounds of the reference's own tests (tests/ops/test_gdn.py:108-200)
REF_TOL = dict(o=0.005, ht=0.005, dq=0.008, dk=0.008, dv=0.008, dh0=0.008, dg=0.02, dbeta=0.02)


def test_full_size_backward_against_oracle_one_head():
    """Headline shape B4 T4096 H16 K=V=128, forward AND backward (with an initial state and a gradient on the final
    state): heads and batch rows are independent, so one (batch row, head) slice of the full-size run is compared
    with the fp64 token-by-token oracle and its autograd gradients over the full 4096 tokens."""
    from b200gdn import chunk_gated_delta_rule
    dev = 'cuda'
    B, T, H, K = 4, 4096, 16, 128
    gen = torch.Generator().manual_seed(0)
    nrm = torch.nn.functional.normalize
    q = nrm(torch.randn(B, T, H, K, generator=gen), dim=-1).to(torch.bfloat16)
    k = nrm(torch.randn(B, T, H, K, generator=gen), dim=-1).to(torch.bfloat16)
    v = torch.randn(B, T, H, K, generator=gen).to(torch.bfloat16)
    g = torch.nn.functional.logsigmoid(torch.randn(B, T, H, generator=gen))
    beta = torch.sigmoid(torch.randn(B, T, H, generator=gen))
    h0 = torch.randn(B, H, K, K, generator=gen) * 0.1
    do = torch.randn(B, T, H, K, generator=gen).to(torch.bfloat16)
    dht = torch.randn(B, H, K, K, generator=gen) * 0.1
    leaves = [x.to(dev).requires_grad_(True) for x in (q, k, v, g, beta, h0)]
    o, ht = chunk_gated_delta_rule(*leaves[:5], initial_state=leaves[5], output_final_state=True)
    torch.autograd.backward([o, ht], [do.to(dev), dht.to(dev)])
    b, h = 2, 5
    sl = lambda x: x[b:b + 1, :, h:h + 1].float()
    ro, rht, rg = O.naive_with_grads(sl(q), sl(k), sl(v), sl(g), sl(beta), K ** -0.5, h0[b:b + 1, h:h + 1],
                                     sl(do), dht[b:b + 1, h:h + 1])
    got = dict(o=o[b:b + 1, :, h:h + 1].float().cpu(), ht=ht[b:b + 1, h:h + 1].cpu())
    for n, leaf in zip(('dq', 'dk', 'dv', 'dg', 'dbeta'), leaves[:5]):
        got[n] = leaf.grad[b:b + 1, :, h:h + 1].float().cpu()
    got['dh0'] = leaves[5].grad[b:b + 1, h:h + 1].cpu()
    want = dict(o=ro, ht=rht, **rg)
    ratios = {n: O.err_ratio(want[n].float(), got[n]) for n in REF_TOL}
    _record('headline_one_head', ratios)
    for n, tol in REF_TOL.items():
        O.assert_close(f'headline (b={b}, h={h}) {n}', want[n].float(), got[n], tol)


def test_full_size_varlen_gva_backward_against_oracle_one_sequence():
    """Packed GVA configuration at full size (16 q/k heads, 32 value heads, 16 sequences, 65536 tokens): one
    sequence and one value head of the packed forward + backward against the fp64 oracle over that whole sequence
    (outputs, final state, all gradients incl. dh0).  dq / dk of a q/k head sum over its group of value heads, so
    they are compared on a run whose other value head of the group receives a zero output gradient."""
    from b200gdn import chunk_gated_delta_rule
    dev = 'cuda'
    cu = O.random_cu_seqlens(16, 65536, 256, 8192, seed=0)
    H, HV, K, V, total = 16, 32, 128, 128, 65536
    gen = torch.Generator().manual_seed(1)
    nrm = torch.nn.functional.normalize
    q = nrm(torch.randn(1, total, H, K, generator=gen), dim=-1).to(torch.bfloat16)
    k = nrm(torch.randn(1, total, H, K, generator=gen), dim=-1).to(torch.bfloat16)
    v = torch.randn(1, total, HV, V, generator=gen).to(torch.bfloat16)
    g = torch.nn.functional.logsigmoid(torch.randn(1, total, HV, generator=gen))
    beta = torch.sigmoid(torch.randn(1, total, HV, generator=gen))
    h0 = torch.randn(16, HV, K, V, generator=gen) * 0.1
    do = torch.randn(1, total, HV, V, generator=gen).to(torch.bfloat16)
    dht = torch.randn(16, HV, K, V, generator=gen) * 0.1
    # the shortest sequence that still spans several chunks keeps the oracle's run time in seconds
    lens = [cu[i + 1] - cu[i] for i in range(16)]
    n = min(range(16), key=lambda i: lens[i])
    s, e = cu[n], cu[n + 1]
    hv = 11
    hq = hv // (HV // H)
    other = hq * (HV // H) + (1 - hv % (HV // H))
    do = do.clone()
    do[:, s:e, other] = 0          # the group's other value head contributes nothing to dq / dk of this sequence
    dht = dht.clone()
    dht[n, other] = 0
    leaves = [x.to(dev).requires_grad_(True) for x in (q, k, v, g, beta, h0)]
    cu_t = torch.tensor(cu, dtype=torch.int32, device=dev)
    o, ht = chunk_gated_delta_rule(*leaves[:5], initial_state=leaves[5], output_final_state=True, cu_seqlens=cu_t)
    torch.autograd.backward([o, ht], [do.to(dev), dht.to(dev)])
    ro, rht, rg = O.naive_with_grads(q[:, s:e, hq:hq + 1].float(), k[:, s:e, hq:hq + 1].float(), v[:, s:e, hv:hv + 1].float(),
                                     g[:, s:e, hv:hv + 1], beta[:, s:e, hv:hv + 1], K ** -0.5, h0[n:n + 1, hv:hv + 1],
                                     do[:, s:e, hv:hv + 1].float(), dht[n:n + 1, hv:hv + 1])
    got = dict(o=o[:, s:e, hv:hv + 1].float().cpu(), ht=ht[n:n + 1, hv:hv + 1].cpu(),
               dq=leaves[0].grad[:, s:e, hq:hq + 1].float().cpu(), dk=leaves[1].grad[:, s:e, hq:hq + 1].float().cpu(),
               dv=leaves[2].grad[:, s:e, hv:hv + 1].float().cpu(), dg=leaves[3].grad[:, s:e, hv:hv + 1].cpu(),
               dbeta=leaves[4].grad[:, s:e, hv:hv + 1].cpu(), dh0=leaves[5].grad[n:n + 1, hv:hv + 1].cpu())
    want = dict(o=ro, ht=rht, **rg)
    ratios = {nme: O.err_ratio(want[nme].float(), got[nme]) for nme in REF_TOL}
    ratios['sequence_length'] = e - s
    _record('varlen_gva_one_sequence', ratios)
    for nme, tol in REF_TOL.items():
        O.assert_close(f'packed GVA (sequence {n}, value head {hv}) {nme}', want[nme].float(), got[nme], tol)


def test_padding_rows_outside_cu_seqlens():
    """A packed buffer with rows before cu_seqlens[0] and after cu_seqlens[-1] (a serving buffer padded to a fixed
    size): the valid rows must equal the run on the unpadded buffer bit for bit, and nothing may turn NaN, although
    the kernels load whole 64-row tiles that reach into the padding."""
    lead, trail = 70, 45
    cu = [0, 37, 101, 165, 300]
    q, k, v, g, beta, do = _inputs(1, 300, 2, 4, 128, 128, seed=11)
    cu_t = torch.tensor(cu, dtype=torch.int32, device='cuda')
    ref = _fwd_bwd(q, k, v, g, beta, do, cu_seqlens=cu_t)

    def pad(x):
        shape = list(x.shape)
        a, b = shape.copy(), shape.copy()
        a[1], b[1] = lead, trail
        # finite but large padding values: they must never reach a valid row
        return torch.cat([torch.full(a, 3.0, dtype=x.dtype, device=x.device), x,
                          torch.full(b, -2.0, dtype=x.dtype, device=x.device)], 1)
    cu_p = torch.tensor([c + lead for c in cu], dtype=torch.int32, device='cuda')
    out = _fwd_bwd(pad(q), pad(k), pad(v), pad(g), pad(beta), pad(do), cu_seqlens=cu_p)
    for nme, a, p in zip(('o', 'ht', 'dq', 'dk', 'dv', 'dg', 'dbeta'), ref, out):
        assert not torch.isnan(p).any(), nme
        got = p if nme == 'ht' else p[:, lead:lead + 300]
        assert torch.equal(a, got), f'{nme} of the valid rows changed with padding around them'


def test_trailing_empty_sequence():
    """cu_seqlens ending in an empty sequence (and one in the middle): it owns no chunk, its final state is its
    initial state and its dh0 is the gradient of the final state."""
    from b200gdn import chunk_gated_delta_rule
    dev = 'cuda'
    cu = [0, 100, 100, 230, 230]
    d = O.make_inputs(1, 230, 2, 2, 128, 128, seed=13, cu_seqlens=cu)
    leaves = [d[n].to(dev).to(torch.bfloat16).requires_grad_(True) for n in ('q', 'k', 'v')]
    leaves += [d[n].to(dev).requires_grad_(True) for n in ('g', 'beta', 'h0')]
    o, ht = chunk_gated_delta_rule(*leaves[:5], initial_state=leaves[5], output_final_state=True,
                                   cu_seqlens=torch.tensor(cu, device=dev))
    torch.autograd.backward([o, ht], [d['do'].to(dev).to(torch.bfloat16), d['dht'].to(dev)])
    ro, rht, rg = O.naive_with_grads(*(d[n].to(torch.bfloat16).float() for n in ('q', 'k', 'v')), d['g'], d['beta'],
                                     128 ** -0.5, d['h0'], d['do'].to(torch.bfloat16).float(), d['dht'], cu_seqlens=cu)
    O.assert_close('o', ro.float(), o.float().cpu(), 0.005)
    O.assert_close('ht', rht.float(), ht.cpu(), 0.005)
    assert torch.equal(ht[1].cpu(), d['h0'][1]) and torch.equal(ht[3].cpu(), d['h0'][3])
    O.assert_close('dh0', rg['dh0'].float(), leaves[5].grad.cpu(), 0.008)
    assert torch.equal(leaves[5].grad[3].cpu(), d['dht'][3])
    import b200gdn
    b200gdn.device_status()


@pytest.mark.parametrize('K,H,HV,more', [(64, 2, 2, 0), (64, 1, 8, 0), (64, 2, 12, 0), (128, 1, 3, 0), (128, 1, 16, 0), (128, 2, 4, 0), (128, 2, 8, 0), (128, 1, 8, 0),
                                         (64, 1, 3, 280), (128, 2, 4, 140), (128, 1, 3, 280)])
def test_chunk_local_backward_by_group_size(K, H, HV, more):
    """Two, four or eight value heads per key head sum their dq and dk in a cluster, any number in turn where there are many
    chunks (here `more` sequences of one token), other group sizes in turn always; sequences of one token up to one past a
    tile, with and without the layer's options."""
    cu = [0, 1, 64, 129, 192, 255, 300] + [301 + i for i in range(more)]
    d = O.make_inputs(1, cu[-1], H, HV, K, K, seed=17, cu_seqlens=cu)
    bf = {n: d[n].to(torch.bfloat16) for n in ('q', 'k', 'v', 'do')}
    cu_t = torch.tensor(cu, dtype=torch.int32, device='cuda')
    _, _, ref = O.naive_with_grads(*(bf[n].float() for n in ('q', 'k', 'v')), d['g'], d['beta'], K ** -0.5, d['h0'],
                                   bf['do'].float(), torch.zeros_like(d['h0']), cu_seqlens=cu)
    from b200gdn import chunk_gated_delta_rule
    for options in (False, True):
        ins = [bf['q'], bf['k'], bf['v'], d['g'], d['beta']]
        kw, extra = {}, []
        if options:   # the same q, k, g and beta through the in-kernel steps
            log_a, dt = torch.zeros(HV, device='cuda', requires_grad=True), torch.zeros(HV, device='cuda', requires_grad=True)
            ins[3] = torch.log(torch.expm1(-d['g'].double()).clamp_min(1e-12)).float()   # g = -softplus(raw)
            ins[4] = torch.logit(d['beta'].double()).float()
            kw = dict(use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, A_log=log_a, dt_bias=dt, use_beta_sigmoid_in_kernel=True)
            extra = [log_a, dt]
        leaves = [x.cuda().requires_grad_(True) for x in ins]
        o, _ = chunk_gated_delta_rule(*leaves, initial_state=d['h0'].cuda(), cu_seqlens=cu_t, **kw)
        got = torch.autograd.grad(o, leaves + extra, bf['do'].cuda())
        want = [ref[n].float() for n in ('dq', 'dk', 'dv', 'dg', 'dbeta')]
        if options:
            for i, x in ((0, bf['q']), (1, bf['k'])):   # backward of x / |x|
                x = x.float().requires_grad_(True)
                want[i], = torch.autograd.grad(torch.nn.functional.normalize(x, dim=-1), x, want[i])
            want[4] = want[4] * d['beta'] * (1 - d['beta'])
            want[3] = want[3] * -torch.sigmoid(ins[3])
            draw = got[3].float().cpu()   # the parameters' gradients are sums over what came out (few and cancelling terms)
            want += [(draw * d['g'] / -torch.sigmoid(ins[3])).sum((0, 1)), draw.sum((0, 1))]
        for n, w, x, tol in zip(('dq', 'dk', 'dv', 'dg', 'dbeta', 'dA_log', 'ddt_bias'), want, got, (0.008,) * 3 + (0.02,) * 2 + (0.002,) * 2):
            O.assert_close(f'{n} options={options}', w, x.float().cpu(), tol)


def test_fp32_and_fp16_inputs_are_rounded_to_bf16_and_keep_their_dtype():
    """q, k, v in fp32 / fp16: the result is the bf16 computation on the rounded inputs (documented), returned in
    the caller's dtype, gradients in each input's dtype."""
    from b200gdn import chunk_gated_delta_rule
    dev = 'cuda'
    d = O.make_inputs(2, 130, 2, 2, 128, 128, seed=17)
    for dt in (torch.float32, torch.float16):
        x = [d[n].to(dev).to(dt).requires_grad_(True) for n in ('q', 'k', 'v')]
        gb = [d[n].to(dev).requires_grad_(True) for n in ('g', 'beta')]
        o, _ = chunk_gated_delta_rule(*x, *gb, use_qk_l2norm_in_kernel=(dt == torch.float32))
        o.float().square().sum().backward()
        assert o.dtype == dt and all(t.grad.dtype == dt for t in x)
        y = [t.detach().to(torch.bfloat16).requires_grad_(True) for t in x]
        gb2 = [t.detach().clone().requires_grad_(True) for t in gb]
        o2, _ = chunk_gated_delta_rule(*y, *gb2, use_qk_l2norm_in_kernel=(dt == torch.float32))
        assert o2.dtype == torch.bfloat16
        # fp16: both runs see identical bf16 operands (only the cast of o to fp16 differs, small values land in fp16's
        # subnormal range); fp32 + norm pass: the normalised q / k are rounded to bf16 from slightly different values
        O.assert_close(f'o {dt} inputs vs bf16 inputs', o2.float().cpu(), o.float().cpu(), 1e-3 if dt == torch.float16 else 0.005)


@pytest.mark.parametrize('name', ['d128_ragged', 'd64_ragged_gva', 'd128_dense'])
def test_forward_stage_by_stage_equals_the_fused_scan(name):
    """The forward pass run one stage per call (scan kernel, then the stand-alone output kernel) against the default
    call, where the scan forms the output itself: both against the oracle, and h / v_new / ht bit-identical."""
    from b200gdn import _lib
    d = make_case(seed=23, **STAGE_CASES[name])
    fwd, _ = oracle_chain(d)
    fused = run_abi(d, do_bwd=False)
    a = run_abi(d, fwd_mask=_lib.FWD_INTRA, do_bwd=False)
    saved = {n: a[n] for n in ('gamma', 'A', 'qk', 'w', 'u')}
    b = run_abi(d, fwd_mask=_lib.FWD_SCAN, do_bwd=False, overrides=dict(saved))
    for n in ('h', 'v_new', 'ht'):
        assert torch.equal(b[n], fused[n]), n
    c = run_abi(d, fwd_mask=_lib.FWD_OUT, do_bwd=False, overrides=dict(saved, h=b['h'], v_new=b['v_new']))
    O.assert_close('o staged', fwd['o'], c['o'], 0.005)
    O.assert_close('o fused', fwd['o'], fused['o'], 0.005)
    O.assert_close('o fused vs staged', c['o'], fused['o'], 0.004)


@pytest.mark.parametrize('pieces', [2, 3, 5])
def test_sequence_split_equals_the_unsplit_scan(pieces):
    """Long sequences cut into pieces that are scanned concurrently (pre-scan of each piece's affine map, prefix chain,
    then the regular scan over all pieces): outputs, final state and every gradient against the oracle and against the
    unsplit run, on ragged packed sequences with grouped value heads, an initial state and a final-state gradient."""
    from b200gdn import chunk_gated_delta_rule, index
    dev = 'cuda'
    cu = [0, 37, 700, 700, 1500, 1563]
    d = O.make_inputs(1, 1563, 2, 4, 128, 128, seed=29, cu_seqlens=cu)
    cu_t = torch.tensor(cu, dtype=torch.int32, device=dev)

    def run():
        leaves = [d[n].to(dev).to(torch.bfloat16).requires_grad_(True) for n in ('q', 'k', 'v')]
        leaves += [d[n].to(dev).requires_grad_(True) for n in ('g', 'beta', 'h0')]
        o, ht = chunk_gated_delta_rule(*leaves[:5], initial_state=leaves[5], output_final_state=True, cu_seqlens=cu_t)
        torch.autograd.backward([o, ht], [d['do'].to(dev).to(torch.bfloat16), d['dht'].to(dev)])
        return [o.float().cpu(), ht.cpu()] + [x.grad.float().cpu() for x in leaves]
    plain = run()
    index.FORCE_PIECES = pieces
    try:
        index._split_cache.clear()
        plan = index.split_plan_for(1, 1563, cu_t, None, torch.device(dev), 4, 2)
        assert plan is not None and max(plan.pieces_per_seq) == pieces
        split = run()
    finally:
        index.FORCE_PIECES = None
        index._split_cache.clear()
    ro, rht, rg = O.naive_with_grads(*(d[n].to(torch.bfloat16).float() for n in ('q', 'k', 'v')), d['g'], d['beta'], 128 ** -0.5,
                                     d['h0'], d['do'].to(torch.bfloat16).float(), d['dht'], cu_seqlens=cu)
    want = [ro, rht, rg['dq'], rg['dk'], rg['dv'], rg['dg'], rg['dbeta'], rg['dh0']]
    names = ('o', 'ht', 'dq', 'dk', 'dv', 'dg', 'dbeta', 'dh0')
    for n, w_, s_, p_ in zip(names, want, split, plain):
        O.assert_close(f'{n} split vs oracle', w_.float(), s_, REF_TOL[n])
        O.assert_close(f'{n} split vs unsplit', p_, s_, 0.004)


@pytest.mark.parametrize('D', [64, 128])
@pytest.mark.parametrize('odd', [None, 'v', 'do'])
def test_pre_scans_leave_out_what_does_not_reach(D, odd):
    """Long pieces whose heads forget nothing, part of a piece, all but two chunks of it, and grow: against the uncut run.  Each of the two
    is within REF_TOL of the exact result, so they are within twice that of one another (heads that forget nothing use most of it, with
    and without anything left out: up to 0.0067 for dk); what a head that forgets shows of the cut is far less.  A value or an output gradient that is not finite in a chunk that is left out still reaches everything that
    it reaches in the uncut run."""
    from b200gdn import chunk_gated_delta_rule, index
    dev, T, H, HV = 'cuda', 64 * 60 + 37, 2, 4
    d = O.make_inputs(1, T, H, HV, D, D, seed=37)
    rate = torch.tensor([-1e-4, -0.2, -1.5, 2e-3])
    g = rate * (0.5 + torch.rand(1, T, HV, generator=torch.Generator().manual_seed(1)))
    v, do = d['v'].clone(), d['do'].clone()
    if odd == 'v':
        v[0, 70, 2, 5] = float('nan')
    if odd == 'do':
        do[0, T - 80, 2, 5] = float('inf')

    def run(pieces):
        index.FORCE_PIECES = pieces
        index._split_cache.clear()
        try:
            leaves = [x.to(dev).to(torch.bfloat16).requires_grad_(True) for x in (d['q'], d['k'], v)]
            leaves += [x.to(dev).requires_grad_(True) for x in (g, d['beta'], d['h0'])]
            o, ht = chunk_gated_delta_rule(*leaves[:5], initial_state=leaves[5], output_final_state=True)
            torch.autograd.backward([o, ht], [do.to(dev).to(torch.bfloat16), d['dht'].to(dev)])
            return [o.float().cpu(), ht.cpu()] + [x.grad.float().cpu() for x in leaves]
        finally:
            index.FORCE_PIECES = None
            index._split_cache.clear()
    names = ('o', 'ht', 'dq', 'dk', 'dv', 'dg', 'dbeta', 'dh0')
    for n, a, b in zip(names, run(1), run(3)):
        if odd is not None:
            bad = ~torch.isfinite(a)
            assert torch.equal(bad, ~torch.isfinite(b)), n
            a, b = a.masked_fill(bad, 0), b.masked_fill(bad, 0)
        O.assert_close(f'{n} cut vs uncut', a, b, 2 * REF_TOL[n])
        if n in ('o', 'dv') and odd is None:
            O.assert_close(f'{n} cut vs uncut, heads that forget', a[:, :, 1:3], b[:, :, 1:3], 1e-3)


@pytest.mark.parametrize('D', [64, 128])
def test_a_query_that_is_not_finite_is_not_left_out(D):
    """An infinite query in a chunk that the reverse pre-scan would leave out, of heads that forget part of a piece and all but two chunks of
    it (and one that forgets nothing): in the cut run the same results are finite as in the uncut one, and these are the same within
    twice the tolerance that each has to the exact result."""
    from b200gdn import chunk_gated_delta_rule, index
    dev, T, H, HV, bf = 'cuda', 64 * 60 + 37, 2, 4, torch.bfloat16
    d = O.make_inputs(1, T, H, HV, D, D, seed=37)
    rate = torch.tensor([-1e-4, -0.2, -1.5, -0.2])
    g = rate * (0.5 + torch.rand(1, T, HV, generator=torch.Generator().manual_seed(1)))
    q = d['q'].clone()
    q[0, T - 80, 1, 5] = float('inf')

    def run(pieces):
        index.FORCE_PIECES = pieces
        index._split_cache.clear()
        try:
            leaves = [x.to(dev).to(bf).requires_grad_(True) for x in (q, d['k'], d['v'])]
            leaves += [x.to(dev).requires_grad_(True) for x in (g, d['beta'], d['h0'])]
            o, ht = chunk_gated_delta_rule(*leaves[:5], initial_state=leaves[5], output_final_state=True)
            return [x.detach().float().cpu() for x in (o, ht, *torch.autograd.grad([o, ht], leaves, [d['do'].to(dev).to(bf), d['dht'].to(dev)]))]
        finally:
            index.FORCE_PIECES = None
            index._split_cache.clear()
    for n, a, b in zip(('o', 'ht', 'dq', 'dk', 'dv', 'dg', 'dbeta', 'dh0'), run(1), run(3)):
        bad = ~torch.isfinite(a)
        assert torch.equal(bad, ~torch.isfinite(b)), n
        assert bad.any() == (n not in ('ht', 'dq'))   # which do not depend on q
        O.assert_close(f'{n} cut vs uncut', a.masked_fill(bad, 0), b.masked_fill(bad, 0), 2 * REF_TOL[n])


@pytest.mark.parametrize('D', [64, 128])
@pytest.mark.parametrize('reverse', [False, True])
def test_pre_scans_where_gates_grow_and_decay(D, reverse):
    """Pieces of 18 chunks whose state grows by 2^116 in nine of them and then decays by 2^129 (reverse: the other way round, so that the
    gradient does, on its way back): what crosses a piece is 2^-13 of what entered it, although the product of its last (first) nine
    transitions alone is below 2^-128.  Head 0 has a start state (end gradient) only, head 1 only what a chunk at the far end of each
    piece adds; against the fp64 recurrence, each result in units of its own size."""
    from b200gdn import chunk_gated_delta_rule, index
    dev, n, pieces = 'cuda', 18 * 64, 3
    T = n * pieces
    d = O.make_inputs(1, T, 1, 2, D, D, seed=43)
    grows, decays = torch.full((n // 2,), 0.14), torch.full((n // 2,), -0.155)
    g = torch.cat([decays, grows] if reverse else [grows, decays]).repeat(pieces)[None, :, None].expand(1, T, 2).contiguous()
    far = (torch.arange(T) % n >= n - 64) if reverse else (torch.arange(T) % n < 64)
    beta, do, h0, dht = d['beta'].clone(), d['do'].clone(), d['h0'].clone(), d['dht'].clone()
    beta[:, ~far] = 0
    do[:, ~far] = 0
    if reverse:
        beta[:] = 0
        do[:, :, 0] = 0
        dht[:, 1] = 0
    else:
        beta[:, :, 0] = 0
        h0[:, 1] = 0
        do[:] = 0
    bf = torch.bfloat16
    q, k, v = (d[x].to(bf) for x in ('q', 'k', 'v'))
    leaf = h0.to(dev).requires_grad_(reverse)
    index.FORCE_PIECES = pieces
    index._split_cache.clear()
    try:
        o, ht = chunk_gated_delta_rule(*(x.to(dev) for x in (q, k, v, g, beta)), initial_state=leaf, output_final_state=True)
        if reverse:
            torch.autograd.backward([o, ht], [do.to(dev).to(bf), dht.to(dev)])
    finally:
        index.FORCE_PIECES = None
        index._split_cache.clear()
    ro, rht, rg = O.naive_with_grads(q, k, v, g, beta, D ** -0.5, h0, do.to(bf), dht)
    got, want = (leaf.grad.cpu(), rg['dh0']) if reverse else (ht.cpu(), rht)
    for hv in range(2):
        size = want[:, hv].abs().max()
        O.assert_close(f'head {hv}', want[:, hv] / size, got[:, hv].double() / size, REF_TOL['dh0' if reverse else 'ht'])
    if not reverse:
        size = ro[:, -64:].abs().max()
        O.assert_close('o', ro[:, -64:] / size, o[:, -64:].cpu().double() / size, REF_TOL['o'])


def _walked(bounds, reverse):
    """From the bounds [chunks] of one sequence: how many chunks a pre-scan walks, whether the whole transition counts as zero, how close a
    sum comes to the line, and the first one below it (for the test's own sake)."""
    sums = np.cumsum((bounds if reverse else bounds[::-1]).astype(np.float64))
    above = np.nonzero(sums[:-1] >= -128)[0]
    return (int(above[-1]) + 2 if len(above) else 1), bool(sums[-1] < -128), np.abs(sums + 128).min(), int((sums >= -128).argmin()) + 1


@pytest.mark.parametrize('D', [64, 128])
@pytest.mark.parametrize('reverse', [False, True])
def test_pre_scan_against_itself(D, reverse):
    """A pre-scan of 66 chunks with and without the transition bounds, through the C ABI, for heads that forget nothing, most of the
    piece (the line is crossed in the second round of 32 chunks), part of it, all but two chunks, that grow, and that grow and decay in turn:
    * the bounds are gamma_last + sum log2 max(1, |1 - beta |k|^2|), their lowest bits clear;
    * results are the same up to the share that may be left out (2^-128 of values that are below 2^20, and again for what the changed
      values round differently in bf16 on the way), so the same bits wherever they are above 2^-80;
    * exactly the chunks are walked that the rule names: NaN in the operands of the others, written after their bounds, is not
      seen, and in the last one of them it is;
    * a start state (end gradient) is not left out, and values that are not finite more than 32 chunks away are not either.
    The forward pass runs without A (B200GDN_FORWARD_ONLY)."""
    from b200gdn import _lib
    from b200gdn.chunk import new_chunk_args
    from b200gdn.index import build_tables
    H, HV, nc = 2, 6, 66
    rows, dev, st = 64 * (nc - 1) + 21, 'cuda', torch.cuda.current_stream().cuda_stream
    d = O.make_inputs(1, rows, H, HV, D, D, seed=47)
    k = d['k'].clone()
    k[:, ::64, 1] *= 1.6   # |1 - beta |k|^2| above one for some
    in_turn = torch.cat([torch.full((9,), -0.17), torch.full((9,), 0.14)]).repeat(4)[:nc]   # nearest the scan's end first
    in_turn = (in_turn if reverse else in_turn.flip(0)).repeat_interleave(64)[:rows]
    g = torch.stack([torch.full((rows,), r) for r in (-1e-4, -0.03, -0.2, -1.5, 2e-3)] + [in_turn], 1)
    cm, sm = (torch.from_numpy(x).to(dev) for x in build_tables([(0, rows)]))
    bf, f32 = dict(dtype=torch.bfloat16, device=dev), dict(dtype=torch.float32, device=dev)
    q0, k0, v0, do0 = (x.to(**bf).contiguous() for x in (d['q'], k, d['v'], d['do']))
    g0, beta0 = g.to(**f32).contiguous(), d['beta'].to(**f32).contiguous()
    state = (torch.randn(1, HV, D, D, generator=torch.Generator().manual_seed(3))).to(dev)

    def intra(q, v):
        a = new_chunk_args(q, k0, v, D ** -0.5, (cm, sm, (nc, 1)))
        t = dict(gamma=torch.zeros(nc * HV * 65, **f32), qk=torch.zeros(rows, HV, 64, **bf), w=torch.zeros(rows, HV, D, **bf),
                 u=torch.zeros(rows, HV, D, **bf))
        a.g, a.beta, a.stage_mask, a.options = g0.data_ptr(), beta0.data_ptr(), _lib.FWD_INTRA, _lib.TRANSITION_BOUNDS | _lib.FORWARD_ONLY
        for name, x in t.items():
            setattr(a, name, x.data_ptr())
        _lib.call('b200gdn_chunk_fwd', a, st)
        return t

    def scan(t, bounds, q=q0, v=v0, do=do0, start=None):
        a = new_chunk_args(q, k0, v, D ** -0.5, (cm, sm, (nc, 1)))
        out, M = torch.full((1, HV, D, D), float('nan'), **f32), torch.full((1, HV, D, D), float('nan'), **f32)
        a.options = _lib.TRANSITION_BOUNDS if bounds else 0
        a.gamma, a.w = t['gamma'].data_ptr(), t['w'].data_ptr()
        if reverse:
            a.qk, a.d_o, a.dht, a.dh0, a.cp_dM = t['qk'].data_ptr(), do.data_ptr(), _lib.ptr(start), out.data_ptr(), M.data_ptr()
            a.stage_mask = _lib.BWD_DVLOCAL | _lib.BWD_SCAN
            _lib.call('b200gdn_chunk_bwd', a, st)
        else:
            a.u, a.h0, a.ht, a.cp_M, a.stage_mask = t['u'].data_ptr(), _lib.ptr(start), out.data_ptr(), M.data_ptr(), _lib.FWD_SCAN
            _lib.call('b200gdn_chunk_fwd', a, st)
        return out[0].cpu(), M[0].cpu()

    def same(x, y):
        return bool(((x.double() - y.double()).abs() <= 2.0 ** -100).all())

    t = intra(q0, v0)
    bounds = t['gamma'][nc * HV * 64:].reshape(nc, HV).cpu()
    assert not (bounds.view(torch.int32) & 1).any()
    kk = k0[0].double().cpu().square().sum(-1).repeat_interleave(HV // H, 1)
    growth = (1 - beta0[0].double().cpu() * kk).abs().clamp(min=1).log2()
    pad = torch.zeros(64 * nc - rows, HV, dtype=torch.float64)
    want = torch.cat([g.double() * O.RCP_LN2 + growth, pad]).reshape(nc, 64, HV).sum(1)
    assert (want - bounds.double()).abs().max() < 1e-3
    rule = [_walked(bounds[:, hv].numpy(), reverse) for hv in range(HV)]
    assert min(r[2] for r in rule) > 0.01   # 66 fp32 values below 2^8 add up to within 0.001
    assert rule[0][0] == nc and 32 < rule[1][0] < nc and rule[2][0] < 16 and rule[3][0] <= 2 and rule[4][0] == nc
    assert rule[5][3] < 18 and 54 < rule[5][0] < nc
    assert [r[1] for r in rule] == [False, True, True, True, False, True]

    full, M_full = scan(t, False)
    cut, M_cut = scan(t, True)
    assert torch.isfinite(full).all() and same(full, cut) and same(M_full, M_cut)
    assert [bool((M_cut[hv] == 0).all()) for hv in range(HV)] == [r[1] for r in rule]
    for a, b in zip(scan(t, False, start=state), scan(t, True, start=state)):
        assert same(a, b)
    # operands of the chunks that are not walked, then of the farthest one that is
    name = 'w' if reverse else 'u'
    x = t[name].clone()
    poisoned = {**t, name: x}
    for hv in range(HV):
        n = rule[hv][0]
        x[slice(64 * n, None) if reverse else slice(0, 64 * (nc - n)), hv] = float('nan')
    assert torch.equal(scan(poisoned, True)[0], cut)
    for hv in range(HV):
        c = rule[hv][0] - 1 if reverse else nc - rule[hv][0]
        x[64 * c:64 * c + 64, hv] = float('nan')
    assert not torch.isfinite(scan(poisoned, True)[0]).any(-1).any(-1).any()
    # values that are not finite, far away
    if reverse:
        q1, do1 = q0.clone(), do0.clone()
        q1[0, 64 * 60 + 3, :, 5] = float('nan')
        do1[0, 64 * 60 + 3, :, 5] = float('inf')
        t1 = intra(q1, v0)
        odd = t1['gamma'][nc * HV * 64:].reshape(nc, HV).cpu().view(torch.int32) & 1
        assert odd[60].all() and odd.sum() == HV
        pairs = [[scan(t1, b, q=q1)[0] for b in (False, True)], [scan(t, b, do=do1)[0] for b in (False, True)]]
    else:
        v1 = v0.clone()
        v1[0, 64 * 10 + 3, :, 5] = float('nan')
        t1 = intra(q0, v1)
        assert torch.isinf(t1['gamma'][nc * HV * 64:].reshape(nc, HV)[10]).all()
        pairs = [[scan(t1, b, v=v1)[0] for b in (False, True)]]
    for a, b in pairs:
        bad = ~torch.isfinite(a)
        assert bad.flatten(1).any(1).all() and torch.equal(bad, ~torch.isfinite(b))
        assert same(a.masked_fill(bad, 0), b.masked_fill(bad, 0))


@pytest.mark.parametrize('D,H,HV,options', [(128, 16, 16, True), (128, 8, 24, True), (128, 4, 16, True), (64, 16, 16, True), (64, 8, 24, True), (64, 8, 32, False)])
def test_results_by_tma_equal_results_by_rows(D, H, HV, options):
    """From 2049 chunk-heads on, whole chunks of the normalised q and k and of dq, dk and dv leave by TMA; below, and where a chunk is
    ragged, by rows.  150 chunks of full and ragged sequences in one call against the sequences one by one (at most 50 chunks): the same bits.
    8/24 heads: a CTA takes the heads of a group in turn, in both; 4/16: a cluster does, 150 x 4 CTAs in turn being the longer way; 8/32:
    in turn in one call and a cluster in the others, which add in the same order."""
    from b200gdn import chunk_gated_delta_rule, index
    lens = [64 * 40, 64 * 30 + 1, 63, 64, 64 * 50, 64 * 26 + 33]
    cu = [0] + [int(x) for x in np.cumsum(lens)]
    T, N, dev, bf = cu[-1], len(lens), 'cuda', torch.bfloat16
    gen = torch.Generator(device=dev).manual_seed(59)

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device=dev)
    q, k = (torch.nn.functional.normalize(normal(1, T, H, D), dim=-1) * (3 if options else 1) for _ in range(2))
    data = [q.to(bf), k.to(bf), normal(1, T, HV, D).to(bf)]
    data += [normal(1, T, HV).to(bf) for _ in range(2)] if options else [torch.nn.functional.logsigmoid(normal(1, T, HV)), torch.rand(1, T, HV, generator=gen, device=dev)]
    h0, do, dht = normal(N, HV, D, D) * 0.1, normal(1, T, HV, D).to(bf), normal(N, HV, D, D) * 0.1
    A_log, dt_bias = normal(HV) * 0.3, normal(HV) * 0.3
    more = dict(use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, A_log=A_log, dt_bias=dt_bias, use_beta_sigmoid_in_kernel=True) if options else {}

    def run(rows, seqs, cu_t):
        leaves = [x[:, rows].contiguous().requires_grad_(True) for x in data] + [h0[seqs].contiguous().requires_grad_(True)]
        o, ht = chunk_gated_delta_rule(*leaves[:5], initial_state=leaves[5], output_final_state=True, cu_seqlens=cu_t, **more)
        grads = torch.autograd.grad([o, ht], leaves, [do[:, rows].contiguous(), dht[seqs].contiguous()])
        return [x.detach() for x in (o, *grads[:5])], [x.detach() for x in (ht, grads[5])]
    index.FORCE_PIECES = 1
    index._split_cache.clear()
    try:
        by_row, by_seq = run(slice(0, T), slice(0, N), torch.tensor(cu, dtype=torch.int32, device=dev))
        parts = [run(slice(cu[i], cu[i + 1]), slice(i, i + 1), None) for i in range(N)]
    finally:
        index.FORCE_PIECES = None
        index._split_cache.clear()
    for j, n in enumerate(('o', 'dq', 'dk', 'dv', 'dg', 'dbeta')):
        for i in range(N):
            assert torch.equal(by_row[j][:, cu[i]:cu[i + 1]], parts[i][0][j]), f'{n}, sequence {i}'
    for j, n in enumerate(('ht', 'dh0')):
        for i in range(N):
            assert torch.equal(by_seq[j][i:i + 1], parts[i][1][j]), f'{n}, sequence {i}'


@pytest.mark.parametrize('pieces', [None, 3])
def test_state_v_first_layout(pieces):
    """states stored [N,HV,V,K] (the reference's state_v_first, tests/ops/test_gdn.py:385-461): the scans read h0 / dht
    and write ht / dh0 in that layout themselves; the split path transposes at its boundary.  Bit-identical to the run
    on transposed states."""
    from b200gdn import chunk_gated_delta_rule, index
    dev = 'cuda'
    cu = [0, 37, 700, 700, 1500, 1563]
    d = O.make_inputs(1, 1563, 2, 4, 128, 128, seed=33, cu_seqlens=cu)
    cu_t = torch.tensor(cu, dtype=torch.int32, device=dev)

    def run(v_first):
        leaves = [d[n].to(dev).to(torch.bfloat16).requires_grad_(True) for n in ('q', 'k', 'v')]
        leaves += [d[n].to(dev).requires_grad_(True) for n in ('g', 'beta')]
        h0 = d['h0'].to(dev)
        h0 = (h0.transpose(-1, -2).contiguous() if v_first else h0).requires_grad_(True)
        dht = d['dht'].to(dev)
        o, ht = chunk_gated_delta_rule(*leaves, initial_state=h0, output_final_state=True, cu_seqlens=cu_t,
                                       state_v_first=v_first)
        torch.autograd.backward([o, ht], [d['do'].to(dev).to(torch.bfloat16), dht.transpose(-1, -2).contiguous() if v_first else dht])
        outs = [o, ht.transpose(-1, -2) if v_first else ht] + [x.grad for x in leaves]
        return [x.float().cpu() for x in outs + [h0.grad.transpose(-1, -2) if v_first else h0.grad]]
    index.FORCE_PIECES = pieces
    try:
        index._split_cache.clear()
        a, b = run(False), run(True)
    finally:
        index.FORCE_PIECES = None
        index._split_cache.clear()
    for i, (x, y) in enumerate(zip(a, b)):
        assert torch.equal(x, y), f'state_v_first differs in result {i}'


def test_sequence_split_heuristic_on_one_long_sequence():
    """One sequence of 32768 tokens with 4 heads: the planner cuts it (the scans would otherwise occupy 8 of 148 SMs), and
    the result agrees with the token-by-token kernel."""
    from b200gdn import chunk_gated_delta_rule, fused_recurrent_gated_delta_rule, index
    q, k, v, g, beta, do = _inputs(1, 32768, 4, 4, 128, 128, seed=31)
    plan = index.split_plan_for(1, 32768, None, None, q.device, 4, 2)
    assert plan is not None and plan.n_pieces > 1
    o, ht = chunk_gated_delta_rule(q, k, v, g, beta, output_final_state=True)
    o_r, ht_r = fused_recurrent_gated_delta_rule(q, k, v, g, beta=beta, output_final_state=True)
    O.assert_close('o chunk (split) vs recurrent', o_r.float().cpu(), o.float().cpu(), 0.005)
    O.assert_close('ht chunk (split) vs recurrent', ht_r.cpu(), ht.cpu(), 0.005)


@pytest.mark.parametrize('D,HV,lens', [(128, 4, [2048]), (64, 4, [4100]), (64, 2, [700, 1300, 5000, 1]), (128, 16, [4095])])
def test_planned_cuts_equal_the_uncut_scan(D, HV, lens):
    """Shapes that the planner cuts into from three pieces to many: outputs, final states and gradients against the uncut
    run, and the outputs against the token-by-token kernel."""
    from b200gdn import fused_recurrent_gated_delta_rule, index
    cu = [0] + list(np.cumsum(lens))
    chunks = [-(-n // 64) for n in lens]
    assert max(index.piece_counts(chunks, HV, D // 64)) >= 3
    q, k, v, g, beta, do = _inputs(1, cu[-1], HV, HV, D, D, seed=37)
    cu_t = torch.tensor(cu, dtype=torch.int32, device='cuda')
    h0 = torch.randn(len(lens), HV, D, D, device='cuda') * 0.1
    out = {}
    for force in (None, 1):
        index.FORCE_PIECES = force
        try:
            index._split_cache.clear()
            out[force] = _fwd_bwd(q, k, v, g, beta, do, cu_seqlens=cu_t, initial_state=h0)
        finally:
            index.FORCE_PIECES = None
            index._split_cache.clear()
    for n, cut, whole in zip(('o', 'ht', 'dq', 'dk', 'dv', 'dg', 'dbeta'), out[None], out[1]):
        O.assert_close(f'{n} cut vs uncut', whole.float().cpu(), cut.float().cpu(), 0.004)
    o_r, ht_r = fused_recurrent_gated_delta_rule(q, k, v, g, beta=beta, initial_state=h0, output_final_state=True, cu_seqlens=cu_t)
    O.assert_close('o vs recurrent', o_r.float().cpu(), out[None][0].float().cpu(), 0.005)
    O.assert_close('ht vs recurrent', ht_r.cpu(), out[None][1].cpu(), 0.005)


@pytest.mark.parametrize('D,H,limit_dg,limit_sum', [(128, 1, 0.0040, 0.008), (64, 4, 0.0043, 0.011)])
def test_gate_gradients_keep_their_distance_from_fp64(D, H, limit_dg, limit_sum):
    """dg, and its sums over a sequence (dA_log and ddt_bias are such sums, of terms that cancel), with the layer's options
    against the fp64 recurrence, over twelve seeds.  Measured: 0.00378 and 0.0051 (128, group of four), 0.00392 and 0.0088
    (64); with the WY terms of dk inside the dots of the gate's gradient, whose bf16 operands do not cancel, 0.00417 and
    0.0116, 0.00470 and 0.0148.  The limits lie between; results are the same from run to run."""
    from b200gdn import chunk_gated_delta_rule
    HV, T, errs, sums = 4, 384, [], []
    for seed in range(12):
        gen = torch.Generator().manual_seed(seed)
        rn = lambda *s: torch.randn(*s, generator=gen)   # noqa: E731
        q, k, v, do = (rn(1, T, h, D).to(torch.bfloat16) for h in (H, H, HV, HV))
        g, b = rn(1, T, HV), rn(1, T, HV)
        log_a, dt = (torch.rand(HV, generator=gen) * 15 + 1).log(), torch.rand(HV, generator=gen) * 0.1
        dt = dt + torch.log(-torch.expm1(-dt))
        opts = dict(use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True)
        wide = [x.double().requires_grad_(True) for x in (q, k, v, g, b, log_a, dt)]
        ro, _ = O.recurrent_step_options(*wide[:5], scale=D ** -0.5, A_log=wide[5], dt_bias=wide[6], dtype=torch.float64, **opts)
        ref_g, ref_dt = torch.autograd.grad(ro, [wide[3], wide[6]], do.double())
        leaves = [x.cuda().requires_grad_(True) for x in (q, k, v, g, b, log_a, dt)]
        o, _ = chunk_gated_delta_rule(*leaves[:5], A_log=leaves[5], dt_bias=leaves[6], **opts)
        got_g, got_dt = (x.double().cpu() for x in torch.autograd.grad(o, [leaves[3], leaves[6]], do.cuda()))
        errs.append((got_g - ref_g).norm() / ref_g.norm())
        sums.append((got_dt - ref_dt) / ref_g[0].norm(dim=0))
    assert torch.stack(errs).mean() <= limit_dg
    assert torch.stack(sums).square().mean().sqrt() <= limit_sum


@pytest.mark.parametrize('D', [64, 128])
@pytest.mark.parametrize('H,HV,copies', [(2, 2, 1), (1, 2, 1), (1, 3, 1), (2, 4, 24)])
def test_chunk_local_backward_at_chunk_edges(D, H, HV, copies):
    """Chunks of 1, 2, 63 and 64 tokens next to one another, write strengths of exactly 0 and 1 among them, one head, groups that meet in a
    cluster, groups that one CTA takes in turn (three heads, and many chunks): every gradient against the fp64 recurrence."""
    from b200gdn import chunk_gated_delta_rule
    lens = [1, 63, 64, 65, 130, 2] * copies
    cu = [0] + [int(x) for x in np.cumsum(lens)]
    T = cu[-1]
    d = O.make_inputs(1, T, H, HV, D, D, seed=41, cu_seqlens=cu)
    d['beta'][:, ::5] = 0.0
    d['beta'][:, 3::7] = 1.0
    bf = torch.bfloat16
    leaves = [d[n].to('cuda').to(bf).requires_grad_(True) for n in ('q', 'k', 'v')]
    leaves += [d[n].to('cuda').requires_grad_(True) for n in ('g', 'beta', 'h0')]
    cu_t = torch.tensor(cu, dtype=torch.int32, device='cuda')
    o, ht = chunk_gated_delta_rule(*leaves[:5], initial_state=leaves[5], output_final_state=True, cu_seqlens=cu_t)
    torch.autograd.backward([o, ht], [d['do'].to('cuda').to(bf), d['dht'].to('cuda')])
    with torch.no_grad():   # where A is not written
        o_only, ht_only = chunk_gated_delta_rule(*leaves[:5], initial_state=leaves[5], output_final_state=True, cu_seqlens=cu_t)
    assert torch.equal(o, o_only) and torch.equal(ht, ht_only)
    ro, rht, rg = O.naive_with_grads(*(d[n].to(bf).float() for n in ('q', 'k', 'v')), d['g'], d['beta'], D ** -0.5, d['h0'],
                                     d['do'].to(bf).float(), d['dht'], cu_seqlens=cu)
    O.assert_close('o', ro.float(), o.detach().float().cpu(), REF_TOL['o'])
    O.assert_close('ht', rht.float(), ht.detach().cpu(), REF_TOL['ht'])
    for n, leaf in zip(('dq', 'dk', 'dv', 'dg', 'dbeta', 'dh0'), leaves):
        O.assert_close(n, rg[n].float(), leaf.grad.float().cpu(), REF_TOL[n])
