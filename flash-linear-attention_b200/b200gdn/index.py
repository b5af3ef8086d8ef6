"""Host-side chunk tables (the information of fla/ops/utils/index.py:155-172, prepare_chunk_indices /
prepare_chunk_offsets, in the form the kernels read)."""
from __future__ import annotations

import functools
from typing import Optional, Sequence, Tuple

import numpy as np
import torch

from . import _lib

CHUNK = 64
_cache: dict = {}
_bounds_cache: dict = {}


class Tables(tuple):
    """(chunk_meta, seq_meta, (n_chunks, n_seq)) plus ``covered``: False when token rows before the first or after
    the last sequence belong to no sequence (a padded packed buffer).  The kernels never write such rows, so the
    caller zero-fills its intermediates then.  ``native()`` is the same as one handle for the native host path."""
    covered = True
    empty_seqs = False   # some sequence has no token (and so no tile)
    stream = 0           # the stream whose memory the tables are
    order = None      # int32 [n_seq]: sequences by falling length, None when all are of one length
    _native = None

    def native(self):
        if self._native is None:
            self._native = _lib.host().plan(self[0], self[1], self[2][0], self[2][1], self.covered, self.empty_seqs,
                                            self.stream, self.order)
        return self._native


def build_tables(bounds: Sequence[Tuple[int, int]]):
    """chunk_meta [n_chunks,4] = (sequence, first row, valid rows, index inside the sequence) and
    seq_meta [n_seq,2] = (first chunk, number of chunks), as int32 numpy arrays.  Chunking restarts at
    every sequence start; an empty sequence owns zero chunks."""
    bounds = np.asarray(bounds, dtype=np.int64).reshape(-1, 2)
    lens = bounds[:, 1] - bounds[:, 0]
    if (lens < 0).any():
        raise ValueError('cu_seqlens must be non-decreasing')
    nchunks = (lens + CHUNK - 1) // CHUNK
    first = np.concatenate([[0], np.cumsum(nchunks)[:-1]]) if len(nchunks) else np.zeros(0, np.int64)
    total = int(nchunks.sum())
    seq = np.repeat(np.arange(len(lens)), nchunks)
    local = np.arange(total) - np.repeat(first, nchunks)
    row = bounds[seq, 0] + local * CHUNK
    ln = np.minimum(CHUNK, bounds[seq, 1] - row)
    chunk_meta = np.stack([seq, row, ln, local], 1).astype(np.int32).reshape(-1, 4)
    seq_meta = np.stack([first, nchunks], 1).astype(np.int32).reshape(-1, 2)
    return chunk_meta, seq_meta


def device_tables(bounds, device) -> Tables:
    """build_tables on the device, with the order in which the scans take the sequences: a scan CTA walks one sequence,
    so with more CTAs than SMs a long sequence that starts late is what everything else waits for."""
    cm, sm = build_tables(bounds)
    out = Tables((torch.from_numpy(cm).to(device), torch.from_numpy(sm).to(device), (cm.shape[0], sm.shape[0])))
    if out[0].is_cuda:
        out.stream = torch.cuda.current_stream(out[0].device).cuda_stream
    out.empty_seqs = bool((sm[:, 1] == 0).any())
    if len(sm) > 1 and (sm[:, 1] != sm[0, 1]).any():
        out.order = torch.from_numpy(np.argsort(-sm[:, 1], kind='stable').astype(np.int32)).to(device)
    return out


def content_version(cu_seqlens: torch.Tensor):
    """Changes when the tensor is written in place, so that tables of its old contents are not used for the new ones
    (a tensor made under inference_mode keeps no such count: there the caller passes another tensor)."""
    return None if cu_seqlens.is_inference() else cu_seqlens._version


def packed_bounds(cu_seqlens: torch.Tensor, cu_seqlens_cpu: Optional[torch.Tensor], rows: int, version):
    """(start, end) of every sequence of a packed batch, none of them outside its ``rows`` token rows.  The device-to-host copy
    that this costs without ``cu_seqlens_cpu`` (17 us) is made once for the tables, the planner and the convolutions."""
    hit = _bounds_cache.get(id(cu_seqlens))
    if hit is None or hit[1] is not cu_seqlens or hit[2] != version:
        cu = (cu_seqlens_cpu if cu_seqlens_cpu is not None else cu_seqlens.cpu()).tolist()
        hit = ([(int(s), int(e)) for s, e in zip(cu[:-1], cu[1:])], cu_seqlens, version)
        if len(_bounds_cache) > 64:
            _bounds_cache.clear()
        _bounds_cache[id(cu_seqlens)] = hit
    bounds = hit[0]
    if bounds and (bounds[0][0] < 0 or bounds[-1][1] > rows):
        raise ValueError(f'cu_seqlens [{bounds[0][0]}, {bounds[-1][1]}] reaches outside the {rows} token rows')
    return bounds


def tables_for(B: int, T: int, cu_seqlens: Optional[torch.Tensor], cu_seqlens_cpu: Optional[torch.Tensor],
               device: torch.device) -> Tables:
    """Device tables for a dense [B,T] batch or a packed batch; memoised by shape / by the identity and version of
    ``cu_seqlens`` (the reference memoises its index tensors by identity, fla/utils/_decorators.py:33-80).
    A packed batch without ``cu_seqlens_cpu`` costs one device-to-host copy on first use."""
    version = None if cu_seqlens is None else content_version(cu_seqlens)
    if cu_seqlens is None:
        key = ('dense', B, T, device)
        hit = _cache.get(key)
        if hit is not None:
            return hit[0]
        bounds = [(b * T, (b + 1) * T) for b in range(B)]
    else:
        key = ('varlen', id(cu_seqlens), B * T, device)
        hit = _cache.get(key)
        if hit is not None and hit[1] is cu_seqlens and hit[2] == version:
            return hit[0]
        bounds = packed_bounds(cu_seqlens, cu_seqlens_cpu, B * T, version)
    out = device_tables(bounds, device)
    out.covered = bool(bounds) and bounds[0][0] == 0 and bounds[-1][1] == B * T
    if len(_cache) > 64:
        _cache.clear()
    _cache[key] = (out, cu_seqlens, version)
    return out


# ------------------------------------------------------------------------------------------- sequence split
# The state scans walk a sequence chunk by chunk, one CTA per (sequence, value head, 64 value columns).  With few
# sequences and heads that leaves most of the GPU idle, so long sequences are cut into pieces that are scanned
# concurrently (fla/ops/common/intracard_cp.py:139-180 does this for its forward pass): a pre-scan gives every piece
# its affine map, a prefix chain turns the maps into the start state of every piece, and the regular scan then runs
# over all pieces at once.  Pieces are whole numbers of chunks, so the chunking (and every chunk-local kernel) is
# unchanged.
FORCE_PIECES = None          # tests: cut every sequence into (up to) this many pieces regardless of the heuristic
_split_cache: dict = {}


class SplitPlan:
    """Virtual-sequence tables and the index tensors that tie the pieces of a sequence together."""
    __slots__ = ('tables', 'n_pieces', 'n_pre', 'chains', 'n_chains', 'pre_fwd', 'pre_bwd', 'first_piece', 'last_piece',
                 'pieces_per_seq', '_native')

    def native(self):
        """The plan as one handle for the native host path."""
        if self._native is None:
            t = self.tables
            self._native = _lib.host().plan(t[0], t[1], t[2][0], t[2][1], t.covered, t.empty_seqs, t.stream, t.order, self.chains,
                                            self.pre_fwd, self.pre_bwd, self.first_piece, self.last_piece, self.n_chains, self.n_pre)
        return self._native


@functools.lru_cache(maxsize=None)
def sm_count(device) -> int:
    return torch.cuda.get_device_properties(device).multi_processor_count if device.type == 'cuda' else 148


def piece_counts(chunks_per_seq, HV: int, slices: int, sms: int = 148):
    """How many pieces each sequence is cut into (equal pieces, so the longest sequences into the most): the cut with the
    least time by the model below, in microseconds as measured on a B200 with heads of 128 and 64; none unless it saves
    a twentieth.  A scan CTA takes `step` per chunk and the pre-scan, which runs beside twice as many transition-matrix
    CTAs (two per SM forward, one backward), nearly as long (heads that forget are pre-scanned in less, but a plan does not
    see the gates); the prefix chain takes a step per piece.  Two pieces never pay: pre-scan and scan together then walk as far as the uncut scan."""
    if FORCE_PIECES is not None:
        return [max(1, min(int(FORCE_PIECES), int(c))) for c in chunks_per_seq]
    uncut = [1] * len(chunks_per_seq)
    lens = [int(c) for c in chunks_per_seq if c > 0]
    per_seq = max(1, slices * HV)                    # scan CTAs of a piece
    if not lens or per_seq * (len(lens) + 2) > sms:
        return uncut
    longest, step, chain = max(lens), 1.27 if slices > 1 else 1.06, 1.5 if slices > 1 else 0.65
    if 8 * slices * HV * len(lens) > sms:       # the chains' CTAs, eight columns each, share SMs
        chain *= 1.8
    best, length = 0.95 * (3.5 + step * longest), None
    for pieces in range(3, min(longest, sms // per_seq - len(lens) + 1) + 1):
        n = -(-longest // pieces)
        total = sum(-(-c // n) for c in lens)
        pre = (total - len(lens)) * 2 * per_seq      # pre-scan CTAs
        if total * per_seq > sms:
            continue
        rounds = (-(-pre // sms) - (-pre // (2 * sms))) / 2
        cost = 12. + step * n * (1 + 0.92 * rounds) + chain * (-(-longest // n) - 1)
        if cost < best:
            best, length = cost, n
    return uncut if length is None else [max(1, -(-int(c) // length)) for c in chunks_per_seq]


def split_plan(bounds, HV: int, slices: int, device, rows: int) -> Optional[SplitPlan]:
    """None when no sequence is worth cutting; otherwise the plan (device tensors) for these bounds."""
    chunks = [(e - s + CHUNK - 1) // CHUNK for s, e in bounds]
    pieces = piece_counts(chunks, HV, slices, sm_count(device))
    if max(pieces, default=1) <= 1:
        return None
    vbounds, chains, pre_fwd, pre_bwd, first_piece, last_piece = [], [], [], [], [], []
    n_pre = 0
    for (s, e), c, P in zip(bounds, chunks, pieces):
        first = len(vbounds)
        base, rem = divmod(c, P)
        start = s
        for p in range(P):
            n = base + (1 if p < rem else 0)
            end = min(e, start + n * CHUNK) if p < P - 1 else e
            vbounds.append((start, end))
            start = end
        chains.append((first, P, n_pre))
        pre_fwd += list(range(first, first + P - 1))
        pre_bwd += list(range(first + 1, first + P))
        n_pre += P - 1
        first_piece.append(first)
        last_piece.append(first + P - 1)
    plan = SplitPlan()
    tables = device_tables(vbounds, device)
    sm = build_tables(vbounds)[1]
    tables.covered = bool(bounds) and bounds[0][0] == 0 and bounds[-1][1] == rows
    plan.tables, plan.n_pieces, plan.n_pre, plan.n_chains = tables, len(vbounds), n_pre, len(bounds)
    plan.chains = torch.tensor(chains, dtype=torch.int32).to(device)
    plan.pre_fwd = torch.from_numpy(sm[pre_fwd]).contiguous().to(device)
    plan.pre_bwd = torch.from_numpy(sm[pre_bwd]).contiguous().to(device)
    plan.first_piece = torch.tensor(first_piece, dtype=torch.long).to(device)
    plan.last_piece = torch.tensor(last_piece, dtype=torch.long).to(device)
    plan.pieces_per_seq = pieces
    plan._native = None
    return plan


def split_plan_for(B: int, T: int, cu_seqlens, cu_seqlens_cpu, device, HV: int, slices: int) -> Optional[SplitPlan]:
    """Memoised like tables_for (by shape, or by the identity and version of ``cu_seqlens``)."""
    version = None if cu_seqlens is None else content_version(cu_seqlens)
    if cu_seqlens is None:
        key = ('dense', B, T, HV, slices, FORCE_PIECES, device)
        hit = _split_cache.get(key)
        if hit is not None:
            return hit[0]
        bounds = [(b * T, (b + 1) * T) for b in range(B)]
    else:
        key = ('varlen', id(cu_seqlens), B * T, HV, slices, FORCE_PIECES, device)
        hit = _split_cache.get(key)
        if hit is not None and hit[1] is cu_seqlens and hit[2] == version:
            return hit[0]
        bounds = packed_bounds(cu_seqlens, cu_seqlens_cpu, B * T, version)
    plan = split_plan(bounds, HV, slices, device, B * T)
    if len(_split_cache) > 64:
        _split_cache.clear()
    _split_cache[key] = (plan, cu_seqlens, version)
    return plan


def native_plan(B: int, T: int, cu_seqlens, cu_seqlens_cpu, device, HV: int, slices: int):
    """Handle of the split plan of these sequences, or of their chunk tables when none is worth cutting."""
    plan = split_plan_for(B, T, cu_seqlens, cu_seqlens_cpu, device, HV, slices)
    return (plan if plan is not None else tables_for(B, T, cu_seqlens, cu_seqlens_cpu, device)).native()
