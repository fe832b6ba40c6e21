"""Per-topology device structures shared by the operators: the vertex -> (face, corner)
CSR, its cache, and the validation of index arrays.

A level's `face` / `vtMap` tensors are reused by every convolution of that level (4 to 16
operator calls per step in the reference's encoder blocks,
picasso/networks/pi2_blocks.py:88-92), so the CSR is built once per (face, vtMap) pair
and looked up afterwards.

Cache policy (TopologyCache in csrc/torch_ops.cpp).  An entry is named by the memory of the index
tensors (device, data pointer, length, stride, type) and good while those storages live and their version counters
stand still.  A lookup whose versions differ (the tensors were overwritten in place, as a streaming
loader does with its device buffers) rebuilds the structure and REPLACES the entry, so stale entries
never pile up; entries whose tensors are gone are dropped at the next insertion, so neither do those of
past batches.  The cache is bounded by bytes (`set_cache_budget`, default 2 GiB of CSR arrays
per process) and evicts least-recently-used entries; `set_cache_budget(0)` turns it off.
Callers that manage topologies themselves can pass a prebuilt `VertexCSR` to the operator
wrappers (`csr=`) and skip the cache altogether.

Validation.  Building a CSR validates every index of `face` / `vtMap` on the device.  In the
default mode the status word is read back right after the build (ONE device synchronisation
per cache miss, which also answers whether `vtMap` is the identity) and a bad index raises
RuntimeError.  `set_validation("deferred")` removes that synchronisation: status words are
kept and `check_deferred()` reads them all at a point where the caller synchronises anyway
(the end of a step).  Bad indices are never dereferenced in either mode.  Arrays that only a backward pass
reads are made ahead of it, in the forward pass; a bad index in them is reported by the backward pass.

Streams and modes.  A structure found on another stream than the one that made it is waited for there; one made inside a
graph capture is found inside that capture only.  Structures outlive the call that makes them and end up in autograd
graphs, so they are ordinary tensors also when that call runs under torch.inference_mode.
"""
from __future__ import annotations

import contextlib
import threading
from typing import List, Optional

import torch

from . import _lib

_ops = _lib.ops
_VERTEX, _CLUSTER, _PAIRS, _MEANS, _MEANS_SH, _SAMPLES = range(6)      # kinds of cache entries
_lock = threading.Lock()
_validation = "sync"
_deferred: List[tuple] = []          # (status tensor, message)


def stream_ptr(device) -> int:
    return torch.cuda.current_stream(device).cuda_stream


def ptr(t: Optional[torch.Tensor]):
    return None if t is None else t.data_ptr()


def set_cache_budget(nbytes: int) -> None:
    """Upper bound on the bytes of CSR arrays the cache keeps (0 = no caching)."""
    _ops.cache_budget(int(nbytes))


def set_validation(mode: str) -> None:
    """'sync' (default): raise on a bad index at build time, one device sync per cache miss.
    'deferred': no sync; call check_deferred() after the step's own synchronisation."""
    global _validation
    if mode not in ("sync", "deferred"):
        raise ValueError(mode)
    _validation = mode


def check_deferred() -> None:
    """Reads every status word collected in deferred mode (synchronises); raises RuntimeError
    for the first bad one."""
    with _lock:
        items = list(_deferred)
        _deferred.clear()
    if not items:
        return
    codes = torch.stack([s.reshape(-1)[0] for s, _ in items]).tolist()
    for code, (_, msg) in zip(codes, items):
        if code != 0:
            raise RuntimeError(msg)


class BadIndex(RuntimeError):
    """An index array holds an index outside its range."""


class VertexCSR:
    """rowptr (NvOut+1,), entries (3*Nf,) int32: row v lists (f << 2 | corner) ascending."""

    def __init__(self, rowptr, entries):
        self.rowptr = rowptr
        self.entries = entries

    def _tensors(self):
        return [self.rowptr, self.entries]


def _store(kind, a, b, m, n, value, shared=False, validated=True):
    """Puts a structure made from the index tensors a (and b) into the cache; shared: its arrays belong to another entry.
    validated: a status word behind its kernels is looked at, in 'sync' mode before this call."""
    tensors = value._tensors()
    _ops.cache_put(kind, a, b, m, n, tensors, value, 0 if shared else sum(t.numel() * t.element_size() for t in tensors),
                   validated and _validation == "sync")


def _building(device):
    """The device of a structure that is made; not under inference mode, for it is kept."""
    if not torch.is_inference_mode_enabled():
        return torch.cuda.device(device)
    stack = contextlib.ExitStack()
    stack.enter_context(torch.inference_mode(False))
    stack.enter_context(torch.cuda.device(device))
    return stack


def _launch_build(face, vt_map, nv_in, nv_out):
    dev = face.device
    nf = face.shape[0]
    if nf > 0 and (face.dim() != 2 or face.shape[1] != 3):
        raise RuntimeError("face must have shape (NfIn, 3)")
    rowptr = torch.empty(nv_out + 1, dtype=torch.int32, device=dev)
    entries = torch.empty(max(3 * nf, 1), dtype=torch.int32, device=dev)
    status = torch.empty(1, dtype=torch.int32, device=dev)
    wbytes = _lib.query("pb200_vertex_csr_workspace_bytes", nf, nv_out)
    ws = torch.empty(wbytes, dtype=torch.uint8, device=dev)
    _lib.call("pb200_build_vertex_csr", nf, nv_in, nv_out, ptr(face), ptr(vt_map), ptr(rowptr),
              ptr(entries), ptr(status), ptr(ws), wbytes, stream_ptr(dev))
    return rowptr, entries, status


def _bad_index_message(nv_in, nv_out):
    return f"face / vtMap hold an index outside the vertex range (NvIn={nv_in}, NvOut={nv_out})"


def build_vertex_csr(face: torch.Tensor, vt_map: Optional[torch.Tensor], nv_in: int, nv_out: int) -> VertexCSR:
    """Uncached build.  Validates every index: in 'sync' mode a bad one raises RuntimeError here
    (one device synchronisation), in 'deferred' mode at the next check_deferred()."""
    with _building(face.device):
        rowptr, entries, status = _launch_build(face, vt_map, nv_in, nv_out)
        if _validation == "deferred":
            with _lock:
                _deferred.append((status, _bad_index_message(nv_in, nv_out)))
        elif int(status.item()) != 0:
            raise BadIndex(_bad_index_message(nv_in, nv_out))
    return VertexCSR(rowptr, entries)


def vertex_csr(face: torch.Tensor, vt_map: Optional[torch.Tensor], nv_in: int, nv_out: int) -> VertexCSR:
    """Cached CSR keyed by output vertex vo = vtMap[face[f][j]] (identity when vt_map is None).
    In 'sync' mode an identity vtMap over nv_in == nv_out vertices shares the arrays of
    vt_map=None (the identity test rides on the build's one synchronisation); in 'deferred'
    mode nothing is read back and the CSR is built from vtMap as given."""
    hit = _ops.cache_find(_VERTEX, face, vt_map, nv_in, nv_out)
    if hit is not None:
        return hit
    may_be_identity = vt_map is not None and nv_in == nv_out and vt_map.shape[0] == nv_in
    if may_be_identity and _validation == "sync":
        base = _ops.cache_find(_VERTEX, face, None, nv_in, nv_out)
        with _building(face.device):
            ident = (vt_map == torch.arange(nv_in, dtype=vt_map.dtype, device=vt_map.device)).all().to(torch.int32)
            if base is None:
                # build the identity CSR and test vtMap in the same synchronisation
                rowptr, entries, status = _launch_build(face, None, nv_in, nv_out)
                code, is_ident = torch.stack([status[0], ident]).tolist()
                if code != 0:
                    raise BadIndex(_bad_index_message(nv_in, nv_out))
                base = VertexCSR(rowptr, entries)
                _store(_VERTEX, face, None, nv_in, nv_out, base)
            else:
                is_ident = int(ident.item())
        if is_ident:
            _store(_VERTEX, face, vt_map, nv_in, nv_out, base, shared=True)
            return base
    csr = build_vertex_csr(face, vt_map, nv_in, nv_out)
    _store(_VERTEX, face, vt_map, nv_in, nv_out, csr)
    return csr


def prepare_level(vertex: torch.Tensor, face: torch.Tensor, vt_map: Optional[torch.Tensor], nv_out: int, L: int,
                  orient: bool = False, want_geometry: bool = True, want_normals: bool = False):
    """Everything a mesh level's convolutions need, in one library call: triangle geometry
    (picasso/mesh/pi_modules/decimate.py:70-85), the (optionally origin-oriented,
    picasso/networks/scene_seg.py:117-124) face normals, their spherical-harmonic filter coefficients
    (picasso/mesh/layers.py:341-356), nfCount (decimate_gpu.cu:813-836) and the vertex CSR, which is
    put into the cache for the operator calls that follow.  Returns a dict with keys geometry (Nf,5)
    or None, normals (Nf,3) or None, coeff (Nf,(L+1)^2), nf_count (NvOut,), csr."""
    if L >= 6 or L < 0:
        raise NotImplementedError
    if not (vertex.is_cuda and face.is_cuda) or vertex.dtype != torch.float32 or face.dtype != torch.int32:
        raise RuntimeError("vertex must be a float32 and face an int32 CUDA tensor")
    if vertex.dim() != 2 or vertex.shape[1] < 3 or face.dim() != 2 or face.shape[1] != 3:
        raise RuntimeError("vertex must have shape (Nv, >=3) and face (Nf, 3)")
    vertex, face = vertex.contiguous(), face.contiguous()
    nv_in, nf = vertex.shape[0], face.shape[0]
    geometry, normals, coeff, nf_count, rowptr, entries, status = _lib.ops.level_prepare(
        vertex, face, vt_map, nv_out, L, bool(orient), bool(want_geometry), bool(want_normals))
    if _validation == "deferred":
        with _lock:
            _deferred.append((status, _bad_index_message(nv_in, nv_out)))
    elif int(status.item()) != 0:
        raise BadIndex(_bad_index_message(nv_in, nv_out))
    csr = VertexCSR(rowptr, entries)
    _store(_VERTEX, face, vt_map, nv_in, nv_out, csr)
    return dict(geometry=geometry, normals=normals, coeff=coeff, nf_count=nf_count, csr=csr)


def for_backward(structure, *args):
    """structure(*args) that only a backward pass reads, or None when it raises BadIndex: the forward pass, in which such an index
    contributes nothing, is not refused for it; the node's backward pass is."""
    try:
        return structure(*args)
    except BadIndex:
        return None


class ClusterCSR:
    """Decimation clusters of a fine level: key (NvIn,) = coarse id of each fine vertex or -1;
    rowptr (NvOut+1,), members (NvIn,) = member fine vertices of every coarse vertex, ascending."""

    def __init__(self, key, rowptr, members):
        self.key = key
        self.rowptr = rowptr
        self.members = members

    def _tensors(self):
        return [self.key, self.rowptr, self.members]


def cluster_csr(vt_replace: torch.Tensor, vt_map: torch.Tensor, nv_out: int) -> ClusterCSR:
    """Cached cluster structures of (vtReplace, vtMap) (same cache, budget and validation modes as
    vertex_csr).  One pooling level is used by a pool in the encoder and an unpool in the decoder,
    forward and backward: four lookups per step, one build."""
    nv_in = vt_replace.shape[0]
    hit = _ops.cache_find(_CLUSTER, vt_replace, vt_map, nv_out, 0)
    if hit is not None:
        return hit
    dev = vt_replace.device
    with _building(dev):
        key = torch.empty(max(nv_in, 1), dtype=torch.int32, device=dev)
        rowptr = torch.empty(nv_out + 1, dtype=torch.int32, device=dev)
        members = torch.empty(max(nv_in, 1), dtype=torch.int32, device=dev)
        status = torch.empty(1, dtype=torch.int32, device=dev)
        wbytes = _lib.query("pb200_cluster_csr_workspace_bytes", nv_in, nv_out)
        ws = torch.empty(wbytes, dtype=torch.uint8, device=dev)
        _lib.call("pb200_build_cluster_csr", nv_in, nv_out, ptr(vt_replace), ptr(vt_map), ptr(key), ptr(rowptr),
                  ptr(members), ptr(status), ptr(ws), wbytes, stream_ptr(dev))
        msg = f"vtReplace / vtMap hold an index outside the vertex range (NvIn={nv_in}, NvOut={nv_out})"
        if _validation == "deferred":
            with _lock:
                _deferred.append((status, msg))
        elif int(status.item()) != 0:
            raise RuntimeError(msg)
    csr = ClusterCSR(key, rowptr, members)
    _store(_CLUSTER, vt_replace, vt_map, nv_out, 0, csr)
    return csr


class PairCSR:
    """Neighbour pairs grouped by one column of nnIndex: rowptr (rows+1,), members (pairs,) = pair ids
    of every row, ascending."""

    def __init__(self, rowptr, members):
        self.rowptr = rowptr
        self.members = members

    def _tensors(self):
        return [self.rowptr, self.members]


def pair_csr(nn_index: torch.Tensor, column: int, n_rows: int) -> PairCSR:
    """Cached grouping of the neighbour pairs of a point-cloud convolution by their output point
    (column 0) or input point (column 1); same cache, budget and validation modes as vertex_csr."""
    npairs = nn_index.shape[0]
    if npairs > 0 and (nn_index.dim() != 2 or nn_index.shape[1] != 2):
        raise RuntimeError("nn_index must have shape (pairs, 2)")
    hit = _ops.cache_find(_PAIRS, nn_index, None, column, n_rows)
    if hit is not None:
        return hit
    dev = nn_index.device
    with _building(dev):
        rowptr = torch.empty(n_rows + 1, dtype=torch.int32, device=dev)
        members = torch.empty(max(npairs, 1), dtype=torch.int32, device=dev)
        status = torch.empty(1, dtype=torch.int32, device=dev)
        wbytes = _lib.query("pb200_cluster_csr_workspace_bytes", npairs, n_rows)
        ws = torch.empty(wbytes, dtype=torch.uint8, device=dev)
        key_ptr = None if npairs == 0 else nn_index.data_ptr() + 4 * column
        _lib.call("pb200_build_key_csr", npairs, n_rows, key_ptr, 2, ptr(rowptr), ptr(members), ptr(status), ptr(ws), wbytes,
                  stream_ptr(dev))
        msg = f"nn_index column {column} holds an index outside [0, {n_rows})"
        if _validation == "deferred":
            with _lock:
                _deferred.append((status, msg))
        elif int(status.item()) != 0:
            raise BadIndex(msg)
    csr = PairCSR(rowptr, members)
    _store(_PAIRS, nn_index, None, column, n_rows, csr)
    return csr


class FaceMeans:
    """Per-face mean of the sample rows of a batch (Nf, F) and the running count 1, 2, ..., Nf that says
    'one sample per face'."""

    def __init__(self, rows, one_each):
        self.rows = rows
        self.one_each = one_each
        # the copy with rows padded to a multiple of four floats that the tensor-core kernels read (None when the row
        # length is such a multiple already): made once here instead of in every forward and backward call
        self.rows_padded = pad_rows(rows)

    def _tensors(self):
        return [t for t in (self.rows, self.one_each, self.rows_padded) if t is not None]


def pad_rows(rows: torch.Tensor):
    """(N, F) float32 rows -> (N, F rounded up to 4) with zero pad columns, or None when F % 4 == 0."""
    n, F = rows.shape
    if F % 4 == 0 or n == 0:
        return None
    Fp = _lib.query("pb200_padded_row_floats", F)
    dev = rows.device
    with _building(dev):
        out = torch.empty(n, Fp, dtype=torch.float32, device=dev)
        _lib.call("pb200_pad_rows", n, F, ptr(rows), ptr(out), stream_ptr(dev))
    return out


def face_means(sample_rows: torch.Tensor, num_interior: torch.Tensor) -> FaceMeans:
    """Cached mean over every face's samples of sample_rows (NiK, F) (num_interior = inclusive running sample
    count, as facet2facet takes it); same cache and budget as vertex_csr.  Forward and backward of a step share it."""
    nf, nik = num_interior.shape[0], sample_rows.shape[0]
    hit = _ops.cache_find(_MEANS, sample_rows, num_interior, sample_rows.shape[1], 0)
    if hit is not None:
        return hit
    dev = sample_rows.device
    with _building(dev):
        check_num_interior(num_interior, nik)
        rows = torch.empty(nf, sample_rows.shape[1], dtype=torch.float32, device=dev)
        _lib.call("pb200_face_mean_rows", nf, nik, sample_rows.shape[1], ptr(sample_rows), ptr(num_interior), ptr(rows),
                  stream_ptr(dev))
        fm = FaceMeans(rows, torch.arange(1, nf + 1, dtype=torch.int32, device=dev))
    _store(_MEANS, sample_rows, num_interior, sample_rows.shape[1], 0, fm, validated=False)
    return fm


def face_means_sph_harm(L: int, sample_xyz: torch.Tensor, num_interior: torch.Tensor) -> FaceMeans:
    """face_means(sph_harm_coeff(L, sample_xyz), num_interior) in one kernel (identical bits), without the
    (NiK, (L+1)^2) array; cached the same way."""
    nf, nik = num_interior.shape[0], sample_xyz.shape[0]
    hit = _ops.cache_find(_MEANS_SH, sample_xyz, num_interior, L, 0)
    if hit is not None:
        return hit
    if sample_xyz.dim() != 2 or sample_xyz.shape[1] != 3 or sample_xyz.dtype != torch.float32 or not sample_xyz.is_contiguous():
        raise RuntimeError("sample_xyz must be a contiguous float32 tensor of shape (NiK, 3)")
    dev = sample_xyz.device
    with _building(dev):
        check_num_interior(num_interior, nik)
        rows = torch.empty(nf, (L + 1) ** 2, dtype=torch.float32, device=dev)
        _lib.call("pb200_face_mean_sph_harm", nf, nik, int(L), ptr(sample_xyz), ptr(num_interior), ptr(rows), stream_ptr(dev))
        fm = FaceMeans(rows, torch.arange(1, nf + 1, dtype=torch.int32, device=dev))
    _store(_MEANS_SH, sample_xyz, num_interior, L, 0, fm, validated=False)
    return fm


class SampleEnds:
    """Running number of rows up to and including every sample (B,) int64."""

    def __init__(self, ends):
        self.ends = ends

    def _tensors(self):
        return [self.ends]


def sample_ends(counts: torch.Tensor, n_rows: int) -> torch.Tensor:
    """Cached running totals of the samples' row counts; same cache, budget and validation modes as vertex_csr.  They must
    add up to n_rows."""
    hit = _ops.cache_find(_SAMPLES, counts, None, n_rows, 0)
    if hit is not None:
        return hit.ends
    with _building(counts.device):
        ends = torch.cumsum(counts.detach(), 0, dtype=torch.int64)
        bad = ends[-1:] != n_rows if counts.shape[0] else torch.full((1,), n_rows != 0, device=counts.device)
        bad = bad | (counts < 0).any()
    msg = "the samples' row counts must be non-negative and add up to the number of rows"
    if _validation == "deferred":
        with _lock:
            _deferred.append((bad.to(torch.int32), msg))
    elif bool(bad.item()):
        raise RuntimeError(msg)
    _store(_SAMPLES, counts, None, n_rows, 0, SampleEnds(ends))
    return ends


def check_num_interior(num_interior: torch.Tensor, nik: int) -> None:
    """Validates a running sample count (non-decreasing, inside [0, nik], ends at nik) on the
    device: raises in 'sync' mode, queues the status word in 'deferred' mode.  The facet2facet
    kernels trust numInterior as the reference does; run this once per array."""
    dev = num_interior.device
    with _building(dev):
        status = torch.empty(1, dtype=torch.int32, device=dev)
        _lib.call("pb200_check_num_interior", num_interior.shape[0], int(nik), ptr(num_interior), ptr(status),
                  stream_ptr(dev))
        msg = f"numInterior is not a running count that ends at NiK={nik}"
        if _validation == "deferred":
            with _lock:
                _deferred.append((status, msg))
        elif int(status.item()) != 0:
            raise RuntimeError(msg)


def cache_stats():
    slots, nbytes, budget = _ops.cache_stats()
    return {"slots": slots, "bytes": nbytes, "budget": budget}


def clear_cache() -> None:
    _ops.cache_clear()
