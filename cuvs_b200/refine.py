"""Mirror of the reference's ``cuvs.neighbors.refine`` (python/cuvs/cuvs/neighbors/refine/refine.pyx):
re-rank candidate neighbours with exact distances on the original vectors."""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib as L
from .common import CUDA_DEVICES, ELEMENT_TYPES, DLTensorRef, Resources, default_resources, is_cuda_matrix
from .ivf_pq import _METRICS


def _refine_arrays(dataset, queries, candidates, k, metric, indices, distances, resources, sync):
    """The whole call for CUDA tensors in one native call (40 us of a call on 4 queries were mostly descriptors and
    foreign calls).  None where an argument is not what that call takes: the general path then says what is wrong."""
    if type(dataset) is not torch.Tensor:
        return None
    kind, code = dataset.dtype, _METRICS.get(metric)
    word = ELEMENT_TYPES.get(kind)
    if word is None or code is None or not is_cuda_matrix(dataset, kind) or not is_cuda_matrix(queries, kind) or \
            not is_cuda_matrix(candidates, torch.int64):
        return None
    device = torch.cuda.current_device()
    n, dim = queries.shape
    if device >= len(CUDA_DEVICES) or dataset.shape[1] != dim or candidates.shape[0] != n:
        return None
    if indices is None:
        indices = torch.empty((n, k), dtype=torch.int64, device=CUDA_DEVICES[device])
    elif not is_cuda_matrix(indices, torch.int64):
        return None
    if distances is None:
        distances = torch.empty((n, k), dtype=torch.float32, device=CUDA_DEVICES[device])
    elif not is_cuda_matrix(distances, torch.float32):
        return None
    out = indices.shape
    if out != distances.shape or out[0] != n or out.numel() == 0 or dataset.numel() == 0 or candidates.numel() == 0:
        return None
    res = resources or default_resources(device)
    L.check(L.load().cuvsB200RefineArrays(res.handle, res.stream_at_call(device), dataset.data_ptr(), dataset.shape[0],
                                          dim, word[0], word[1], queries.data_ptr(), n, candidates.data_ptr(),
                                          candidates.shape[1], code, indices.data_ptr(), distances.data_ptr(), out[1],
                                          bool(sync)))
    return distances, indices


def refine(dataset, queries, candidates, k=None, metric="sqeuclidean", indices=None, distances=None,
           resources: Resources | None = None, sync: bool = True):
    """Returns ``(distances, indices)`` of the k best candidates per query by exact distance."""
    n = queries.shape[0]
    if k is None:
        if indices is None:
            raise ValueError("Argument k must be specified if both indices and distances arg is None")
        k = indices.shape[1]
    found = _refine_arrays(dataset, queries, candidates, k, metric, indices, distances, resources, sync)
    if found is not None:
        return found
    res = resources or default_resources()
    res.use_current_stream()
    if indices is None:
        indices = torch.empty((n, k), dtype=torch.int64, device="cuda")
    if distances is None:
        distances = torch.empty((n, k), dtype=torch.float32, device="cuda")
    if metric not in _METRICS:
        raise ValueError(f"metric {metric!r} not supported")
    a, b, c, d, e = (DLTensorRef(t) for t in (dataset, queries, candidates, indices, distances))
    L.check(L.load().cuvsRefine(res.handle, a.ref(), b.ref(), c.ref(), C.c_int(_METRICS[metric]),
                                d.ref(), e.ref()))
    if sync:
        res.sync()
    return distances, indices
