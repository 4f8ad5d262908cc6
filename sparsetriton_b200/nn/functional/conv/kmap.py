"""Output coordinates of a sparse convolution (reference: nn/functional/conv/kmap.py).

`build_out_coords` keeps the reference's signature and return triple.  What differs is how the
work is done: the reference materialises all N*K candidate rows, filters them with three
boolean-mask compactions and dedupes through a scratch table of 31-bit keys; here one C-ABI call
enumerates candidates in registers, dedupes on exact 64-bit keys keeping the candidate with the
smallest flat index n*K+k, and a second call writes the survivors in that order.  The order is the
one the reference's sequential CPU path produces (first occurrence, n-major, k-minor), and it does
not depend on thread scheduling.

Two reference behaviours are intentionally not reproduced:
  * coordinates whose 31-bit keys collide are merged by the reference (kmap.py:93); here they stay
    distinct;
  * the transposed path multiplies the batch column by the stride (kmap.py:407), which breaks
    batch indices >= 1; here only the spatial columns are scaled.
"""
from typing import Tuple

import torch

from sparsetriton_b200 import _lib

__all__ = ["build_out_coords", "out_coords_and_map", "PendingOutCoordsAndMap", "kernel_offsets", "output_shape"]


def kernel_offsets(kernel_size: int, dilation: int, padding: int, transposed: bool):
    """(K,3) python list of offsets, K = kernel_size^3, k = (ix*ks + iy)*ks + iz.

    base = (i - ks//2) * dilation per axis (kmap.py:104-132);
    normal: -base + padding - ((ks-1)*dilation)//2 (:135-156); transposed: the negation (:159-180).
    """
    ks, half = kernel_size, ((kernel_size - 1) * dilation) // 2
    axis = [(i - ks // 2) * dilation for i in range(ks)]
    sign, shift = (1, half - padding) if transposed else (-1, padding - half)
    one = [sign * a + shift for a in axis]
    return [(one[ix], one[iy], one[iz]) for ix in range(ks) for iy in range(ks) for iz in range(ks)]


def output_shape(spatial_shape, kernel_size, stride, dilation, padding, transposed):
    """New spatial shape: kmap.py:254-258 (normal), :373-377 (transposed)."""
    if transposed:
        return tuple((int(s) - 1) * stride + (kernel_size - 1) * dilation - 2 * padding + 1 for s in spatial_shape)
    return tuple((int(s) - (kernel_size - 1) * dilation + 2 * padding - 1) // stride + 1 for s in spatial_shape)


_CONSTANTS = {}


def _constant_tensor(values, dtype, device, shape):
    """Small constant device tensor, made once per (values, dtype, device): building one from a python list is a
    pageable host->device copy, which waits for everything its stream holds."""
    key = (tuple(values), dtype, device.type, device.index, shape)
    t = _CONSTANTS.get(key)
    if t is None:
        if len(_CONSTANTS) > 256:
            _CONSTANTS.clear()
        t = _CONSTANTS[key] = torch.tensor(list(values), dtype=dtype, device=device).reshape(shape)
    return t


def _offsets_tensor(offsets, like):
    """(K,3) device tensor of the offsets in the coordinate dtype.  Shared between calls: treat as read-only."""
    t = _constant_tensor([v for o in offsets for v in o], like.dtype, like.device, (-1, 3))
    return t.view(t.shape)            # a fresh tensor object per call (callers attach attributes), same storage


def build_out_coords(
    in_coords: torch.Tensor,
    spatial_shape: Tuple[int, int, int],
    kernel_size: int,
    stride: int = 1,
    dilation: int = 1,
    padding: int = 1,
    transposed: bool = False,
    submanifold: bool = True,
    chunk_size: int = None,
):
    """Returns (out_coords, new_spatial_shape, kernel_offsets) as kmap.py:447-495 does.

    out_coords has the dtype of in_coords; new_spatial_shape is an int64 device tensor of 3
    values, or `spatial_shape` itself on the submanifold shortcut; kernel_offsets is a (K,3)
    device tensor of the coordinate dtype.  `chunk_size` is accepted and ignored (nothing is
    materialised per chunk).
    """
    device = in_coords.device
    offsets = kernel_offsets(kernel_size, dilation, padding, transposed)
    koff = _offsets_tensor(offsets, in_coords).clone()          # the caller's own copy (a device-side copy: no wait)
    new_shape = output_shape(spatial_shape, kernel_size, stride, dilation, padding, transposed)

    # kmap.py:261-262 / :380-381
    if submanifold and stride == 1 and ((kernel_size - 1) * dilation) // 2 == padding:
        return in_coords, spatial_shape, koff

    new_shape_t = _constant_tensor(new_shape, torch.int64, device, (3,)).clone()
    new_shape_t._st_host = new_shape      # spares callers in this package a device->host read
    out, _ = _run_out_coords(in_coords, kernel_size, dilation, padding, new_shape, stride, transposed, with_map=False)
    return out, new_shape_t, koff


def out_coords_and_map(in_coords, spatial_shape, kernel_size, stride, dilation, padding, transposed, batch_bound=0):
    """Output coordinates AND the (N_out, K) neighbour map of a strided / transposed convolution in
    one pass over the candidates (the map is scattered from the same dedupe table instead of probing
    the input table N_out*K times).  Returns (out_coords, new_shape tuple, kernel_offsets tensor, nbr).
    Same results as build_out_coords followed by compute_neighbor_indices.  `batch_bound`: the number of samples in
    the batch (every batch index below it) if the caller knows it, else 0; it lets the library dedupe by direct
    addressing instead of hashing."""
    return PendingOutCoordsAndMap(in_coords, spatial_shape, kernel_size, stride, dilation, padding, transposed,
                                  batch_bound).finish()


def _run_out_coords(in_coords, kernel_size, dilation, padding, new_shape, stride, transposed, with_map, in_shape=(0, 0, 0),
                    batch_bound=0):
    """(out_coords, nbr or None) of a strided / transposed layer, through the native two-pass build."""
    return _begin_out_coords(in_coords, kernel_size, dilation, padding, new_shape, stride, transposed, with_map, in_shape,
                             batch_bound).finish()[:2]


def _begin_out_coords(in_coords, kernel_size, dilation, padding, new_shape, stride, transposed, with_map, in_shape, batch_bound):
    """First half: candidates counted and deduplicated on the current stream, the count on its way to pinned host
    memory.  `.finish()` waits for that alone (not for the stream), sizes the outputs, launches the second half on the same
    stream and returns (out_coords, nbr, state of the map)."""
    if in_coords.shape[0] > 0:
        _lib.require_cuda(in_coords, "build_out_coords")
    return _lib.host().OutCoords(in_coords, kernel_size, stride, dilation, padding, bool(transposed), list(new_shape),
                                 [int(v) for v in in_shape], int(batch_bound or 0), with_map)


class PendingOutCoordsAndMap:
    """`out_coords_and_map` in two halves: construction launches the counting half, `finish()` returns what
    `out_coords_and_map` returns.  Lets a caller put other work between the launch and the wait for the count."""

    def __init__(self, in_coords, spatial_shape, kernel_size, stride, dilation, padding, transposed, batch_bound=0):
        self.geometry = (kernel_size, dilation, padding, transposed)
        self.like = in_coords
        self.new_shape = output_shape(spatial_shape, kernel_size, stride, dilation, padding, transposed)
        self.pending = _begin_out_coords(in_coords, kernel_size, dilation, padding, self.new_shape, stride, transposed, True,
                                         spatial_shape, batch_bound)

    def finish_map(self):
        """(out_coords, new_shape, nbr): `finish` without the offsets tensor."""
        out, nbr, state = self.pending.finish()
        nbr._st_map = state
        return out, self.new_shape, nbr

    def finish(self):
        out, new_shape, nbr = self.finish_map()
        offsets = kernel_offsets(*self.geometry)
        koff = _offsets_tensor(offsets, self.like)
        koff._st_host = [v for o in offsets for v in o]
        return out, new_shape, koff, nbr
