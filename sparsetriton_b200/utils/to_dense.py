"""Sparse -> dense conversion (reference: utils/to_dense.py:143-282).

`to_dense(feats, coords, spatial_range)` keeps the reference's signature and its (B, X, Y, Z, C)
result.  Forward is one scatter kernel (st_to_dense_fwd, which also clears the volume), backward one
gather kernel (st_to_dense_bwd): both move 16-byte pieces of feature rows and are bound by HBM.

`batch_size` (no reference counterpart) lets a caller that already knows the batch size skip the
device->host read of `coords[:, 0].max()`; SparseTensor.dense() passes its own.
"""
import torch

from sparsetriton_b200 import _lib

__all__ = ["to_dense", "ToDenseFunction"]


class ToDenseFunction(torch.autograd.Function):
    """feats (N, C), coords (N, 4) -> dense (batch, X, Y, Z, C); backward gives grad_feats only.  `apply` makes the native
    node (host/spatial.cpp)."""

    @staticmethod
    def apply(feats, coords, spatial_range, batch_size):
        _lib.require_cuda(feats, "to_dense")
        return _lib.host().to_dense(feats, coords, [int(v) for v in spatial_range], int(batch_size))


def to_dense(feats, coords, spatial_range, batch_size=None):
    """Dense (B, X, Y, Z, C) copy of the sparse rows; B = largest batch index + 1 (1 for an empty tensor)
    unless `batch_size` is given."""
    if batch_size is None:
        batch_size = int(coords[:, 0].max().item()) + 1 if coords.shape[0] > 0 else 1
    return ToDenseFunction.apply(feats, coords, tuple(spatial_range), batch_size)
