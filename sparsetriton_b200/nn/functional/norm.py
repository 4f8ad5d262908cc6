"""Per-sample batch normalisation of sparse features (reference: nn/functional/norm.py:20-112).

Statistics are taken per (batch index, channel), exactly as in the reference, so sharding a batch by
sample over GPUs needs no cross-GPU statistics.  On the GPU the layer runs as four streaming kernels
behind the C ABI (st_bn_forward_stats + st_bn_apply forward, st_bn_backward backward: one pass over the features
for the statistics, one for the output, two for the gradient; no elementwise torch ops in between), with the
ReLU that follows it in the reference's networks optionally folded in (`relu=True`; the reference has
no fused form, its ReLU is a separate module).  Unlike the reference, half / bfloat16 features are
accepted: statistics are fp32 and the result is cast back to the feature dtype.  The autograd node is native (host/norm.cpp).
"""
import torch

from sparsetriton_b200 import _lib
from sparsetriton_b200.tensor import SparseTensor

__all__ = ["sparse_batch_norm"]


def _batch_info(tensor: SparseTensor):
    """(int32 batch index per row, fp32 1/count per sample, int32 status word, int32 first row per sample), memoised with the coordinate
    set.  The kernels OR ST_DEV_BAD_INDEX into the status word for rows whose batch index is not in
    [0, batch_size) -- such rows join no statistic and come out as zeros; `bad_batch_index(tensor)` reads it."""
    cache = tensor._cache.kmaps
    hit = cache.get("batch_info")
    if hit is None or hit[0].shape[0] != tensor.C.shape[0]:
        hit = cache["batch_info"] = _lib.host().batch_info(tensor.C, int(tensor.batch_size))
    return hit


def bad_batch_index(tensor: SparseTensor) -> bool:
    """True if a batch-norm kernel has met a batch index outside [0, batch_size) on this tensor's
    coordinate set (one device->host read)."""
    hit = tensor._cache.kmaps.get("batch_info")
    return bool(hit is not None and int(hit[2].item()) & _lib.DEV_BAD_INDEX)


def sparse_batch_norm(tensor: SparseTensor, weight=None, bias=None, running_mean=None, running_var=None,
                      training=True, eps=1e-5, momentum=0.1, relu=False) -> SparseTensor:
    feats = tensor.F
    if feats.shape[0] == 0:
        return tensor.replace(feats)
    if training:
        if (running_mean is not None and running_mean.dtype != torch.float32) or \
                (running_var is not None and running_var.dtype != torch.float32):
            raise TypeError("running_mean / running_var must be float32 tensors")
        batch, inv_count, status, first_row = _batch_info(tensor)
        # the running buffers are updated by the statistics kernel itself (norm.py:91-94)
        y = _lib.host().batch_norm_train(feats, weight, bias, batch, inv_count, status, first_row, running_mean, running_var,
                                         int(tensor.batch_size), float(eps), float(momentum), bool(relu))
    else:
        y = _lib.host().batch_norm_running(feats, weight, bias, running_mean, running_var, float(eps), bool(relu))
    return tensor.replace(y)
