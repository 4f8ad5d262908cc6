"""Thin torch wrappers that act on SparseTensor.F (reference: nn/modules/linear.py:23-73,
nn/modules/activation.py:23-65)."""
import torch
from torch import nn

from sparsetriton_b200 import _lib
from sparsetriton_b200.tensor import SparseTensor

__all__ = ["SparseLinear", "ReLU"]

_SPLIT_ROWS = 8192          # rows per partial product of the weight gradient
_TALL = 1 << 16             # from this many rows on the weight gradient is split


class _TallLinear(torch.autograd.Function):
    """y = x W^T + b for a matrix of very many rows and few columns (a per-voxel head).  Only the weight gradient
    differs from torch's: dW = dY^T X reduces over all N rows into an (out, in) result of a few hundred entries, a shape
    for which the library GEMM runs on a handful of SMs (0.65 ms for 1.7 M x 32 -> 20 in fp32).  Here the rows are cut
    into pieces of 8192, the pieces multiplied as one batched product and the partial results added in a fixed order."""

    @staticmethod
    def forward(ctx, x, weight, bias):
        ctx.save_for_backward(x, weight)
        ctx.has_bias = bias is not None
        return torch.addmm(bias, x, weight.t()) if bias is not None else x @ weight.t()

    @staticmethod
    def backward(ctx, dy):
        x, weight = ctx.saved_tensors
        dy = dy.contiguous()
        dx = dy @ weight if ctx.needs_input_grad[0] else None
        dw = db = None
        if ctx.needs_input_grad[1]:
            n = x.shape[0]
            full = n // _SPLIT_ROWS * _SPLIT_ROWS
            dw = torch.zeros_like(weight)
            if full:
                parts = torch.bmm(dy[:full].view(-1, _SPLIT_ROWS, dy.shape[1]).transpose(1, 2),
                                  x[:full].view(-1, _SPLIT_ROWS, x.shape[1]))
                dw = parts.sum(0)
            if full < n:
                dw = dw + dy[full:].t() @ x[full:]
        if ctx.has_bias and ctx.needs_input_grad[2]:
            db = dy.sum(0)
        return dx, dw, db


class _RowLinear(torch.autograd.Function):
    """y = x.float() W^T + b by the library's own kernels, x read in its own type."""

    @staticmethod
    def forward(ctx, x, weight, bias):
        n, c = x.shape
        o = weight.shape[0]
        w = weight.detach().contiguous()
        y = torch.empty((n, o), dtype=torch.float32, device=x.device)
        p = _lib.ptr
        with torch.cuda.device(x.device):
            _lib.check(_lib.lib().st_linear_fwd(_lib.feat_code(x), p(x), p(w), p(bias), p(y), n, c, o, _lib.stream_ptr(x.device)),
                       "st_linear_fwd")
        ctx.save_for_backward(x, w)
        ctx.has_bias = bias is not None
        return y

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        n, c = x.shape
        o = w.shape[0]
        dy = dy.contiguous()
        L, p, code = _lib.lib(), _lib.ptr, _lib.feat_code(x)
        dx = dw = db = None
        with torch.cuda.device(x.device):
            s = _lib.stream_ptr(x.device)
            if ctx.needs_input_grad[0]:
                dx = torch.empty_like(x)
                _lib.check(L.st_linear_dgrad(code, p(dy), p(w), p(dx), n, c, o, s), "st_linear_dgrad")
            if ctx.needs_input_grad[1] or (ctx.has_bias and ctx.needs_input_grad[2]):
                dw = torch.empty_like(w)
                db = torch.empty(o, dtype=torch.float32, device=w.device) if ctx.has_bias else None
                size = L.st_linear_workspace_bytes(n, c, o)
                ws = torch.empty(size, dtype=torch.uint8, device=w.device)
                _lib.check(L.st_linear_wgrad(code, p(x), p(dy), p(dw), p(db), n, c, o, p(ws), size, s), "st_linear_wgrad")
        return dx, dw, db


class SparseLinear(nn.Linear):
    def float_rows(self, feats):
        """self(feats.float()), the conversion and the product in one pass where the kernels take the widths.  (From one row on:
        with few rows it saves launches, with many the passes over memory.)"""
        w, b = self.weight, self.bias
        if feats.is_cuda and feats.ndim == 2 and feats.shape[0] > 0 and feats.is_contiguous() and w.is_cuda and \
                w.dtype == torch.float32 and (b is None or b.dtype == torch.float32) and feats.data_ptr() % 16 == 0 and \
                feats.dtype in (torch.float32, torch.float16, torch.bfloat16) and \
                _lib.lib().st_linear_supported(_lib.feat_code(feats), w.shape[1], w.shape[0]):
            return _RowLinear.apply(feats, w, b)
        return self._apply_rows(feats.float())

    def _apply_rows(self, feats):
        if feats.is_cuda and feats.ndim == 2 and feats.shape[0] >= _TALL and feats.is_contiguous() and \
                feats.dtype == self.weight.dtype and torch.is_grad_enabled() and self.weight.requires_grad:
            return _TallLinear.apply(feats, self.weight, self.bias)
        return super().forward(feats)

    def forward(self, input):
        if isinstance(input, SparseTensor):
            return input.replace(self._apply_rows(input.F))
        return self._apply_rows(input)


class ReLU(nn.ReLU):
    def forward(self, input):
        if isinstance(input, SparseTensor):
            return input.replace(super().forward(input.F))
        return super().forward(input)
