"""Stored-map form of the convolution: autograd node over the C ABI.

Reference: nn/functional/conv/funcs/implicit_precomputed_gemm.py:233-324
(ConvPrecomputedNeighborGEMM).  Same call signature and return values:

    out = ConvPrecomputedNeighborGEMM.apply(features, weights, neighbor_indices)
    backward -> (d_features, d_weights, None)

The node itself, the three products it launches and what is derived from a map (tile plans, inverse) are native code
(host/conv.cpp, host/geometry.cpp); what a map has derived so far hangs on the map tensor, so layers that share a map
share its plans.
"""
import torch

from sparsetriton_b200 import _lib
from sparsetriton_b200.config import get_row_order

__all__ = ["ConvPrecomputedNeighborGEMM", "inverse_map", "inverse_plan", "map_plan", "map_state", "MapPlan", "prepare_plans"]


def map_state(neighbor_indices, state=None):
    """The native object that holds what is derived from a map, kept on the map tensor (made on first use)."""
    if state is None:
        state = getattr(neighbor_indices, "_st_map", None)
        if state is not None:
            return state
        state = _lib.host().MapState()
    neighbor_indices._st_map = state
    return state


class MapPlan:
    """Tile plan of a (forward or inverse) neighbour map: row order, re-laid map, tile masks
    (st_map_plan).  `ptrs()` are the three pointers the *_planned entry points take."""
    __slots__ = ("order", "tmap", "tmask")

    def __init__(self, order, tmap, tmask):
        self.order, self.tmap, self.tmask = order, tmap, tmask

    def ptrs(self):
        return _lib.ptr(self.order), _lib.ptr(self.tmap), _lib.ptr(self.tmask)


def map_plan(map_tensor):
    """The tile plan of a map, memoised with it.  Rows are sorted by occupied offsets unless
    config.set_row_order(False) or the map is small."""
    return MapPlan(*map_state(map_tensor).plan(map_tensor, get_row_order()))


def inverse_map(neighbor_indices, n_in):
    """inv (n_in, K) with inv[nbr[o,k], k] = o, memoised with the map."""
    state = map_state(neighbor_indices)
    inv = state.inverse(neighbor_indices, n_in)
    if getattr(inv, "_st_map", None) is None:
        inv._st_map = state.inverse_state(neighbor_indices, n_in)
    return inv


def inverse_plan(neighbor_indices, n_in):
    """Tile plan of the inverse map built straight from the forward map (st_map_plan_inverse), or None
    when that form does not apply (more than 32 offsets, row order switched off, small maps)."""
    plan = map_state(neighbor_indices).inverse_plan(neighbor_indices, n_in, get_row_order())
    return None if plan is None else MapPlan(*plan)


_AUX_STREAMS = {}


def _aux_stream(device, like):
    """A second stream per device (and priority of the stream it helps) for work that is independent of what the
    current stream does next."""
    key = (device.index if device.index is not None else torch.cuda.current_device(), like.priority)
    s = _AUX_STREAMS.get(key)
    if s is None:
        s = _AUX_STREAMS[key] = torch.cuda.Stream(device=device, priority=like.priority)
    return s


def prepare_plans(nbr, n_in, backward=True):
    """Builds (and memoises on the map) what the tensor-core products read besides the map: the tile plan, and with
    `backward` the feature gradient's side (nothing more for a symmetric submanifold map, else the inverse map's plan).
    The two plans depend on the map alone and each is a chain of short kernels, so the inverse map's plan is built on
    a second stream beside the forward one; the current stream waits for it before this returns.
    Returns the tensors made, for callers that manage streams."""
    made = []
    fork = None
    if backward and not map_state(nbr).symmetric(nbr, n_in):
        cur = torch.cuda.current_stream(nbr.device)
        aux = _aux_stream(nbr.device, cur)
        aux.wait_stream(cur)
        with torch.cuda.stream(aux):
            inv_plan = inverse_plan(nbr, n_in)
            if inv_plan is None:
                inv = inverse_map(nbr, n_in)
                inv_plan = map_plan(inv)
                made.append(inv)
        fork = (cur, aux)
        made += [inv_plan.order, inv_plan.tmap, inv_plan.tmask]
    plan = map_plan(nbr)
    made += [plan.order, plan.tmap, plan.tmask]
    if fork is not None:
        cur, aux = fork
        cur.wait_stream(aux)
        for t in made:
            if t is not None and t.is_cuda and t.numel() > 0:
                t.record_stream(cur)
    return made


class ConvPrecomputedNeighborGEMM(torch.autograd.Function):
    """The differentiable product over a stored map; `apply` makes the native node."""

    @staticmethod
    def apply(features, weights, neighbor_indices):
        _lib.require_cuda(features, "ConvPrecomputedNeighborGEMM")
        assert weights.shape[1] == features.shape[1], \
            f"weights expect {weights.shape[1]} input channels, features have {features.shape[1]}"
        assert neighbor_indices.shape[1] == weights.shape[0], "neighbor_indices must be (N_out, K)"
        assert neighbor_indices.dtype == torch.int32, "neighbor_indices must be int32"
        return _lib.host().conv(features, weights, neighbor_indices, map_state(neighbor_indices), get_row_order())
