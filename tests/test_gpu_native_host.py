"""The native host side and the kernels behind it at the sizes where they can go wrong: edges of tiles and rings, remainders,
the smallest and largest of a range.  References are plain PyTorch in fp32, or the slower form of the same entry point."""
import ctypes

import pytest
import torch

from sparsetriton_b200 import _lib, synthetic
from sparsetriton_b200.config import get_coords_dtype, set_coords_dtype
from sparsetriton_b200.nn.functional.conv.conv import compute_neighbor_indices
from sparsetriton_b200.nn.functional.conv.kmap import build_out_coords
from sparsetriton_b200.tensor import SparseTensor
from sparsetriton_b200.utils.hash import HashTable

pytestmark = pytest.mark.gpu
TOL = {torch.float32: 2e-3, torch.bfloat16: 1e-2, torch.float16: 1e-2}


def _rel(got, want):
    got, want = got.double(), want.double()
    return float((got - want).norm() / want.norm().clamp(min=1e-30))


def _map(n_rows, n_src, K, density, seed):
    g = torch.Generator().manual_seed(seed)
    m = torch.randint(0, n_src, (n_rows, K), generator=g, dtype=torch.int32)
    m[torch.rand(n_rows, K, generator=g) >= density] = -1
    # at most one output per (input, offset), as in a convolution
    for k in range(K):
        seen = {}
        col = m[:, k].tolist()
        for o, i in enumerate(col):
            if i >= 0 and i in seen:
                m[o, k] = -1
            seen[i] = o
    return m


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("n_rows,n_src,K,cin,cout,density", [
    (1, 1, 1, 16, 16, 1.0), (127, 40, 27, 32, 64, 0.2), (128, 128, 8, 64, 32, 0.5), (129, 200, 27, 96, 48, 0.3),
    (900, 700, 27, 256, 256, 0.4), (700, 900, 33, 48, 80, 0.1), (500, 500, 125, 128, 16, 0.05), (20000, 17000, 27, 64, 128, 0.15),
    (300, 300, 27, 144, 240, 0.0)])
def test_products_at_the_edges(cuda_device, dtype, n_rows, n_src, K, cin, cout, density):
    H = _lib.host()
    nbr = _map(n_rows, n_src, K, density, n_rows + K)
    g = torch.Generator().manual_seed(cin)
    x, w, dy = (torch.randn(s, generator=g).to(cuda_device, dtype) for s in ((n_src, cin), (K, cin, cout), (n_rows, cout)))
    x.requires_grad_(True)
    w.requires_grad_(True)
    nbr = nbr.to(cuda_device)
    y = H.conv(x, w, nbr, H.MapState(), True)
    dx, dw = torch.autograd.grad(y, [x, w], dy)
    torch.cuda.synchronize()
    assert _lib.device_status(cuda_device)[0] == 0
    xf, wf, dyf, have = x.detach().float(), w.detach().float(), dy.float(), nbr >= 0
    want_y, want_dx, want_dw = torch.zeros(n_rows, cout, device=cuda_device), torch.zeros_like(xf), torch.zeros_like(wf)
    for k in range(K):
        o = have[:, k].nonzero()[:, 0]
        i = nbr[o, k].long()
        want_y[o] += xf[i] @ wf[k]
        want_dx.index_add_(0, i, dyf[o] @ wf[k].t())
        want_dw[k] = xf[i].t() @ dyf[o]
    for got, want in ((y, want_y), (dx, want_dx), (dw, want_dw)):
        assert got.dtype == dtype
        assert _rel(got, want) < TOL[dtype] if want.abs().sum() > 0 else float(got.abs().sum()) == 0


def test_fp32_weights_take_fp32_sums(cuda_device):
    """16-bit features with fp32 master weights: dW arrives in fp32, unrounded."""
    H = _lib.host()
    nbr = _map(600, 500, 27, 0.3, 5).to(cuda_device)
    x = torch.randn(500, 32, device=cuda_device).bfloat16()
    w = torch.randn(27, 32, 64, device=cuda_device, requires_grad=True)
    dy = torch.randn(600, 64, device=cuda_device).bfloat16()
    (dw,) = torch.autograd.grad(H.conv(x, w, nbr, H.MapState(), True), [w], dy)
    want = torch.zeros_like(w)
    for k in range(27):
        o = (nbr[:, k] >= 0).nonzero()[:, 0]
        want[k] = x[nbr[o, k].long()].float().t() @ dy[o].float()
    assert dw.dtype == torch.float32 and _rel(dw, want) < 1e-5


@pytest.mark.parametrize("k,d,n,grid,dtype", [(3, 1, 230_000, 64, torch.int32), (3, 2, 230_000, 97, torch.int16),
                                              (5, 1, 60_000, 40, torch.int32), (7, 1, 20_000, 33, torch.int32)])
def test_map_by_columns_equals_full_probing(cuda_device, k, d, n, grid, dtype):
    """From half a million probes on the symmetric map goes through the column filter; duplicates, negative cells and cells outside
    the grid included."""
    coords = synthetic.random_cells(n, 2, grid, seed=k)
    coords[5] = coords[n // 2]
    coords[7, 3] = -1
    coords[9, 1] = grid + 40
    coords = coords.to(cuda_device, dtype)
    assert _lib.lib().st_map_build_symmetric_workspace_bytes(n, k ** 3) > 0
    table = HashTable(1 << 20, device=cuda_device)
    table.insert(coords)
    _, _, off = build_out_coords(coords, (grid,) * 3, k, 1, d, (k - 1) * d // 2, submanifold=True)
    want = compute_neighbor_indices(table, coords, off, (grid,) * 3, 1)
    got = compute_neighbor_indices(table, coords, off, (grid,) * 3, 1, queries_are_table_rows=True)
    assert torch.equal(got, want)


@pytest.mark.parametrize("n", [1, 255, 1024, 1025, 700_001])
@pytest.mark.parametrize("dtype", [torch.int16, torch.int32])
def test_extent(cuda_device, n, dtype):
    c = torch.randint(-500, 30_000, (n, 4), dtype=dtype, device=cuda_device)
    for _ in range(3):                                        # the scratch has to be left as it was found
        assert _lib.host().extent(c) == c.max(dim=0).values.tolist()


@pytest.mark.parametrize("n,samples,order", [(1, 1, "sorted"), (2047, 3, "sorted"), (2049, 70, "mixed"), (300_000, 1500, "mixed")])
def test_batch_info(cuda_device, n, samples, order):
    b = torch.randint(-1, samples + 1, (n,), device=cuda_device)
    b = b.sort().values if order == "sorted" else b
    coords = torch.stack([b] + [torch.zeros_like(b)] * 3, 1).int()
    ids, inv, status, first = _lib.host().batch_info(coords, samples)
    ok = (b >= 0) & (b < samples)
    counts = torch.bincount(b[ok], minlength=samples)
    want_first = torch.full((samples,), n, device=cuda_device).scatter_reduce(0, b[ok], ok.nonzero()[:, 0], "amin")
    assert torch.equal(ids.long(), b) and int(status) == 0
    assert torch.equal(inv, 1.0 / counts.clamp(min=1).float())
    assert torch.equal(first.long(), torch.where(counts > 0, want_first, -1))


@pytest.mark.parametrize("C", [8, 20, 64])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
def test_batch_norm_over_running_statistics(cuda_device, C, dtype):
    g = torch.Generator().manual_seed(C)
    x, w, b, m = (torch.randn(s, generator=g).to(cuda_device) for s in ((333, C), (C,), (C,), (C,)))
    v = torch.rand(C, generator=g).to(cuda_device) + 0.1
    x = x.to(dtype).requires_grad_(True)
    w.requires_grad_(True)
    y = _lib.host().batch_norm_running(x, w, b, m, v, 1e-5, True)
    xr = x.detach().float().requires_grad_(True)
    wr = w.detach().clone().requires_grad_(True)
    want = torch.relu((xr - m) * torch.rsqrt(v + 1e-5) * wr + b)
    dy = torch.randn_like(want).to(dtype)
    got_g, want_g = torch.autograd.grad(y, [x, w], dy), torch.autograd.grad(want, [xr, wr], dy.float())
    for a, c in zip((y,) + got_g, (want,) + want_g):
        assert _rel(a, c) < (1e-5 if dtype == torch.float32 else 1e-2)


@pytest.mark.parametrize("mode", ["max", "avg"])
@pytest.mark.parametrize("C", [5, 8, 64])
@pytest.mark.parametrize("grid,n", [(9, 300), (40, 30_000)])
def test_pooling_forward_and_gradient(cuda_device, mode, C, grid, n):
    """Whole 16-byte rows (C = 8, 64) and others (C = 5) against a reduction by cell."""
    from sparsetriton_b200.nn.functional.spatial import sparse_pooling
    before = get_coords_dtype()
    set_coords_dtype(torch.int32)
    try:
        c = synthetic.random_cells(n, 2, grid, seed=n).to(cuda_device)
        x = (torch.randperm(n * C, device=cuda_device).float() * 2.0 ** -20 - 0.5).view(n, C)      # no ties under a maximum
        x.requires_grad_(True)
        out = sparse_pooling(SparseTensor(x, c, (grid,) * 3, 2), 4, 2, 4, mode)
        key = ((c[:, 0].long() * 64 + c[:, 1] // 4) * 64 + c[:, 2] // 4) * 64 + c[:, 3] // 4
        cells, inv = torch.unique(key, return_inverse=True)
        want = torch.zeros(cells.shape[0], C, device=cuda_device).scatter_reduce(
            0, inv[:, None].expand(-1, C), x, "amax" if mode == "max" else "mean", include_self=False)
        dy = torch.randn_like(want)
        assert torch.allclose(out.F, want, atol=1e-6)
        assert torch.allclose(torch.autograd.grad(out.F, x, dy)[0], torch.autograd.grad(want, x, dy)[0], atol=1e-6)
    finally:
        set_coords_dtype(before)


@pytest.mark.parametrize("n_rows,n_src,K", [(1, 1, 1), (127, 90, 8), (128, 300, 9), (129, 129, 16), (5000, 4000, 27),
                                            (40001, 30000, 32), (70000, 70001, 27), (1100000, 5000, 8)])
def test_balanced_plans(cuda_device, n_rows, n_src, K):
    """The plans that the products walk are those of st_map_plan(sorted) with whole tiles moved: most offsets first."""
    L, dev, p = _lib.lib(), cuda_device, _lib.ptr
    g = torch.Generator().manual_seed(n_rows + K)
    nbr = torch.randint(0, n_src, (n_rows, K), generator=g, dtype=torch.int32)
    nbr[torch.rand(n_rows, K, generator=g) > torch.rand(n_rows, 1, generator=g)] = -1
    nbr = nbr.to(dev)
    # a map that an inverse exists of: no source twice under one offset
    fwd = torch.full((n_rows, K), -1, dtype=torch.int32, device=dev)
    for k in range(K):
        m = min(n_rows, n_src) // (1 + k % 5)
        fwd[torch.randperm(n_rows, generator=g)[:m].to(dev), k] = torch.randperm(n_src, generator=g)[:m].to(dev, torch.int32)
    inv = torch.empty((n_src, K), dtype=torch.int32, device=dev)
    with torch.cuda.device(dev):
        s = _lib.stream_ptr()
        _lib.check(L.st_map_invert(p(fwd), n_rows, K, n_src, p(inv), s), "invert")
        for of, n, call in ((nbr, n_rows, lambda b, w: L.st_map_plan_balanced(p(nbr), n_rows, K, *b, p(w), w.numel(), s)),
                            (inv, n_src, lambda b, w: L.st_map_plan_inverse_balanced(p(fwd), n_rows, K, n_src, *b, p(w), w.numel(), s))):
            tiles = (n + 127) // 128
            plain, got = [[torch.full((m,), -7, dtype=torch.int32, device=dev) for m in (n, tiles * K * 128, tiles)] for _ in "ab"]
            ws = _lib.workspace(L.st_map_plan_workspace_bytes(n, K), dev)
            _lib.check(L.st_map_plan(p(of), n, K, 1, *[p(t) for t in plain], p(ws), ws.numel(), s), "plan")
            ws = _lib.workspace(L.st_map_plan_balanced_workspace_bytes(n, K), dev)
            _lib.check(call([p(t) for t in got], ws), "balanced")
            bits = (plain[2][:, None] >> torch.arange(K, device=dev)) & 1
            full = n // 128
            place = torch.arange(tiles)
            place[:full] = torch.sort(-bits[:full].sum(1).clamp(max=31).cpu(), stable=True).indices
            place = place.to(dev)
            assert torch.equal(got[2], plain[2][place])
            assert torch.equal(got[0][:full * 128].view(-1, 128), plain[0][:full * 128].view(-1, 128)[place[:full]])
            assert torch.equal(got[0][full * 128:], plain[0][full * 128:])
            lines, want = got[1].view(tiles, K, 128), plain[1].view(tiles, K, 128)[place]
            occupied = (bits[place] > 0)[:, :, None]
            assert torch.equal(lines, torch.where(occupied, want, torch.full_like(want, -7)))


@pytest.mark.parametrize("ks,n", [(3, 1500000), (5, 200000), (7, 60000)])
def test_filtered_map_is_the_probed_map(cuda_device, ks, n):
    """st_map_build_symmetric_ws with the column filter's workspace and without it, over tables whose chains differ from one
    build to the next (rows claim their slots in any order)."""
    L, dev, p = _lib.lib(), cuda_device, _lib.ptr
    g = torch.Generator(device=dev).manual_seed(ks)
    flat = torch.randint(0, 16 * 400 * 400, (n // 4,), generator=g, device=dev)              # short columns: surfaces
    z0 = torch.randint(0, 37, (n // 4,), generator=g, device=dev)
    c = torch.stack([flat // 160000, flat // 400 % 400, flat % 400, z0], 1).repeat_interleave(4, 0)
    c[:, 3] += torch.arange(4, device=dev).repeat(n // 4)
    c = torch.unique(c, dim=0).int().contiguous()
    n = c.shape[0]
    r, K = ks // 2, ks ** 3
    offs = [v for x in range(r, -r - 1, -1) for y in range(r, -r - 1, -1) for z in range(r, -r - 1, -1) for v in (x, y, z)]
    off, shape = (ctypes.c_int32 * (3 * K))(*offs), (ctypes.c_int32 * 3)(400, 400, 41)
    need = L.st_map_build_symmetric_workspace_bytes(n, K)
    assert need > 0
    ws = torch.empty(need, dtype=torch.uint8, device=dev)
    cap = 1 << (2 * n - 1).bit_length()
    keys, vals = torch.empty(cap, dtype=torch.int64, device=dev), torch.empty(cap, dtype=torch.int32, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    a, b = (torch.empty((n, K), dtype=torch.int32, device=dev) for _ in "ab")
    code = _lib.coord_code(c)
    with torch.cuda.device(dev):
        s = _lib.stream_ptr()
        for _ in range(8):
            _lib.check(L.st_hash_clear(p(keys), p(vals), cap, s), "clear")
            _lib.check(L.st_hash_build(p(c), n, code, p(keys), p(vals), cap, p(status), s), "build")
            for out, w in ((a, ws), (b, None)):
                _lib.check(L.st_map_build_symmetric_ws(p(c), n, code, off, K, shape, p(keys), p(vals), cap, p(out), None,
                                                       p(w) if w is not None else None, need if w is not None else 0, s), "map")
            assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("n,C,O,bias", [(1, 16, 4, True), (63, 32, 20, True), (65, 64, 64, False), (5000, 32, 20, True),
                                        (70001, 16, 64, True), (300000, 64, 12, False)])
def test_row_linear(cuda_device, dtype, n, C, O, bias):
    from sparsetriton_b200.nn.modules import SparseLinear
    torch.manual_seed(n)
    lin = SparseLinear(C, O, bias=bias).to(cuda_device)
    x = torch.randn(n, C, device=cuda_device).to(dtype).requires_grad_(True)
    y = lin.float_rows(x)
    assert y.dtype == torch.float32
    dy = torch.randn(n, O, device=cuda_device)
    got = torch.autograd.grad(y, [x] + list(lin.parameters()), dy)
    xd, w = x.detach().double(), lin.weight.detach().double()
    want = [dy.double() @ w, dy.double().t() @ xd] + ([dy.double().sum(0)] if bias else [])
    assert _rel(y, xd @ w.t() + (lin.bias.detach().double() if bias else 0)) < 1e-6
    assert got[0].dtype == dtype and _rel(got[0], want[0]) < (1e-6 if dtype == torch.float32 else 3e-3)
    for a, b in zip(got[1:], want[1:]):
        assert _rel(a, b) < 1e-5
