"""What a user of the package has it do, as cases that can be timed.

Four kinds of pass, each through the public entry points and each on coordinates the package has not seen before
(a `SparseTensor` is constructed in every pass, so its table, maps and plans are built in every pass, as they are
for every new batch of a training or serving program):

    layer   one convolution layer: forward alone, or forward and both gradients
    net     the sparse U-Net: inference (running statistics), or a training step with SGD
    maps    hash table, submanifold maps of kernels 3 and 5 and a strided layer's coordinates and map
    pool    a lidar detector's neck: pooling to coarse cells, dense volume, and the gradient of both

Scenes: `surface` (ground sheet, spherical and box shells: indoor and city scans), `lidar` (one sweep of a spinning
sensor over boxes on a plane), `random` (cells drawn uniformly: the densest and the sparsest neighbourhoods).  A case
has one set of scenes, so that every pass of it has the same number of rows in and out; a seed moves them (whole cells
of the coarsest level, away from the grid's border), swaps their axes and samples, and draws all values."""
import math

import torch

import sparsetriton_b200 as st
from sparsetriton_b200.config import ConvAlgo, set_conv_algo, set_coords_dtype
from sparsetriton_b200.distributed import GradientBucket
from sparsetriton_b200.nn import SparseConv3D, SparseConvTransposed3D, SparsePooling, SubMConv3D
from sparsetriton_b200.nn.functional.conv.conv import compute_neighbor_indices
from sparsetriton_b200.nn.functional.conv.kmap import build_out_coords, out_coords_and_map
from sparsetriton_b200.unet import SparseUNet
from sparsetriton_b200.utils.hash import HashTable

DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
ALGOS = {"stored": ConvAlgo.PrecomputedNeighborGEMM, "hashfly": ConvAlgo.ImplicitHashFlyGEMM}
LIDAR_GRID = (1440, 1440, 41)
WIDTHS = (32, 64, 128, 256)


def _layer(name, conv, scene, samples, voxels, grid, cin, cout, k=3, s=1, p=0, dtype="bf16", coords="int32",
           algo="stored", train=True, bias=False):
    return {"name": name, "kind": "layer", "conv": conv, "scene": scene, "samples": samples, "voxels": voxels, "grid": grid,
            "cin": cin, "cout": cout, "k": k, "s": s, "p": p, "dtype": dtype, "coords": coords, "algo": algo,
            "train": train, "bias": bias}


def _net(name, samples, rings, azimuths, train, dtype="bf16"):
    return {"name": name, "kind": "net", "samples": samples, "rings": rings, "azimuths": azimuths, "train": train,
            "dtype": dtype}


def listed():
    return [
        # A layer of a few thousand voxels: what one sees when stepping through a model; launches and host time.
        _layer("subm-4k-fp32-train", "subm", "random", 2, 2048, 64, 16, 32, dtype="fp32", bias=True),
        # A densely filled small grid in single precision, default coordinate type: the shape layers are compared at.
        _layer("subm-200k-fp32-train", "subm", "random", 2, 100_000, 64, 16, 32, dtype="fp32", coords="int16", bias=True),
        # The large downsampling layer of a scan backbone in training: every product direction, half precision.
        _layer("down-1200k-bf16-train", "down", "surface", 4, 300_000, 512, 64, 128, s=2, p=1),
        # The same geometry on one ragged scene with the algorithm that stores no map between calls.
        _layer("down-87k-hashfly-fp16-train", "down", "surface", 1, 87_431, 274, 64, 128, s=2, p=1, dtype="fp16",
               algo="hashfly"),
        # The widest level of a backbone: few voxels, tensor-core work.
        _layer("subm-95k-wide-bf16-train", "subm", "surface", 3, 31_847, 165, 256, 256),
        # A decoder's upsampling layer in serving: every child of every voxel is made.
        _layer("up-40k-bf16-infer", "up", "surface", 2, 20_011, 131, 128, 64, k=2, s=2, train=False, coords="int16"),
        # Coordinate work alone at the scale of a fused multi-sweep map.
        {"name": "maps-2m", "kind": "maps", "scene": "random", "samples": 4, "voxels": 500_000, "grid": 2048,
         "coords": "int32"},
        # One sweep through the network: the latency of a perception stack.
        _net("net-1-infer", 1, 64, 2048, False),
        # A batch of eight sweeps: offline inference.
        _net("net-8-infer", 8, 64, 2048, False),
        # A training step of two sweeps: the share of one of eight GPUs.
        _net("net-2-train", 2, 64, 2048, True),
        # The whole training batch on one GPU.
        _net("net-16-train", 16, 64, 2048, True),
        # Detector neck: maximum over 8-cell columns, then the dense grid that 2-D layers read.
        {"name": "neck-4-bf16-train", "kind": "pool", "samples": 4, "rings": 64, "azimuths": 2048, "channels": 64,
         "cell": 8, "mode": "max", "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["layer"] * 4 + ["net"] * 3 + ["maps", "pool"])
    if kind == "layer":
        conv = rng.choice(["subm", "subm", "down", "up"])
        scene = rng.choice(["random", "surface"])
        samples = rng.randint(1, 4)
        voxels = _log_int(rng, 1500, 40_000 if conv == "up" else 300_000)
        # random cells fill 1 to 35 % of their grid (4 k and 200 k voxels in two 64^3 grids: 1 and 38 %); a surface
        # scene's ground sheet is most of its voxels
        grid = int((voxels / math.exp(rng.uniform(math.log(0.01), math.log(0.35)))) ** (1 / 3)) + 9 if scene == "random" \
            else int(math.sqrt(0.87 * voxels)) + 8
        k, s, p = {"subm": (3, 1, 0), "down": rng.choice([(3, 2, 1), (2, 2, 0)]), "up": (2, 2, 0)}[conv]
        most = 256 if samples * voxels < 100_000 else 128
        cin, cout = (rng.choice([w for w in (16, 32, 64, 96, 128, 256) if w <= most]) for _ in range(2))
        case = _layer("", conv, scene, samples, voxels, grid, cin, cout, k, s, p, rng.choice(["fp32", "fp16", "bf16", "bf16"]),
                      rng.choice(["int16", "int32"]), rng.choice(["stored", "stored", "hashfly"]), rng.random() < 0.7,
                      rng.random() < 0.5)
    elif kind == "net":
        train = rng.random() < 0.5
        case = _net("", _log_int(rng, 1, 16 if train else 8), rng.randint(24, 64), rng.randint(900, 2048), train)
    elif kind == "maps":
        voxels = _log_int(rng, 5000, 500_000)
        case = {"kind": "maps", "scene": rng.choice(["random", "surface"]), "samples": 4, "voxels": voxels,
                "grid": 0, "coords": "int32"}
        case["grid"] = int(voxels ** 0.58) + 8 if case["scene"] == "random" else int(math.sqrt(0.87 * voxels)) + 8
    else:
        case = {"kind": "pool", "samples": rng.randint(1, 4), "rings": rng.randint(24, 64), "azimuths": rng.randint(900, 2048),
                "channels": rng.choice([16, 32, 64, 128]), "cell": rng.choice([6, 8, 10]), "mode": rng.choice(["max", "avg"]),
                "dtype": rng.choice(["fp32", "fp16", "bf16"])}
    case.pop("name", None)
    return case


# ------------------------------------------------------------------------------------------------- scenes
def _margin(grid):
    """Cells left free at every border of a cubic grid."""
    return 2 * (grid // 64) + 4


def _moved(cells, gen, samples, steps, unit, turn_z):
    """The scenes of `cells` (N, 4) somewhere else: every sample shifted by up to `steps` times `unit` cells along each axis
    (along z where `turn_z`), its x and y swapped or not, the samples in another order; rows in cell order."""
    shift = torch.randint(-steps, steps + 1, (samples, 3), generator=gen, device="cuda") * unit
    if not turn_z:
        shift[:, 2] = 0
    swap = torch.rand(samples, generator=gen, device="cuda") < 0.5
    place = torch.randperm(samples, generator=gen, device="cuda")
    b, xyz = cells[:, 0], cells[:, 1:]
    xyz = torch.where(swap[b][:, None], xyz[:, [1, 0, 2]], xyz) + shift[b]
    key = (place[b] << 48 | xyz[:, 0] << 32 | xyz[:, 1] << 16 | xyz[:, 2]).sort().values
    return torch.stack([key >> 48, key >> 32 & 0xFFFF, key >> 16 & 0xFFFF, key & 0xFFFF], 1)


def _random_cells(gen, samples, voxels, grid):
    """`voxels` distinct cells of each of `samples` cubic grids; rows (b, x, y, z)."""
    m = _margin(grid)
    side = grid - 2 * m
    cells = side ** 3
    rows = []
    for b in range(samples):
        if cells <= 1 << 24:
            flat = torch.randperm(cells, generator=gen, device="cuda")[:voxels]
        else:
            flat = torch.unique(torch.randint(0, cells, (int(voxels * 1.1) + 64,), generator=gen, device="cuda"))
            flat = flat[torch.randperm(flat.shape[0], generator=gen, device="cuda")[:voxels]]
        rows.append(torch.stack([torch.full_like(flat, b)] + [v + m for v in (flat // (side * side), flat // side % side, flat % side)], 1))
    return torch.cat(rows)


def _shell(kind, centre, size, grid):
    """Cells (x*grid + y)*grid + z of a one-voxel spherical shell or of the faces of a box, clipped to the grid within its
    margin."""
    m = _margin(grid)
    size = [size[0]] * 3 if kind == "sphere" else size
    lo = [max(m, int(c - r) - 1) for c, r in zip(centre, size)]
    hi = [min(grid - 1 - m, int(c + r) + 1) for c, r in zip(centre, size)]
    if any(a > b for a, b in zip(lo, hi)):
        return torch.empty(0, dtype=torch.int64, device="cuda")
    x, y, z = (torch.arange(a, b + 1, device="cuda") for a, b in zip(lo, hi))
    x, y, z = x[:, None, None], y[None, :, None], z[None, None, :]
    if kind == "sphere":
        d = ((x - centre[0]) ** 2 + (y - centre[1]) ** 2 + (z - centre[2]) ** 2).float().sqrt()
        hit = (d - size[0]).abs() < 0.5
    else:
        dx, dy, dz = ((v - int(c)).abs() - int(r) for v, c, r in zip((x, y, z), centre, size))
        hit = torch.maximum(torch.maximum(dx, dy), dz) == 0
    return ((x * grid + y) * grid + z).expand(hit.shape)[hit]


def _surface_cells(gen, samples, voxels, grid):
    """A ground sheet z = 20 + {-1, 0, 1} over the whole grid, then whole spherical and box shells in turn, the last one
    cut, to `voxels` cells a sample (the sheet alone is about 80 % of them)."""
    rows, m = [], _margin(grid)
    side = torch.arange(m, grid - m, device="cuda")
    cols = (side[:, None] * grid + side).reshape(-1)
    for b in range(samples):
        flat = cols * grid + (20 + torch.randint(-1, 2, cols.shape, generator=gen, device="cuda")).clamp(max=grid - 1 - m)
        flat = flat[:voxels]
        for turn in range(400):
            if flat.shape[0] >= voxels:
                break
            r = torch.rand(6, generator=gen, device="cuda").tolist()
            scale = grid / 512
            kind = "sphere" if turn % 2 == 0 else "box"
            size = [(r[3] * 100 + 20) * scale] if kind == "sphere" else [(v * 55 + 5) * scale for v in r[3:]]
            new = _shell(kind, [v * grid for v in r[:3]], size, grid)
            new = new[~torch.isin(new, flat)]
            flat = torch.cat([flat, new[: voxels - flat.shape[0]]])
        rows.append(torch.stack([torch.full_like(flat, b), flat // (grid * grid), flat // grid % grid, flat % grid], 1))
    return torch.cat(rows)


def _lidar_cells(gen, samples, rings, azimuths):
    """Cells hit by one sweep a sample: `rings` elevation rings x `azimuths` headings from the grid's centre, each ray
    ending at the nearest of the ground plane and 40 boxes; duplicates merged."""
    gx, gy, gz = LIDAR_GRID
    origin = torch.tensor([gx / 2.0, gy / 2.0, 38.0], device="cuda")
    el = -torch.atan((origin[2] - 2.5) / torch.linspace(250.0, 680.0, rings, device="cuda"))
    az = torch.arange(azimuths, device="cuda") * (2 * math.pi / azimuths)
    ce, se = torch.cos(el)[:, None], torch.sin(el)[:, None]
    d = torch.stack([ce * torch.cos(az), ce * torch.sin(az), se.expand(-1, azimuths)], -1).reshape(-1, 3)
    inv = 1.0 / torch.where(d.abs() < 1e-9, torch.full_like(d, 1e-9), d)
    rows = []
    for b in range(samples):
        r = torch.rand(40, 5, generator=gen, device="cuda")
        centre, half, height = r[:, :2] * 1240 + 100, r[:, 2:4] * 36 + 4, r[:, 4] * 26 + 4
        lo = torch.cat([centre - half, torch.full_like(height, 2.0)[:, None]], 1)
        hi = torch.cat([centre + half, 2.0 + height[:, None]], 1)
        t1, t2 = (lo - origin) * inv[:, None], (hi - origin) * inv[:, None]
        near, far = torch.minimum(t1, t2).amax(2), torch.maximum(t1, t2).amin(2)
        t = torch.where((near <= far) & (near > 0), near, math.inf).amin(1)
        t = torch.minimum(t, torch.where(d[:, 2] < -1e-6, (2.5 - origin[2]) / d[:, 2], math.inf))
        q = torch.floor(origin + d * (t[:, None] + 1e-3)).to(torch.int64)
        ok = torch.isfinite(t) & (q >= 0).all(1) & (q < torch.tensor(LIDAR_GRID, device="cuda")).all(1)
        q = q[ok]
        flat = torch.unique((q[:, 0] * gy + q[:, 1]) * gz + q[:, 2])
        rows.append(torch.stack([torch.full_like(flat, b), flat // (gy * gz), flat // gz % gy, flat % gz], 1))
    return torch.cat(rows)


def _cells(case, gen):
    scenes = torch.Generator(device="cuda").manual_seed(7)
    if case["kind"] in ("net", "pool"):
        cells = _lidar_cells(scenes, case["samples"], case["rings"], case["azimuths"])
        return _moved(cells, gen, case["samples"], 4, 8, False)
    make = _random_cells if case["scene"] == "random" else _surface_cells
    cells = _moved(make(scenes, case["samples"], case["voxels"], case["grid"]), gen, case["samples"],
                   _margin(case["grid"]) // 2 - 1, 2, True)
    if case["kind"] == "maps" and case["scene"] == "random":       # points as they come, in no order
        cells = cells[torch.randperm(cells.shape[0], generator=gen, device="cuda")]
    return cells


def _tensor(s, feats):
    return st.SparseTensor(feats, s["coords"], spatial_shape=s["shape"], batch_size=s["samples"])


# ------------------------------------------------------------------------------------------------- prepare
def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    torch.manual_seed(seed)
    set_conv_algo(ALGOS[case.get("algo", "stored")])
    coord_dtype = torch.int16 if case.get("coords") == "int16" else torch.int32
    set_coords_dtype(coord_dtype)
    s = {"case": case, "samples": case["samples"]}

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device="cuda").to(dtype)

    if case["kind"] == "maps":
        s["coords"] = _cells(case, gen).to(coord_dtype)
        s["shape"] = (case["grid"],) * 3
        return s
    dtype = DTYPES[case["dtype"]]
    if case["kind"] == "layer":
        s["coords"] = _cells(case, gen).to(coord_dtype)
        s["shape"] = (case["grid"],) * 3
        s["feats"] = normal(s["coords"].shape[0], case["cin"])
        if case["conv"] == "subm":
            s["layer"] = SubMConv3D(case["cin"], case["cout"], case["k"], bias=case["bias"]).cuda()
        else:
            make = SparseConv3D if case["conv"] == "down" else SparseConvTransposed3D
            s["layer"] = make(case["cin"], case["cout"], case["k"], stride=case["s"], padding=case["p"],
                              bias=case["bias"]).cuda()
        if case["train"]:
            s["feats"].requires_grad_(True)
            if case["conv"] == "subm":
                rows = s["coords"].shape[0]
            else:
                with torch.no_grad():
                    rows = s["layer"](_tensor(s, s["feats"].detach())).F.shape[0]
            s["dy"] = normal(rows, case["cout"])
        return s
    s["coords"] = _cells(case, gen).to(coord_dtype)
    s["shape"] = LIDAR_GRID
    n = s["coords"].shape[0]
    if case["kind"] == "pool":
        s["feats"] = normal(n, case["channels"]).requires_grad_(True)
        s["layer"] = SparsePooling(case["cell"], mode=case["mode"], stride=case["cell"], padding=case["cell"] // 2)
        with torch.no_grad():
            s["dvol"] = normal(*s["layer"](_tensor(s, s["feats"].detach())).dense().shape)
        return s
    # the network's inputs: normalised position and an intensity
    position = s["coords"][:, 1:].float() / torch.tensor([float(v) for v in LIDAR_GRID], device="cuda")
    s["feats"] = torch.cat([position, torch.rand(n, 1, generator=gen, device="cuda")], 1).to(dtype)
    net = s["net"] = SparseUNet(in_channels=4, widths=WIDTHS, num_classes=20).cuda()
    norms = [m for m in net.modules() if hasattr(m, "running_mean")]
    flat = s["running"] = torch.empty(2 * sum(m.num_features for m in norms), device="cuda")
    at = 0
    for m in norms:                            # running statistics as views of one buffer, of plausible values
        for b, mean, spread in ((m.running_mean, 0.0, 0.1), (m.running_var, 0.3, 0.1)):
            v = flat[at:at + m.num_features]
            v.copy_(mean + spread * (torch.rand(m.num_features, generator=gen, device="cuda") * 2 - 1))
            setattr(m, "running_mean" if b is m.running_mean else "running_var", v)
            at += m.num_features
    net.train(case["train"])
    if case["train"]:
        # classes by height and distance, one voxel in ten labelled otherwise
        far = (s["coords"][:, 1:3].float() - 720).norm(dim=1)
        labels = (s["coords"][:, 3] // 6).clamp(max=4) * 4 + (far / 180).long().clamp(max=3)
        noise = torch.randint(0, 200, (n,), generator=gen, device="cuda")
        s["labels"] = torch.where(noise < 20, noise, labels.long())
        # parameters and gradients each in one flat buffer, as data-parallel training keeps them
        flat = s["parameters"] = torch.cat([p.detach().reshape(-1) for p in net.parameters()])
        at = 0
        for p in net.parameters():
            p.data = flat[at:at + p.numel()].view_as(p)
            at += p.numel()
        s["bucket"] = GradientBucket(net.parameters())
        s["sgd"] = torch.optim.SGD(net.parameters(), lr=0.01, momentum=0.9)
    return s


# ------------------------------------------------------------------------------------------------- run
def run(s):
    case = s["case"]
    if case["kind"] == "layer":
        layer, x = s["layer"], s["feats"]
        if not case["train"]:
            with torch.no_grad():
                out = layer(_tensor(s, x))
            return {"coords": out.C, "y": out.F}
        out = layer(_tensor(s, x))
        grads = torch.autograd.grad(out.F, [x] + list(layer.parameters()), s["dy"])
        return {"coords": out.C, "y": out.F.detach(), "grads": grads}
    if case["kind"] == "maps":
        coords, shape = s["coords"], s["shape"]
        table = HashTable(2 * coords.shape[0], device=coords.device)
        table.insert(coords)
        maps = []
        for k in (3, 5):
            _, _, offsets = build_out_coords(coords, shape, k, 1, 1, k // 2, submanifold=True)
            maps.append(compute_neighbor_indices(table, coords, offsets, shape, 1, queries_are_table_rows=True))
        down, _, _, down_map = out_coords_and_map(coords, shape, 3, 2, 1, 1, False, s["samples"])
        return {"rows": table.query(coords), "subm": maps, "down": down, "down_map": down_map}
    if case["kind"] == "pool":
        x = s["feats"]
        volume = s["layer"](_tensor(s, x)).dense()
        (dx,) = torch.autograd.grad(volume, [x], s["dvol"])
        return {"volume": volume.detach(), "dx": dx}
    net = s["net"]
    if not case["train"]:
        with torch.no_grad():
            return net(_tensor(s, s["feats"])).F
    out = net(_tensor(s, s["feats"])).F
    loss = torch.nn.functional.cross_entropy(out, s["labels"], reduction="none").sum() / out.shape[0]
    s["bucket"].zero()
    loss.backward()
    grads = s["bucket"].all_reduce()
    s["sgd"].step()
    return {"loss": loss.detach(), "logits": out.detach(), "grads": grads, "running": s["running"],
            "parameters": s["parameters"]}


# ------------------------------------------------------------------------------------------------- work
# Shape of the scenes, counted once: neighbours a voxel has under a kernel, output rows and pairs of a strided layer
# per input voxel.  Random cells follow from how full their grid is.
_SURFACE = {"subm3": 7.5, "subm5": 25.0, "down3": (0.69, 3.7), "down2": (0.42, 1.0), "up2": (7.0, 8.0)}
# The U-Net's levels on a lidar sweep: voxels per input voxel, neighbours of a voxel under kernel 3.
_LIDAR = ((1.0, 2.9), (0.70, 3.9), (0.37, 5.4), (0.15, 8.7))
_LIDAR_HITS = 0.79                             # distinct cells per ray


def _strided(case, k):
    """(output rows, pairs) per input voxel of a stride-2 layer."""
    if case["scene"] == "surface":
        return _SURFACE["down%d" % k]
    fill = case["voxels"] / case["grid"] ** 3
    pairs = (k / 2.0) ** 3
    return pairs * (1 - (1 - fill) ** (k ** 3)) / (fill * k ** 3), pairs


def _neighbours(case, k):
    return _SURFACE["subm%d" % k] if case["scene"] == "surface" else 1 + case["voxels"] / case["grid"] ** 3 * (k ** 3 - 1)


def _conv_flops(pairs, cin, cout, train):
    return 2.0 * pairs * cin * cout * (3 if train else 1)


def work(case):
    es = 4 if case.get("dtype") == "fp32" else 2
    cs = 8 if case.get("coords") == "int16" else 16
    if case["kind"] == "layer":
        n, k, cin, cout = case["samples"] * case["voxels"], case["k"], case["cin"], case["cout"]
        if case["conv"] == "subm":
            rows, pairs = 1.0, _neighbours(case, k)
        elif case["conv"] == "down":
            rows, pairs = _strided(case, k)
        else:
            rows, pairs = _SURFACE["up2"]
        n_out = n * rows
        weights = k ** 3 * cin * cout + (cout if case["bias"] else 0)
        out_cells = 0 if case["conv"] == "subm" else cs * n_out
        once = cs * n + out_cells + es * (n * cin + n_out * cout) + 4 * weights
        if case["train"]:                      # dY in, dX and the weights' gradients out
            once += es * (n_out * cout + n * cin) + 4 * weights
        return {"bytes": once, "flops": _conv_flops(n * pairs, cin, cout, case["train"])}
    if case["kind"] == "maps":
        n = case["samples"] * case["voxels"]
        rows, _ = _strided(case, 3)
        return {"bytes": 16 * n + 4 * n + 4 * n * (27 + 125) + n * rows * (16 + 4 * 27), "flops": 0}
    n = case["samples"] * case["rings"] * case["azimuths"] * _LIDAR_HITS
    if case["kind"] == "pool":
        a = [g // case["cell"] + 1 for g in LIDAR_GRID]
        volume = case["samples"] * a[0] * a[1] * a[2] * case["channels"]
        return {"bytes": 16 * n + es * (2 * n * case["channels"] + 2 * volume), "flops": 0}
    # every layer's features are written once and read once (a layer needs all rows of the one before it), and with
    # gradients once more each way
    passes = 3 if case["train"] else 1
    flops, values, c = 0.0, 0.0, 4
    for i, w in enumerate(WIDTHS):
        rows, near = _LIDAR[i][0] * n, _LIDAR[i][1]
        enc = c if i == 0 else w
        flops += _conv_flops(rows * near, enc, w, False) + _conv_flops(rows * near, w, w, False)
        values += 2 * rows * w
        if i + 1 < len(WIDTHS):                # down-convolution, its mirror image, and the decoder's block
            flops += 2 * _conv_flops(rows, w, WIDTHS[i + 1], False)
            flops += _conv_flops(rows * near, 2 * w, w, False) + _conv_flops(rows * near, w, w, False)
            values += 3 * rows * w + _LIDAR[i + 1][0] * n * WIDTHS[i + 1]
    flops += 2.0 * n * WIDTHS[0] * 20
    return {"bytes": 16 * n + es * n * 4 + 4 * n * 20 + 2 * es * values * passes, "flops": flops * passes}


def tolerance(case):
    if case["kind"] == "maps":
        return "exact"
    if case["kind"] == "pool":                 # one rounding to the features' type
        return {"rel": {"fp32": 1e-6, "fp16": 1e-3, "bf16": 5e-3}[case["dtype"]]}
    if case["kind"] == "layer":                # fp32 layers multiply in tf32
        return {"rel": {"fp32": 1e-3, "fp16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
    # a network of 20 layers in bf16; gradients jump where a ReLU's input changes sign
    return {"rel": 0.03, "max": 0.9} if case["train"] else {"rel": 0.02, "max": 0.8}
