"""Performance cases: the work that a user of this framework has it do.

Every case goes through the public entry points (GeometryTensorQO.ProjectRays and its autograd
adjoint, ComputeImage, SampleVolumeIndirect, ProposalSampler, recon.node_errors, the grid-sample
operators, SiddonProject, optim.Adam). Model shapes are the repository's configurations C1 (rank 8,
depth-2 octree, 8 -> 32 -> 1), C2 (rank 16, depth 4, 16 -> 64 -> 64 -> 1) and C5 (rank 24 on an
adaptive depth-6 octree of a thin slab), with 17^2 planes and parallel-beam rays.

  listed()            the cases          draw(rng)       one more case of the same ranges
  prepare(case, seed) inputs and model   run(state)      one pass, its outputs
  work(case)          bytes and operations that one pass cannot do without
  exact(case, seed)   the outputs in 64 bits from plain torch (none of this package's code)
"""

from __future__ import annotations

import math

import numpy as np
import torch

DEV = "cuda"


# ----------------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------------
def _model(channels, hidden, depth, grid=17, leaves=0, op="add"):
    return {"channels": channels, "hidden": hidden, "depth": depth, "grid": grid, "leaves": leaves, "op": op}


def listed():
    c1, c2 = _model(8, "32", 2), _model(16, "64,64", 4)
    c5 = _model(24, "64,64", 6, leaves=4096)
    return [
        # a user looks at a few detector rows of a small field while it trains: the smallest call,
        # bound by launches and host work
        {"name": "preview_fp32", "kind": "project", **c1, "rays": 256, "samples": 32, "precision": "fp32",
         "grad": False},
        # one training step (projection, loss, adjoint) of the small configuration in the plain form
        {"name": "train_fp32_small", "kind": "project", **c1, "rays": 4096, "samples": 32, "precision": "fp32",
         "grad": True},
        # one training step of the standard configuration in the plain FP32 form (the parity path
        # and what "seconds to a PSNR" is compared with)
        {"name": "train_fp32", "kind": "project", **c2, "rays": 16384, "samples": 24, "precision": "fp32",
         "grad": True},
        # the same step in the BF16 tensor-core form that training uses by default
        {"name": "train_bf16", "kind": "project", **c2, "rays": 16384, "samples": 24, "precision": "bf16",
         "grad": True},
        # one training step of the largest configuration: adaptive octree, rank 24, 119 samples per leaf diagonal
        {"name": "train_bf16_adaptive", "kind": "project", **c5, "rays": 16384, "samples": 119, "precision": "bf16",
         "grad": True},
        # the same step through the learned proposal at its 64 samples per ray
        {"name": "train_proposal", "kind": "proposal", **c5, "rays": 16384, "budget": 64},
        # a program built on the reference's separate operators: sample list, ComputeImage, autograd
        {"name": "train_operators", "kind": "operators", **c1, "rays": 4096, "samples": 32},
        # evaluation: density at the voxel centres of a slice stack of the 256^3 volume (PSNR, export)
        {"name": "volume", "kind": "volume", **c2, "points": 1 << 21},
        # per-leaf errors that drive the octree refinement, over a subset of the tilt series
        {"name": "node_errors", "kind": "node_errors", **c2, "rays": 65536, "samples": 24, "precision": "bf16"},
        # the two grid-sample operators on their own, forward and backward (planes in torch's default order)
        {"name": "grid_sample", "kind": "grid_sample", "slots": 4096, "channels": 16, "grid": 17, "line": 256,
         "points": 1 << 20, "channels_last": False},
        # making a tilt series: line integrals of four 256^2 images through a 256^3 volume
        {"name": "tilt_series", "kind": "siddon", "volume": 256, "rays": 4 * 65536},
        # the optimizer step over the standard configuration's parameters, writing the BF16 copies
        {"name": "adam", "kind": "adam", **c2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# decoders that the fused FP32 projection takes, by channels and feature operation
_FP32_DECODERS = {(8, "add"): ("32", "64", "64,64"), (16, "add"): ("32", "64", "64,64"), (8, "cat"): ("32", "64,64")}


def draw(rng):
    kind = rng.choice(["fp32", "fp32", "bf16", "bf16", "adaptive", "proposal", "operators", "volume", "node_errors",
                       "grid_sample", "siddon", "adam"])
    if kind == "fp32":
        channels, op = rng.choice(sorted(_FP32_DECODERS))
        m = _model(channels, rng.choice(_FP32_DECODERS[channels, op]), rng.randint(1, 4), rng.randint(9, 17), op=op)
        return {"kind": "project", **m, "rays": _log_int(rng, 64, 16384), "samples": rng.randint(8, 24),
                "precision": "fp32", "grad": rng.random() < 0.75}
    if kind == "bf16":
        m = _model(rng.choice([16, 24]), "64,64", rng.randint(2, 4), rng.randint(13, 17))
        return {"kind": "project", **m, "rays": _log_int(rng, 64, 16384), "samples": rng.randint(8, 32),
                "precision": "bf16", "grad": rng.random() < 0.75}
    if kind == "adaptive":
        m = _model(rng.choice([16, 24]), "64,64", rng.randint(5, 6), leaves=_log_int(rng, 400, 4096))
        return {"kind": "project", **m, "rays": _log_int(rng, 1000, 16384), "samples": rng.randint(40, 119),
                "precision": "bf16", "grad": rng.random() < 0.75}
    if kind == "proposal":
        m = _model(rng.choice([16, 24]), "64,64", rng.randint(5, 6), leaves=_log_int(rng, 400, 4096))
        return {"kind": "proposal", **m, "rays": _log_int(rng, 1000, 16384), "budget": rng.randint(32, 128)}
    if kind == "operators":
        m = _model(rng.choice([8, 12, 16]), rng.choice(["32", "64", "48"]), rng.randint(1, 3), rng.randint(9, 17))
        return {"kind": "operators", **m, "rays": _log_int(rng, 64, 2048), "samples": rng.randint(4, 16)}
    if kind == "volume":
        channels = rng.choice([8, 16, 24])
        m = _model(channels, rng.choice(["32", "64", "64,64"]), rng.randint(2, 4), rng.randint(9, 17))
        return {"kind": "volume", **m, "points": _log_int(rng, 1 << 12, 1 << 21)}
    if kind == "node_errors":
        m = _model(rng.choice([16, 24]), "64,64", rng.randint(2, 4))
        return {"kind": "node_errors", **m, "rays": 8192 * rng.randint(1, 8), "samples": rng.randint(8, 24),
                "precision": "bf16"}
    if kind == "grid_sample":
        return {"kind": "grid_sample", "slots": _log_int(rng, 64, 4096), "channels": rng.choice([4, 7, 8, 16, 24]),
                "grid": rng.randint(9, 17), "line": rng.randint(17, 256), "points": _log_int(rng, 1 << 12, 1 << 20),
                "channels_last": rng.random() < 0.5}
    if kind == "siddon":
        return {"kind": "siddon", "volume": rng.randint(48, 256), "rays": _log_int(rng, 1 << 12, 1 << 18)}
    return {"kind": "adam", **_model(rng.choice([8, 16, 24]), "64,64", rng.randint(2, 3), rng.randint(9, 17))}


# ----------------------------------------------------------------------------
# inputs, from the seed alone
# ----------------------------------------------------------------------------
def _gen(seed, stream):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 64 + stream)


def _uniform(g, lo, hi, *shape):
    return torch.rand(*shape, generator=g, device=DEV) * (hi - lo) + lo


def _level_start(depth):
    """Id of the first node of a level: the octree's nodes are numbered level by level."""
    return (8**depth - 1) // 7


def _node_boxes(nodes):
    """Depth and float64 boxes [n, 3] of octree nodes of [-1, 1]^3 (child i of a node: bit 0 of i is the
    upper half in x, bit 1 in y, bit 2 in z)."""
    nodes = np.asarray(nodes, np.int64)
    depth = np.zeros(len(nodes), np.int64)
    d = 1
    while _level_start(d) <= nodes.max():
        depth[nodes >= _level_start(d)] = d
        d += 1
    code = nodes - np.array([_level_start(int(k)) for k in range(d)])[depth]
    cell = np.zeros((len(nodes), 3), np.int64)
    for b in range(d):
        for k in range(3):
            cell[:, k] |= ((code >> (3 * b + k)) & 1) << b
    size = 2.0 / (1 << depth)[:, None]
    lo = -1.0 + cell * size
    return depth, lo, lo + size


_SLAB = 0.25  # half thickness of the adaptive trees' specimen


def _leaves(case):
    """Node ids of the active leaves, ascending: a whole level, or (leaves > 0) a tree refined around the
    surfaces of random ellipsoids in a slab, with the empty children left out (one specimen for each case:
    the seed changes the field and the rays)."""
    if not case["leaves"]:
        return np.arange(_level_start(case["depth"]), _level_start(case["depth"] + 1))
    rng = np.random.default_rng(1000 + case["leaves"])
    n = 30
    centre = rng.uniform(-0.8, 0.8, (n, 3)) * [1, 1, _SLAB]
    axes = rng.uniform(0.05, 0.25, (n, 3)) * [1, 1, _SLAB]

    def look(nodes):
        """(nodes that hold density, how much surface each may hold)"""
        _, lo, hi = _node_boxes(nodes)
        mid, half = (lo + hi) / 2, (hi - lo)[:, 0] / 2
        q = np.sqrt((((mid[:, None] - centre[None]) / axes[None]) ** 2).sum(-1))
        reach = half[:, None] * np.sqrt((1 / axes**2).sum(1))[None]
        keep = ((q < 1 + reach).any(1)) & (lo[:, 2] < _SLAB) & (hi[:, 2] > -_SLAB)
        score = (np.abs(q - 1) < reach / 2).sum(1).astype(float)
        return np.asarray(nodes)[keep], score[keep]

    leaves, score = look(np.arange(_level_start(3), _level_start(4)))
    last = _level_start(case["depth"])
    while len(leaves) < case["leaves"]:
        cand = np.nonzero((leaves < last) & (score > 0))[0]
        if len(cand) == 0:
            break
        pick = cand[np.lexsort((leaves[cand], -score[cand]))[:max(1, min(len(cand) // 5, (case["leaves"] - len(leaves)) // 7 + 1))]]
        kids, ks = look((8 * leaves[pick][:, None] + 1 + np.arange(8)[None]).reshape(-1))
        rest = np.ones(len(leaves), bool)
        rest[pick] = False
        leaves, score = np.concatenate([leaves[rest], kids]), np.concatenate([score[rest], ks])
    return np.sort(leaves)


def _rays(case, seed):
    """Parallel-beam rays of random pixels of 61 tilts (2 degrees apart, about the y axis): origin, direction."""
    g, n = _gen(seed, 1), case["rays"]
    th = torch.deg2rad((torch.randint(0, 61, (n,), generator=g, device=DEV).double() - 30) * 2)
    pix = (torch.randint(0, 256, (2, n), generator=g, device=DEV).double() + 0.5) / 128 - 1
    c, s = th.cos(), th.sin()
    d = torch.stack([s, torch.zeros_like(s), c], 1)
    o = torch.stack([pix[0] * c, pix[1], -pix[0] * s], 1) - math.sqrt(2.0) * d
    return o.float().contiguous(), d.float().contiguous()


def _factors(case, slots, seed):
    """Planes [slots, C, G, G] (channels-last), lines [1, C, L, 1], decoder weights and biases: the
    framework's initialisation (factors U(-0.5, 0.5), Kaiming-normal weights)."""
    g, C, G = _gen(seed, 2), case["channels"], case["grid"]
    n = (G - 1) << min(case["depth"], 4)
    planes = [_uniform(g, -0.5, 0.5, slots, G, G, C).permute(0, 3, 1, 2) for _ in range(3)]
    lines = [_uniform(g, -0.5, 0.5, 1, L, 1, C).permute(0, 3, 1, 2) for L in (n, G, n)]
    dims = [C * (3 if case["op"] == "cat" else 1)] + [int(h) for h in case["hidden"].split(",")] + [1]
    W = [torch.randn(b, a, generator=g, device=DEV) * math.sqrt(2.0 / a) for a, b in zip(dims, dims[1:])]
    B = [_uniform(g, -1 / math.sqrt(a), 1 / math.sqrt(a), b) for a, b in zip(dims, dims[1:])]
    return planes, lines, W, B


def _target(case, seed):
    return _uniform(_gen(seed, 3), 0.0, 2.0, case["rays"])


def _jitter(seed):
    return 0x9E3779B1 * (int(seed) % 1000003 + 1)


def _points(case, seed):
    """Voxel centres of the 256^3 volume, slice by slice from a seeded one on."""
    N = 256
    first = (int(seed) * 7919) % (N**3 - case["points"] + 1)
    i = torch.arange(first, first + case["points"], device=DEV)
    return torch.stack([(torch.remainder(v, N).double() + 0.5) / N * 2 - 1 for v in (i, i // N, i // (N * N))], 1).float().contiguous()


def _grid_inputs(case, seed):
    g, N, C, G, S = _gen(seed, 4), case["slots"], case["channels"], case["grid"], case["points"]
    grid = _uniform(g, -0.5, 0.5, N, C, G, G)
    line = _uniform(g, -0.5, 0.5, 1, C, case["line"], 1)
    if case["channels_last"]:
        grid = grid.contiguous(memory_format=torch.channels_last)
        line = line.contiguous(memory_format=torch.channels_last)
    index = torch.randint(0, N, (S,), generator=g, device=DEV)
    uv, u = _uniform(g, -1, 1, S, 2), _uniform(g, -1, 1, S, 1)
    return grid, line, index, uv, u, _uniform(g, -1, 1, S, C), _uniform(g, -1, 1, S, C)


def _siddon_inputs(case, seed):
    g, N = _gen(seed, 5), case["volume"]
    vol = (_uniform(g, -1, 1, N, N, N)).clamp_min(0)
    o, d = _rays(case, seed)
    return vol, o, d


# ----------------------------------------------------------------------------
# prepare and run
# ----------------------------------------------------------------------------
class _Series:
    """What recon.node_errors reads of a tilt series."""

    def __init__(self, origin, direction, target):
        self.origin, self.direction, self.target, self.num_rays = origin, direction, target, origin.shape[0]


def _geometry(case, seed):
    import adaptivetensordf_b200 as ab
    from adaptivetensordf_b200 import synthetic as syn

    tree = syn.tree_from_leaves(case["depth"], _leaves(case), device=DEV)
    planes, lines, W, B = _factors(case, tree.NumActiveNodes(), seed)
    geo = ab.GeometryTensorQO()
    geo.planes = [p.requires_grad_(True) for p in planes]
    geo.lines = [p.requires_grad_(True) for p in lines]
    geo.leaf_slot = tree.node_active_prefix_sum
    geo.tensor_op = case["op"]
    geo.decoder_weight = [w.requires_grad_(True) for w in W]
    geo.decoder_bias = [b.requires_grad_(True) for b in B]
    geo.activation, geo.last_activation, geo.softplus_beta = "silu", "softplus", 2.0
    geo.precision = case.get("precision", "fp32")
    if geo.precision == "bf16":
        geo.RefreshLowPrecision()
    return tree, geo


def prepare(case, seed):
    import adaptivetensordf_b200 as ab

    s = {"case": case, "seed": _jitter(seed)}
    kind = case["kind"]
    if kind == "grid_sample":
        s["inputs"] = _grid_inputs(case, seed)
        for i in (0, 1, 3, 4):
            s["inputs"][i].requires_grad_(True)
        return s
    if kind == "siddon":
        s["inputs"] = _siddon_inputs(case, seed)
        return s
    if kind == "proposal":
        case = {**case, "precision": "bf16"}
    elif kind == "adam":
        case = {**case, "precision": "bf16"}
    s["tree"], s["geo"] = _geometry(case, seed)
    geo = s["geo"]
    s["params"] = list(geo.planes) + list(geo.lines) + list(geo.decoder_weight) + list(geo.decoder_bias)
    if kind == "volume":
        s["points"] = _points(case, seed)
    elif kind == "adam":
        from adaptivetensordf_b200.optim import Adam

        g = _gen(seed, 6)
        for p in s["params"]:
            p.grad = torch.empty_like(p).normal_(0.0, 1e-3, generator=g)
        s["adam"] = Adam([{"params": s["params"][:6], "lr": 0.01}, {"params": s["params"][6:], "lr": 5e-4}],
                         geometry=geo)
    else:
        o, d = _rays(case, seed)
        s["rays"], s["target"] = ab.RayList(o, d), _target(case, seed)
        if kind == "node_errors":
            s["series"] = _Series(o, d, s["target"])
        if kind == "proposal":
            s["sampler"] = ab.ProposalSampler(s["tree"].NumNodes(), 64, 3, 1005, DEV)
            s["sampler"].budget = case["budget"]
            s["sampler"].precision = "bf16"
            s["sampler"].occupancy = _uniform(_gen(seed, 7), 0.0, 1.0, *s["sampler"].occupancy.shape)
    return s


def _step(s, image):
    """Loss and gradients of a training step on `image`."""
    loss = (image.view(-1) - s["target"]).pow(2).mean()
    for p in s["params"]:
        p.grad = None
    loss.backward()
    return {"image": image.detach(), "loss": loss.detach(), "grad": [p.grad for p in s["params"]]}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "project":
        if not case["grad"]:
            with torch.no_grad():
                return s["geo"].ProjectRays(s["tree"], s["rays"], case["samples"], s["seed"])
        return _step(s, s["geo"].ProjectRays(s["tree"], s["rays"], case["samples"], s["seed"]))
    if kind == "proposal":
        return _step(s, s["sampler"].Project(s["tree"], s["geo"], s["rays"], s["seed"]))
    if kind == "operators":
        samples = s["tree"].CreateSamplesForRaysWithRnd(s["rays"], case["samples"], None, s["seed"])
        image, _, _ = s["geo"].ComputeImage(s["tree"], samples, 1, case["rays"])
        return _step(s, image)
    if kind == "volume":
        with torch.no_grad():
            node, inside = s["tree"].NodeIdForPositionGPU(s["points"])
            return {"node": node, "inside": inside, "density": s["geo"].SampleVolumeIndirect(s["tree"], s["points"], node)}
    if kind == "node_errors":
        from adaptivetensordf_b200 import recon

        recon.node_errors(s["tree"], s["geo"], s["series"], case["samples"], rays=case["rays"], batch=min(16384, case["rays"]))
        return s["tree"].node_error
    if kind == "grid_sample":
        import adaptivetensordf_b200 as ab

        grid, line, index, uv, u, w2, w1 = s["inputs"]
        for p in (grid, line, uv, u):
            p.grad = None
        a = ab.IndirectGridSample2D(grid, index, uv)
        b = ab.IndirectGridSample1D(line, torch.zeros_like(index), u)
        torch.autograd.backward([a, b], [w2, w1])
        return {"plane": a.detach(), "line": b.detach(), "grad": [p.grad for p in (grid, uv, line, u)]}
    if kind == "siddon":
        import adaptivetensordf_b200 as ab

        return ab.SiddonProject(*s["inputs"])
    if kind == "adam":
        s["adam"].step()
        st = s["adam"].state
        return {"param": [p.detach() for p in s["params"]], "bf16": list(s["geo"].planes_bf16) + list(s["geo"].lines_bf16),
                "moment": [st[p]["exp_avg"] for p in s["params"]], "square": [st[p]["exp_avg_sq"] for p in s["params"]]}
    raise ValueError(kind)


# ----------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------
def _decoder_macs(case):
    dims = [case["channels"] * (3 if case["op"] == "cat" else 1)] + [int(h) for h in case["hidden"].split(",")] + [1]
    return sum(a * b for a, b in zip(dims, dims[1:]))


def _samples_per_ray(case):
    """Expected samples of a ray: a mean chord of 1.87 of the [-1, 1]^3 cube (the adaptive slab: about 0.3 of
    occupied length) over the leaf diagonal, and half a sample per leaf for the rounding up."""
    if case["leaves"]:
        return case["samples"] * 2.1
    edge = 2.0 / (1 << case["depth"])
    return case["samples"] * 1.87 / (edge * math.sqrt(3)) + 0.61 * (1 << case["depth"])


def _slots(case):
    return case["leaves"] or 8 ** case["depth"]


def work(case):
    kind = case["kind"]
    if kind == "grid_sample":
        S, C = case["points"], case["channels"]
        planes = case["slots"] * C * case["grid"] ** 2 * 4
        return {"bytes": 3 * planes + S * (2 * 8 + 4 * 3 * 2 + 4 * C * 4), "flops": S * C * 60}
    if kind == "siddon":
        return {"bytes": case["volume"] ** 3 * 4 + case["rays"] * 32, "flops": case["rays"] * case["volume"] * 12}
    feats = 12 * 2 * case["channels"]  # gathers, products and sums of a sample's features
    factors = _slots(case) * 3 * case["channels"] * case["grid"] ** 2
    if kind == "adam":
        return {"bytes": factors * 30, "flops": factors * 12}
    if kind == "volume":
        P = case["points"]
        return {"bytes": P * (12 + 8 + 4 + 4) + factors * 4 * min(1.0, P / 256**3), "flops": P * (2 * _decoder_macs(case) + feats)}
    bf16 = case.get("precision", "fp32") == "bf16" or kind == "proposal"
    S = case["rays"] * (case["budget"] if kind == "proposal" else _samples_per_ray(case))
    grad = kind in ("proposal", "operators") or (kind == "project" and case["grad"])
    touched = min(1.0, S / 32 / _slots(case))  # few rays do not meet every leaf
    return {"bytes": case["rays"] * 32 + factors * ((2 if bf16 else 4) * touched + (4 if grad else 0)),
            "flops": S * (2 * _decoder_macs(case) + feats) * (3 if grad else 1)}


# ----------------------------------------------------------------------------
# the outputs in 64 bits, from plain torch
# ----------------------------------------------------------------------------
def _mix64(z):
    """SplitMix64's finaliser on int64 tensors (wrapping products, logical shifts)."""

    def shr(v, k):
        return (v >> k) & ((1 << (64 - k)) - 1)

    def wrap(c):
        return c - (1 << 64) if c >= 1 << 63 else c

    z = (z ^ shr(z, 30)) * wrap(0xBF58476D1CE4E5B9)
    z = (z ^ shr(z, 27)) * wrap(0x94D049BB133111EB)
    return z ^ shr(z, 31)


def _exact_samples(leaves, o, d, M, seed):
    """The uniform per-leaf samples of every ray, float32 with one rounding per operation as the sampler
    defines them (jittered, or at the interval's middle for seed 0): ray, slot, leaf boxes, weight and
    position of each sample."""
    _, lo, hi = _node_boxes(leaves)
    lo = torch.from_numpy(lo).float().to(DEV)
    hi = torch.from_numpy(hi).float().to(DEV)
    node = torch.from_numpy(np.asarray(leaves)).to(DEV)
    parts = []
    step = max(1, (1 << 24) // len(leaves))
    for r0 in range(0, o.shape[0], step):
        oo, dd = o[r0:r0 + step], d[r0:r0 + step]
        n = torch.full((oo.shape[0], len(leaves)), -236436436.0, device=DEV)
        f = torch.full_like(n, 43637575.0)
        ok = torch.ones_like(n, dtype=torch.bool)
        for k in range(3):
            ox, dx = oo[:, k:k + 1], dd[:, k:k + 1]
            flat = dx == 0
            t1, t2 = (lo[None, :, k] - ox) / dx, (hi[None, :, k] - ox) / dx
            a, b = torch.minimum(t1, t2), torch.maximum(t1, t2)
            n = torch.where(flat, n, torch.maximum(n, a))
            f = torch.where(flat, f, torch.minimum(f, b))
            ok &= torch.where(flat, (ox >= lo[None, :, k]) & (ox < hi[None, :, k]), (n <= f) & (f >= 0))
        ok &= ~((f - n).double() < 1e-5)
        r, s = ok.nonzero(as_tuple=True)
        parts.append((r + r0, s, n[r, s], f[r, s]))
    r, s, t0, t1 = (torch.cat(x) for x in zip(*parts))
    size = hi - lo
    sq = size * size
    diag = ((sq[:, 0] + sq[:, 1]) + sq[:, 2]).sqrt()
    cnt = torch.ceil(((t1 - t0) / diag[s]) * torch.tensor(float(M), device=DEV)).long()
    seg = torch.repeat_interleave(torch.arange(len(r), device=DEV), cnt)
    j = torch.arange(len(seg), device=DEV) - (cnt.cumsum(0) - cnt)[seg]
    golden = 0x9E3779B97F4A7C15 - (1 << 64)
    key = _mix64(seed + golden * r)[seg]
    inc = ((t1 - t0) / cnt.float())[seg]
    a0, nn = t0[seg], node[s][seg]

    def t_of(i):
        if seed:
            a = (((_mix64(key ^ ((nn << 32) | i)) >> 40) & 0xFFFFFF).float()) * (1.0 / 16777216.0)
        else:
            a = torch.full_like(a0, 0.5)
        u, v = a0 + i.float() * inc, a0 + (i + 1).float() * inc
        return u * (1.0 - a) + v * a

    t = t_of(j)
    half = torch.tensor(0.5, device=DEV)
    w_lo = torch.where(j == 0, a0, (t_of((j - 1).clamp_min(0)) + t) * half)
    w_hi = torch.where(j == cnt[seg] - 1, t1[seg], (t_of(j + 1) + t) * half)
    ray = r[seg]
    pos = o[ray] + d[ray] * t[:, None]
    return ray, s[seg], lo, hi, w_hi - w_lo, pos


def _lerp2(grid, slot, u, v):
    """Bilinear samples (align_corners, clamped) of grid [N, C, H, W] at u along W, v along H."""
    N, C, H, W = grid.shape
    flat = grid.permute(0, 2, 3, 1).reshape(-1, C)
    x, y = (u + 1) / 2 * (W - 1), (v + 1) / 2 * (H - 1)
    x0, y0 = x.floor(), y.floor()
    out = 0
    for dy in (0, 1):
        for dx in (0, 1):
            w = (x - x0 if dx else x0 + 1 - x) * (y - y0 if dy else y0 + 1 - y)
            at = (slot * H + (y0 + dy).long().clamp(0, H - 1)) * W + (x0 + dx).long().clamp(0, W - 1)
            out = out + w[:, None] * flat.index_select(0, at)
    return out


def _lerp1(line, u):
    C, L = line.shape[1], line.shape[2]
    flat = line[0, :, :, 0].t()
    x = (u + 1) / 2 * (L - 1)
    x0 = x.floor()
    return sum((x - x0 if dx else x0 + 1 - x)[:, None] * flat.index_select(0, (x0 + dx).long().clamp(0, L - 1)) for dx in (0, 1))


def _density(case, P, slot, lo, hi, pos):
    planes, lines, W, B = P
    p = pos.double()
    loc = (p - lo[slot].double()) / (hi - lo)[slot].double() * 2 - 1
    pl = ((loc[:, 1], loc[:, 2]), (loc[:, 0], loc[:, 2]), (loc[:, 0], loc[:, 1]))
    ln = (p[:, 0], loc[:, 1], p[:, 2])  # the region of interest is [-1, 1]: its x coordinate is x itself
    feats = [_lerp2(planes[m], slot, *pl[m]) * _lerp1(lines[m], ln[m]) for m in range(3)]
    x = torch.cat(feats, 1) if case["op"] == "cat" else feats[0] + feats[1] + feats[2]
    for i, (w, b) in enumerate(zip(W, B)):
        x = x @ w.t() + b
        x = x * torch.sigmoid(x) if i + 1 < len(W) else torch.nn.functional.softplus(x, 2.0)
    return x[:, 0]


def _double(case, slots, seed):
    planes, lines, W, B = _factors(case, slots, seed)
    if case.get("precision") == "bf16":  # the working copies that the BF16 form holds
        planes, lines = [p.bfloat16() for p in planes], [p.bfloat16() for p in lines]
    return [[t.double().requires_grad_(True) for t in v] for v in (planes, lines, W, B)]


def _exact_image(case, P, samples, rays, grad_image=None):
    """The image; with grad_image also adds the parameters' gradients, a part of the samples at a time."""
    ray, slot, lo, hi, w, pos = samples
    image = torch.zeros(rays, dtype=torch.float64, device=DEV)
    for i in range(0, len(ray), 1 << 19):
        k = slice(i, i + (1 << 19))
        with torch.set_grad_enabled(grad_image is not None):
            v = _density(case, P, slot[k], lo, hi, pos[k]) * w[k].double()
            if grad_image is not None:
                (v * grad_image[ray[k]]).sum().backward()
        image.index_add_(0, ray[k], v.detach())
    return image


def exact(case, seed):
    kind = case["kind"]
    if kind == "proposal":
        return None  # where its samples lie depends on the proposal network's own roundings
    if kind == "grid_sample":
        grid, line, index, uv, u, w2, w1 = _grid_inputs(case, seed)
        grid, line, uv, u = (t.double().requires_grad_(True) for t in (grid, line, uv, u))
        a = _lerp2(grid, index, uv[:, 0], uv[:, 1])
        b = _lerp1(line, u[:, 0])
        torch.autograd.backward([a, b], [w2.double(), w1.double()])
        # the 1D operator weights each end's share of the coordinate gradient by the distance to the
        # other end, as the reference's does (IndirectGridSample1D.cu)
        x = (u.detach()[:, 0] + 1) / 2 * (case["line"] - 1)
        x0, v = x.floor(), line.detach()[0, :, :, 0].t()
        ends = [v.index_select(0, (x0 + i).long().clamp(0, case["line"] - 1)) for i in (0, 1)]
        du = (((x - x0)[:, None] * ends[1] - (x0 + 1 - x)[:, None] * ends[0]) * w1.double()).sum(1)
        u_grad = (du * (case["line"] - 1) / 2)[:, None]
        return {"plane": a.detach(), "line": b.detach(), "grad": [grid.grad, uv.grad, line.grad, u_grad]}
    if kind == "siddon":
        return _exact_siddon(case, seed)
    leaves = _leaves(case)
    if kind == "adam":
        planes, lines, W, B = _factors(case, len(leaves), seed)
        g, out = _gen(seed, 6), {"param": [], "bf16": [None] * 6, "moment": [], "square": []}
        for i, p in enumerate(planes + lines + W + B):
            grad = torch.empty_like(p).normal_(0.0, 1e-3, generator=g).double()
            m, v = 0.1 * grad, 0.001 * grad * grad
            out["param"].append(p.double() - (0.01 if i < 6 else 5e-4) * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8))
            out["moment"].append(m)
            out["square"].append(v)
        return out
    P = _double(case, len(leaves), seed)
    if kind == "volume":
        pts = _points(case, seed)
        n = 1 << case["depth"]
        cell = torch.floor((pts.double() + 1) / 2 * n).long()
        slot = torch.zeros(len(pts), dtype=torch.int64, device=DEV)
        for b in range(case["depth"]):
            for k in range(3):
                slot |= ((cell[:, k] >> b) & 1) << (3 * b + k)
        _, lo, hi = _node_boxes(leaves)
        lo, hi = (torch.from_numpy(v).float().to(DEV) for v in (lo, hi))
        with torch.no_grad():
            dens = torch.cat([_density(case, P, slot[i:i + (1 << 19)], lo, hi, pts[i:i + (1 << 19)])
                              for i in range(0, len(pts), 1 << 19)])
        return {"node": None, "inside": None, "density": dens[:, None]}
    if kind == "node_errors":
        o, d = _rays(case, seed)
        idx = torch.randint(0, case["rays"], (case["rays"],), device=DEV, generator=torch.Generator(device=DEV).manual_seed(1006))
        o, d, target = o[idx], d[idx], _target(case, seed)[idx]
        ls = torch.zeros(_level_start(case["depth"] + 1), dtype=torch.float64, device=DEV)
        ws = torch.zeros_like(ls)
        node = torch.from_numpy(leaves).to(DEV)
        for i in range(0, case["rays"], 16384):
            smp = _exact_samples(leaves, o[i:i + 16384], d[i:i + 16384], case["samples"], 0)
            img = _exact_image(case, P, smp, len(o[i:i + 16384]))
            per_ray = (img - target[i:i + 16384].double()) ** 2
            ws.index_add_(0, node[smp[1]], smp[4].double())
            ls.index_add_(0, node[smp[1]], smp[4].double() * per_ray[smp[0]])
        out = torch.full_like(ls, -1.0)  # inner nodes keep the value that says "no error yet"
        out[node] = torch.where(ws > 0, ls / ws.clamp_min(1e-30), torch.zeros_like(ls))[node]
        return out
    o, d = _rays(case, seed)
    samples = _exact_samples(leaves, o, d, case["samples"], _jitter(seed))
    image = _exact_image(case, P, samples, case["rays"])
    if kind == "project" and not case["grad"]:
        return image[None]
    off = image - _target(case, seed).double()
    _exact_image(case, P, samples, case["rays"], 2 * off / case["rays"])
    return {"image": image[None], "loss": (off * off).mean(), "grad": [t.grad for v in P for t in v]}


def _exact_siddon(case, seed):
    """Line integrals through the voxels of [-1, 1]^3: the crossings of all voxel planes, sorted."""
    vol, o, d = _siddon_inputs(case, seed)
    N = case["volume"]
    flat = vol.reshape(-1).double()
    out = []
    edges = torch.arange(N + 1, device=DEV, dtype=torch.float64) * (2.0 / N) - 1
    for i in range(0, len(o), 1 << 14):
        oo, dd = o[i:i + (1 << 14)].double(), d[i:i + (1 << 14)].double()
        near = torch.full((len(oo),), -math.inf, dtype=torch.float64, device=DEV)
        far = -near
        ts = []
        for k in range(3):
            flat_k = dd[:, k] == 0
            inv = 1 / torch.where(flat_k, torch.ones_like(far), dd[:, k])
            t = (edges[None] - oo[:, k:k + 1]) * inv[:, None]
            a, b = torch.minimum(t[:, 0], t[:, -1]), torch.maximum(t[:, 0], t[:, -1])
            outside = (oo[:, k] < -1) | (oo[:, k] > 1)
            near = torch.where(flat_k, torch.where(outside, torch.full_like(near, math.inf), near), torch.maximum(near, a))
            far = torch.where(flat_k, far, torch.minimum(far, b))
            ts.append(torch.where(flat_k[:, None], torch.zeros_like(t), t))
        hit = far > near
        near, far = torch.where(hit, near, torch.zeros_like(near)), torch.where(hit, far, torch.zeros_like(far))
        t = torch.cat(ts, 1).clamp(near[:, None], far[:, None]).sort(1).values
        length = t[:, 1:] - t[:, :-1]
        mid = (t[:, 1:] + t[:, :-1]) / 2
        cell = [((oo[:, k:k + 1] + dd[:, k:k + 1] * mid + 1) / 2 * N).floor().long().clamp(0, N - 1) for k in range(3)]
        out.append((length * flat[(cell[2] * N + cell[1]) * N + cell[0]]).sum(1))
    return torch.cat(out)
