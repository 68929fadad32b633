"""The two tensor-core forwards (by runs of segments for small calls, by slot with
staged planes for large ones) against the FP64 oracle on the BF16-rounded
parameters. A call counts as large by the segments that its rays could have
(3 * 2^depth + 3 each), so rays that miss the volume take a small set of rays,
which the oracle can project, to the form by slot."""

import ctypes as ct

import numpy as np
import pytest
import torch

from oracle import proposal_oracle as po
from tests.scene import gpu_scene, oracle_views, rel_err

pytestmark = pytest.mark.gpu

LINE = 1 << 18       # segments by capacity up to which a call goes by runs
LINE24 = 1 << 22     # the same for 24 channels on 2048 slots or more
# Relative L2 of the image. WIDE: the benchmark's shapes, three times the
# measured 1.4e-5 (hundreds of samples a ray average the decoder's BF16
# rounding). FEW: three times the 1.3e-4 of scenes with few samples a ray.
WIDE, FEW = 5e-5, 4e-4
RAY = 2.0**-8        # of one ray, and of the bins in L2: one BF16 rounding of every activation
BIN = 0.05           # of one bin, in parts of the largest: a sample more or less is far beyond


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


def _bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(torch.bfloat16).to(torch.float64).numpy()


def _views(tree, geo):
    geo.precision = "bf16"
    geo.RefreshLowPrecision()
    td, fd, md = oracle_views(tree, geo)
    fd = {**fd, "planes": [_bf16(p) for p in fd["planes"]], "lines": [_bf16(x) for x in fd["lines"]]}
    layers = [(_bf16(w), b.astype(np.float64)) for w, b in md["layers"]]
    layers[-1] = (md["layers"][-1][0].astype(np.float64), layers[-1][1])  # the last layer runs in FP32
    return td, fd, {**md, "layers": layers}


def _with_misses(o, d, total):
    """The rays and, behind them, rays beside the volume up to `total`."""
    n = max(0, total - len(o))
    far, along = np.full((n, 3), 5.0, np.float32), np.tile(np.array([[0.0, 0.0, 1.0]], np.float32), (n, 1))
    return np.concatenate([o, far]), np.concatenate([d, along])


def _check(img, ref, tol):
    img, n = img.detach().cpu().numpy().reshape(-1), ref.size
    assert rel_err(img[:n], ref.reshape(-1)) < tol
    assert (np.abs(img[:n] - ref.reshape(-1)) <= RAY * np.abs(ref).reshape(-1) + 1e-6 * np.abs(ref).max()).all()
    assert (img[n:] == 0.0).all()


def _project(tree, geo, o, d, M, seed):
    import adaptivetensordf_b200 as ab

    img = geo.ProjectRays(tree, ab.RayList(torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()), M, seed)
    geo.CheckErrors()
    return img


@pytest.mark.parametrize("M", [24, 96])
def test_standard_configuration_by_slot(oracle, M):
    """16 channels at the standard configuration's shapes through a window of
    the detector: slots of several items, and (M = 96) items beyond the sample
    map."""
    from adaptivetensordf_b200 import synthetic as syn

    cfg = syn.CONFIGS["C2"]
    tree = syn.make_tree(cfg.tree_depth, device="cuda")
    geo = syn.make_geometry(tree, cfg.channels, cfg.grid, cfg.lines(), cfg.hidden, seed=1003)
    td, fd, md = _views(tree, geo)
    R, w = (2048, 64) if M == 24 else (512, 16)
    rng = np.random.default_rng(M)
    img, px, py = rng.integers(0, cfg.angles, R), *(128 - w // 2 + rng.integers(0, w, (2, R)))
    o, d = syn.parallel_beam_rays(syn.tilt_angles(cfg), cfg.detector, img, py * cfg.detector + px)
    segs = oracle.ray_segments(td, o, d, M)
    assert np.bincount(segs["node"]).max() > 128
    so = oracle.emit_samples(segs, o, d, oracle.jitter_for_segments(57, segs))
    ref = oracle.project_forward(fd, md, td, so, R, np.float64)
    per = 3 * 2**cfg.tree_depth + 3
    o, d = _with_misses(o, d, LINE // per + 1)
    assert len(o) * per > LINE
    _check(_project(tree, geo, o, d, M, 57), ref, WIDE)


def test_largest_configuration_by_slot(oracle):
    """24 channels on the adaptive tree through a window of the detector, in a
    call beyond the line of many slots: leaves of several depths, slots of many
    items, windows of the lines."""
    from adaptivetensordf_b200 import synthetic as syn

    cfg = syn.CONFIGS["C5"]
    tree = syn.adaptive_tree(cfg, syn.config_phantom(cfg, 1001), device="cuda")
    geo = syn.make_geometry(tree, cfg.channels, cfg.grid, cfg.lines(), cfg.hidden, seed=1003)
    td, fd, md = _views(tree, geo)
    R, w, M = 1024, 32, cfg.max_samples_per_node
    rng = np.random.default_rng(78)
    img, px, py = rng.integers(0, cfg.angles, R), *(cfg.detector // 2 - w // 2 + rng.integers(0, w, (2, R)))
    o, d = syn.parallel_beam_rays(syn.tilt_angles(cfg), cfg.detector, img, py * cfg.detector + px, cfg.off_axis_deg)
    segs = oracle.ray_segments(td, o, d, M)
    assert np.bincount(segs["node"]).max() > 3 * 128
    so = oracle.emit_samples(segs, o, d, oracle.jitter_for_segments(61, segs))
    ref = oracle.project_forward(fd, md, td, so, R, np.float64)
    per = min(3 * 2**tree.max_depth + 3, 256)
    o, d = _with_misses(o, d, LINE24 // per + 1)
    assert len(o) * per > LINE24
    _check(_project(tree, geo, o, d, M, 61), ref, WIDE)


@pytest.mark.parametrize("C,depth", [(16, 4), (24, 3)])
@pytest.mark.parametrize("by_slot", [False, True])
def test_every_kind_of_samples(oracle, C, depth, by_slot):
    """Jittered uniform samples, the same t and weights placed by the caller, and
    the bins of rho * w, by runs and by slot (24 channels: few slots, so that
    the line is the common one)."""
    from adaptivetensordf_b200 import capi

    R, M, seed, per = 1200, 12, 31, 3 * 2**depth + 3
    L = 16 << depth
    tree, geo, o, d = gpu_scene(depth, C, 17, (L, 17, L), [64, 64], R, seed=C)
    td, fd, md = _views(tree, geo)
    segs = oracle.ray_segments(td, o, d, M)
    so = oracle.emit_samples(segs, o, d, oracle.jitter_for_segments(seed, segs))
    feat = oracle.vm_features(fd, td, so["global_coordinate"], so["node_id"], np.float64)
    rho = oracle.mlp_forward(md, feat, np.float64)[:, 0] * so["weight"]
    ref = np.zeros(R)
    np.add.at(ref, so["ray_index"], rho)
    if by_slot:
        o, d = _with_misses(o, d, LINE // per + 1)
    R = len(o)
    assert (R * per > LINE) == by_slot
    _check(_project(tree, geo, o, d, M, seed), ref, FEW)

    Lb, t = capi.lib(), capi.tree_struct(tree)
    f, keep_f = capi.field_struct_bf16(geo)
    m, keep_m = capi.mlp_struct(geo)
    ot, dt = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    size = ct.c_size_t()
    assert Lb.atdf_project_workspace_size(R, t.max_depth, t.ns, f.num_slots, 1, ct.byref(size)) == 0
    ws = torch.empty(size.value, dtype=torch.uint8, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    view, img = capi.Segments(), torch.empty(1, R, device="cuda")
    # placed
    assert Lb.atdf_project_segments(ct.byref(t), capi.ptr(ot), capi.ptr(dt), R, M, f.num_slots, capi.ptr(ws),
                                    size.value, ct.byref(view), capi.ptr(err), None) == 0
    xt, xw = torch.from_numpy(so["ray_t"]).cuda(), torch.from_numpy(so["weight"]).cuda()
    assert Lb.atdf_project_forward_samples(ct.byref(t), ct.byref(f), ct.byref(m), capi.ptr(ot), capi.ptr(dt), R,
                                           capi.ptr(xt), capi.ptr(xw), capi.ptr(img), capi.ptr(ws), size.value,
                                           capi.ptr(err), None) == 0
    torch.cuda.synchronize()
    _check(img, ref, FEW)
    # binned
    bins = torch.empty(view.capacity, po.BINS, device="cuda")
    assert Lb.atdf_project_forward_binned(ct.byref(t), ct.byref(f), ct.byref(m), capi.ptr(ot), capi.ptr(dt), R, M, seed,
                                          capi.ptr(img), capi.ptr(bins), capi.ptr(ws), size.value, capi.ptr(err),
                                          None) == 0
    torch.cuda.synchronize()
    assert err.item() == 0
    _check(img, ref, FEW)
    G = len(segs["n"])
    seg = np.repeat(np.arange(G), segs["n"])
    x = (so["ray_t"] - segs["tmin"][seg]) / (segs["tmax"] - segs["tmin"])[seg] * np.float32(po.BINS)
    want = np.zeros((G, po.BINS))
    np.add.at(want, (seg, np.clip(x.astype(np.int64), 0, po.BINS - 1)), rho)
    edge = np.abs(x - np.rint(x)) < 1e-3  # t at the edge of a bin may round to either side
    clear = np.ones(G, bool)
    clear[seg[edge]] = False
    got = bins[:G].double().cpu().numpy()
    assert clear.mean() > 0.5 and not bins[G:].any()
    assert rel_err(got[clear], want[clear]) < RAY
    assert np.abs(got - want)[clear].max() < BIN * want.max()
