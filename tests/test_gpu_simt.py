"""The FP32 fused kernels (csrc/fused_simt.cuh) at the sizes where their tiling
can go wrong, against the FP64 oracle: every decoder variant, items of one
sample up to just past a tile and a geometry pass, few and many copies of the
line gradients, and a hidden activation other than the inlined one."""

import numpy as np
import pytest
import torch

from tests.scene import gpu_scene, oracle_views, rel_err

pytestmark = pytest.mark.gpu

REL_TOL = 1e-5  # the FP32 form's parity tolerance


@pytest.fixture(scope="module")
def oracle():
    from oracle import oracle as O

    return O


def _check(oracle, tree, geo, o, d, M, seed):
    import adaptivetensordf_b200 as ab

    R = o.shape[0]
    td, fd, md = oracle_views(tree, geo)
    img = geo.ProjectRays(tree, ab.RayList(torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()), M, seed)
    segs = oracle.ray_segments(td, o, d, M)
    so = oracle.emit_samples(segs, o, d, oracle.jitter_for_segments(seed, segs) if seed else None)
    ref = oracle.project_forward(fd, md, td, so, R, np.float64)
    assert rel_err(img.detach().cpu().numpy(), ref) < REL_TOL
    gi = np.random.default_rng(4).normal(size=ref.shape)
    img.backward(torch.from_numpy(gi.astype(np.float32)).cuda())
    geo.CheckErrors()
    gr = oracle.project_backward(fd, md, td, so, R, gi.astype(np.float32).astype(np.float64), np.float64)
    for m in range(3):
        assert rel_err(geo.planes[m].grad.cpu().numpy(), gr["planes"][m]) < REL_TOL, f"plane {m}"
        assert rel_err(geo.lines[m].grad.cpu().numpy(), gr["lines"][m]) < REL_TOL, f"line {m}"
    for li in range(len(md["layers"])):
        assert rel_err(geo.decoder_weight[li].grad.cpu().numpy(), gr["W"][li]) < REL_TOL, f"W{li}"
        assert rel_err(geo.decoder_bias[li].grad.cpu().numpy(), gr["b"][li]) < REL_TOL, f"b{li}"
    return len(so["weight"])


@pytest.mark.parametrize("C,hidden,op", [(8, [32], "add"), (8, [64], "add"), (8, [64, 64], "add"), (16, [32], "add"),
                                         (16, [64], "add"), (16, [64, 64], "add"), (8, [64, 64], "cat"),
                                         (8, [32], "cat")])
@pytest.mark.parametrize("R,depth,M,G", [(1, 3, 1, 17), (37, 1, 5, 9), (900, 2, 13, 12)])
def test_variants(oracle, C, hidden, op, R, depth, M, G):
    tree, geo, o, d = gpu_scene(depth, C, G, (G + 5, G, 3 * G), hidden, R, seed=C + R, tensor_op=op)
    _check(oracle, tree, geo, o, d, M, 77)


@pytest.mark.parametrize("hidden", [[32], [64, 64]])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 129, 257])
def test_tile_edges(oracle, hidden, n):
    """One axis-parallel ray through a single leaf with n samples (length 2 of
    a diagonal of 2 sqrt(3))."""
    tree, geo, _, _ = gpu_scene(0, 16, 17, (40, 17, 33), hidden, 1, seed=n)
    o, d = np.array([[0.13, -0.37, -2.0]], np.float32), np.array([[0.0, 0.0, 1.0]], np.float32)
    M = int(np.floor(n * np.sqrt(3.0)))
    assert _check(oracle, tree, geo, o, d, M, 5) == n


@pytest.mark.parametrize("activation", ["relu", "tanh", "softplus"])
def test_other_activations(oracle, activation):
    tree, geo, o, d = gpu_scene(2, 8, 9, (32, 9, 32), [64, 64], 200, seed=21, activation=activation)
    _check(oracle, tree, geo, o, d, 9, 0)


@pytest.mark.parametrize("C", [8, 16])
@pytest.mark.parametrize("n", [65, 127, 128, 129, 257])
def test_tile_edges_one_wide_layer(oracle, C, n):
    """As test_tile_edges for one hidden layer of 64 units: two tiles of 64
    samples share a geometry pass and the feature tile."""
    tree, geo, _, _ = gpu_scene(0, C, 17, (40, 17, 33), [64], 1, seed=n)
    o, d = np.array([[0.13, -0.37, -2.0]], np.float32), np.array([[0.0, 0.0, 1.0]], np.float32)
    assert _check(oracle, tree, geo, o, d, int(np.floor(n * np.sqrt(3.0))), 5) == n


# Largest error of one value of the FP32 form: its features, 80 products and
# sums and the activations at a few ulp each (2^-24 of the largest terms), far
# below a feature row taken from another sample.
MAX_TOL = 1e-4


@pytest.mark.parametrize("C", [8, 16])
def test_tiles_of_a_pass_keep_their_features(oracle, C):
    """One hidden layer of 64 units on every SM, several times: density at
    points where every second tile is outside the ROI (no texels to wait for,
    so its warps run ahead) and the projection, each value against the FP64
    oracle."""
    import adaptivetensordf_b200 as ab

    n = 128 * 148 * 6 + 77
    tree, geo, o, d = gpu_scene(1, C, 17, (33, 17, 33), [64], 3000, seed=C)
    slot = geo.leaf_slot.clone()
    slot[tree.active_node_ids[0]] = -1
    geo.leaf_slot = slot
    td, fd, md = oracle_views(tree, geo)
    rng = np.random.default_rng(C)
    pts = rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)
    outside = np.arange(n) // 64 % 2 == 1
    pts[outside] -= 1.0  # the lowest leaf
    pt = torch.from_numpy(pts).cuda()
    node, _ = tree.NodeIdForPositionGPU(pt)
    so = {"global_coordinate": pts, "node_id": node.cpu().numpy(), "weight": np.ones(n, np.float32),
          "ray_index": np.arange(n)}
    ref = oracle.project_forward(fd, md, td, so, n, np.float64).reshape(n)
    segs = oracle.ray_segments(td, o, d, 300)
    ref_img = oracle.project_forward(fd, md, td, oracle.emit_samples(segs, o, d, None), len(o), np.float64).reshape(-1)
    rays = ab.RayList(torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda())
    for _ in range(5):
        with torch.no_grad():
            got = geo.SampleVolumeIndirect(tree, pt, node).cpu().numpy().reshape(n)
            img = geo.ProjectRays(tree, rays, 300, 0).cpu().numpy().reshape(-1)
        assert np.abs(got - ref).max() < MAX_TOL * np.abs(ref).max()
        assert np.abs(img - ref_img).max() < MAX_TOL * np.abs(ref_img).max()
