"""The unfused operators' kernels at the sizes where their tiling, vector width
and shared-memory paths can go wrong."""

import numpy as np
import pytest
import torch

from tests.scene import gpu_scene, oracle_views, rel_err

pytestmark = pytest.mark.gpu

REL_TOL = 1e-5  # the FP32 operators' parity tolerance


@pytest.fixture(scope="module")
def oracle():
    from oracle import oracle as O

    return O


def _mlp64(x, ws, bs, hidden, last):
    act = {"silu": torch.nn.functional.silu, "relu": torch.relu, "id": lambda v: v, "tanh": torch.tanh,
           "softplus": lambda v: torch.nn.functional.softplus(v, 2.0)}
    for i, (w, b) in enumerate(zip(ws, bs)):
        x = act[last if i + 1 == len(ws) else hidden](x @ w.t() + b)
    return x


@pytest.mark.parametrize("dims,hidden,last", [
    ([8, 32, 1], "silu", "softplus"), ([16, 64, 64, 1], "silu", "softplus"), ([48, 64, 64, 1], "silu", "softplus"),
    ([12, 48, 3], "relu", "id"), ([7, 5, 2], "tanh", "id"), ([3, 1], "silu", "softplus"),
    ([24, 65, 33, 4], "silu", "id"), ([20, 12, 20, 12], "silu", "tanh"), ([200, 130, 17], "silu", "softplus"),
    ([256, 256, 256, 1], "silu", "softplus"),
])
@pytest.mark.parametrize("S", [1, 33, 64, 129, 5000])
def test_decoder(dims, hidden, last, S):
    """DecodeFeatures and its gradients against torch in FP64: widths around
    the 4-, 16-, 32- and 64-column blocks, several outputs, networks too wide
    for the tile kernels, rows around the tile heights."""
    import adaptivetensordf_b200 as ab

    g = torch.Generator().manual_seed(sum(dims) + S)
    ws = [torch.randn(b, a, generator=g) * (2.0 / a) ** 0.5 for a, b in zip(dims, dims[1:])]
    bs = [torch.rand(b, generator=g) - 0.5 for b in dims[1:]]
    x, gy = torch.randn(S, dims[0], generator=g), torch.randn(S, dims[-1], generator=g)
    cu = [[t.cuda().requires_grad_(True) for t in v] for v in (ws, bs, [x])]
    y = ab.DecodeFeatures(cu[0], cu[1], hidden, last, 2.0, cu[2][0])
    y.backward(gy.cuda())
    ref = [[t.double().requires_grad_(True) for t in v] for v in (ws, bs, [x])]
    y64 = _mlp64(ref[2][0], ref[0], ref[1], hidden, last)
    y64.backward(gy.double())
    assert rel_err(y.detach().cpu().numpy(), y64.detach().numpy()) < REL_TOL
    assert rel_err(cu[2][0].grad.cpu().numpy(), ref[2][0].grad.numpy()) < REL_TOL
    # a layer's weight and bias gradients as one vector: the last bias alone is
    # one sum whose terms cancel, which has no relative accuracy of its own
    for l in range(len(ws)):
        got, want = (np.concatenate([v[k][l].grad.double().cpu().numpy().ravel() for k in (0, 1)]) for v in (cu, ref))
        assert rel_err(got, want) < REL_TOL, f"layer {l}"


@pytest.mark.parametrize("C,op", [(4, "add"), (6, "cat"), (7, "add"), (8, "cat"), (12, "add"), (16, "add"), (24, "cat")])
@pytest.mark.parametrize("beam", [False, True])
def test_field_channels(oracle, C, op, beam):
    """Features and their adjoint through ComputeImage for channel counts with
    8, 4 and 1 channels a thread; beam: rays normal to y, whose samples share
    the entries of the y line."""
    import adaptivetensordf_b200 as ab

    R, M = 300, 9
    tree, geo, o, d = gpu_scene(2, C, 9, (32, 9, 32), [32], R, seed=C, tensor_op=op)
    if beam:
        d[:, 1] = 0.0
        d /= np.linalg.norm(d, axis=1, keepdims=True)
    td, fd, md = oracle_views(tree, geo)
    rays = ab.RayList(torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda())
    s = tree.CreateSamplesForRays(rays, M, False)
    so = {k: getattr(s, k).cpu().numpy() for k in ["global_coordinate", "weight", "ray_index", "node_id"]}
    feat = geo.SampleVolumeIndirect_feature(tree, s.global_coordinate, s.node_id)
    assert np.array_equal(feat.detach().cpu().numpy(),
                          oracle.vm_features(fd, td, so["global_coordinate"], so["node_id"], np.float32))
    img, _, _ = geo.ComputeImage(tree, s, 1, R)
    gi = np.random.default_rng(3).normal(size=(1, R)).astype(np.float32)
    img.backward(torch.from_numpy(gi).cuda())
    gr = oracle.project_backward(fd, md, td, so, R, gi.astype(np.float64), np.float64)
    for m in range(3):
        assert rel_err(geo.planes[m].grad.cpu().numpy(), gr["planes"][m]) < REL_TOL, f"plane {m}"
        assert rel_err(geo.lines[m].grad.cpu().numpy(), gr["lines"][m]) < REL_TOL, f"line {m}"


def test_field_long_lines(oracle):
    """Lines whose gradients do not fit in shared memory go to global memory."""
    import adaptivetensordf_b200 as ab

    R = 200
    tree, geo, o, d = gpu_scene(1, 8, 9, (2500, 9, 1500), [32], R, seed=2)
    td, fd, md = oracle_views(tree, geo)
    s = tree.CreateSamplesForRays(ab.RayList(torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()), 20, False)
    so = {k: getattr(s, k).cpu().numpy() for k in ["global_coordinate", "weight", "ray_index", "node_id"]}
    img, _, _ = geo.ComputeImage(tree, s, 1, R)
    img.backward(torch.ones_like(img))
    # the FP32 oracle: at 2500 entries the tap weights themselves are rounded by 1e-4
    gr = oracle.project_backward(fd, md, td, so, R, np.ones((1, R)), np.float32)
    for m in range(3):
        assert rel_err(geo.lines[m].grad.cpu().numpy(), gr["lines"][m]) < REL_TOL, f"line {m}"
