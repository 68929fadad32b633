"""Tensor-core forward by runs of segments (small calls: planes read from global
memory) against the forward by slot (large calls: planes staged in shared
memory): the same rays projected in one call beyond the line between the two
and in calls on the other side of it, down to a single ray."""

import pytest
import torch

from tests.scene import gpu_scene, rel_err

pytestmark = pytest.mark.gpu

# Both compute a sample's features in FP32 in the same order and round them to
# BF16 for the decoder; a difference in FP32 contraction could move a feature
# by one unit in the last place of BF16 (2^-8 of it).
TOL = 2.0**-8


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


# segments by capacity: 3 * 2^depth + 3 a ray; the line is at 2^18
@pytest.mark.parametrize("C,depth,M", [(16, 4, 24), (16, 3, 3), (24, 3, 24)])
def test_forward_by_runs_equals_by_slot(C, depth, M):
    import adaptivetensordf_b200 as ab

    per = 3 * (1 << depth) + 3
    R = (1 << 18) // per + 301
    L = 16 << depth
    tree, geo, o, d = gpu_scene(depth, C, 17, (L, 17, L), [64, 64], R, seed=depth + C)
    geo.precision = "bf16"
    geo.RefreshLowPrecision()
    o, d = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()

    def project(lo, hi):
        with torch.no_grad():
            return geo.ProjectRays(tree, ab.RayList(o[lo:hi].contiguous(), d[lo:hi].contiguous()), M, 0).reshape(-1)

    whole = project(0, R)
    at, parts = 0, []
    for n in (1, 2, 7, 33, 257, (1 << 18) // per):
        parts.append(project(at, at + n))
        at += n
    assert at <= R
    got = torch.cat(parts)
    ref = whole[:at]
    assert bool((ref > 0).any())
    assert rel_err(got.double().cpu().numpy(), ref.double().cpu().numpy()) < TOL
    assert bool(((got - ref).abs() <= 4 * TOL * ref.abs() + 1e-6 * ref.abs().max()).all())
