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


@pytest.mark.parametrize("shape,S", [((5, 8, 17, 17), 1), ((5, 8, 17, 17), 300), ((5, 8, 17, 17), 361),
                                     ((5, 8, 17, 17), 4000), ((3, 4, 6, 9), 777), ((2, 7, 5, 8), 500),
                                     ((9, 24, 3, 2), 65)])
@pytest.mark.parametrize("layout", ["contiguous", "channels_last", "sliced"])
def test_grid_sample_layouts(oracle, shape, S, layout):
    """The 2D operator's channels-last kernels and the strided ones (channel
    counts of 4 or not, samples around one per 4 texels, other strides): the
    forward and the coordinate gradient bit for bit."""
    import adaptivetensordf_b200 as ab

    rng = np.random.default_rng(S)
    g = rng.normal(size=shape).astype(np.float32)
    idx = rng.integers(0, shape[0], S)
    uv = rng.uniform(-1.2, 1.2, (S, 2)).astype(np.float32)
    go = rng.normal(size=(S, shape[1])).astype(np.float32)
    gt = torch.from_numpy(g).cuda()
    if layout == "channels_last":
        gt = gt.contiguous(memory_format=torch.channels_last)
    elif layout == "sliced":
        gt = torch.cat([gt, gt], 3)[..., :shape[3]]
    gt = gt.requires_grad_(True)
    ut = torch.from_numpy(uv).cuda().requires_grad_(True)
    out = ab.IndirectGridSample2D(gt, torch.from_numpy(idx).cuda(), ut)
    assert np.array_equal(out.detach().cpu().numpy(), oracle.grid_sample2d(g, idx, uv, np.float32))
    gg, gu = torch.autograd.grad(out, [gt, ut], torch.from_numpy(go).cuda())
    assert gg.shape == gt.shape and gg.is_contiguous()
    assert rel_err(gg.cpu().numpy(), oracle.grid_sample2d_bwd(g, idx, uv, go, np.float64)[0]) < REL_TOL
    assert np.array_equal(gu.cpu().numpy(), oracle.grid_sample2d_bwd(g, idx, uv, go, np.float32)[1])


@pytest.mark.parametrize("shape,S", [((1, 16, 256, 1), 5000), ((2, 7, 33, 1), 65), ((2, 7, 33, 1), 66),
                                     ((40, 8, 64, 1), 3000), ((3, 4, 1, 1), 100)])
def test_grid_sample_lines(oracle, shape, S):
    """The 1D operator's gradient summed in shared memory (few entries) and in
    global memory (more than 64 KB, or more entries than samples)."""
    import adaptivetensordf_b200 as ab

    rng = np.random.default_rng(S)
    g = rng.normal(size=shape).astype(np.float32)
    idx = rng.integers(0, shape[0], S)
    u = rng.uniform(-1.1, 1.1, (S, 1)).astype(np.float32)
    go = rng.normal(size=(S, shape[1])).astype(np.float32)
    gt, ut = torch.from_numpy(g).cuda().requires_grad_(True), torch.from_numpy(u).cuda().requires_grad_(True)
    out = ab.IndirectGridSample1D(gt, torch.from_numpy(idx).cuda(), ut)
    assert np.array_equal(out.detach().cpu().numpy(), oracle.grid_sample1d(g, idx, u, np.float32))
    out.backward(torch.from_numpy(go).cuda())
    assert rel_err(gt.grad.cpu().numpy(), oracle.grid_sample1d_bwd(g, idx, u, go, np.float64)[0]) < REL_TOL
    assert np.array_equal(ut.grad.cpu().numpy(), oracle.grid_sample1d_bwd(g, idx, u, go, np.float32)[1])


@pytest.mark.parametrize("M,seed", [(1, 0), (27, 0), (28, 9), (56, 9), (90, 3)])
def test_node_error_segment_lengths(oracle, M, seed):
    """Segments of up to 1, 16, 17, 33 and more samples (16 lanes a segment)."""
    import adaptivetensordf_b200 as ab

    R = 333
    tree, geo, o, d = gpu_scene(2, 8, 9, (32, 9, 32), [32], R, seed=M)
    td, _, _ = oracle_views(tree, geo)
    y = np.random.default_rng(0).uniform(0, 2, (1, R)).astype(np.float32)
    rays = ab.RayList(torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda())
    img, ls, ws = geo.ProjectNodeError(tree, rays, M, seed, torch.from_numpy(y).cuda())
    segs = oracle.ray_segments(td, o, d, M)
    so = oracle.emit_samples(segs, o, d, oracle.jitter_for_segments(seed, segs) if seed else None)
    ls_o, ws_o = oracle.accumulate_loss_per_node(so, (img.cpu().numpy() - y) ** 2, len(td["node_depth"]))
    assert rel_err(ws.cpu().numpy(), ws_o) < 1e-12
    assert rel_err(ls.cpu().numpy(), ls_o) < 1e-9


@pytest.mark.parametrize("C,hidden,op", [(8, [32], "add"), (16, [64, 64], "add"), (8, [64, 64], "cat"), (16, [64], "add"),
                                         (24, [64, 64], "add")])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 3000])
def test_density_without_gradients(oracle, C, hidden, op, n):
    """The one-kernel density (no gradients wanted) against the FP64 oracle:
    points counts around its tiles, leaves outside the ROI, a decoder it does
    not take (24 channels), and a node id out of range."""
    tree, geo, _, _ = gpu_scene(2, C, 9, (32, 9, 32), hidden, 1, seed=n, tensor_op=op)
    slot = geo.leaf_slot.clone()
    slot[tree.active_node_ids[::5]] = -1
    geo.leaf_slot = slot
    td, fd, md = oracle_views(tree, geo)
    pts = np.random.default_rng(n).uniform(-1, 1, (n, 3)).astype(np.float32)
    node, _ = tree.NodeIdForPositionGPU(torch.from_numpy(pts).cuda())
    with torch.no_grad():
        got = geo.SampleVolumeIndirect(tree, torch.from_numpy(pts).cuda(), node)
    assert got.shape == (n, 1) and not got.requires_grad
    # each point as one sample of weight 1 on a ray of its own
    so = {"global_coordinate": pts, "node_id": node.cpu().numpy(), "weight": np.ones(n, np.float32),
          "ray_index": np.arange(n)}
    ref = oracle.project_forward(fd, md, td, so, n, np.float64).reshape(n, 1)
    assert rel_err(got.cpu().numpy(), ref) < REL_TOL
    node[0] = tree.NumNodes()
    with torch.no_grad(), pytest.raises(RuntimeError, match="index out of range"):
        geo.SampleVolumeIndirect(tree, torch.from_numpy(pts).cuda(), node)


def test_decoder_parameters_of_another_rank():
    """Weights [out, in, 1, 1], biases [1, out] and a scalar last bias give
    what [out, in] and [out] give, and gradients of their own shapes."""
    import adaptivetensordf_b200 as ab

    tree, geo, o, d = gpu_scene(2, 8, 9, (32, 9, 32), [32], 300, seed=3)
    rays = ab.RayList(torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda())
    x = torch.randn(77, 8, generator=torch.Generator().manual_seed(1)).cuda()
    w, b = [t.detach() for t in geo.decoder_weight], [t.detach() for t in geo.decoder_bias]
    other = ([t[:, :, None, None] for t in w], [b[0][None], b[1].reshape([])])
    res = []
    for ws, bs in ((w, b), other):
        ws, bs = ([t.clone().requires_grad_(True) for t in v] for v in (ws, bs))
        y = ab.DecodeFeatures(ws, bs, "silu", "softplus", 1.0, x)
        geo.decoder_weight, geo.decoder_bias = ws, bs
        img = geo.ProjectRays(tree, rays, 9, 0)
        out = [y, img]
        for v in (y, img):
            gs = torch.autograd.grad(v, ws + bs, torch.ones_like(v))
            assert [g.shape for g in gs] == [p.shape for p in ws + bs]
            out += gs
        res.append([v.detach().cpu().numpy().reshape(-1) for v in out])
    for got, want in zip(res[1], res[0]):
        assert rel_err(got, want) < REL_TOL


@pytest.mark.parametrize("N,batch_stride", [(1, 8 * 9 * 6 + 5), (3, 8 * 9 * 6)])
@pytest.mark.parametrize("S", [5, 700])
@pytest.mark.parametrize("start", [0, 1])
def test_grid_sample_unaligned_channels_last(oracle, N, batch_stride, S, start):
    """Channels-last grids that start off a 16-byte boundary, and one slot
    whose batch stride is any number (a dimension of one entry)."""
    import adaptivetensordf_b200 as ab

    C, H, W = 8, 9, 6
    rng = np.random.default_rng(S + N)
    g = rng.normal(size=(N, C, H, W)).astype(np.float32)
    idx = rng.integers(0, N, S)
    uv = rng.uniform(-1.2, 1.2, (S, 2)).astype(np.float32)
    go = rng.normal(size=(S, C)).astype(np.float32)
    gt = torch.zeros(start + N * batch_stride, device="cuda").as_strided(
        (N, C, H, W), (batch_stride, 1, C * W, C), start)
    gt = gt.copy_(torch.from_numpy(g)).detach().requires_grad_(True)
    assert gt.is_contiguous(memory_format=torch.channels_last) and gt.data_ptr() % 16 == 4 * start
    ut = torch.from_numpy(uv).cuda().requires_grad_(True)
    out = ab.IndirectGridSample2D(gt, torch.from_numpy(idx).cuda(), ut)
    assert np.array_equal(out.detach().cpu().numpy(), oracle.grid_sample2d(g, idx, uv, np.float32))
    gg, gu = torch.autograd.grad(out, [gt, ut], torch.from_numpy(go).cuda())
    assert rel_err(gg.cpu().numpy(), oracle.grid_sample2d_bwd(g, idx, uv, go, np.float64)[0]) < REL_TOL
    assert np.array_equal(gu.cpu().numpy(), oracle.grid_sample2d_bwd(g, idx, uv, go, np.float32)[1])


def test_grid_sample_without_memory_for_copies():
    """The channels-last copies of a large grid are taken only where they fit:
    with memory for no more than the results the operator reads the grid as it
    is, with the same values."""
    import adaptivetensordf_b200 as ab

    N, C, H, W, S = 1024, 16, 64, 64, 1 << 20  # the grid: 256 MiB, a sample per 4 texels
    gen = torch.Generator(device="cuda").manual_seed(5)
    grid = torch.randn(N, C, H, W, generator=gen, device="cuda").requires_grad_(True)
    idx = torch.randint(0, N, (S,), generator=gen, device="cuda")
    uv = (torch.rand(S, 2, generator=gen, device="cuda") * 2 - 1).requires_grad_(True)
    go = torch.randn(S, C, generator=gen, device="cuda")
    total = torch.cuda.get_device_properties(0).total_memory
    res = []
    for more in (None, (64 + 128, 256 + 64)):  # MiB beyond what is held: out and half a copy; the gradient and a quarter
        out = None
        try:
            for step in range(2):
                torch.cuda.synchronize()
                torch.cuda.empty_cache()
                if more:
                    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (more[step] << 20)) / total)
                if step == 0:
                    out = ab.IndirectGridSample2D(grid, idx, uv)
                else:
                    grads = torch.autograd.grad(out, [grid, uv], go)
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
        res.append([out.detach().cpu()] + [g.cpu() for g in grads])
        del out, grads
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][2], res[1][2])
    assert rel_err(res[1][1].numpy(), res[0][1].numpy()) < REL_TOL


@pytest.mark.parametrize("which", ["position", "plane", "line", "weight", "bias"])
@pytest.mark.parametrize("no_grad", [False, True])
def test_density_refuses_tangents(which, no_grad):
    """A forward-mode tangent is refused (the operators have no jvp), not
    dropped, also where no reverse-mode gradient is wanted."""
    import torch.autograd.forward_ad as fwd

    tree, geo, _, _ = gpu_scene(1, 8, 9, (16, 9, 16), [32], 1)
    pts = torch.rand(50, 3, generator=torch.Generator().manual_seed(2)).cuda()
    node, _ = tree.NodeIdForPositionGPU(pts)
    geo.planes, geo.lines = [t.detach() for t in geo.planes], [t.detach() for t in geo.lines]
    geo.decoder_weight = [t.detach() for t in geo.decoder_weight]
    geo.decoder_bias = [t.detach() for t in geo.decoder_bias]

    def dual(v, i):
        return [fwd.make_dual(t, torch.ones_like(t)) if k == i else t for k, t in enumerate(v)]

    with fwd.dual_level(), torch.set_grad_enabled(not no_grad):
        if which == "position":
            pts = fwd.make_dual(pts, torch.ones_like(pts))
        elif which == "plane":
            geo.planes = dual(geo.planes, 2)
        elif which == "line":
            geo.lines = dual(geo.lines, 1)
        elif which == "weight":
            geo.decoder_weight = dual(geo.decoder_weight, 1)
        else:
            geo.decoder_bias = dual(geo.decoder_bias, 0)
        with pytest.raises(RuntimeError, match="jvp"):
            geo.SampleVolumeIndirect(tree, pts, node)


@pytest.mark.parametrize("dims", [[8, 32, 1], [16, 64, 64, 3], [12, 20, 17], [256, 256, 256, 1]])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
def test_decoder_rows_without_gradient(dims, value):
    """Rows that are not finite and want no gradient leave the weights'
    gradients as they are without them (relu, whose derivative is finite
    everywhere)."""
    import adaptivetensordf_b200 as ab

    S = 333
    g = torch.Generator().manual_seed(sum(dims))
    ws = [torch.randn(b, a, generator=g) * (2.0 / a) ** 0.5 for a, b in zip(dims, dims[1:])]
    bs = [torch.rand(b, generator=g) - 0.5 for b in dims[1:]]
    x, gy = torch.randn(S, dims[0], generator=g), torch.randn(S, dims[-1], generator=g)
    masked = torch.arange(S) % 7 == 3
    gy[masked] = 0.0
    res = []
    for fill in (0.0, value):
        x[masked, : dims[0] // 2] = fill
        leaf = [t.clone().cuda().requires_grad_(True) for t in ws + bs]
        y = ab.DecodeFeatures(leaf[: len(ws)], leaf[len(ws):], "relu", "id", 1.0, x.cuda())
        y.backward(gy.cuda())
        res.append([t.grad.cpu().numpy() for t in leaf])
    for got, want in zip(res[1], res[0]):
        assert rel_err(got, want) < REL_TOL


@pytest.mark.parametrize("S", [50, 7300 * 289 // 18 - 1, 7300 * 289 // 18 + 1])
def test_grid_sample_adjoint_of_a_large_channels_last_grid(oracle, S):
    """Both sides of the line from which a channels-last grid of more than 2 M
    texels takes the channels-last adjoint: a sample per 10 + 2 C texels."""
    import adaptivetensordf_b200 as ab

    shape = (7300, 4, 17, 17)
    rng = np.random.default_rng(S)
    g = rng.normal(size=shape).astype(np.float32)
    idx = rng.integers(0, shape[0], S)
    uv = rng.uniform(-1.2, 1.2, (S, 2)).astype(np.float32)
    go = rng.normal(size=(S, 4)).astype(np.float32)
    gt = torch.from_numpy(g).cuda().contiguous(memory_format=torch.channels_last).requires_grad_(True)
    ut = torch.from_numpy(uv).cuda().requires_grad_(True)
    out = ab.IndirectGridSample2D(gt, torch.from_numpy(idx).cuda(), ut)
    assert np.array_equal(out.detach().cpu().numpy(), oracle.grid_sample2d(g, idx, uv, np.float32))
    gg, gu = torch.autograd.grad(out, [gt, ut], torch.from_numpy(go).cuda())
    assert gg.is_contiguous()
    assert rel_err(gg.cpu().numpy(), oracle.grid_sample2d_bwd(g, idx, uv, go, np.float64)[0]) < REL_TOL
    assert np.array_equal(gu.cpu().numpy(), oracle.grid_sample2d_bwd(g, idx, uv, go, np.float32)[1])


@pytest.mark.parametrize("shape,S", [((2, 7, 33, 1), 4095), ((2, 7, 33, 1), 4096), ((2, 7, 33, 1), 30001),
                                     ((1, 5, 700, 1), 16799), ((1, 5, 700, 1), 16800), ((1, 3, 6000, 1), 144000)])
def test_grid_sample_line_sums(oracle, shape, S):
    """The line gradient's sums on both sides of 4096 samples and 24 an entry
    (shared memory from there on), and lines beyond 64 KB."""
    import adaptivetensordf_b200 as ab

    rng = np.random.default_rng(S)
    g = rng.normal(size=shape).astype(np.float32)
    idx = rng.integers(0, shape[0], S)
    u = rng.uniform(-1.1, 1.1, (S, 1)).astype(np.float32)
    go = rng.normal(size=(S, shape[1])).astype(np.float32)
    gt, ut = torch.from_numpy(g).cuda().requires_grad_(True), torch.from_numpy(u).cuda().requires_grad_(True)
    out = ab.IndirectGridSample1D(gt, torch.from_numpy(idx).cuda(), ut)
    assert np.array_equal(out.detach().cpu().numpy(), oracle.grid_sample1d(g, idx, u, np.float32))
    out.backward(torch.from_numpy(go).cuda())
    # the FP32 oracle's weights: at thousands of entries they are rounded by 1e-4 by definition
    assert rel_err(gt.grad.cpu().numpy(), oracle.grid_sample1d_bwd(g, idx, u, go, np.float32)[0]) < REL_TOL
    assert np.array_equal(ut.grad.cpu().numpy(), oracle.grid_sample1d_bwd(g, idx, u, go, np.float32)[1])
