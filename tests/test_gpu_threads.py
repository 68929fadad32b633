"""Operators called from several host threads with different sizes through the C
ABI (ctypes releases the interpreter lock): a kernel's shared-memory limit
belongs to the kernel, so no call may lower it under another's launch."""

import ctypes as ct
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

CALLS = 3000


def _decoder(capi, dims, S, seed):
    g = torch.Generator().manual_seed(seed)
    ws = [(torch.randn(b, a, generator=g) * (2.0 / a) ** 0.5).cuda() for a, b in zip(dims, dims[1:])]
    bs = [torch.rand(b, generator=g).cuda() for b in dims[1:]]
    m = capi.Mlp()
    m.num_layers = len(ws)
    for i, d in enumerate(dims):
        m.dims[i] = d
    for i in range(len(ws)):
        m.weight[i], m.bias[i] = ws[i].data_ptr(), bs[i].data_ptr()
    m.hidden_activation, m.last_activation, m.softplus_beta = capi.ACT["silu"], capi.ACT["softplus"], 1.0
    x = torch.randn(S, dims[0], generator=g).cuda()
    return m, x, torch.empty(S, dims[-1], device="cuda"), (ws, bs)


def _run(calls):
    """Each call CALLS times in a thread of its own, in step with the others'
    start; the statuses that were not 0."""
    bad, gate = [], threading.Barrier(len(calls))

    def work(call):
        gate.wait()
        bad.extend(s for s in (call() for _ in range(CALLS)) if s != 0)

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    return bad


def test_decoders_of_different_widths():
    from adaptivetensordf_b200 import capi

    L = capi.lib()
    nets = [_decoder(capi, dims, 256, k) for k, dims in enumerate(([16, 64, 64, 1], [64, 96, 96, 1], [8, 32, 1]))]
    streams = [torch.cuda.Stream() for _ in nets]
    torch.cuda.synchronize()

    def call(k):
        m, x, y, _ = nets[k]
        return lambda: L.atdf_mlp_forward(ct.byref(m), capi.ptr(x), 256, capi.ptr(y),
                                          ct.c_void_p(streams[k].cuda_stream))

    alone = []
    for k in range(len(nets)):
        assert call(k)() == 0
        torch.cuda.synchronize()
        alone.append(nets[k][2].clone())
    assert _run([call(k) for k in range(len(nets))]) == []
    assert all(torch.equal(a, n[2]) for a, n in zip(alone, nets))


def test_line_gradients_of_different_lengths():
    from adaptivetensordf_b200 import capi

    L = capi.lib()
    C, S = 4, 24 * 3900  # 24 samples an entry and more: summed in shared memory
    work = []
    for W in (17, 1024, 3900):
        grid, uv, go = torch.randn(1, C, W, 1, device="cuda"), torch.zeros(S, device="cuda"), torch.ones(S, C, device="cuda")
        work.append((W, grid, torch.zeros(S, dtype=torch.int64, device="cuda"), uv, go, torch.zeros_like(grid),
                     torch.zeros(1, dtype=torch.int32, device="cuda"), (ct.c_int64 * 3)(C * W, W, 1), torch.cuda.Stream()))
    torch.cuda.synchronize()

    def call(k):
        W, grid, idx, uv, go, gg, err, stride, st = work[k]
        return lambda: L.atdf_grid_sample1d_backward(capi.ptr(grid), 1, C, W, stride, capi.ptr(idx), capi.ptr(uv), S,
                                                     capi.ptr(go), capi.ptr(gg), None, capi.ptr(err),
                                                     ct.c_void_p(st.cuda_stream))

    assert _run([call(k) for k in range(len(work))]) == []
    for k, w in enumerate(work):  # the middle of the line takes every sample's weights, which sum to 1
        w[5].zero_()
        torch.cuda.synchronize()
        assert call(k)() == 0
        torch.cuda.synchronize()
        assert w[6].item() == 0
        assert torch.equal(w[5].sum((0, 2, 3)), torch.full((C,), float(S), device="cuda"))
