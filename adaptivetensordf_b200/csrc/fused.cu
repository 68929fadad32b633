// Fused leaf-major forward projection and its hand-written adjoint (FP32,
// CUDA cores) for sm_100a.
//
// One training step of the reference runs CreateSamplesForRays, then
// SampleVolumeIndirect (six gathers + products), DecodeFeatures (FCBlock +
// softplus) and IntegrateSamplesXRay (index_add_), materialising every [S, .]
// intermediate in HBM, and autograd replays them backwards with atomics into
// the factor-grid gradients (hyperacorn/csrc/geometry/geometry.cpp:828-1019,
// geometry_tensor_qo.cpp:257-380, modules/IndirectGridSample2D.cu:175-393).
//
// Here:
//  1. ray_segments (sampler.cu) lists every ray's leaf segments in canonical
//     order; no per-sample array is ever written.
//  2. Segments are bucketed by plane slot and cut into work items of at most
//     kSegItem segments.
//  3. A persistent kernel takes items from a queue and runs each item's
//     samples through features, decoder and per-segment sums (FP32:
//     fused_simt.cuh; BF16 on the tensor cores: fused_tc.cu, fused_tc24.cu).
//  4. A per-ray pass adds the segment partials in t order.
//  The backward kernels recompute each sample (no stored activations).

#include <algorithm>
#include <mutex>
#include <vector>

#include "fused_simt.cuh"

namespace atdf {

// The segment pass's scratch: the kept hits in the workspace's bucket and
// segment-partial arrays (R * per entries, idle until the segments exist), the
// block sums (2 R bytes) in the item queue's (at least 6 R).
static int launch_ray_segments_ws(const atdf_tree_t& tree, const float* origin, const float* dir, int64_t R, int M,
                                  const Ws& w, int32_t* err, cudaStream_t st)
{
    SegScratch sc;
    sc.kept_lo = reinterpret_cast<uint32_t*>(w.bucket);
    sc.kept_hi = reinterpret_cast<uint32_t*>(w.seg_partial);
    sc.kept_per = R > 0 ? w.cap / R : 0;
    sc.block_sums = reinterpret_cast<longlong2*>(w.item_queue);
    return launch_ray_segments(tree, origin, dir, R, M, ws_segments(w), err, st, &sc);
}

// ---------------------------------------------------------------------------
// bucketing by plane slot
// ---------------------------------------------------------------------------
// Counts the segments of each slot; a segment keeps its rank there (in the
// segment partials, idle until the forward). A segment whose node id or plane
// slot is out of range sets the index bit and joins the out-of-ROI bucket
// (zero features, no gradient).
__device__ __forceinline__ void count_segments(const Ws& w, const atdf_field_t& f, int64_t num_nodes, int32_t* err,
                                               int64_t first, int64_t step)
{
    const int64_t nseg = min(w.totals[0], w.cap);
    int32_t* rank = reinterpret_cast<int32_t*>(w.seg_partial);
    for (int64_t i = first; i < nseg; i += step) {
        const int32_t nd = w.node[i];
        if (nd < 0 || nd >= num_nodes || f.leaf_slot[nd] >= f.num_slots) set_err(err, ATDF_DEVERR_INDEX);
        rank[i] = atomicAdd(&w.slot_offset[seg_slot(f, num_nodes, nd)], 1);
    }
}

__device__ __forceinline__ void scatter_segments(const Ws& w, const atdf_field_t& f, int64_t num_nodes, int64_t first,
                                                 int64_t step)
{
    const int64_t nseg = min(w.totals[0], w.cap);
    const int32_t* rank = reinterpret_cast<const int32_t*>(w.seg_partial);
    for (int64_t i = first; i < nseg; i += step) {
        const int64_t s = seg_slot(f, num_nodes, w.node[i]);
        w.bucket[w.slot_offset[s] + rank[i]] = (int32_t)i;
    }
}

__global__ void bucket_count_kernel(Ws w, atdf_field_t f, int64_t num_nodes, int32_t* err)
{
    count_segments(w, f, num_nodes, err, (int64_t)blockIdx.x * blockDim.x + threadIdx.x,
                   (int64_t)gridDim.x * blockDim.x);
}

__global__ void bucket_scatter_kernel(Ws w, atdf_field_t f, int64_t num_nodes)
{
    scatter_segments(w, f, num_nodes, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}

// From the slots' segment counts, in one block and launch (each step is a few
// microseconds of latency on a few thousand slots; as five kernels they took
// 40 us a call):
//  * slot offsets (exclusive scan) and items per slot: equal shares of at most
//    kSegItem segments. items > 0 (the FP32 kernels): also small enough that
//    the call makes about that many items, but not below kMinItem segments;
//  * the slot queue's order (slot_order): slots by descending segment count,
//    so that the largest start first and the kernels' tail holds the smallest
//    (longest-processing-time-first), a counting sort on min(count / 2, 255);
//  * the item queue: each slot's items in the slot queue's order;
//    counters[4] = the number of items.
// SMALL (at most kSmallCap segments by capacity: small calls, whose time is
// launches): the block also clears, counts and scatters, in place of a memset
// and the two bucket kernels.
constexpr int64_t kSmallCap = 16384;

template <bool SMALL>
__global__ void __launch_bounds__(1024) plan_kernel(Ws w, int items, atdf_field_t f, int64_t num_nodes, int32_t* err)
{
    __shared__ int warp_sum[32];
    __shared__ int hist[256];
    __shared__ int s_base;
    const int n = (int)w.nslot + 1;  // plane slots and the out-of-ROI bucket
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (SMALL) {
        for (int i = tid; i < n; i += 1024) w.slot_offset[i] = 0;
        if (tid < 8) w.counters[tid] = 0;
        __syncthreads();
        count_segments(w, f, num_nodes, err, tid, 1024);
        __syncthreads();
    }
    int per = kSegItem;
    if (items > 0) per = (int)max((int64_t)kMinItem, min((int64_t)kSegItem, min(w.totals[0], w.cap) / items));
    for (int i = tid; i < 256; i += 1024) hist[i] = 0;
    if (tid == 0) s_base = 0;
    __syncthreads();
    for (int s = tid; s < n; s += 1024) {
        const int cnt = w.slot_offset[s];
        w.item_offset[s] = (cnt + per - 1) / per;
        atomicAdd(&hist[255 - min(cnt >> 1, 255)], 1);
    }
    if (tid == 0) w.slot_offset[n] = w.item_offset[n] = 0;
    __syncthreads();
    if (wid == 0) {  // exclusive scan of the 256 bins, 8 a lane
        int v[8], sum = 0;
        for (int k = 0; k < 8; ++k) {
            v[k] = hist[8 * lane + k];
            sum += v[k];
        }
        int incl = sum;
        for (int off = 1; off < 32; off <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += x;
        }
        int run = incl - sum;
        for (int k = 0; k < 8; ++k) {
            hist[8 * lane + k] = run;
            run += v[k];
        }
    }
    __syncthreads();
    for (int s = tid; s < n; s += 1024) w.slot_order[atomicAdd(&hist[255 - min(w.slot_offset[s] >> 1, 255)], 1)] = s;
    __syncthreads();
    // the items in the order of the queue, before the scan of their counts
    for (int c0 = 0; c0 < n; c0 += 1024) {
        const int q = c0 + tid;
        int sl = -1, ni = 0;
        if (q < n) {
            sl = w.slot_order[q];
            ni = w.item_offset[sl];
        }
        int incl = ni;
        for (int off = 1; off < 32; off <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += x;
        }
        if (lane == 31) warp_sum[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            int v = warp_sum[lane];
            for (int off = 1; off < 32; off <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, v, off);
                if (lane >= off) v += x;
            }
            warp_sum[lane] = v;  // inclusive over warps
        }
        __syncthreads();
        const int pos = s_base + (wid > 0 ? warp_sum[wid - 1] : 0) + incl - ni;
        for (int i = 0; i < ni; ++i) w.item_queue[pos + i] = make_int2(sl, i);
        __syncthreads();
        if (tid == 0) s_base += warp_sum[31];
        __syncthreads();
    }
    if (tid == 0) w.counters[4] = s_base;
    block_scan_exclusive<int32_t>(w.slot_offset, n + 1, nullptr, warp_sum);
    block_scan_exclusive<int32_t>(w.item_offset, n + 1, nullptr, warp_sum);
    if (SMALL) scatter_segments(w, f, num_nodes, tid, 1024);
}

// Zeroes the plane gradients of the slots that no segment touches; the
// tensor-core backward writes every touched slot's gradient itself.
__global__ void zero_untouched_slots_kernel(Ws w, atdf_field_grad_t g, atdf_field_t f)
{
    for (int64_t s = blockIdx.x; s < w.nslot; s += gridDim.x) {
        if (w.item_offset[s + 1] > w.item_offset[s]) continue;
        for (int m = 0; m < 3; ++m) {
            const int64_t pf = (int64_t)f.plane_h[m] * f.plane_w[m] * f.channels;
            float* dst = g.plane[m] + s * pf;
            for (int64_t i = threadIdx.x; i < pf; i += blockDim.x) dst[i] = 0.0f;
        }
    }
}

// End of the FP32 adjoint: the sum of the line gradients' copies (n_rep > 0)
// and the last bias' gradient, both in FP64 with one rounding at the end. The
// last bias is one sum over every sample whose terms largely cancel.
__global__ void adjoint_end_kernel(const float* __restrict__ rep, int n_rep, int n, int n0, int n1, float* g0,
                                   float* g1, float* g2, const double* __restrict__ last_sum, float* last_bias)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *last_bias = (float)*last_sum;
    if (n_rep == 0 || i >= n) return;
    double acc = 0.0;
    for (int r = 0; r < n_rep; ++r) acc += (double)rep[(int64_t)r * n + i];
    (i < n0 ? g0[i] : i < n0 + n1 ? g1[i - n0] : g2[i - n0 - n1]) = (float)acc;
}

// Per-ray sum of the segment partials, in segment (t) order.
__global__ void ray_reduce_kernel(Ws w, int64_t R, float* image)
{
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= R) return;
    const int64_t b = w.ray_seg_offset[r], e = w.ray_seg_offset[r + 1];
    float acc = 0.0f;
    if (e <= w.cap)
        for (int64_t s = b; s < e; ++s) acc = __fadd_rn(acc, w.seg_partial[s]);
    image[r] = acc;
}

// ---------------------------------------------------------------------------
// node-error scoring: 16 lanes per segment, a lane per sample, FP64 sums. The
// weights come from the neighbours' t, which the neighbouring lanes hold (a
// warp per segment with three t per sample was bound by its instructions: 127
// us for 319 k segments of 11 samples).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) node_error_kernel(Ws w, const float* __restrict__ prl, int cout, int64_t R,
                                                         uint64_t seed, double* ls, double* wsum, int64_t num_nodes,
                                                         int32_t* err)
{
    constexpr int G = 16;
    const int lane = threadIdx.x & (G - 1);
    const int64_t nseg = min(w.totals[0], w.cap);
    const int64_t groups = (int64_t)gridDim.x * blockDim.x / G;
    // every lane of a warp makes the same number of rounds (full-warp shuffles)
    for (int64_t s0 = 0; s0 < nseg; s0 += groups) {
        const int64_t sidx = s0 + ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
        const bool have = sidx < nseg;
        const int n = have ? w.nsamp[sidx] : 0, node = have ? w.node[sidx] : 0, r = have ? w.ray[sidx] : 0;
        const float tmin = have ? w.tmin[sidx] : 0.0f, tmax = have ? w.tmax[sidx] : 0.0f;
        const float step = n > 0 ? __fdiv_rn(__fsub_rn(tmax, tmin), (float)n) : 0.0f;
        auto t_of = [&](int j) { return sample_t_step(tmin, step, j, sample_a(nullptr, 0, seed, r, node, j)); };
        int most = n;  // rounds of the warp's longer segment
        most = max(most, __shfl_xor_sync(0xffffffffu, most, G));
        double acc = 0.0;
        for (int j0 = 0; j0 < most; j0 += G) {
            const int j = j0 + lane;
            const float t = j < n ? t_of(j) : 0.0f;
            float tp = __shfl_up_sync(0xffffffffu, t, 1, G), tn = __shfl_down_sync(0xffffffffu, t, 1, G);
            if (lane == 0 && j > 0 && j < n) tp = t_of(j - 1);
            if (lane == G - 1 && j < n - 1) tn = t_of(j + 1);
            if (j < n) acc += (double)sample_w(tmin, tmax, n, j, tp, t, tn);
        }
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
        if (lane == 0 && have) {
            if (node < 0 || node >= num_nodes) {
                set_err(err, ATDF_DEVERR_INDEX);
                continue;
            }
            double l = 0.0;
            for (int c = 0; c < cout; ++c) l += (double)prl[c * R + r];
            l /= (double)cout;
            atomicAdd(&ls[node], l * acc);
            atomicAdd(&wsum[node], acc);
        }
    }
}

// ---------------------------------------------------------------------------
// dispatch
// ---------------------------------------------------------------------------
using KernelFn = void (*)(FusedParams);

using PointsFn = void (*)(FusedParams, simt::PointArgs);

struct Variant {
    int C, mode, H, NH;
    KernelFn fwd, bwd;
    PointsFn points;
    int (*smem)(bool);
};

template <int C, int MODE, int H, int NH>
static int smem_bytes(bool bwd)
{
    return (bwd ? simt::Smem<C, MODE, H, NH, true>::total : simt::Smem<C, MODE, H, NH, false>::total) * 4;
}

// Largest total size (floats) of a slot's three planes that the FP32 form
// takes: what fits in 227 KB of shared memory beside a 32-sample tile, for the
// adjoint together with the gradients. The kernels no longer stage planes, but
// a caller that was refused a size still is.
static int plane_limit(int C, int F, int H, int NH, bool bwd)
{
    const int n = bwd ? 2 : 1, two = NH == 2;
    int fixed = n * F * H + two * (n * H * H + H) + 2 * H + 4 + n * F * 32 + 4 * 32 + kSegTabFloats;
    fixed += bwd ? 3 * 64 * C + (3 + 2 * two) * H * 32 : (1 + two) * H * 32;
    return (232448 / 4 - fixed) / n;
}

#define ATDF_VARIANT(C, M, H, NH) \
    {C, M, H, NH, simt::forward_kernel<C, M, H, NH>, simt::backward_kernel<C, M, H, NH>, \
     simt::points_kernel<C, M, H, NH>, smem_bytes<C, M, H, NH>}

static const Variant kVariants[] = {
    ATDF_VARIANT(8, 0, 32, 1),  ATDF_VARIANT(8, 0, 64, 1),  ATDF_VARIANT(8, 0, 64, 2),
    ATDF_VARIANT(16, 0, 32, 1), ATDF_VARIANT(16, 0, 64, 1), ATDF_VARIANT(16, 0, 64, 2),
    ATDF_VARIANT(8, 1, 64, 2),  ATDF_VARIANT(8, 1, 32, 1),
};

static const Variant* find_variant(const atdf_field_t* f, const atdf_mlp_t* m)
{
    const int nh = m->num_layers - 1;
    if (nh < 1 || nh > 2 || m->dims[m->num_layers] != 1) return nullptr;
    const int H = m->dims[1];
    if (nh == 2 && m->dims[2] != H) return nullptr;
    const int F = f->mode ? 3 * f->channels : f->channels;
    if (m->dims[0] != F) return nullptr;
    for (const Variant& v : kVariants)
        if (v.C == f->channels && v.mode == f->mode && v.H == H && v.NH == nh) return &v;
    return nullptr;
}

// Work items that the FP32 kernels aim at per call (two to three blocks an SM
// take them): few items leave blocks idle, many small ones pay the item set-up.
constexpr int kSimtItems = 4 * 148;
constexpr int kLineRep = 64;  // most copies of the line gradients in the FP32 adjoint

static int max_smem_optin()
{
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return v;
}

static int prepare(const atdf_tree_t* tree, const atdf_field_t* field, const atdf_mlp_t* mlp, const float* origin,
                   const float* dir, int64_t R, void* workspace, size_t ws_bytes, FusedParams& p,
                   const Variant*& var)
{
    if (!tree || !field || !mlp || !workspace || R < 0 || (R > 0 && (!origin || !dir)))
        return ATDF_ERR_INVALID_ARGUMENT;
    if (!field->leaf_slot) return ATDF_ERR_INVALID_ARGUMENT;
    var = nullptr;
    if (field->dtype == ATDF_BF16) {
        if (!tc_supported(field, mlp)) return ATDF_ERR_UNSUPPORTED;
    } else if (field->dtype == ATDF_F32) {
        var = find_variant(field, mlp);
        if (!var) return ATDF_ERR_UNSUPPORTED;
    } else {
        return ATDF_ERR_UNSUPPORTED;
    }
    for (int l = 0; l < mlp->num_layers; ++l)
        if (!mlp->weight[l] || !mlp->bias[l]) return ATDF_ERR_INVALID_ARGUMENT;
    // The 16-channel BF16 tensor-core kernels keep each plane in shared
    // memory with rows padded to a pitch of 2 mod 4 texels (texel = 16
    // channels = 32 bytes): the four corners of a bilinear footprint then
    // have texel indices of all four residues mod 4 and fill distinct bank
    // groups. The 24-channel ones keep the planes unpadded.
    int off = 0, goff = 0;
    for (int m = 0; m < 3; ++m) {
        if (!field->plane[m] || !field->line[m] || ((uintptr_t)field->plane[m] & 15) ||
            ((uintptr_t)field->line[m] & 15))
            return ATDF_ERR_UNSUPPORTED;
        const int W = field->plane_w[m];
        p.plane_pitch[m] = (field->dtype == ATDF_BF16 && field->channels == 16) ? W + ((2 - W) & 3) : W;
        p.plane_off[m] = off;
        off += field->plane_h[m] * p.plane_pitch[m] * field->channels;
        p.gplane_off[m] = goff;
        goff += field->plane_h[m] * W * field->channels;
    }
    p.plane_off[3] = off;
    p.gplane_off[3] = goff;
    p.roi_inv = pow2_reciprocal(field->roi_max[0] - field->roi_min[0]);
    const size_t need = ws_layout(R, tree->max_depth, field->num_slots, nullptr, nullptr);
    if (ws_bytes < need) return ATDF_ERR_WORKSPACE;
    ws_layout(R, tree->max_depth, field->num_slots, (char*)workspace, &p.ws);
    p.tree = *tree;
    p.field = *field;
    p.mlp = *mlp;
    p.origin = origin;
    p.dir = dir;
    p.R = R;
    p.grad_image = nullptr;
    p.xt = nullptr;
    p.xw = nullptr;
    p.bins = nullptr;
    p.line_rep = 0;
    return ATDF_OK;
}

// What the device's limits say about a kernel: blocks per SM and the shared
// memory carve-out (percent) they need, the rest of the L1 holding texels. Asked
// once per kernel and device; the answers depend on nothing else.
struct LaunchShape {
    const void* fn;
    int dev, sms, per, carveout;
};

static int launch_shape(const void* fn, int smem, LaunchShape& out)
{
    static std::mutex lock;
    static std::vector<LaunchShape> known;
    int dev = 0;
    ATDF_CUDA_TRY(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> g(lock);
        for (const LaunchShape& k : known)
            if (k.fn == fn && k.dev == dev) {
                out = k;
                return ATDF_OK;
            }
    }
    int per_sm = 0;
    out.fn = fn;
    out.dev = dev;
    ATDF_CUDA_TRY(cudaDeviceGetAttribute(&out.sms, cudaDevAttrMultiProcessorCount, dev));
    ATDF_CUDA_TRY(cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    ATDF_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       (int)cudaSharedmemCarveoutMaxShared));
    ATDF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&out.per, fn, simt::kThreads, smem));
    if (out.per < 1) return ATDF_ERR_UNSUPPORTED;
    out.carveout = std::min(100, (int)((int64_t)out.per * (smem + 1536) * 100 / per_sm) + 1);  // 1 KB a block is the system's
    std::lock_guard<std::mutex> g(lock);
    known.push_back(out);
    return ATDF_OK;
}

static int launch_persistent(KernelFn fn, int smem, const FusedParams& p, cudaStream_t st)
{
    if (smem > max_smem_optin()) return ATDF_ERR_UNSUPPORTED;
    ATDF_CUDA_TRY(cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    LaunchShape k;
    if (const int e = launch_shape((const void*)fn, smem, k)) return e;
    ATDF_CUDA_TRY(cudaFuncSetAttribute((const void*)fn, cudaFuncAttributePreferredSharedMemoryCarveout, k.carveout));
    fn<<<k.sms * k.per, simt::kThreads, smem, st>>>(p);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}


// Forward projection. compute_segments: derive the ray/leaf segments (and the
// uniform per-node sample counts) into the workspace; otherwise use the
// segments already there (atdf_project_segments) with caller-placed samples.
static int project_forward(const atdf_tree_t* tree, const atdf_field_t* field, const atdf_mlp_t* mlp,
                           const float* ray_origin, const float* ray_direction, int64_t num_rays,
                           int32_t max_samples_per_node, uint64_t jitter_seed, bool compute_segments,
                           const float* xt, const float* xw, float* bins, float* image, void* workspace,
                           size_t workspace_bytes, int32_t* dev_error, cudaStream_t s)
{
    FusedParams p;
    const Variant* var = nullptr;
    int st = prepare(tree, field, mlp, ray_origin, ray_direction, num_rays, workspace, workspace_bytes, p, var);
    if (st != ATDF_OK) return st;
    if (var && p.plane_off[3] > plane_limit(var->C, mlp->dims[0], var->H, var->NH, false)) return ATDF_ERR_UNSUPPORTED;
    if (!image) return ATDF_ERR_INVALID_ARGUMENT;
    if (num_rays >= ((int64_t)1 << 31)) return ATDF_ERR_UNSUPPORTED;
    p.seed = jitter_seed;
    p.err = dev_error;
    p.xt = xt;
    p.xw = xw;
    p.bins = bins;
    const Ws& w = p.ws;
    if (compute_segments) {
        st = launch_ray_segments_ws(*tree, ray_origin, ray_direction, num_rays, max_samples_per_node, w, dev_error,
                                    s);
        if (st != ATDF_OK) return st;
    }
    if (bins) ATDF_CUDA_TRY(cudaMemsetAsync(bins, 0, (size_t)w.cap * kBins * sizeof(float), s));
    const int items = var ? kSimtItems : 0;
    if (w.cap <= kSmallCap) {
        plan_kernel<true><<<1, 1024, 0, s>>>(w, items, *field, tree->num_nodes, dev_error);
        ATDF_LAUNCH_CHECK();
    } else {
        // counters and slot counts lie side by side
        ATDF_CUDA_TRY(cudaMemsetAsync(w.counters, 0, 256 + (w.nslot + 2) * 4, s));
        bucket_count_kernel<<<592, 256, 0, s>>>(w, *field, tree->num_nodes, dev_error);
        ATDF_LAUNCH_CHECK();
        plan_kernel<false><<<1, 1024, 0, s>>>(w, items, *field, tree->num_nodes, dev_error);
        ATDF_LAUNCH_CHECK();
        bucket_scatter_kernel<<<592, 256, 0, s>>>(w, *field, tree->num_nodes);
        ATDF_LAUNCH_CHECK();
    }
    st = var ? launch_persistent(var->fwd, var->smem(false), p, s) : launch_tc_forward(p, s);
    if (st != ATDF_OK) return st;
    if (num_rays > 0) {
        ray_reduce_kernel<<<(unsigned)div_up(num_rays, 256), 256, 0, s>>>(w, num_rays, image);
        ATDF_LAUNCH_CHECK();
    }
    return ATDF_OK;
}

// Backward (recomputes every sample; reuses the forward's workspace).
static int project_backward(const atdf_tree_t* tree, const atdf_field_t* field, const atdf_mlp_t* mlp,
                            const float* ray_origin, const float* ray_direction, int64_t num_rays,
                            uint64_t jitter_seed, const float* xt, const float* xw, const float* grad_image,
                            const atdf_field_grad_t* grad_field, const atdf_mlp_grad_t* grad_mlp, void* workspace,
                            size_t workspace_bytes, int32_t* dev_error, cudaStream_t s)
{
    FusedParams p;
    const Variant* var = nullptr;
    int st = prepare(tree, field, mlp, ray_origin, ray_direction, num_rays, workspace, workspace_bytes, p, var);
    if (st != ATDF_OK) return st;
    if (var && p.plane_off[3] > plane_limit(var->C, mlp->dims[0], var->H, var->NH, true)) return ATDF_ERR_UNSUPPORTED;
    if (!grad_image || !grad_field || !grad_mlp) return ATDF_ERR_INVALID_ARGUMENT;
    for (int m = 0; m < 3; ++m)
        if (!grad_field->plane[m] || !grad_field->line[m] || ((uintptr_t)grad_field->plane[m] & 15))
            return ATDF_ERR_INVALID_ARGUMENT;
    for (int l = 0; l < mlp->num_layers; ++l)
        if (!grad_mlp->weight[l] || !grad_mlp->bias[l]) return ATDF_ERR_INVALID_ARGUMENT;
    p.seed = jitter_seed;
    p.err = dev_error;
    p.grad_image = grad_image;
    p.gfield = *grad_field;
    p.gmlp = *grad_mlp;
    p.xt = xt;
    p.xw = xw;
    // Line gradients are sums of tens of thousands of samples per entry: each
    // block adds to one of up to kLineRep copies (in the workspace's segment
    // partials, idle after the forward), summed at the end. One shared copy
    // would lose digits to its long running FP32 sums (3e-6 instead of 1e-6
    // relative on 290 k samples) and serialise the reductions on hot entries.
    const int ll[3] = {field->line_len[0] * field->channels, field->line_len[1] * field->channels,
                       field->line_len[2] * field->channels};
    const int64_t n = (int64_t)ll[0] + ll[1] + ll[2];
    if (var) p.line_rep = (int)std::min<int64_t>(kLineRep, p.ws.cap / n);
    for (int m = 0; m < 3; ++m) {
        // the tensor-core backward writes the plane gradient of every slot
        // it touches (zeroing it first) and the rest is zeroed below
        if (var) {
            const size_t pf = (size_t)field->plane_h[m] * field->plane_w[m] * field->channels * field->num_slots;
            ATDF_CUDA_TRY(cudaMemsetAsync(grad_field->plane[m], 0, pf * 4, s));
        }
        if (p.line_rep == 0)
            ATDF_CUDA_TRY(
                cudaMemsetAsync(grad_field->line[m], 0, (size_t)field->line_len[m] * field->channels * 4, s));
    }
    if (!var && p.ws.nslot > 0) {
        zero_untouched_slots_kernel<<<(unsigned)std::min<int64_t>(p.ws.nslot, 592), 256, 0, s>>>(p.ws, *grad_field,
                                                                                                *field);
        ATDF_LAUNCH_CHECK();
    }
    // the decoder's gradients, neighbouring arrays (one flat vector) at once
    float* from = grad_mlp->weight[0];
    float* to = from;
    for (int l = 0; l < mlp->num_layers; ++l) {
        float* part[2] = {grad_mlp->weight[l], grad_mlp->bias[l]};
        const size_t n[2] = {(size_t)mlp->dims[l] * mlp->dims[l + 1], (size_t)mlp->dims[l + 1]};
        for (int k = 0; k < 2; ++k) {
            if (part[k] != to) {
                ATDF_CUDA_TRY(cudaMemsetAsync(from, 0, (to - from) * sizeof(float), s));
                from = to = part[k];
            }
            to += n[k];
        }
    }
    ATDF_CUDA_TRY(cudaMemsetAsync(from, 0, (to - from) * sizeof(float), s));
    ATDF_CUDA_TRY(cudaMemsetAsync(p.ws.counters + 1, 0, 4, s));
    if (!var) return launch_tc_backward(p, s);
    if (p.line_rep > 0) ATDF_CUDA_TRY(cudaMemsetAsync(p.ws.seg_partial, 0, (size_t)p.line_rep * n * 4, s));
    ATDF_CUDA_TRY(cudaMemsetAsync(p.ws.last_sum, 0, sizeof(double), s));
    st = launch_persistent(var->bwd, var->smem(true), p, s);
    if (st != ATDF_OK) return st;
    adjoint_end_kernel<<<p.line_rep > 0 ? (unsigned)div_up(n, 128) : 1, 128, 0, s>>>(
        p.ws.seg_partial, p.line_rep, (int)n, ll[0], ll[1], grad_field->line[0], grad_field->line[1],
        grad_field->line[2], p.ws.last_sum, grad_mlp->bias[mlp->num_layers - 1]);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

}  // namespace atdf

using namespace atdf;

extern "C" {

int atdf_field_density(const atdf_field_t* field, const atdf_mlp_t* mlp, const float* pmin, const float* pmax,
                       int64_t num_nodes, const float* position, const int64_t* node_id, int64_t num_points, float* out,
                       int32_t* dev_error, atdf_stream_t stream)
{
    if (!field || !mlp || !pmin || !pmax || num_points < 0 || (num_points > 0 && (!position || !node_id || !out)) ||
        !field->leaf_slot)
        return ATDF_ERR_INVALID_ARGUMENT;
    const Variant* var = field->dtype == ATDF_F32 ? find_variant(field, mlp) : nullptr;
    if (!var || field->num_slots > INT32_MAX) return ATDF_ERR_UNSUPPORTED;
    for (int l = 0; l < mlp->num_layers; ++l)
        if (!mlp->weight[l] || !mlp->bias[l]) return ATDF_ERR_INVALID_ARGUMENT;
    for (int m = 0; m < 3; ++m)
        if (!field->plane[m] || !field->line[m] || ((uintptr_t)field->plane[m] & 15) || ((uintptr_t)field->line[m] & 15))
            return ATDF_ERR_UNSUPPORTED;
    if (num_points == 0) return ATDF_OK;
    FusedParams p = {};
    p.field = *field;
    p.mlp = *mlp;
    p.tree.node_position_min = pmin;
    p.tree.node_position_max = pmax;
    p.tree.num_nodes = num_nodes;
    p.err = dev_error;
    const int smem = var->smem(false);
    if (smem > max_smem_optin()) return ATDF_ERR_UNSUPPORTED;
    ATDF_CUDA_TRY(cudaFuncSetAttribute((const void*)var->points, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    LaunchShape k;
    if (const int e = launch_shape((const void*)var->points, smem, k)) return e;
    ATDF_CUDA_TRY(
        cudaFuncSetAttribute((const void*)var->points, cudaFuncAttributePreferredSharedMemoryCarveout, k.carveout));
    const int64_t tiles = div_up(num_points, simt::kGeo);
    var->points<<<(unsigned)std::min<int64_t>(tiles, (int64_t)k.sms * k.per), simt::kThreads, smem,
                  (cudaStream_t)stream>>>(p, simt::PointArgs{position, node_id, num_points, out});
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

int atdf_project_workspace_size(int64_t num_rays, int32_t max_depth, int32_t ns, int64_t num_slots,
                                int32_t out_channels, size_t* bytes)
{
    if (!bytes || num_rays < 0 || max_depth < 0 || num_slots < 0 || (ns != 4 && ns != 8) || out_channels != 1)
        return ATDF_ERR_INVALID_ARGUMENT;
    *bytes = ws_layout(num_rays, max_depth, num_slots, nullptr, nullptr);
    return ATDF_OK;
}

int atdf_project_forward(const atdf_tree_t* tree, const atdf_field_t* field, const atdf_mlp_t* mlp,
                         const float* ray_origin, const float* ray_direction, int64_t num_rays,
                         int32_t max_samples_per_node, uint64_t jitter_seed, float* image, void* workspace,
                         size_t workspace_bytes, int32_t* dev_error, atdf_stream_t stream)
{
    return project_forward(tree, field, mlp, ray_origin, ray_direction, num_rays, max_samples_per_node, jitter_seed,
                           true, nullptr, nullptr, nullptr, image, workspace, workspace_bytes, dev_error,
                           (cudaStream_t)stream);
}

int atdf_project_forward_segmented(const atdf_tree_t* tree, const atdf_field_t* field, const atdf_mlp_t* mlp,
                                   const float* ray_origin, const float* ray_direction, int64_t num_rays,
                                   uint64_t jitter_seed, float* image, void* workspace, size_t workspace_bytes,
                                   int32_t* dev_error, atdf_stream_t stream)
{
    return project_forward(tree, field, mlp, ray_origin, ray_direction, num_rays, 0, jitter_seed, false, nullptr,
                           nullptr, nullptr, image, workspace, workspace_bytes, dev_error, (cudaStream_t)stream);
}

int atdf_project_forward_binned(const atdf_tree_t* tree, const atdf_field_t* field, const atdf_mlp_t* mlp,
                                const float* ray_origin, const float* ray_direction, int64_t num_rays,
                                int32_t max_samples_per_node, uint64_t jitter_seed, float* image, float* seg_bins,
                                void* workspace, size_t workspace_bytes, int32_t* dev_error, atdf_stream_t stream)
{
    if (!seg_bins) return ATDF_ERR_INVALID_ARGUMENT;
    return project_forward(tree, field, mlp, ray_origin, ray_direction, num_rays, max_samples_per_node, jitter_seed,
                           true, nullptr, nullptr, seg_bins, image, workspace, workspace_bytes, dev_error,
                           (cudaStream_t)stream);
}

int atdf_project_segments(const atdf_tree_t* tree, const float* ray_origin, const float* ray_direction,
                          int64_t num_rays, int32_t max_samples_per_node, int64_t num_slots, void* workspace,
                          size_t workspace_bytes, atdf_segments_t* view, int32_t* dev_error, atdf_stream_t stream)
{
    if (!tree || !workspace || !view || num_rays < 0 || num_slots < 0 ||
        (num_rays > 0 && (!ray_origin || !ray_direction)))
        return ATDF_ERR_INVALID_ARGUMENT;
    if (num_rays >= ((int64_t)1 << 31)) return ATDF_ERR_UNSUPPORTED;
    const size_t need = ws_layout(num_rays, tree->max_depth, num_slots, nullptr, nullptr);
    if (workspace_bytes < need) return ATDF_ERR_WORKSPACE;
    Ws w;
    ws_layout(num_rays, tree->max_depth, num_slots, (char*)workspace, &w);
    *view = ws_segments(w);
    return launch_ray_segments_ws(*tree, ray_origin, ray_direction, num_rays, max_samples_per_node, w, dev_error,
                                  (cudaStream_t)stream);
}

int atdf_project_segment_view(int64_t num_rays, int32_t max_depth, int64_t num_slots, void* workspace,
                              size_t workspace_bytes, atdf_segments_t* view)
{
    if (!workspace || !view || num_rays < 0 || max_depth < 0 || num_slots < 0) return ATDF_ERR_INVALID_ARGUMENT;
    const size_t need = ws_layout(num_rays, max_depth, num_slots, nullptr, nullptr);
    if (workspace_bytes < need) return ATDF_ERR_WORKSPACE;
    Ws w;
    ws_layout(num_rays, max_depth, num_slots, (char*)workspace, &w);
    *view = ws_segments(w);
    return ATDF_OK;
}

int atdf_project_forward_samples(const atdf_tree_t* tree, const atdf_field_t* field, const atdf_mlp_t* mlp,
                                 const float* ray_origin, const float* ray_direction, int64_t num_rays,
                                 const float* sample_t, const float* sample_w, float* image, void* workspace,
                                 size_t workspace_bytes, int32_t* dev_error, atdf_stream_t stream)
{
    if (num_rays > 0 && (!sample_t || !sample_w)) return ATDF_ERR_INVALID_ARGUMENT;
    return project_forward(tree, field, mlp, ray_origin, ray_direction, num_rays, 0, 0, false, sample_t, sample_w,
                           nullptr, image, workspace, workspace_bytes, dev_error, (cudaStream_t)stream);
}

int atdf_project_backward(const atdf_tree_t* tree, const atdf_field_t* field, const atdf_mlp_t* mlp,
                          const float* ray_origin, const float* ray_direction, int64_t num_rays,
                          int32_t max_samples_per_node, uint64_t jitter_seed, const float* grad_image,
                          const atdf_field_grad_t* grad_field, const atdf_mlp_grad_t* grad_mlp, void* workspace,
                          size_t workspace_bytes, int32_t* dev_error, atdf_stream_t stream)
{
    (void)max_samples_per_node;
    return project_backward(tree, field, mlp, ray_origin, ray_direction, num_rays, jitter_seed, nullptr, nullptr,
                            grad_image, grad_field, grad_mlp, workspace, workspace_bytes, dev_error,
                            (cudaStream_t)stream);
}

int atdf_project_backward_samples(const atdf_tree_t* tree, const atdf_field_t* field, const atdf_mlp_t* mlp,
                                  const float* ray_origin, const float* ray_direction, int64_t num_rays,
                                  const float* sample_t, const float* sample_w, const float* grad_image,
                                  const atdf_field_grad_t* grad_field, const atdf_mlp_grad_t* grad_mlp,
                                  void* workspace, size_t workspace_bytes, int32_t* dev_error, atdf_stream_t stream)
{
    if (num_rays > 0 && (!sample_t || !sample_w)) return ATDF_ERR_INVALID_ARGUMENT;
    return project_backward(tree, field, mlp, ray_origin, ray_direction, num_rays, 0, sample_t, sample_w, grad_image,
                            grad_field, grad_mlp, workspace, workspace_bytes, dev_error, (cudaStream_t)stream);
}

int atdf_project_node_error(const atdf_tree_t* tree, const float* ray_origin, const float* ray_direction,
                            int64_t num_rays, int32_t max_samples_per_node, uint64_t jitter_seed,
                            const float* per_ray_loss, int32_t out_channels, double* loss_sum, double* weight_sum,
                            void* workspace, size_t workspace_bytes, int32_t* dev_error, atdf_stream_t stream)
{
    (void)ray_origin;
    (void)ray_direction;
    (void)max_samples_per_node;
    if (!tree || !per_ray_loss || !loss_sum || !weight_sum || !workspace || out_channels <= 0 || num_rays < 0)
        return ATDF_ERR_INVALID_ARGUMENT;
    Ws w;
    // the slot count does not move the segment arrays; any value gives them
    const size_t need = ws_layout(num_rays, tree->max_depth, 0, nullptr, nullptr);
    if (workspace_bytes < need) return ATDF_ERR_WORKSPACE;
    ws_layout(num_rays, tree->max_depth, 0, (char*)workspace, &w);
    cudaStream_t s = (cudaStream_t)stream;
    ATDF_CUDA_TRY(cudaMemsetAsync(loss_sum, 0, tree->num_nodes * sizeof(double), s));
    ATDF_CUDA_TRY(cudaMemsetAsync(weight_sum, 0, tree->num_nodes * sizeof(double), s));
    node_error_kernel<<<1184, 256, 0, s>>>(w, per_ray_loss, out_channels, num_rays, jitter_seed, loss_sum, weight_sum,
                                           tree->num_nodes, dev_error);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

}  // extern "C"
