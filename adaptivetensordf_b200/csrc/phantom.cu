// Line integrals of a voxel volume along rays, in FP64 with exact
// intersection lengths (Siddon's method, traversed voxel by voxel in the
// incremental form of Amanatides & Woo). This generates the training
// projections of the synthetic tilt series from a voxelised phantom; the
// reference reads measured tilt series instead
// (hyperacorn/csrc/data/SceneBase.cpp:904-1000).
#include <cuda_runtime.h>
#include <math.h>

#include "atdf.h"
#include "atdf_common.cuh"

namespace atdf {

struct SiddonGrid {
    const float* vol;  // [nz][ny][nx]
    int n[3];          // nx, ny, nz
    double bmin[3], bmax[3], h[3];
};

constexpr int kAhead = 4;  // voxel reads in flight per ray

__global__ void __launch_bounds__(128) siddon_kernel(SiddonGrid g, const float* __restrict__ origin, const float* __restrict__ dir,
                              int64_t R, double* __restrict__ out)
{
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= R) return;
    double o[3], d[3];
    for (int a = 0; a < 3; ++a) {
        o[a] = (double)origin[3 * r + a];
        d[a] = (double)dir[3 * r + a];
    }
    double t0 = -INFINITY, t1 = INFINITY;
    for (int a = 0; a < 3; ++a) {
        if (d[a] == 0.0) {
            if (o[a] < g.bmin[a] || o[a] >= g.bmax[a]) {
                out[r] = 0.0;
                return;
            }
        } else {
            const double ta = (g.bmin[a] - o[a]) / d[a], tb = (g.bmax[a] - o[a]) / d[a];
            t0 = fmax(t0, fmin(ta, tb));
            t1 = fmin(t1, fmax(ta, tb));
        }
    }
    if (!(t0 < t1)) {
        out[r] = 0.0;
        return;
    }
    // voxel containing the point just inside the entry face, and per axis the
    // parameter of the next voxel face crossed there: recomputed from the face's
    // number (kept as a double, exact), so rounding does not accumulate, only on
    // the axis that moved, and with the direction's reciprocal. What
    // bounds the walk is the latency of its voxel reads and of its FP64 chain:
    // 262144 rays through 256^3 voxels took 0.76 ms with three FP64 divides a
    // step, 0.47 ms without, each read waited for before the next step, and
    // 0.42 ms with kAhead reads in flight. (Voxels in 2^3 bricks, read once per
    // brick with a 32-byte load, were slower: 0.59 ms with the copy.)
    int idx[3], step[3];
    double tf[3], inv[3], off[3], face[3], dir1[3];
    int64_t v = 0, stride[3];
    const double tin = t0 + 1e-9 * (t1 - t0);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double u = (o[a] + d[a] * tin - g.bmin[a]) / g.h[a];
        int i = (int)floor(u);
        idx[a] = i < 0 ? 0 : (i >= g.n[a] ? g.n[a] - 1 : i);
        const bool up = d[a] > 0;
        step[a] = up ? 1 : -1;
        dir1[a] = up ? 1.0 : -1.0;
        inv[a] = d[a] != 0.0 ? 1.0 / d[a] : 0.0;
        off[a] = g.bmin[a] - o[a];
        face[a] = (double)(idx[a] + (up ? 1 : 0));
        tf[a] = d[a] != 0.0 ? fma(face[a], g.h[a], off[a]) * inv[a] : INFINITY;
        const int64_t s = a == 0 ? 1 : a == 1 ? g.n[0] : (int64_t)g.n[0] * g.n[1];
        v += idx[a] * s;
        stride[a] = up ? s : -s;
    }
    double acc = 0.0, t = t0;
    const int max_steps = g.n[0] + g.n[1] + g.n[2] + 3;
    bool going = true;
    // kAhead steps at a time: their voxel reads are in flight together, and
    // are added, in order, once the group is through
    for (int it = 0; going && it < max_steps; it += kAhead) {
        double len[kAhead];
        float density[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            going = going && t < t1 && it + k < max_steps;
            // the nearest face (ties: the lower axis), or the exit
            const bool y = tf[1] < tf[0];
            const double txy = y ? tf[1] : tf[0];
            const bool z = tf[2] < txy;
            const double near = z ? tf[2] : txy;
            const bool inside = near < t1;
            const double tn = inside ? near : t1;
            const bool some = going && tn > t;
            len[k] = some ? tn - t : 0.0;
            density[k] = some ? __ldg(&g.vol[v]) : 0.0f;
            if (some) t = tn;
            going = going && inside;
            bool left = false;
#pragma unroll
            for (int a = 0; a < 3; ++a) {  // selects, not branches: the lanes of a warp move along different axes
                const bool mine = going && (a == 2 ? z : a == 1 ? y && !z : !y && !z);
                const double next = face[a] + dir1[a], t_next = fma(next, g.h[a], off[a]) * inv[a];
                idx[a] += mine ? step[a] : 0;
                v += mine ? stride[a] : 0;
                face[a] = mine ? next : face[a];
                tf[a] = mine ? t_next : tf[a];
                left = left || (unsigned)idx[a] >= (unsigned)g.n[a];
            }
            going = going && !left;
        }
#pragma unroll
        for (int k = 0; k < kAhead; ++k) acc = fma(len[k], (double)density[k], acc);
    }
    out[r] = acc;
}

}  // namespace atdf

using namespace atdf;

extern "C" int atdf_siddon_project(const float* volume, int32_t nx, int32_t ny, int32_t nz, const double* box_min,
                                   const double* box_max, const float* ray_origin, const float* ray_direction,
                                   int64_t num_rays, double* out, atdf_stream_t stream)
{
    if (num_rays < 0 || nx <= 0 || ny <= 0 || nz <= 0 || !box_min || !box_max) return ATDF_ERR_INVALID_ARGUMENT;
    if (num_rays == 0) return ATDF_OK;
    if (!volume || !ray_origin || !ray_direction || !out) return ATDF_ERR_INVALID_ARGUMENT;
    SiddonGrid g;
    g.vol = volume;
    g.n[0] = nx;
    g.n[1] = ny;
    g.n[2] = nz;
    for (int a = 0; a < 3; ++a) {
        if (!(box_max[a] > box_min[a])) return ATDF_ERR_INVALID_ARGUMENT;
        g.bmin[a] = box_min[a];
        g.bmax[a] = box_max[a];
        g.h[a] = (box_max[a] - box_min[a]) / g.n[a];
    }
    const int threads = 128;
    siddon_kernel<<<(unsigned)((num_rays + threads - 1) / threads), threads, 0, (cudaStream_t)stream>>>(
        g, ray_origin, ray_direction, num_rays, out);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}
