// maxflow_tile.cuh -- the single solve over tile_sweep.cuh: two iterations per
// launch, the residual of either of them.  Included by maxflow.cu.
//
// Iterations run in pairs (0, 1), (2, 3), ..., a last odd one alone.  A pair
// with a check sums |err| of both its iterations; where the check of its first
// iteration stops the solve, the state before the pair is still in the buffer
// the pair read, and the first iteration is run again alone.
#pragma once

#include "common.cuh"
#include "tile_sweep.cuh"

namespace m16 {
namespace {

struct MfTileArgs {
    CUtensorMap mh, mu, mdir, meig, mcaps, mrad;
    TileView V;
    int nx, ny, zc;
    float *partials;        // per block: iteration 0, then iteration 1
    const int *stopped;     // null: run whatever the solve's state
    TileFail fail;
};

template <int K, int METRIC, int ASRC, bool SUP, bool CHECK>
__global__ void __launch_bounds__(kTileLanes *kTileNW, kTileBlocks) mf_tile_kernel(const __grid_constant__ MfTileArgs a)
{
    extern __shared__ __align__(128) unsigned char tile_mem[];
    __shared__ float red[32];
    TileMem<METRIC, ASRC> &M = *reinterpret_cast<TileMem<METRIC, ASRC> *>(tile_mem);
    tile_init(M);
    TileView V = a.V;
    V.mh = &a.mh; V.mu = &a.mu; V.mdir = &a.mdir; V.meig = &a.meig; V.mcaps = &a.mcaps; V.mrad = &a.mrad;
    V.fail = &a.fail;
    const int bx = blockIdx.x % a.nx, t = blockIdx.x / a.nx;
    const int by = t % a.ny, za = t / a.ny * a.zc;
    float acc[2] = {0.f, 0.f};
    const bool ran = tile_sweep<K, METRIC, ASRC, false, SUP, CHECK>(V, M, bx, by, za, min(za + a.zc, V.d0), acc, [] {
        pdl_wait();
        pdl_launch_next();
    }, a.stopped);
    if (!ran) return;
    if (CHECK) {
        const float s0 = block_sum(acc[0], red);
        __syncthreads();
        const float s1 = block_sum(acc[1], red);
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            a.partials[blockIdx.x] = s0;
            a.partials[gridDim.x + blockIdx.x] = s1;
        }
    }
}

// the padded fields: h4 = (0, 0, 0, -u rcc), u2 = (u, fmin(cs, ct)) with u =
// img / denom (continuous_cut_anisotropic_gpu.py:276-289), caps; where given,
// dir (column `axis` of the rotation and the radius, or the quaternion for
// axis < 0), eig (square roots of the eigenvalues and the radius) and rad
__global__ void mf_tile_init_kernel(const float *__restrict__ img, const float *__restrict__ quat3,
                                    const float *__restrict__ sqeigs, const float *__restrict__ alpha,
                                    float alpha_scalar, const float *__restrict__ cs, const float *__restrict__ ct,
                                    int d2, int64_t rows, float rcc, int axis, const MfCtrl *ctrl,
                                    float4 *__restrict__ h4, float2 *__restrict__ u2, float2 *__restrict__ caps,
                                    float4 *__restrict__ dir, float4 *__restrict__ eig, float *__restrict__ rad)
{
    const float denom = ctrl->denom;
    const int pitch = tile_pitch(d2);
    const int64_t np = rows * pitch;
    for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < np; o += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = o / pitch;
        const int x = (int)(o - row * pitch);
        if (x >= d2) {   // never part of a result; kept finite
            h4[o] = make_float4(0.f, 0.f, 0.f, 0.f);
            u2[o] = caps[o] = make_float2(0.f, 0.f);
            if (dir) dir[o] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (eig) eig[o] = make_float4(1.f, 1.f, 1.f, 0.f);
            if (rad) rad[o] = 0.f;
            continue;
        }
        const int64_t i = row * d2 + x;
        const float u = img[i] / denom, c = cs[i], t = ct[i];
        h4[o] = make_float4(0.f, 0.f, 0.f, -(u * rcc));
        u2[o] = make_float2(u, fminf(c, t));
        caps[o] = make_float2(c, t);
        const float r = alpha ? alpha[i] : alpha_scalar;
        if (dir) dir[o] = axis < 0 ? qexpand(quat3[3 * i], quat3[3 * i + 1], quat3[3 * i + 2])
                                   : tile_direction(quat3 + 3 * i, axis, r);
        if (eig) eig[o] = make_float4(sqeigs[3 * i], sqeigs[3 * i + 1], sqeigs[3 * i + 2], r);
        if (rad) rad[o] = r;
    }
}

__global__ void mf_tile_result_kernel(const float2 *__restrict__ u2, int d2, int64_t n, float *__restrict__ u)
{
    const int pitch = tile_pitch(d2);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        u[i] = u2[i / d2 * pitch + i % d2].x;
}

// the residuals of a pair's iterations first and first + 1, each where it is a
// check (continuous_cut_anisotropic_gpu.py:321-337)
__global__ void mf_tile_check_kernel(const float *__restrict__ part, int nparts, double inv_norm, double bound,
                                     int first, int count, int update, int resid_cap, MfCtrl *ctrl, double *resid)
{
    __shared__ double s[2][256];
    pdl_wait();
    pdl_launch_next();
    if (__ldcg(&ctrl->stopped)) return;
    double a0 = 0.0, a1 = 0.0;
    for (int k = threadIdx.x; k < nparts; k += blockDim.x) {
        a0 += (double)part[k];
        a1 += (double)part[nparts + k];
    }
    s[0][threadIdx.x] = a0;
    s[1][threadIdx.x] = a1;
    __syncthreads();
    for (int w = blockDim.x >> 1; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            s[0][threadIdx.x] += s[0][threadIdx.x + w];
            s[1][threadIdx.x] += s[1][threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    for (int k = 0; k < count; ++k) {
        const int it = first + k;
        if (it % update) continue;
        const double err = s[k][0] * inv_norm;
        const int idx = it / update;
        if (idx < resid_cap) resid[idx] = err;
        ctrl->n_checks = idx + 1;
        if (isnan(err) || err < bound) {
            ctrl->stopped = 1;
            ctrl->iterations = it + 1;
            return;
        }
    }
}

struct MfTileLayout {
    size_t h[2], u[2], dir, eig, caps, partials, maxpart, ctrl, resid, total;
    int nx, ny, zc, nblocks, resid_cap;
};

inline MfTileLayout mf_tile_layout(int d0, int d1, int d2, int num_iter, int update, bool field)
{
    MfTileLayout L;
    const size_t np = (size_t)tile_voxels(d0, d1, d2);
    L.nx = tile_count_x(d2);
    L.ny = tile_count_y(d1, kTileRows);
    L.zc = tile_zc(d0, (int64_t)L.nx * L.ny);
    L.nblocks = (int)(L.nx * L.ny * div_up(d0, L.zc));
    L.resid_cap = num_iter / (update > 0 ? update : 1) + 2;
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off = align_up(off + bytes, 256); return o; };
    for (int k = 0; k < 2; ++k) {
        L.h[k] = take(np * 16);
        L.u[k] = take(np * 8);
    }
    L.dir = take(np * 16);
    L.eig = take(np * (field ? 16 : 4));   // the eigenvalues' field, or the radius alone
    L.caps = take(np * 8);
    L.partials = take((size_t)L.nblocks * 8);
    L.maxpart = take(kMaxBlocks * 4);
    L.ctrl = take(sizeof(MfCtrl));
    L.resid = take((size_t)L.resid_cap * 8);
    L.total = off;
    return L;
}

typedef void (*MfTileKernel)(const MfTileArgs);

struct MfTileLaunch {
    MfTileKernel kernel;
    size_t smem;
};

template <int METRIC, int ASRC, bool SUP>
MfTileLaunch mf_tile_kernel_of(int k, bool check)
{
    MfTileLaunch L;
    L.smem = sizeof(TileMem<METRIC, ASRC>);
    if (k == 2) L.kernel = check ? mf_tile_kernel<2, METRIC, ASRC, SUP, true> : mf_tile_kernel<2, METRIC, ASRC, SUP, false>;
    else L.kernel = check ? mf_tile_kernel<1, METRIC, ASRC, SUP, true> : mf_tile_kernel<1, METRIC, ASRC, SUP, false>;
    return L;
}

template <bool SUP>
MfTileLaunch mf_tile_pick(int metric, int k, bool check)
{
    switch (metric) {
        case kMetricIso: return mf_tile_kernel_of<kMetricIso, kRadPlanar, SUP>(k, check);
        case kMetricAxis: return mf_tile_kernel_of<kMetricAxis, kRadPacked, SUP>(k, check);
        case kMetricConst: return mf_tile_kernel_of<kMetricConst, kRadPlanar, SUP>(k, check);
        default: return mf_tile_kernel_of<kMetricField, kRadPacked, SUP>(k, check);
    }
}

}  // namespace
}  // namespace m16
