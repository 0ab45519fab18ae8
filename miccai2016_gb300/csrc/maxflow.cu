// maxflow.cu -- continuous max-flow with anisotropic total variation (ATV),
// the GB300 replacement of the reference's update_p / update_u / update_tmp
// kernels (src/clcode-anisotropic/update_qp.cl:150-316) and of the solve loop
// in CmfCutQAnisotropicGpu._execute
// (src/processing/continuous_cut_anisotropic_gpu.py:198-344).
//
// A solve runs two iterations per pass over memory (maxflow_tile.cuh,
// tile_sweep.cuh).  Volumes beyond 32-bit indexes and callers with a small
// workspace take two sweeps per iteration:
//   P: hp <- project_alpha(H^-1 hp + steps * H^T grad(tmp)), hp <- H p
//   U: div(hp), p_s, p_t, u and tmp = err - u / cc (update_tmp fused), and on
//      check iterations the |err| partial sums of the residual.
// Data layout in HBM of the two sweeps (N voxels, all fp32, C order z-y-x):
//   caller:    img, quat3 (N x 3), alpha (N or scalar), cs, ct, labels (u8), u (output/state)
//   workspace: hp0, hp1, hp2, pt, tmp (N each), q4 (N x float4, the expanded
//              quaternion), block partials, control word, residual log.
// Each thread marches along z through a column of the volume; x/y neighbours
// come from L1, the z neighbour is carried in a register.  The quaternion is
// expanded once per solve so the iterations need no trigonometry.
#include <cuda_runtime.h>
#include <math.h>
#include <float.h>

#include <algorithm>
#include <atomic>
#include <memory>
#include <vector>

#include "common.cuh"
#include "sweeps.cuh"

namespace m16 {
namespace {

struct MfCtrl {
    int stopped;      // 1 once a check stopped the solve
    int iterations;   // iterations executed
    int n_checks;     // residual checks done
    int error;        // a copy of the tile sweeps did not arrive in time
    float denom;      // max(img) + FLT_MIN
    float pad1[3];
};

struct MfArgs {
    int d0, d1, d2, zc;
    float rcc, rs0, rs1, rs2, ss0, ss1, ss2;
    float sq0, sq1, sq2, isq0, isq1, isq2;
    float alpha_scalar;
    float *hp0, *hp1, *hp2, *tmp, *pt, *u;
    const float4 *q4;
    const float *alpha, *sqeigs, *cs, *ct;
    const uint8_t *labels;
    float *partials;
    MfCtrl *ctrl;
};

constexpr int kBX = 32, kBY = 8;

// ---- initialisation ------------------------------------------------------

__global__ void mf_max_kernel(const float *__restrict__ img, int64_t n, float *__restrict__ part)
{
    __shared__ float sm[32];
    __shared__ int snan;
    if (threadIdx.x == 0) snan = 0;
    __syncthreads();
    float m = -INFINITY;
    int nan = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float v = img[i];
        if (v != v) nan = 1; else m = fmaxf(m, v);
    }
    if (nan) snan = 1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        float r = sm[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) r = fmaxf(r, sm[w]);
        part[blockIdx.x] = snan ? NAN : r;
    }
}

__global__ void __launch_bounds__(256) mf_init_ctrl_kernel(const float *__restrict__ part, int nparts, int num_iter,
                                                           MfCtrl *ctrl)
{
    __shared__ float sm[8];
    __shared__ int snan;
    if (threadIdx.x == 0) snan = 0;
    __syncthreads();
    float m = -INFINITY;
    for (int k = threadIdx.x; k < nparts; k += blockDim.x) {
        const float v = part[k];
        if (v != v) snan = 1; else m = fmaxf(m, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < 8; ++w) m = fmaxf(m, sm[w]);
    const bool nan = snan != 0;
    ctrl->denom = (nan ? NAN : m) + FLT_MIN;   // np.max(img) + np.finfo(float32).tiny
    ctrl->stopped = 0;
    ctrl->iterations = num_iter;
    ctrl->n_checks = 0;
    ctrl->error = 0;
}

// hp = 0, p_t = fmin(cs, ct), u = img / denom, tmp = -u * rcc, q4 = qexpand(quat3)
// (continuous_cut_anisotropic_gpu.py:276-289)
__global__ void mf_init_kernel(MfArgs a, const float *__restrict__ img, const float *__restrict__ quat3, int64_t n)
{
    const float denom = a.ctrl->denom;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        a.hp0[i] = 0.f;
        a.hp1[i] = 0.f;
        a.hp2[i] = 0.f;
        a.pt[i] = fminf(a.cs[i], a.ct[i]);
        const float ui = img[i] / denom;
        a.u[i] = ui;
        a.tmp[i] = -(ui * a.rcc);
        const float *s = quat3 + 3 * i;
        const_cast<float4 *>(a.q4)[i] = qexpand(s[0], s[1], s[2]);
    }
}

// ---- P and U sweeps (bodies in sweeps.cuh, shared with the batched engine) --

// resident blocks per SM the sweeps are compiled for: 4 caps them at 64
// registers (the flow sweep needs 69 uncapped, which allows 3); measured on
// GB300 at 256^3 the capped flow sweep runs 0.861 of the HBM copy rate
// against 0.794 uncapped, the label sweep is unchanged
#ifndef M16_MF_MINB
#define M16_MF_MINB 4
#endif
constexpr int kZB = kMfZB > kMfUZB ? kMfZB : kMfUZB;   // z-chunks are whole load batches of both sweeps

__device__ __forceinline__ FlowView flow_view(const MfArgs &a)
{
    FlowView f;
    f.d0 = a.d0; f.d1 = a.d1; f.d2 = a.d2;
    f.ss0 = a.ss0; f.ss1 = a.ss1; f.ss2 = a.ss2;
    f.sq0 = a.sq0; f.sq1 = a.sq1; f.sq2 = a.sq2; f.isq0 = a.isq0; f.isq1 = a.isq1; f.isq2 = a.isq2;
    f.alpha_scalar = a.alpha_scalar; f.alpha = a.alpha; f.grad2 = nullptr; f.w = 0.f; f.neg_inv_decay2 = 0.f;
    f.sqeigs = a.sqeigs; f.q4 = a.q4; f.tmp = a.tmp; f.hp0 = a.hp0; f.hp1 = a.hp1; f.hp2 = a.hp2;
    return f;
}

__device__ __forceinline__ LabelView label_view(const MfArgs &a)
{
    LabelView l;
    l.d0 = a.d0; l.d1 = a.d1; l.d2 = a.d2;
    l.rcc = a.rcc; l.rs0 = a.rs0; l.rs1 = a.rs1; l.rs2 = a.rs2;
    l.hp0 = a.hp0; l.hp1 = a.hp1; l.hp2 = a.hp2; l.cs = a.cs; l.ct = a.ct; l.labels = a.labels;
    l.pt = a.pt; l.u = a.u; l.tmp = a.tmp;
    return l;
}

template <bool POINTWISE, bool ALPHA_ARR>
__global__ void __launch_bounds__(kBX * kBY, M16_MF_MINB) mf_update_p_kernel(MfArgs a)
{
    pdl_wait();
    pdl_launch_next();
    if (__ldcg(&a.ctrl->stopped)) return;
    const int x = blockIdx.x * kBX + threadIdx.x;
    const int y = blockIdx.y * kBY + threadIdx.y;
    if (x >= a.d2 || y >= a.d1) return;
    const int z0 = blockIdx.z * a.zc;
    flow_column<POINTWISE, ALPHA_ARR ? kAlphaArray : kAlphaScalar>(flow_view(a), x, y, z0, min(z0 + a.zc, a.d0));
}

template <bool SUPERVISED, bool CHECK>
__global__ void __launch_bounds__(kBX * kBY, M16_MF_MINB) mf_update_u_kernel(MfArgs a)
{
    __shared__ float red[32];
    pdl_wait();
    pdl_launch_next();
    if (__ldcg(&a.ctrl->stopped)) return;
    const int x = blockIdx.x * kBX + threadIdx.x;
    const int y = blockIdx.y * kBY + threadIdx.y;
    float acc = 0.f;
    if (x < a.d2 && y < a.d1) {
        const int z0 = blockIdx.z * a.zc;
        acc = label_column<SUPERVISED>(label_view(a), x, y, z0, min(z0 + a.zc, a.d0));
    }
    if (CHECK) {
        const float s = block_sum(acc, red);
        if (threadIdx.x == 0 && threadIdx.y == 0)
            a.partials[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = s;
    }
}

// residual = sum(partials) / (N * rcc); stop on NaN or below the bound
// (continuous_cut_anisotropic_gpu.py:321-337)
__global__ void mf_check_kernel(const float *__restrict__ part, int nparts, double inv_norm, double bound,
                                int iter, int check_idx, int resid_cap, MfCtrl *ctrl, double *resid)
{
    __shared__ double s[256];
    pdl_wait();
    pdl_launch_next();
    if (__ldcg(&ctrl->stopped)) return;
    double acc = 0.0;
    for (int k = threadIdx.x; k < nparts; k += blockDim.x) acc += (double)part[k];
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int w = blockDim.x >> 1; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double err = s[0] * inv_norm;
        if (check_idx < resid_cap) resid[check_idx] = err;
        ctrl->n_checks = check_idx + 1;
        if (isnan(err) || err < bound) {
            ctrl->stopped = 1;
            ctrl->iterations = iter + 1;
        }
    }
}

// ---- host side --------------------------------------------------------------

struct MfLayout {
    size_t hp0, hp1, hp2, pt, tmp, q4, partials, maxpart, ctrl, resid, total;
    int nparts, resid_cap;
};

constexpr int kMaxBlocks = 4 * kSMs;

// z-slices per thread: enough blocks for 8 per SM, at most 16, a multiple of
// the load batch once it reaches it
inline int choose_zc(int d0, int d1, int d2)
{
    const int64_t cols = div_up(d2, kBX) * div_up(d1, kBY);
    int64_t zc = (int64_t)d0 * cols / (8 * kSMs);
    if (zc < 1) zc = 1;
    if (zc > 16) zc = 16;
    if (zc >= kZB) zc = zc / kZB * kZB;
    return (int)zc;
}

// the two-sweep state, the expanded quaternions, the block partials and the
// residual log
inline MfLayout mf_layout(int d0, int d1, int d2, int num_iter, int update)
{
    MfLayout L;
    const int64_t n = (int64_t)d0 * d1 * d2;
    const int zc = choose_zc(d0, d1, d2);
    L.nparts = (int)(div_up(d2, kBX) * div_up(d1, kBY) * div_up(d0, zc));
    L.resid_cap = num_iter / (update > 0 ? update : 1) + 2;
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off = align_up(off + bytes, 256); return o; };
    L.hp0 = take(n * 4); L.hp1 = take(n * 4); L.hp2 = take(n * 4);
    L.pt = take(n * 4); L.tmp = take(n * 4);
    L.q4 = take(n * 16);
    L.partials = take((size_t)L.nparts * 4);
    L.maxpart = take(kMaxBlocks * 4);
    L.ctrl = take(sizeof(MfCtrl));
    L.resid = take((size_t)L.resid_cap * 8);
    L.total = off;
    return L;
}

inline bool finite_pos(double v) { return v > 0.0 && v < 1e300; }

}  // namespace
}  // namespace m16

#include "maxflow_tile.cuh"

using namespace m16;

extern "C" size_t m16_maxflow_workspace_bytes_min(int32_t d0, int32_t d1, int32_t d2, const m16_cut_params *params)
{
    if (d0 < 1 || d1 < 1 || d2 < 1 || !params) return 0;
    return mf_layout(d0, d1, d2, params->num_iter, params->update).total;
}

static size_t maxflow_workspace(int d0, int d1, int d2, const m16_cut_params *params, bool field)
{
    const size_t two_sweeps = m16_maxflow_workspace_bytes_min(d0, d1, d2, params);
    if (!two_sweeps || !tile_shape_ok(d0, d1, d2)) return two_sweeps;
    return std::max(two_sweeps, mf_tile_layout(d0, d1, d2, params->num_iter, params->update, field).total);
}

extern "C" size_t m16_maxflow_workspace_bytes(int32_t d0, int32_t d1, int32_t d2, const m16_cut_params *params)
{
    return maxflow_workspace(d0, d1, d2, params, true);
}

extern "C" size_t m16_maxflow_workspace_bytes_const(int32_t d0, int32_t d1, int32_t d2, const m16_cut_params *params)
{
    return maxflow_workspace(d0, d1, d2, params, false);
}

extern "C" int m16_maxflow_solve(const float *img, const float *quat3, const double *sqevals3,
                                 const float *sqeigs, const float *alpha, float alpha_scalar,
                                 const float *cs, const float *ct, const uint8_t *labels,
                                 int32_t d0, int32_t d1, int32_t d2, const m16_cut_params *params,
                                 float *u, int32_t *iterations, double *residuals, int32_t residuals_cap,
                                 int32_t *n_residuals, void *workspace, size_t workspace_bytes, void *stream)
{
    return m16_maxflow_solve_ex(img, quat3, sqevals3, sqeigs, alpha, alpha_scalar, cs, ct, labels, d0, d1, d2,
                                params, u, iterations, residuals, residuals_cap, n_residuals, workspace,
                                workspace_bytes, stream, nullptr);
}

namespace {
// A pool of CUDA events bracketing the P/U launches of one chunk of iterations.
struct EventPool {
    std::vector<cudaEvent_t> ev;
    int used = 0;
    bool ok = true;
    explicit EventPool(int n) : ev(n, nullptr)
    {
        for (auto &e : ev)
            if (cudaEventCreate(&e) != cudaSuccess) { ok = false; e = nullptr; }
    }
    ~EventPool()
    {
        for (auto e : ev)
            if (e) cudaEventDestroy(e);
    }
};

// Iterations between two looks at the stopping state: whole check intervals, at
// least `least` iterations, a multiple of `unit`, no more than the solve has.
// 64-bit until it is cut: an update of 2^31 - 1 ("check once") is in order.
inline int mf_chunk(int num_iter, int update, int least, int unit)
{
    int64_t c = std::max<int64_t>((int64_t)update * std::max(1, 64 / update), least);
    c = (c + unit - 1) / unit * unit;
    return (int)std::min<int64_t>(c, std::max(num_iter, 1));
}
inline int mf_chunk_end(int it, int chunk, int num_iter) { return (int)std::min<int64_t>(num_iter, (int64_t)it + chunk); }
}  // namespace

namespace {

// The solve over the tile sweeps (maxflow_tile.cuh); the arguments have been
// checked.
int maxflow_solve_tiles(const float *img, const float *quat3, const double *sqevals3, const float *sqeigs,
                        const float *alpha, float alpha_scalar, const float *cs, const float *ct,
                        const uint8_t *labels, int d0, int d1, int d2, const m16_cut_params *params, float *u,
                        int32_t *iterations, double *residuals, int32_t residuals_cap, int32_t *n_residuals,
                        const MfTileLayout &L, char *ws, cudaStream_t st, m16_solve_stats *stats)
{
    const int64_t n = (int64_t)d0 * d1 * d2;
    TileView V = TileView();
    int axis = -1;
    const int metric = sqevals3 ? tile_metric(sqevals3, V, &axis) : kMetricField;
    const double *sc = params->scaling;
    const double smin = fmin(sc[0], fmin(sc[1], sc[2]));
    const double rcc = 1.0 / (params->cc * (smin * smin));
    MfCtrl *ctrl = (MfCtrl *)(ws + L.ctrl);
    double *resid = (double *)(ws + L.resid);
    V.d0 = d0; V.d1 = d1; V.d2 = d2; V.pitch = tile_pitch(d2);
    V.ss0 = (float)(params->steps / sc[0] * (smin * smin));
    V.ss1 = (float)(params->steps / sc[1] * (smin * smin));
    V.ss2 = (float)(params->steps / sc[2] * (smin * smin));
    V.rs0 = (float)(1.0 / sc[0]); V.rs1 = (float)(1.0 / sc[1]); V.rs2 = (float)(1.0 / sc[2]);
    V.rcc = (float)rcc;
    V.ircc = (float)(1.0 / rcc);
    V.labels = labels;
    // the two directions of a sweep: buffer k read, the other written
    MfTileArgs args[2];
    for (int k = 0; k < 2; ++k) {
        MfTileArgs &a = args[k];
        a.V = V;
        a.V.ho = (float4 *)(ws + L.h[1 - k]);
        a.V.uo = (float2 *)(ws + L.u[1 - k]);
        a.nx = L.nx; a.ny = L.ny; a.zc = L.zc;
        a.partials = (float *)(ws + L.partials);
        a.stopped = &ctrl->stopped;
        a.fail = TileFail{&ctrl->error, &ctrl->stopped};
        bool ok = tile_map(&a.mh, ws + L.h[k], d0, d1, V.pitch, 4, kTileRows + 1) &&
                  tile_map(&a.mu, ws + L.u[k], d0, d1, V.pitch, 2, kTileRows) &&
                  tile_map(&a.mcaps, ws + L.caps, d0, d1, V.pitch, 2, kTileRows);
        if (metric != kMetricIso) ok = ok && tile_map(&a.mdir, ws + L.dir, d0, d1, V.pitch, 4, kTileRows);
        if (metric == kMetricField) ok = ok && tile_map(&a.meig, ws + L.eig, d0, d1, V.pitch, 4, kTileRows);
        else ok = ok && tile_map(&a.mrad, ws + L.eig, d0, d1, V.pitch, 1, kTileRows);
        if (!ok) return M16_ERR_CUDA;
    }
    MfTileLaunch kernels[2][2];   // [iterations - 1][check]
    for (int k = 0; k < 2; ++k)
        for (int c = 0; c < 2; ++c) {
            kernels[k][c] = labels ? mf_tile_pick<true>(metric, k + 1, c != 0) : mf_tile_pick<false>(metric, k + 1, c != 0);
            M16_CUDA_TRY(cudaFuncSetAttribute(kernels[k][c].kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)kernels[k][c].smem));
        }

    const int init_blocks = (int)std::min<int64_t>(kMaxBlocks, div_up(n, 256));
    mf_max_kernel<<<init_blocks, 256, 0, st>>>(img, n, (float *)(ws + L.maxpart));
    mf_init_ctrl_kernel<<<1, 256, 0, st>>>((float *)(ws + L.maxpart), init_blocks, params->num_iter, ctrl);
    const bool planar = metric == kMetricIso || metric == kMetricConst;
    mf_tile_init_kernel<<<init_blocks, 256, 0, st>>>(
        img, quat3, sqeigs, alpha, alpha_scalar, cs, ct, d2, (int64_t)d0 * d1, V.rcc, axis, ctrl,
        (float4 *)(ws + L.h[0]), (float2 *)(ws + L.u[0]), (float2 *)(ws + L.caps),
        metric != kMetricIso ? (float4 *)(ws + L.dir) : nullptr,
        metric == kMetricField ? (float4 *)(ws + L.eig) : nullptr, planar ? (float *)(ws + L.eig) : nullptr);
    M16_CUDA_TRY(cudaGetLastError());
    int launches = 3;

    const int num_iter = params->num_iter, update = params->update;
    // even, so that pairs start at even iterations; without a bound only a NaN
    // residual stops
    const int chunk = mf_chunk(num_iter, update, params->error_bound > 0.0 ? 1 : 1024, 2);
    const bool timing = stats && stats->time_kernels;
    const bool pdl = !(stats && (stats->flags & M16_SOLVE_NO_PDL));
    std::unique_ptr<EventPool> pool;
    if (timing) {
        pool.reset(new EventPool(chunk + 2));
        if (!pool->ok) return M16_ERR_CUDA;
    }
    int it = 0;
    auto sweep = [&](int count, bool check, int buf, bool always) -> cudaError_t {
        const MfTileLaunch &K = kernels[count - 1][check];
        MfTileArgs a = args[buf];
        if (always) a.stopped = nullptr;
        // the first one reads what the set-up kernel wrote before it waits: not early
        return launch_pdl_smem(K.kernel, dim3(L.nblocks), dim3(kTileLanes, kTileNW), K.smem, st, pdl && it > 0, a);
    };
    int pair_n = 0;
    double pair_ms = 0.0;
    MfCtrl hctrl;
    hctrl.stopped = 0;
    while (it < num_iter) {
        const int end = mf_chunk_end(it, chunk, num_iter), begin = it;
        int slots = 0;
        while (it < end) {
            const int count = std::min(2, num_iter - it);
            const bool check = it % update == 0 || (count == 2 && (it + 1) % update == 0);
            const bool time_it = timing && count == 2;
            if (time_it) cudaEventRecord(pool->ev[2 * slots], st);
            M16_CUDA_TRY(sweep(count, check, (it >> 1) & 1, false));
            if (time_it) cudaEventRecord(pool->ev[2 * slots++ + 1], st);
            ++launches;
            if (check) {
                M16_CUDA_TRY(launch_pdl(mf_tile_check_kernel, dim3(1), dim3(256), st, pdl,
                                        (const float *)(ws + L.partials), L.nblocks, 1.0 / ((double)n * rcc),
                                        params->error_bound, it, count, update, L.resid_cap, ctrl, resid));
                ++launches;
            }
            it += count;
        }
        M16_CUDA_TRY(cudaGetLastError());
        M16_CUDA_TRY(cudaMemcpyAsync(&hctrl, ctrl, sizeof(MfCtrl), cudaMemcpyDeviceToHost, st));
        M16_CUDA_TRY(cudaStreamSynchronize(st));
        for (int j = 0; j < slots; ++j) {
            // only pairs that ran (not the no-op launches after a stop) count
            if (hctrl.stopped && begin + 2 * j >= hctrl.iterations) break;
            float ms = 0.f;
            M16_CUDA_TRY(cudaEventElapsedTime(&ms, pool->ev[2 * j], pool->ev[2 * j + 1]));
            pair_ms += ms;
            ++pair_n;
        }
        if (hctrl.stopped) break;
    }
    if (num_iter == 0) {
        M16_CUDA_TRY(cudaMemcpyAsync(&hctrl, ctrl, sizeof(MfCtrl), cudaMemcpyDeviceToHost, st));
        M16_CUDA_TRY(cudaStreamSynchronize(st));
    }
    if (hctrl.error) return M16_ERR_TIMEOUT;
    const int ran = hctrl.stopped ? hctrl.iterations : it;
    // stopped by the check of a pair's first iteration: that one again, alone,
    // from the buffer the pair read
    const bool again = ran & 1 && ran < num_iter;
    if (again) {
        M16_CUDA_TRY(sweep(1, false, (ran >> 1) & 1, true));
        ++launches;
    }
    mf_tile_result_kernel<<<init_blocks, 256, 0, st>>>((const float2 *)(ws + L.u[((ran + 1) >> 1) & 1]), d2, n, u);
    ++launches;
    M16_CUDA_TRY(cudaGetLastError());
    if (stats) {
        stats->launches = launches;
        stats->p_launches = stats->u_launches = 0;   // no separate flow and label launches
        stats->p_ms = stats->u_ms = 0.0;
        stats->pair_launches = timing ? pair_n : ran / 2;
        stats->pair_ms = pair_ms;
        stats->pair_zc = L.zc;
    }
    *iterations = hctrl.iterations;
    if (n_residuals) *n_residuals = hctrl.n_checks;
    if (residuals && residuals_cap > 0) {
        const int cnt = std::min(std::min(hctrl.n_checks, residuals_cap), L.resid_cap);
        if (cnt > 0) M16_CUDA_TRY(cudaMemcpyAsync(residuals, resid, (size_t)cnt * 8, cudaMemcpyDeviceToHost, st));
    }
    int late = 0;   // a copy of the iteration that ran again
    if (again) M16_CUDA_TRY(cudaMemcpyAsync(&late, &ctrl->error, sizeof(int), cudaMemcpyDeviceToHost, st));
    M16_CUDA_TRY(cudaStreamSynchronize(st));
    return late ? M16_ERR_TIMEOUT : M16_OK;
}

}  // namespace

// The solve: over the tile sweeps where the workspace holds their fields, else
// every iteration a flow and a label launch.
static int maxflow_solve_impl(const float *img, const float *quat3, const double *sqevals3, const float *sqeigs,
                              const float *alpha, float alpha_scalar, const float *cs, const float *ct,
                              const uint8_t *labels, int32_t d0, int32_t d1, int32_t d2,
                              const m16_cut_params *params, float *u, int32_t *iterations, double *residuals,
                              int32_t residuals_cap, int32_t *n_residuals, void *workspace, size_t workspace_bytes,
                              void *stream, m16_solve_stats *stats)
{
    if (d0 < 1 || d1 < 1 || d2 < 1) return M16_ERR_BAD_SHAPE;
    if ((int64_t)d0 * d1 * d2 > ((int64_t)1 << 34)) return M16_ERR_BAD_SHAPE;
    if (!params || !img || !quat3 || !cs || !ct || !u || !iterations) return M16_ERR_BAD_ARG;
    if (!sqevals3 && !sqeigs) return M16_ERR_BAD_ARG;
    if (params->update < 1 || params->num_iter < 0) return M16_ERR_BAD_ARG;
    if (!(params->cc > 0.0) || !(params->steps >= 0.0)) return M16_ERR_BAD_ARG;
    for (int k = 0; k < 3; ++k)
        if (!finite_pos(params->scaling[k])) return M16_ERR_BAD_ARG;
    if (sqevals3)
        for (int k = 0; k < 3; ++k)
            if (!finite_pos(sqevals3[k])) return M16_ERR_BAD_ARG;
    const MfLayout L = mf_layout(d0, d1, d2, params->num_iter, params->update);
    if (!workspace || workspace_bytes < L.total || ((uintptr_t)workspace & 255)) return M16_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    char *ws = (char *)workspace;
    const int64_t n = (int64_t)d0 * d1 * d2;
    // Two iterations a pass over 72 bytes a voxel (256^3: 95 us an iteration)
    // against two passes an iteration over 88 (228 us); the two sweeps take half
    // the workspace and any volume size.
    TileView view = TileView();
    int axis;
    const int metric = sqevals3 ? tile_metric(sqevals3, view, &axis) : kMetricField;
    if (tile_shape_ok(d0, d1, d2) && tile_rows_ok(metric, d0, d1, d2, kSmallSolve) &&
        !(stats && stats->path == M16_PATH_TWO_SWEEPS)) {
        const MfTileLayout T = mf_tile_layout(d0, d1, d2, params->num_iter, params->update, sqevals3 == nullptr);
        if (workspace_bytes >= T.total)
            return maxflow_solve_tiles(img, quat3, sqevals3, sqeigs, alpha, alpha_scalar, cs, ct, labels, d0, d1, d2,
                                       params, u, iterations, residuals, residuals_cap, n_residuals, T, ws, st, stats);
    }

    // constants as _reinit_clprograms derives them (continuous_cut_anisotropic_gpu.py:104-129)
    const double *sc = params->scaling;
    const double smin = fmin(sc[0], fmin(sc[1], sc[2]));
    const double rcc = 1.0 / (params->cc * (smin * smin));
    MfArgs a;
    a.d0 = d0; a.d1 = d1; a.d2 = d2; a.zc = choose_zc(d0, d1, d2);
    a.rcc = (float)rcc;
    a.rs0 = (float)(1.0 / sc[0]); a.rs1 = (float)(1.0 / sc[1]); a.rs2 = (float)(1.0 / sc[2]);
    a.ss0 = (float)(params->steps / sc[0] * (smin * smin));
    a.ss1 = (float)(params->steps / sc[1] * (smin * smin));
    a.ss2 = (float)(params->steps / sc[2] * (smin * smin));
    const double sqd[3] = {sqevals3 ? sqevals3[0] : 1.0, sqevals3 ? sqevals3[1] : 1.0, sqevals3 ? sqevals3[2] : 1.0};
    a.sq0 = (float)sqd[0]; a.sq1 = (float)sqd[1]; a.sq2 = (float)sqd[2];
    a.isq0 = (float)(1.0 / sqd[0]); a.isq1 = (float)(1.0 / sqd[1]); a.isq2 = (float)(1.0 / sqd[2]);
    a.alpha_scalar = alpha_scalar;
    a.hp0 = (float *)(ws + L.hp0); a.hp1 = (float *)(ws + L.hp1); a.hp2 = (float *)(ws + L.hp2);
    a.pt = (float *)(ws + L.pt); a.tmp = (float *)(ws + L.tmp); a.u = u;
    a.q4 = (const float4 *)(ws + L.q4);
    a.alpha = alpha; a.sqeigs = sqeigs; a.cs = cs; a.ct = ct; a.labels = labels;
    a.partials = (float *)(ws + L.partials);
    a.ctrl = (MfCtrl *)(ws + L.ctrl);
    double *resid = (double *)(ws + L.resid);

    const int init_blocks = (int)std::min<int64_t>(kMaxBlocks, div_up(n, 256));
    mf_max_kernel<<<init_blocks, 256, 0, st>>>(img, n, (float *)(ws + L.maxpart));
    mf_init_ctrl_kernel<<<1, 256, 0, st>>>((float *)(ws + L.maxpart), init_blocks, params->num_iter, a.ctrl);
    mf_init_kernel<<<init_blocks, 256, 0, st>>>(a, img, quat3, n);
    M16_CUDA_TRY(cudaGetLastError());

    const dim3 block(kBX, kBY, 1);
    const dim3 grid((unsigned)div_up(d2, kBX), (unsigned)div_up(d1, kBY), (unsigned)div_up(d0, a.zc));
    const int nparts_sweep = (int)(grid.x * grid.y * grid.z);
    const bool pointwise = sqevals3 == nullptr;
    const bool alpha_arr = alpha != nullptr;
    const bool sup = labels != nullptr;
    const double inv_norm = 1.0 / ((double)n * rcc);
    const int update = params->update;
    const int chunk = mf_chunk(params->num_iter, update, 1, 1);

    const bool timing = stats && stats->time_kernels;
    const bool pdl = !(stats && (stats->flags & M16_SOLVE_NO_PDL));
    std::unique_ptr<EventPool> pool;
    if (timing) {
        pool.reset(new EventPool(3 * chunk));
        if (!pool->ok) return M16_ERR_CUDA;
    }
    int launches = 3, p_launches = 0, u_launches = 0;
    double p_ms = 0.0, u_ms = 0.0;

    MfCtrl hctrl;
    hctrl.stopped = 0;
    int it = 0;
    while (it < params->num_iter) {
        const int end = mf_chunk_end(it, chunk, params->num_iter);
        // per launch slot: its iteration, for the timing
        std::vector<int> slot_it;
        while (it < end) {
            const int j = (int)slot_it.size();
            if (timing) cudaEventRecord(pool->ev[3 * j], st);
            slot_it.push_back(it);
            const MfArgs &s = a;
            if (pointwise) {
                if (alpha_arr) M16_CUDA_TRY(launch_pdl(mf_update_p_kernel<true, true>, grid, block, st, pdl, s));
                else M16_CUDA_TRY(launch_pdl(mf_update_p_kernel<true, false>, grid, block, st, pdl, s));
            } else {
                if (alpha_arr) M16_CUDA_TRY(launch_pdl(mf_update_p_kernel<false, true>, grid, block, st, pdl, s));
                else M16_CUDA_TRY(launch_pdl(mf_update_p_kernel<false, false>, grid, block, st, pdl, s));
            }
            if (timing) cudaEventRecord(pool->ev[3 * j + 1], st);
            const bool check = (it % update) == 0;
            if (check) {
                if (sup) M16_CUDA_TRY(launch_pdl(mf_update_u_kernel<true, true>, grid, block, st, pdl, s));
                else M16_CUDA_TRY(launch_pdl(mf_update_u_kernel<false, true>, grid, block, st, pdl, s));
                if (timing) cudaEventRecord(pool->ev[3 * j + 2], st);
                M16_CUDA_TRY(launch_pdl(mf_check_kernel, dim3(1), dim3(256), st, pdl, (const float *)a.partials,
                                          nparts_sweep, inv_norm, params->error_bound, it, it / update, L.resid_cap,
                                          a.ctrl, resid));
                ++launches;
            } else {
                if (sup) M16_CUDA_TRY(launch_pdl(mf_update_u_kernel<true, false>, grid, block, st, pdl, s));
                else M16_CUDA_TRY(launch_pdl(mf_update_u_kernel<false, false>, grid, block, st, pdl, s));
                if (timing) cudaEventRecord(pool->ev[3 * j + 2], st);
            }
            launches += 2;
            ++it;
        }
        M16_CUDA_TRY(cudaGetLastError());
        M16_CUDA_TRY(cudaMemcpyAsync(&hctrl, a.ctrl, sizeof(MfCtrl), cudaMemcpyDeviceToHost, st));
        M16_CUDA_TRY(cudaStreamSynchronize(st));
        if (timing) {
            // only launches that ran (not the no-op launches after a stop) count
            const int ran_end = hctrl.stopped ? std::min(end, hctrl.iterations) : end;
            for (size_t j = 0; j < slot_it.size(); ++j) {
                if (slot_it[j] >= ran_end) break;
                float a_ms = 0.f, b_ms = 0.f;
                M16_CUDA_TRY(cudaEventElapsedTime(&a_ms, pool->ev[3 * j], pool->ev[3 * j + 1]));
                M16_CUDA_TRY(cudaEventElapsedTime(&b_ms, pool->ev[3 * j + 1], pool->ev[3 * j + 2]));
                p_ms += a_ms;
                u_ms += b_ms;
                ++p_launches;
                ++u_launches;
            }
        }
        if (hctrl.stopped) break;
    }
    M16_CUDA_TRY(cudaMemcpyAsync(&hctrl, a.ctrl, sizeof(MfCtrl), cudaMemcpyDeviceToHost, st));
    M16_CUDA_TRY(cudaStreamSynchronize(st));
    const int ran = hctrl.stopped ? hctrl.iterations : it;
    if (stats) {
        stats->launches = launches;
        if (!timing) p_launches = u_launches = ran;
        stats->p_launches = p_launches;
        stats->u_launches = u_launches;
        stats->p_ms = p_ms;
        stats->u_ms = u_ms;
        stats->pair_launches = 0;
        stats->pair_ms = 0.0;
        stats->pair_zc = 0;
    }
    *iterations = hctrl.iterations;
    if (n_residuals) *n_residuals = hctrl.n_checks;
    if (residuals && residuals_cap > 0) {
        const int cnt = std::min(std::min(hctrl.n_checks, residuals_cap), L.resid_cap);
        if (cnt > 0) {
            M16_CUDA_TRY(cudaMemcpyAsync(residuals, resid, (size_t)cnt * 8, cudaMemcpyDeviceToHost, st));
            M16_CUDA_TRY(cudaStreamSynchronize(st));
        }
    }
    return M16_OK;
}

extern "C" int m16_maxflow_solve_ex(const float *img, const float *quat3, const double *sqevals3,
                                    const float *sqeigs, const float *alpha, float alpha_scalar,
                                    const float *cs, const float *ct, const uint8_t *labels,
                                    int32_t d0, int32_t d1, int32_t d2, const m16_cut_params *params,
                                    float *u, int32_t *iterations, double *residuals, int32_t residuals_cap,
                                    int32_t *n_residuals, void *workspace, size_t workspace_bytes, void *stream,
                                    m16_solve_stats *stats)
{
    if (stats && stats->path != M16_PATH_DEFAULT && stats->path != M16_PATH_TWO_SWEEPS) return M16_ERR_BAD_ARG;
    return maxflow_solve_impl(img, quat3, sqevals3, sqeigs, alpha, alpha_scalar, cs, ct, labels, d0, d1, d2, params,
                              u, iterations, residuals, residuals_cap, n_residuals, workspace, workspace_bytes,
                              stream, stats);
}

// ---- fixed-footprint variant: no allocation by anyone --------------------------
//
// m16_maxflow_solve takes its scratch from a workspace the caller allocates.
// Some callers cannot allocate device memory at all: a plugin whose host owns
// every byte of device memory through its own pool and hands it no allocator,
// a language binding (Go, Java, ...) that wants a fixed device footprint known
// at load time, or a service that must not allocate once it is serving.  For
// them m16_maxflow_solve_static runs the same solve with its scratch in the
// file-scope array below, which the CUDA module reserves on every device that
// loads this library and which stays reserved until the process exits.
//
// Limits: at most kStaticMaxVoxels voxels (e.g. 64 x 64 x 64) and at most
// kStaticMaxChecks residual checks (num_iter / update + 2 <= kStaticMaxChecks).

namespace m16 {
namespace {
constexpr int64_t kStaticMaxVoxels = 262144;
constexpr int kStaticMaxChecks = 4096;
// The largest workspace of the tile sweeps at the limits, of all shapes: 88 B per
// padded voxel (at most 294,912 of them, tile_shape_ok), 8 B per block (a block of
// a volume of few columns or planes writes as few as 52 voxels: 5041 blocks at 1 x
// 65536 x 4), max partials, control and residual log, each region rounded up to 256
// B: 25,874,176 B (2097 x 5 x 25).  The two sweeps take less than half of it.
constexpr size_t kStaticBytes = 25u << 20;

}  // namespace
}  // namespace m16

static __device__ __align__(256) unsigned char m16_static_scratch[m16::kStaticBytes];

namespace m16 {
namespace {
// Device address of the scratch array on the current device.  Host code cannot
// use the array's name as a device address, so every call asks the runtime for
// it, with the calling device current.  The lookup is cheap once the module is
// loaded, and it is never stale: a device reset, or any teardown and
// re-creation of the context, reloads the module and may move the array, and
// the next lookup returns the new address.
int static_scratch_on_current_device(void **out)
{
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, m16_static_scratch) != cudaSuccess || !p) return M16_ERR_CUDA;
    *out = p;
    return M16_OK;
}
}  // namespace
}  // namespace m16

extern "C" int m16_maxflow_solve_static(const float *img, const float *quat3, const double *sqevals3,
                                        const float *sqeigs, const float *alpha, float alpha_scalar,
                                        const float *cs, const float *ct, const uint8_t *labels,
                                        int32_t d0, int32_t d1, int32_t d2, const m16_cut_params *params,
                                        float *u, int32_t *iterations, double *residuals, int32_t residuals_cap,
                                        int32_t *n_residuals, void *stream)
{
    // size checks first: nothing touches the GPU for a request that cannot fit
    if (d0 < 1 || d1 < 1 || d2 < 1 || !params) return d0 < 1 || d1 < 1 || d2 < 1 ? M16_ERR_BAD_SHAPE : M16_ERR_BAD_ARG;
    if (params->update < 1 || params->num_iter < 0) return M16_ERR_BAD_ARG;
    if ((int64_t)d0 * d1 * d2 > kStaticMaxVoxels) return M16_ERR_TOO_LARGE;
    if (params->num_iter / params->update + 2 > kStaticMaxChecks) return M16_ERR_TOO_LARGE;
    const MfLayout L = mf_layout(d0, d1, d2, params->num_iter, params->update);
    if (L.total > kStaticBytes) return M16_ERR_TOO_LARGE;
    void *scratch = nullptr;
    const int st = static_scratch_on_current_device(&scratch);
    if (st != M16_OK) return st;
    // The solve's initialisation kernels write every scratch word before it is
    // read (flow state, control word, partial sums), so nothing of the previous
    // call's contents leaks into this one.
    return maxflow_solve_impl(img, quat3, sqevals3, sqeigs, alpha, alpha_scalar, cs, ct, labels, d0, d1, d2, params,
                              u, iterations, residuals, residuals_cap, n_residuals, scratch, kStaticBytes, stream,
                              nullptr);
}
