// batch_kernels.cuh -- device side of the batched ATV max-flow: descriptors,
// set-up kernels, the sweeps over a work list of (instance, tile) items, the
// per-instance residual check and the output of u.  Included by batched.cu
// (m16_batch_solve: a fixed batch run to completion) and serve.cu
// (m16_server_*: requests admitted and retired while others iterate).
//
// The reference runs its (weighting, decay) grid search as one
// CmfCutQAnisotropicGpu.execute() per grid point and cut type
// (src/phantom_experiment.py:350-368), each with three launches per iteration
// and a blocking residual read every `update` iterations.  Here a batch of
// instances -- any mix of volumes, weightings, decays and eigenvalue sets --
// advances together: a launch runs two iterations (tile_sweep.cuh) of every
// active instance of one kind, the residual check of every instance is one
// block of one launch, and an instance stops on its own at its threshold.
//
// Layout.  An instance has its own state, double-buffered.  The direction
// field with |grad I|^2, the capacities and, for isotropic and three-valued
// metrics, |grad I|^2 alone belong to the volume; the work list puts the
// instances of a volume side by side for every tile, so these fields come from
// L2 for all but the first of them.  The projection radius is an instance's
// own alpha field or w * exp(-|grad I|^2 / decay^2) (phantom_experiment.py:359)
// computed in the sweep.
//
// An instance's state word holds its stop flag and which buffer is current.
// Within a run of launches between two checks the buffers alternate by the
// launch's number; the check that ends the run stores the buffer it ends in,
// so captured launches can be replayed.
//
// Measured on GB300: 16 grid points at 128^3, anisotropic and isotropic (32
// instances), 358 -> 155 ms against groups of four interleaved instances in a
// flow and a label launch per iteration; eight uneven volumes 39.6 -> 20.0 ms;
// ten served requests 113 -> 52 ms; 16 single planes of 256^2 alone are slower
// (120 iterations 2.60 -> 3.16 ms).  Bound by HBM where the tiles fit the
// volume (48 bytes of state per voxel and two iterations), by the march's
// instructions on the halo where they do not (128^3: 1.56 times the voxels).
//
// The compact sweeps at the end (one buffer, planar fields, a flow and a label
// launch per iteration) take the instances whose double-buffered state does
// not fit.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <float.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "sweeps.cuh"
#include "tile_sweep.cuh"

namespace m16 {
namespace {

constexpr int kBX = 32, kBY = 8, kTile = kBX * kBY;
constexpr int kSetupBlocks = 4 * kSMs;

constexpr unsigned kStopped = 1u, kBuffer = 2u;   // bits of an instance's state word (kStopped: also tile_fail's)

struct InstCtrl {
    int stopped;
    int iterations;
    int n_checks;
    int pad;
    double resid;   // last checked residual
};

// what the check and the output need of an instance
struct InstDev {
    int64_t n;
    int64_t part_off;        // float index of its first partial sum
    int nparts, d2;
    float rcc;
    const float2 *u2[2];     // padded (tile sweeps), or null:
    const float *u1;         // the compact sweeps' u
    float *u_out;
};

// an instance of the tile sweeps
struct TileDev {
    TileView V;              // all but the buffers and fail
    TileFail fail;
    const CUtensorMap *mh[2], *mu[2];
    float4 *h[2];
    float2 *u[2];
    int64_t part_off, rows;
    int nx, ny, zc;
    // set-up inputs
    const float *img, *cs, *ct, *alpha, *denom;
    float *rad;              // its own padded radius field (alpha instances), or null
};

// kinds of launches: the tile sweeps' instantiations, then the compact sweeps
enum BatchKind { kAxisPacked = 0, kAxisPlanar, kIsoPlanar, kConstPlanar, kTileKinds, kCompactAlpha = kTileKinds,
                 kCompactExp, kKinds };

// ---- initialisation ---------------------------------------------------------

__global__ void bt_max_kernel(const float *__restrict__ img, int64_t n, float *__restrict__ part)
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

// *denom = np.max(img) + np.finfo(float32).tiny (one block)
__global__ void __launch_bounds__(256) bt_denom_kernel(const float *__restrict__ part, int nparts, float *denom)
{
    __shared__ float s[256];
    __shared__ int snan;
    if (threadIdx.x == 0) snan = 0;
    __syncthreads();
    float m = -INFINITY;
    for (int k = threadIdx.x; k < nparts; k += blockDim.x) {
        const float v = part[k];
        if (v != v) snan = 1; else m = fmaxf(m, v);
    }
    s[threadIdx.x] = m;
    __syncthreads();
    for (int w = blockDim.x >> 1; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) s[threadIdx.x] = fmaxf(s[threadIdx.x], s[threadIdx.x + w]);
        __syncthreads();
    }
    if (threadIdx.x == 0) *denom = (snan ? NAN : s[0]) + FLT_MIN;
}

// the volume's padded fields: caps and, where given, the direction of each
// axis with `value` (|grad I|^2 or alpha), the quaternion, and value alone
struct VolumeFields {
    float2 *caps;
    float4 *dir[3], *q4;
    float *rad;
};

__global__ void bt_volume_kernel(const float *__restrict__ quat3, const float *__restrict__ value,
                                 const float *__restrict__ cs, const float *__restrict__ ct, int d2, int64_t rows,
                                 VolumeFields F)
{
    const int pitch = tile_pitch(d2);
    const int64_t np = rows * pitch;
    for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < np; o += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = o / pitch;
        const int x = (int)(o - row * pitch);
        const bool in = x < d2;   // the padding is never part of a result; kept finite
        const int64_t i = row * d2 + (in ? x : 0);
        const float v = in && value ? value[i] : 0.f;
        F.caps[o] = in ? make_float2(cs[i], ct[i]) : make_float2(0.f, 0.f);
        for (int k = 0; k < 3; ++k)
            if (F.dir[k]) F.dir[k][o] = tile_direction(quat3 + 3 * i, k, v);
        if (F.q4) F.q4[o] = qexpand(quat3[3 * i], quat3[3 * i + 1], quat3[3 * i + 2]);
        if (F.rad) F.rad[o] = v;
    }
}

// every instance (blockIdx.y): h4 = (0, 0, 0, -u rcc), u2 = (u, fmin(cs, ct))
// with u = img / denom (continuous_cut_anisotropic_gpu.py:276-289) in buffer 0,
// and its own radius field
__global__ void bt_state_kernel(const TileDev *tiles, int first)
{
    const TileDev &T = tiles[first + blockIdx.y];
    const float denom = *T.denom, rcc = T.V.rcc;
    const int d2 = T.V.d2, pitch = T.V.pitch;
    const int64_t np = T.rows * pitch;
    for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < np; o += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = o / pitch;
        const int x = (int)(o - row * pitch);
        const bool in = x < d2;
        const int64_t i = row * d2 + (in ? x : 0);
        const float u = in ? T.img[i] / denom : 0.f;
        T.h[0][o] = make_float4(0.f, 0.f, 0.f, -(u * rcc));
        T.u[0][o] = make_float2(u, in ? fminf(T.cs[i], T.ct[i]) : 0.f);
        if (T.rad) T.rad[o] = in ? T.alpha[i] : 0.f;
    }
}

// u of every instance (blockIdx.y) into its output; flip: the buffer is the
// other one than the state word says
__global__ void bt_result_kernel(const InstDev *insts, const unsigned *state, int first, int flip)
{
    const InstDev &I = insts[first + blockIdx.y];
    const int b = ((state[first + blockIdx.y] & kBuffer) ? 1 : 0) ^ flip;
    const float2 *u2 = I.u2[b];
    const int pitch = tile_pitch(I.d2);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < I.n; i += (int64_t)gridDim.x * blockDim.x)
        I.u_out[i] = u2 ? u2[i / I.d2 * pitch + i % I.d2].x : I.u1[i];
}

// ---- the tile sweeps ----------------------------------------------------------

// K iterations of the work items' tiles; work == NULL: block b is tile b of
// instance `first`.  The launch reads the current buffer, or with `odd` (an odd
// launch since the state word was set) the other one.
template <int K, int METRIC, int ASRC, bool CHECK>
__global__ void __launch_bounds__(kTileLanes *kTileNW, kTileBlocks) bt_tile_kernel(const int2 *__restrict__ work,
                                                                                  int first, const TileDev *tiles,
                                                                                  const unsigned *__restrict__ state,
                                                                                  float *__restrict__ partials,
                                                                                  int odd)
{
    extern __shared__ __align__(128) unsigned char tile_mem[];
    __shared__ float red[32];
    TileMem<METRIC, ASRC> &M = *reinterpret_cast<TileMem<METRIC, ASRC> *>(tile_mem);
    tile_init(M);
    pdl_wait();
    pdl_launch_next();
    const int2 wk = work ? work[blockIdx.x] : make_int2(first, (int)blockIdx.x);
    const unsigned s = __ldcg(state + wk.x);
    if (s & kStopped) return;   // uniform over the block
    const int b = ((s & kBuffer) ? 1 : 0) ^ odd;
    const TileDev &T = tiles[wk.x];
    TileView V = T.V;
    V.mh = T.mh[b];
    V.mu = T.mu[b];
    V.ho = T.h[1 - b];
    V.uo = T.u[1 - b];
    V.fail = &T.fail;
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        tile_acquire(V.mh);
        tile_acquire(V.mu);
        tile_acquire(V.mcaps);
        if (METRIC != kMetricIso) tile_acquire(V.mdir);
        if (ASRC == kRadPlanar) tile_acquire(V.mrad);
    }
    const int nx = T.nx, ny = T.ny, zc = T.zc;
    const int bx = wk.y % nx, t = wk.y / nx, by = t % ny, za = t / ny * zc;
    float acc[2] = {0.f, 0.f};
    tile_sweep<K, METRIC, ASRC, true, false, CHECK>(V, M, bx, by, za, min(za + zc, V.d0), acc, [] {}, nullptr);
    if (CHECK) {
        const float sum = block_sum(acc[K - 1], red);
        if (threadIdx.x == 0 && threadIdx.y == 0) partials[T.part_off + wk.y] = sum;
    }
}

typedef void (*BatchTileKernel)(const int2 *, int, const TileDev *, const unsigned *, float *, int);

struct BatchTileLaunch {
    BatchTileKernel kernel;
    size_t smem;
};

template <int METRIC, int ASRC>
BatchTileLaunch batch_tile_kernel(int k, bool check)
{
    BatchTileLaunch L;
    L.smem = sizeof(TileMem<METRIC, ASRC>);
    if (k == 2) L.kernel = check ? bt_tile_kernel<2, METRIC, ASRC, true> : bt_tile_kernel<2, METRIC, ASRC, false>;
    else L.kernel = check ? bt_tile_kernel<1, METRIC, ASRC, true> : bt_tile_kernel<1, METRIC, ASRC, false>;
    return L;
}

inline BatchTileLaunch batch_tile_pick(int kind, int k, bool check)
{
    switch (kind) {
        case kAxisPacked: return batch_tile_kernel<kMetricAxis, kRadPacked>(k, check);
        case kAxisPlanar: return batch_tile_kernel<kMetricAxis, kRadPlanar>(k, check);
        case kIsoPlanar: return batch_tile_kernel<kMetricIso, kRadPlanar>(k, check);
        default: return batch_tile_kernel<kMetricConst, kRadPlanar>(k, check);
    }
}

// once per device and call, before any launch (not while capturing)
inline cudaError_t batch_tile_prepare(int kind)
{
    for (int k = 1; k <= 2; ++k)
        for (int c = 0; c < 2; ++c) {
            const BatchTileLaunch L = batch_tile_pick(kind, k, c != 0);
            const cudaError_t e =
                cudaFuncSetAttribute(L.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

// TileView constants of a volume (scaling sc) under the solve's parameters
inline void tile_view(TileView &V, int d0, int d1, int d2, const double *sc, const m16_cut_params &p)
{
    const double smin = fmin(sc[0], fmin(sc[1], sc[2]));
    const double rcc = 1.0 / (p.cc * (smin * smin));
    V.d0 = d0; V.d1 = d1; V.d2 = d2; V.pitch = tile_pitch(d2);
    V.ss0 = (float)(p.steps / sc[0] * (smin * smin));
    V.ss1 = (float)(p.steps / sc[1] * (smin * smin));
    V.ss2 = (float)(p.steps / sc[2] * (smin * smin));
    V.rs0 = (float)(1.0 / sc[0]); V.rs1 = (float)(1.0 / sc[1]); V.rs2 = (float)(1.0 / sc[2]);
    V.rcc = (float)rcc;
    V.ircc = (float)(1.0 / rcc);
}

// one block per instance: residual = sum of its partial sums / (N * rcc); below
// the bound (or NaN) the instance stops.  Every instance is checked at its own
// iterations 0, update, 2 update, ..., so the n-th check (from 0) follows
// iteration n * update and a stop there counts n * update + 1 iterations,
// wherever the instance joined the batch.  flip: the run of launches that the
// check ends was odd, so the other buffer is the current one now.
__global__ void bt_check_kernel(const InstDev *insts, InstCtrl *ctrl, unsigned *state,
                                const float *__restrict__ partials, double bound, int update, int flip,
                                const int *__restrict__ list, int first)
{
    pdl_wait();
    pdl_launch_next();
    __shared__ double s[256];
    const int inst = list ? list[blockIdx.x] : first + (int)blockIdx.x;   // list: the instances to check
    const unsigned word = __ldcg(state + inst);
    if (word & kStopped) return;
    const InstDev &I = insts[inst];
    InstCtrl &C = ctrl[inst];
    const float *p = partials + I.part_off;
    double acc = 0.0;
    for (int k = threadIdx.x; k < I.nparts; k += blockDim.x) acc += (double)p[k];
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int w = blockDim.x >> 1; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double err = s[0] / ((double)I.n * (double)I.rcc);
        C.resid = err;
        const int n = C.n_checks;
        C.n_checks = n + 1;
        unsigned w = flip ? word ^ kBuffer : word;
        if (isnan(err) || err < bound) {
            C.stopped = 1;
            C.iterations = n * update + 1;
            w |= kStopped;
        }
        state[inst] = w;
    }
}

// the end of an odd run of launches without a check
__global__ void bt_flip_kernel(unsigned *state, int n)
{
    pdl_wait();
    pdl_launch_next();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && !(state[i] & kStopped)) state[i] ^= kBuffer;
}

// ---- the compact sweeps: the single solve's two sweeps over the work list ------

struct VolDev {
    int d0, d1, d2, zc, tx, ty, tz, pad;
    float rcc, rs0, rs1, rs2, ss0, ss1, ss2;
    const float4 *q4;
    const float *grad2, *cs, *ct;
};

struct GroupDev {
    int vol, pad;
    int64_t part_off;
    float w, nid2;           // radius = w * exp(nid2 * |grad I|^2), nid2 = -1 / decay^2
    float sq0, sq1, sq2, isq0, isq1, isq2;
    float *state;            // hp0 hp1 hp2 pt tmp u: slabs of `slab` floats
    int64_t slab;
    const float *alpha;      // the instance's own radius, or NULL
    const float *img, *denom;
};

constexpr int kFields = 6;

__global__ void bt_expand_kernel(const float *__restrict__ quat3, float4 *__restrict__ q4, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        q4[i] = qexpand(quat3[3 * i], quat3[3 * i + 1], quat3[3 * i + 2]);
}

__global__ void bt1_state_kernel(const VolDev *vols, const GroupDev *groups, int first)
{
    const GroupDev &G = groups[first + blockIdx.y];
    const VolDev &V = vols[G.vol];
    const float denom = *G.denom;
    const int64_t S = G.slab, n = (int64_t)V.d0 * V.d1 * V.d2;
    float *st = G.state;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float ui = G.img[i] / denom;
        st[i] = 0.f;
        st[S + i] = 0.f;
        st[2 * S + i] = 0.f;
        st[3 * S + i] = fminf(V.cs[i], V.ct[i]);
        st[4 * S + i] = -(ui * V.rcc);
        st[5 * S + i] = ui;
    }
}

__device__ __forceinline__ void decode_tile(const VolDev &V, int tile, int &bx, int &by, int &bz)
{
    bx = tile % V.tx;
    by = (tile / V.tx) % V.ty;
    bz = tile / (V.tx * V.ty);
}

// resident blocks per SM of the compact sweeps: 4 (64 registers) measured
// fastest on GB300
constexpr int kCompactBlocks = 4;

template <int ALPHA>
__global__ void __launch_bounds__(kTile, kCompactBlocks) bt1_flow_kernel(const int2 *__restrict__ work, int first,
                                                                        const VolDev *vols, const GroupDev *groups,
                                                                        const unsigned *__restrict__ state)
{
    pdl_wait();
    pdl_launch_next();
    const int2 wk = work ? work[blockIdx.x] : make_int2(first, (int)blockIdx.x);
    if (__ldcg(state + wk.x) & kStopped) return;
    const GroupDev &G = groups[wk.x];
    const VolDev &V = vols[G.vol];
    int bx, by, bz;
    decode_tile(V, wk.y, bx, by, bz);
    const int x = bx * kBX + threadIdx.x, y = by * kBY + threadIdx.y;
    // the view in shared memory: its fields are read where used instead of
    // held in registers for the whole column
    __shared__ FlowView sf;
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        float *st = G.state;
        const int64_t S = G.slab;
        sf.d0 = V.d0; sf.d1 = V.d1; sf.d2 = V.d2;
        sf.ss0 = V.ss0; sf.ss1 = V.ss1; sf.ss2 = V.ss2;
        sf.sq0 = G.sq0; sf.sq1 = G.sq1; sf.sq2 = G.sq2; sf.isq0 = G.isq0; sf.isq1 = G.isq1; sf.isq2 = G.isq2;
        sf.alpha_scalar = 0.f;
        sf.alpha = G.alpha;
        sf.grad2 = V.grad2;
        sf.w = G.w;
        sf.neg_inv_decay2 = G.nid2;
        sf.sqeigs = nullptr;
        sf.q4 = V.q4;
        sf.tmp = st + 4 * S;
        sf.hp0 = st; sf.hp1 = st + S; sf.hp2 = st + 2 * S;
    }
    __syncthreads();
    if (x >= sf.d2 || y >= sf.d1) return;
    const int z0 = bz * V.zc;
    flow_column<false, ALPHA>(sf, x, y, z0, min(z0 + V.zc, sf.d0));
}

template <bool CHECK>
__global__ void __launch_bounds__(kTile, CHECK ? 3 : kCompactBlocks) bt1_label_kernel(const int2 *__restrict__ work, int first,
                                                                         const VolDev *vols, const GroupDev *groups,
                                                                         const unsigned *__restrict__ state,
                                                                         float *__restrict__ partials)
{
    pdl_wait();
    pdl_launch_next();
    __shared__ float red[32];
    const int2 wk = work ? work[blockIdx.x] : make_int2(first, (int)blockIdx.x);
    if (__ldcg(state + wk.x) & kStopped) return;   // uniform over the block
    const GroupDev &G = groups[wk.x];
    const VolDev &V = vols[G.vol];
    int bx, by, bz;
    decode_tile(V, wk.y, bx, by, bz);
    const int x = bx * kBX + threadIdx.x, y = by * kBY + threadIdx.y;
    const int z0 = bz * V.zc, z1 = min(z0 + V.zc, V.d0);
    float acc = 0.f;
    if (x < V.d2 && y < V.d1) {
        float *st = G.state;
        const int64_t S = G.slab;
        LabelView l;
        l.d0 = V.d0; l.d1 = V.d1; l.d2 = V.d2;
        l.rcc = V.rcc; l.rs0 = V.rs0; l.rs1 = V.rs1; l.rs2 = V.rs2;
        l.hp0 = st; l.hp1 = st + S; l.hp2 = st + 2 * S;
        l.cs = V.cs; l.ct = V.ct; l.labels = nullptr;
        l.pt = st + 3 * S; l.tmp = st + 4 * S; l.u = st + 5 * S;
        acc = label_column<false>(l, x, y, z0, z1);
    }
    if (CHECK) {
        const float s = block_sum(acc, red);
        if (threadIdx.x == 0 && threadIdx.y == 0) partials[G.part_off + wk.y] = s;
    }
}

inline void compact_volume(VolDev &d, int d0, int d1, int d2, int zc, const TileView &V)
{
    d.d0 = d0; d.d1 = d1; d.d2 = d2;
    d.zc = zc;
    d.tx = (int)div_up(d2, kBX); d.ty = (int)div_up(d1, kBY); d.tz = (int)div_up(d0, zc);
    d.pad = 0;
    d.rcc = V.rcc; d.rs0 = V.rs0; d.rs1 = V.rs1; d.rs2 = V.rs2; d.ss0 = V.ss0; d.ss1 = V.ss1; d.ss2 = V.ss2;
}

// z-slices per block of the compact sweeps: four blocks per SM for the volume
// alone, at least two slices, whole load batches
inline int compact_zc(int d0, int d1, int d2)
{
    const int64_t cols = div_up(d2, kBX) * div_up(d1, kBY);
    const int64_t zc = (int64_t)d0 * cols / (4 * kSMs);
    return (int)std::max<int64_t>(std::min<int64_t>(2, d0), std::min<int64_t>(32, zc));
}

inline int compact_tiles(int d0, int d1, int d2)
{
    return (int)(div_up(d2, kBX) * div_up(d1, kBY) * div_up(d0, compact_zc(d0, d1, d2)));
}

// ---- launches --------------------------------------------------------------------

// the device tables and the work list of a batch or a server step
struct BatchTables {
    const int2 *work = nullptr;
    int first = 0;               // work == NULL: tiles of this instance
    int seg[kKinds + 1] = {};    // items seg[k] .. seg[k + 1] - 1 are of kind k
    const TileDev *tiles = nullptr;
    const VolDev *vols = nullptr;
    const GroupDev *groups = nullptr;
    const InstDev *insts = nullptr;
    InstCtrl *ctrl = nullptr;
    unsigned *state = nullptr;
    float *partials = nullptr;
};

// events around the launches of two iterations of a run, and how many there were
// (all kinds' launches of the same two iterations count as one)
struct PairTimer {
    cudaEvent_t begin = nullptr, end = nullptr;
    int pairs = 0;
};

// Enqueues m iterations of the work items; `check` computes the residual sums
// of the last one (the caller launches the check).  Returns the number of sweep
// launches of the tile kinds (their buffers alternated that often) or -1 on a
// launch error.
inline int enqueue_iterations(const BatchTables &T, int m, bool check, cudaStream_t st, int &launches,
                              PairTimer *timer = nullptr)
{
    cudaError_t e = cudaSuccess;
    auto keep = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
    int done = 0, sweeps = 0;
    while (done < m) {
        const int k = (m - done) & 1 ? 1 : 2;
        const bool last = done + k == m;
        const bool timed = timer && k == 2 && T.seg[kTileKinds] > T.seg[0];
        if (timed && timer->pairs++ == 0) keep(cudaEventRecord(timer->begin, st));
        for (int kind = 0; kind < kTileKinds; ++kind) {
            const int items = T.seg[kind + 1] - T.seg[kind];
            if (items <= 0) continue;
            const BatchTileLaunch L = batch_tile_pick(kind, k, check && last);
            keep(launch_pdl_smem(L.kernel, dim3(items), dim3(kTileLanes, kTileNW), L.smem, st, true,
                                 T.work ? T.work + T.seg[kind] : nullptr, T.first, T.tiles,
                                 (const unsigned *)T.state, T.partials, sweeps & 1));
            ++launches;
        }
        if (timed && last) keep(cudaEventRecord(timer->end, st));
        done += k;
        ++sweeps;
    }
    const int na = T.seg[kCompactAlpha + 1] - T.seg[kCompactAlpha];
    const int ne = T.seg[kCompactExp + 1] - T.seg[kCompactExp];
    if (na + ne > 0) {
        const dim3 block(kBX, kBY, 1);
        const int2 *wa = T.work ? T.work + T.seg[kCompactAlpha] : nullptr;
        const int2 *we = T.work ? T.work + T.seg[kCompactExp] : nullptr;
        const unsigned *state = T.state;
        for (int i = 0; i < m; ++i) {
            if (na > 0) keep(launch_pdl(bt1_flow_kernel<kAlphaArray>, dim3(na), block, st, true, wa, T.first, T.vols, T.groups, state));
            if (ne > 0) keep(launch_pdl(bt1_flow_kernel<kAlphaFromGrad2>, dim3(ne), block, st, true, we, T.first, T.vols, T.groups, state));
            if (check && i == m - 1)
                keep(launch_pdl(bt1_label_kernel<true>, dim3(na + ne), block, st, true, wa, T.first, T.vols, T.groups, state, T.partials));
            else
                keep(launch_pdl(bt1_label_kernel<false>, dim3(na + ne), block, st, true, wa, T.first, T.vols, T.groups, state, T.partials));
            launches += (na > 0) + (ne > 0) + 1;
        }
    }
    return e == cudaSuccess ? sweeps : -1;
}

}  // namespace
}  // namespace m16
