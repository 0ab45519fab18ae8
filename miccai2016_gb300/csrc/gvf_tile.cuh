// gvf_tile.cuh -- K iterations of the gradient vector flow in one pass over
// memory (the equations: gvf.cu).  Included by gvf.cu.
//
// Fields are planar and padded (tile_pitch), the components one behind the
// other, so that one tensor copy brings all three.  A block marches along z
// with 32 columns and GvfShape::Rows rows; stage k (the k-th iteration) works a plane
// behind stage k - 1.  A lane keeps kGvfRT rows of two adjacent columns
// (f32x2.cuh), half a warp a row, three planes of each stage's input in
// registers.  Stage 1 reads the x and y neighbours of its plane from the copied
// tile (one column and row wider on every side); later stages take x neighbours
// by shuffle and y neighbours from the lane's rows or, at their edge, from the
// rows stored a step before, so one barrier a step is enough.  A block writes
// all but K - 1 rows (and as many columns, rounded up to a pair) on each side.
//
// Bound: 36 bytes a voxel for K iterations (40 with a response), and about 66
// instructions a computed voxel and iteration.  Measured on GB300 at 256^3 (100
// iterations, set-up and output included): one iteration a pass over 40 bytes
// 124 us an iteration; K = 1 here 94, K = 2 66 (0.72 of the copy rate, issue 54
// %, shared memory 60 % busy), K = 3 73 (its slots leave one block per SM); K =
// 2 with scalar arithmetic 76.  2 x 12 half-warps of rows, 2 blocks per SM; 16
// rows and 3 blocks 66, 32 rows and one block 79, one row a lane 93, four rows
// 109 (spills).
//
// With a response that shape's slots fill more than half of an SM's shared
// memory, so one block of six warps ran on each (256^3 102 us an iteration, 97 x
// 161 x 203 27.2, 75 x 93 x 110 8.2).  There one block of 8 warps (32 rows) and K
// = 3 take 73, 17.5 and 6.3; two blocks of 20 rows and K = 2 82, 18.3 and 6.7; of
// 16 rows 80, 19.0 and 6.3.
#pragma once

#include "common.cuh"
#include "f32x2.cuh"
#include "tile_sweep.cuh"

namespace m16 {
namespace {

constexpr int kGvfRT = 2;                            // rows per lane
// iterations of a pass, warps of a block and blocks per SM
template <bool RESP>
struct GvfShape {
    static constexpr int K = RESP ? 3 : 2, NW = RESP ? 8 : 6, Blocks = RESP ? 1 : 2;
    static constexpr int Groups = 2 * NW, Rows = kGvfRT * Groups;   // half-warps, rows of a block
};
constexpr int kGvfMaxK = 3;
constexpr int kGvfGW = 40, kGvfVW = 32;              // copied row lengths
// columns a block leaves out on each inner side: K - 1, pairs of them, with
// starts on a 16-byte boundary
__host__ __device__ constexpr int gvf_halo(int k) { return k & ~1; }

struct GvfTileArgs {
    CUtensorMap mg, mv, mr;
    int d0, d1, d2, pitch, nx, ny, zc;
    float rss0, rss1, rss2, nmu, ndt;   // 1 / spacing^2, -mu, -dt
    int64_t comp;                   // voxels of a padded component
    const float *gi;
    float *go;
    float *partials;                // per iteration: per block
    int checks;                     // bit k: |delta| of iteration k is summed
    const GvfCtrl *ctrl;            // null: run whatever the state
    TileFail fail;
};

template <int K, bool RESP>
struct GvfMem {
    static constexpr int H = GvfShape<RESP>::Rows, Lag = K < 2 ? 2 : K, S = Lag + 2;
    struct Slot {   // v of plane p, g of plane p + 1
        alignas(128) float g[3][H + 2][kGvfGW];
        alignas(128) float v[3][H][kGvfVW];
        alignas(128) float r[RESP ? H : 1][kGvfVW];
    } slot[S];
    // [stage][step parity][half-warp][first, last row] of each later stage's input
    f2 edge[K > 1 ? K - 1 : 1][2][GvfShape<RESP>::Groups + 2][2][3][16];
    uint64_t full[S];
};

__device__ __forceinline__ void gvf_copy(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *b)
{
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, "
                 "%4, %5}], [%6];" ::"r"(smem_addr(dst)),
                 "l"(map), "r"(x), "r"(y), "r"(z), "r"(0), "r"(smem_addr(b))
                 : "memory");
}

// FLAT: fewer rows than a block has, so that the last row of the volume may be
// any row of a lane; otherwise the last tile ends on it.
template <int K, bool RESP, bool CHECK, bool FLAT>
__global__ void __launch_bounds__(kTileLanes *GvfShape<RESP>::NW, GvfShape<RESP>::Blocks)
    gvf_tile_kernel(const __grid_constant__ GvfTileArgs a)
{
    extern __shared__ __align__(128) unsigned char gvf_mem[];
    __shared__ float red[32];
    typedef GvfMem<K, RESP> Mem;
    Mem &M = *reinterpret_cast<Mem *>(gvf_mem);
    constexpr int RT = kGvfRT, H = Mem::H, S = Mem::S, Lag = Mem::Lag;
    const int lane = threadIdx.x, warp = threadIdx.y;
    const bool copier = lane == 0 && warp == 0;
    if (copier) {
        for (int k = 0; k < S; ++k) bar_init(&M.full[k]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    pdl_wait();
    pdl_launch_next();
    if (a.ctrl && __ldcg(&a.ctrl->stopped)) return;

    constexpr int HX = gvf_halo(K), OW = kTileLanes - 2 * HX, OH = H - 2 * (K - 1);
    const int bx = blockIdx.x % a.nx, bt = blockIdx.x / a.nx, by = bt % a.ny;
    const int d0 = a.d0, d1 = a.d1, d2 = a.d2;
    const int za = bt / a.ny * a.zc, zb = min(za + a.zc, d0);
    // the region's origin and this lane's pair of columns and rows
    const int xr = bx * OW, yr = FLAT ? 0 : min(by * OH, d1 - H);
    const int lx = 2 * (lane & 15), group = 2 * warp + (lane >> 4);
    const int x = xr + lx, row0 = group * RT, y0 = yr + row0;
    const bool xlast = xr + kTileLanes >= d2;
    const bool xout = lx >= (bx ? HX : 0) && (xlast ? x < d2 : lx < kTileLanes - HX);
    const bool pair = x + 1 < d2;                       // the second column is inside
    const int ylo = by * OH + (by ? K - 1 : 0), yhi = by == a.ny - 1 ? d1 : by * OH + H - (K - 1);
    // mirrored neighbours (d2 >= 2): the column before the pair and the one
    // after it; where the pair's first column is the last, its own neighbour
    const bool xfirst = x == 0, xend = x + 1 >= d2 - 1, ghost = x == d2 - 1;
    const int srcl = xfirst ? lane : max(lane - 1, 0), srcg = xend ? lane : min(lane + 1, kTileLanes - 1);
    const int coll = lx + 4 + (xfirst ? 1 : -1), colg = lx + 4 + (xend ? 0 : 2);
    const bool top = y0 == 0, bottom = y0 + RT == d1;
    const f2 m2 = both2(-2.f), rss0 = both2(a.rss0), rss1 = both2(a.rss1), rss2 = both2(a.rss2), nmu = both2(a.nmu),
             ndt = both2(a.ndt);
    auto at2 = [](const float *p) { return *reinterpret_cast<const f2 *>(p); };

    const int zs = max(za - K + 1, 0);                  // first plane of stage 1
    const int zl = min(zb + K - 2, d0 - 1);             // its last
    auto fill = [&](int p) {
        const unsigned f = (unsigned)(p - (zs - 1));
        auto &slot = M.slot[f % S];
        uint64_t *bar = &M.full[f % S];
        const bool whole = p >= zs;
        bar_expect(bar, (unsigned)(sizeof(slot.g) + (whole ? sizeof(slot.v) + (RESP ? sizeof(slot.r) : 0) : 0)));
        gvf_copy(slot.g, &a.mg, xr - 4, yr - 1, p + 1, bar);
        if (!whole) return;
        gvf_copy(slot.v, &a.mv, xr, yr, p, bar);
        if (RESP) tile_copy(slot.r, &a.mr, xr, yr, p, bar);
    };
    bool ok = true;
    auto wait = [&](int p) {
        const unsigned f = (unsigned)(p - (zs - 1));
        ok = bar_wait(&M.full[f % S], (f / S) & 1u) && ok;
    };
    if (copier)
        for (int p = zs - 1; p <= min(zl, zs + S - 2); ++p) fill(p);

    // [stage][plane mod 3][row][component]: three planes of the stage's input
    f2 G[K][3][RT][3] = {};
    if (zs > 0) {   // the plane before stage 1's first
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                G[0][0][r][c] = __ldg(reinterpret_cast<const f2 *>(
                    a.gi + c * a.comp + ((int64_t)(zs - 1) * d1 + min(y0 + r, d1 - 1)) * a.pitch + min(x, a.pitch - 2)));
    }
    wait(zs - 1);
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) G[0][1][r][c] = at2(&M.slot[0].g[c][row0 + r + 1][lx + 4]);
    float acc[K] = {};

    const int zend = zb - 1 + K - 1;
    for (int zz = zs; zz <= zend; zz += 3) {
#pragma unroll
        for (int ph = 0; ph < 3; ++ph) {
            const int z = zz + ph;
            if (z > zend) break;
            constexpr int kNext[3] = {2, 0, 1}, kHere[3] = {1, 2, 0}, kLast[3] = {0, 1, 2};
            __syncthreads();   // the last step's edges are stored, its slots read
            const unsigned f = (unsigned)(z - (zs - 1));
            // the slot last read a step ago: v of the last stage, g of the first
            if (copier && z - Lag >= zs - 1 && z - Lag + S <= zl) {
                if (ok) fill(z - Lag + S);
                else bar_release(&M.full[(f - Lag) % S], ((f - Lag + S) / S) & 1u);
            }
            if (z <= zl) {
                wait(z);
                const auto &cur = M.slot[f % S];
#pragma unroll
                for (int r = 0; r < RT; ++r)
#pragma unroll
                    for (int c = 0; c < 3; ++c) G[0][kNext[ph]][r][c] = at2(&cur.g[c][row0 + r + 1][lx + 4]);
            }
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int pz = z - k;
                if (pz < max(za - K + k + 1, 0) || pz > min(zb - 1 + K - 1 - k, d0 - 1)) continue;
                f2(&P)[RT][3] = G[k][kLast[ph]], (&C)[RT][3] = G[k][kHere[ph]], (&N)[RT][3] = G[k][kNext[ph]];
                if (pz == 0) {   // mirrored planes
#pragma unroll
                    for (int r = 0; r < RT; ++r)
#pragma unroll
                        for (int c = 0; c < 3; ++c) P[r][c] = d0 == 1 ? C[r][c] : N[r][c];
                }
                if (pz == d0 - 1) {
#pragma unroll
                    for (int r = 0; r < RT; ++r)
#pragma unroll
                        for (int c = 0; c < 3; ++c) N[r][c] = d0 == 1 ? C[r][c] : P[r][c];
                }
                const auto &slot = M.slot[(f + S - k) % S];
                const auto &gslot = M.slot[(f + S - 1) % S];   // g of plane z (stage 1)
                f2 w[RT][3], resp[RT], nrm[RT];
#pragma unroll
                for (int r = 0; r < RT; ++r) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) w[r][c] = at2(&slot.v[c][row0 + r][lx]);
                    resp[r] = RESP ? at2(&slot.r[RESP ? row0 + r : 0][lx])
                                   : fma2(w[r][2], w[r][2], fma2(w[r][1], w[r][1], mul2(w[r][0], w[r][0])));
                    nrm[r] = 0;
                }
                f2 O[RT][3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    f2 up, dn;   // the rows before and after the lane's
                    if (k == 0) {
                        up = at2(&gslot.g[c][row0][lx + 4]);
                        dn = at2(&gslot.g[c][row0 + RT + 1][lx + 4]);
                    } else {
                        up = M.edge[k > 0 ? k - 1 : 0][(z - 1) & 1][group][1][c][lane & 15];
                        dn = M.edge[k > 0 ? k - 1 : 0][(z - 1) & 1][group + 2][0][c][lane & 15];
                    }
                    if (!FLAT) {
                        if (top) up = RT > 1 ? C[RT > 1 ? 1 : 0][c] : dn;
                        if (bottom) dn = RT > 1 ? C[RT > 1 ? RT - 2 : 0][c] : up;
                    }
#pragma unroll
                    for (int r = 0; r < RT; ++r) {
                        const f2 ctr = C[r][c];
                        f2 ya = r > 0 ? C[r > 0 ? r - 1 : 0][c] : up;
                        f2 yb = r + 1 < RT ? C[r + 1 < RT ? r + 1 : r][c] : dn;
                        if (FLAT) {
                            if (y0 + r == 0) ya = d1 == 1 ? ctr : yb;
                            if (y0 + r >= d1 - 1) yb = d1 == 1 ? ctr : ya;
                        }
                        float xa, xb;   // the columns before and after the pair
                        if (k == 0) {
                            const float *row = gslot.g[c][row0 + r + 1];
                            xa = row[coll];
                            xb = row[colg];
                        } else {
                            xa = __shfl_sync(0xffffffffu, hi2(ctr), srcl);
                            xb = __shfl_sync(0xffffffffu, lo2(ctr), srcg);
                        }
                        const f2 xs = pack2(__fadd_rn(xa, ghost ? xa : hi2(ctr)), __fadd_rn(lo2(ctr), xb));
                        const f2 t0 = fma2(m2, ctr, add2(P[r][c], N[r][c]));
                        const f2 t1 = fma2(m2, ctr, add2(ya, yb));
                        const f2 t2 = fma2(m2, ctr, xs);
                        const f2 lap = fma2(t2, rss2, fma2(t1, rss1, mul2(t0, rss0)));
                        const f2 e = fma2(resp[r], sub2(ctr, w[r][c]), mul2(nmu, lap));
                        O[r][c] = fma2(ndt, e, ctr);
                        if (CHECK) nrm[r] = fma2(e, e, nrm[r]);
                    }
                }
                // |delta| of the voxels this block writes
                if (CHECK && ((a.checks >> k) & 1) && pz >= za && pz < zb && xout) {
#pragma unroll
                    for (int r = 0; r < RT; ++r)
                        if (y0 + r >= ylo && y0 + r < yhi)
                            acc[k] += sqrtf(lo2(nrm[r])) + (pair ? sqrtf(hi2(nrm[r])) : 0.f);
                }
                if (k == K - 1) {
                    if (xout) {
#pragma unroll
                        for (int r = 0; r < RT; ++r) {
                            const int y = y0 + r;
                            if (y >= ylo && y < yhi) {   // rows are padded: the pair always fits
                                const int64_t o = ((int64_t)pz * d1 + y) * a.pitch + x;
#pragma unroll
                                for (int c = 0; c < 3; ++c)
                                    *reinterpret_cast<f2 *>(a.go + c * a.comp + o) = O[r][c];
                            }
                        }
                    }
                } else {
                    constexpr int k1 = K > 1 ? K - 1 : 1;   // (the last stage has no next)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        M.edge[k % k1][z & 1][group + 1][0][c][lane & 15] = O[0][c];
                        M.edge[k % k1][z & 1][group + 1][1][c][lane & 15] = O[RT - 1][c];
#pragma unroll
                        for (int r = 0; r < RT; ++r) G[(k + 1) % K][kNext[ph]][r][c] = O[r][c];
                    }
                }
            }
        }
    }
    if (!ok) tile_fail(a.fail);
    if (CHECK) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (!((a.checks >> k) & 1)) continue;
            __syncthreads();
            const float s = block_sum(acc[k], red);
            if (lane == 0 && warp == 0) a.partials[k * gridDim.x + blockIdx.x] = s;
        }
    }
}

}  // namespace
}  // namespace m16
