// lost_copies.cu -- bulk copies that do not arrive, for the tile sweeps of the
// max-flow (PART 0), the gradient vector flow (PART 1) and the batch (PART 2).
//
// A copy is lost by a tensor map whose box is a row short: the copy itself is in
// order, in bounds and completes, but its bytes are fewer than the slot's barrier
// expects, so the barrier never completes and the sweep's wait has to run out.
// (Nothing traps and nothing spins without a limit.)
#if PART == 0
#include "maxflow.cu"
#elif PART == 1
#include "gvf.cu"
#else
#include "batch_kernels.cuh"
#endif

#include <algorithm>
#include <chrono>
#include <vector>

using namespace m16;

struct Outcome {
    int error, stop;       // after the call
    int untouched;         // the written buffers hold what they held before the call
    float ms;              // the launches, host clock
};

namespace {

double now_ms()
{
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// device memory full of one byte
char *filled(size_t bytes, int value)
{
    char *p = nullptr;
    if (cudaMalloc((void **)&p, bytes) != cudaSuccess || cudaMemset(p, value, bytes) != cudaSuccess) return nullptr;
    return p;
}

bool all_bytes(const char *dev, size_t bytes, unsigned char value)
{
    std::vector<unsigned char> h(bytes);
    if (cudaMemcpy(h.data(), dev, bytes, cudaMemcpyDeviceToHost) != cudaSuccess) return false;
    return std::all_of(h.begin(), h.end(), [&](unsigned char v) { return v == value; });
}

template <typename Launch>
bool timed(Launch launch, float *ms)
{
    if (cudaDeviceSynchronize() != cudaSuccess) return false;
    const double t0 = now_ms();
    launch();
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) return false;
    *ms = (float)(now_ms() - t0);
    return true;
}

}  // namespace

// out[0]: launches whose copies are lost; out[1]: a launch after them; out[2]: a
// launch with whole copies and a clean state.  Returns 0 when all ran.
#if PART == 0
namespace {
template <int METRIC, int ASRC, int K>
int lose(int d0, int d1, int d2, Outcome *out)
{
    const size_t np = (size_t)tile_voxels(d0, d1, d2);
    char *in = filled(np * 64, 0), *ho = filled(np * 16, 0x41), *uo = filled(np * 8, 0x41);
    MfCtrl *ctrl = (MfCtrl *)filled(sizeof(MfCtrl), 0);
    if (!in || !ho || !uo || !ctrl) return 1;
    MfTileArgs a = {};
    double sq[3] = {1.0, 0.5, METRIC == kMetricAxis ? 0.5 : 0.25};
    int axis;
    tile_metric(sq, a.V, &axis);
    a.V.d0 = d0; a.V.d1 = d1; a.V.d2 = d2; a.V.pitch = tile_pitch(d2);
    a.V.ss0 = a.V.ss1 = a.V.ss2 = 0.1f;
    a.V.rs0 = a.V.rs1 = a.V.rs2 = 1.f;
    a.V.rcc = 5.f; a.V.ircc = 0.2f;
    a.V.ho = (float4 *)ho; a.V.uo = (float2 *)uo;
    a.fail = TileFail{&ctrl->error, &ctrl->stopped};
    a.nx = tile_count_x(d2); a.ny = tile_count_y(d1, kTileRows); a.zc = d0;
    a.stopped = &ctrl->stopped;
    const int pitch = a.V.pitch;
    const MfTileLaunch k = mf_tile_kernel_of<METRIC, ASRC, false>(K, false);
    if (cudaFuncSetAttribute(k.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem) != cudaSuccess) return 2;
    for (int run = 0; run < 3; ++run) {
        const int rows = run < 2 ? kTileRows - 1 : kTileRows;
        if (!tile_map(&a.mh, in, d0, d1, pitch, 4, kTileRows + 1) || !tile_map(&a.mu, in, d0, d1, pitch, 2, rows) ||
            !tile_map(&a.mcaps, in, d0, d1, pitch, 2, kTileRows) || !tile_map(&a.mdir, in, d0, d1, pitch, 4, kTileRows) ||
            !tile_map(&a.mrad, in, d0, d1, pitch, 1, kTileRows))
            return 3;
        if (run == 2 && cudaMemset(ctrl, 0, sizeof(MfCtrl)) != cudaSuccess) return 4;
        if (cudaMemset(ho, 0x41, np * 16) != cudaSuccess || cudaMemset(uo, 0x41, np * 8) != cudaSuccess) return 4;
        if (!timed([&] { k.kernel<<<a.nx * a.ny, dim3(kTileLanes, kTileNW), k.smem>>>(a); }, &out[run].ms)) return 5;
        MfCtrl h;
        if (cudaMemcpy(&h, ctrl, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 6;
        out[run].error = h.error;
        out[run].stop = h.stopped;
        out[run].untouched = all_bytes(ho, np * 16, 0x41) && all_bytes(uo, np * 8, 0x41);
    }
    cudaFree(in); cudaFree(ho); cudaFree(uo); cudaFree(ctrl);
    return 0;
}
}  // namespace

extern "C" int lost_copies(int variant, int d0, int d1, int d2, Outcome *out)
{
    switch (variant) {
        case 0: return lose<kMetricAxis, kRadPacked, 2>(d0, d1, d2, out);
        case 1: return lose<kMetricAxis, kRadPacked, 1>(d0, d1, d2, out);
        default: return lose<kMetricConst, kRadPlanar, 2>(d0, d1, d2, out);
    }
}
#elif PART == 1
extern "C" int lost_copies(int variant, int d0, int d1, int d2, Outcome *out)
{
    const bool resp = variant == 1;
    const int k = gvf_iterations(resp), rows = gvf_rows(resp);
    const size_t np = (size_t)tile_voxels(d0, d1, d2);
    char *in = filled(np * 32, 0), *go = filled(np * 12, 0x41);
    GvfCtrl *ctrl = (GvfCtrl *)filled(sizeof(GvfCtrl), 0);
    if (!in || !go || !ctrl) return 1;
    GvfTileArgs a = {};
    a.d0 = d0; a.d1 = d1; a.d2 = d2; a.pitch = tile_pitch(d2);
    a.rss0 = a.rss1 = a.rss2 = 1.f;
    a.nmu = -0.2f; a.ndt = -0.1f;
    a.comp = (int64_t)np;
    a.gi = (const float *)in; a.go = (float *)go;
    a.fail = TileFail{&ctrl->error, &ctrl->stopped};
    a.ctrl = ctrl;
    GvfTileGrid G = gvf_tile_grid(d0, d1, d2, k, resp);
    G.zc = d0;   // one block marches through all planes
    G.blocks = G.nx * G.ny;
    a.nx = G.nx; a.ny = G.ny; a.zc = G.zc;
    size_t smem;
    const GvfTileKernel kernel = resp ? gvf_kernel<GvfShape<true>::K, true>(k, false, d1 < rows, &smem)
                                      : gvf_kernel<GvfShape<false>::K, false>(k, false, d1 < rows, &smem);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 2;
    for (int run = 0; run < 3; ++run) {
        const cuuint64_t dims[3] = {(cuuint64_t)a.pitch, (cuuint64_t)d1, (cuuint64_t)d0};
        const cuuint64_t row = (cuuint64_t)a.pitch * 4, strides[2] = {row, row * d1};
        const cuuint32_t box[3] = {kGvfVW, (cuuint32_t)rows, 1};
        if (!gvf_map(&a.mg, in, d0, d1, a.pitch, kGvfGW, rows + 2) ||
            !gvf_map(&a.mv, in, d0, d1, a.pitch, kGvfVW, run < 2 ? rows - 1 : rows) ||
            !tile_map_encode(&a.mr, in, 3, dims, strides, box))
            return 3;
        if (run == 2 && cudaMemset(ctrl, 0, sizeof(GvfCtrl)) != cudaSuccess) return 4;
        if (cudaMemset(go, 0x41, np * 12) != cudaSuccess) return 4;
        if (!timed([&] { kernel<<<G.blocks, dim3(kTileLanes, gvf_warps(resp)), smem>>>(a); }, &out[run].ms)) return 5;
        GvfCtrl h;
        if (cudaMemcpy(&h, ctrl, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 6;
        out[run].error = h.error;
        out[run].stop = h.stopped;
        out[run].untouched = all_bytes(go, np * 12, 0x41);
    }
    cudaFree(in); cudaFree(go); cudaFree(ctrl);
    return 0;
}
#else
extern "C" int lost_copies(int variant, int d0, int d1, int d2, Outcome *out)
{
    const size_t np = (size_t)tile_voxels(d0, d1, d2);
    char *in = filled(np * 64, 0), *ho = filled(np * 16, 0x41), *uo = filled(np * 8, 0x41);
    int *err = (int *)filled(256, 0);
    unsigned *state = (unsigned *)filled(256, 0);
    TileDev *tiles = (TileDev *)filled(sizeof(TileDev), 0);
    CUtensorMap *maps = (CUtensorMap *)filled(4 * sizeof(CUtensorMap), 0);
    float *partials = (float *)filled(1 << 16, 0);
    if (!in || !ho || !uo || !err || !state || !tiles || !maps || !partials) return 1;
    TileDev t = TileDev();
    double sq[3] = {1.0, 0.5, 0.5}, sc[3] = {1.0, 1.0, 1.0};
    int axis;
    tile_metric(sq, t.V, &axis);
    m16_cut_params p = {};
    p.cc = 0.2; p.steps = 0.11;
    tile_view(t.V, d0, d1, d2, sc, p);
    t.V.exp_radius = 1;
    t.V.w = 0.1f; t.V.nid2 = -0.01f;
    t.fail = TileFail{err, (int *)state};
    for (int k = 0; k < 2; ++k) {
        t.mh[k] = maps; t.mu[k] = maps + 1;
        t.h[k] = (float4 *)ho; t.u[k] = (float2 *)uo;
    }
    t.V.mdir = maps + 2; t.V.mcaps = maps + 3;
    t.nx = tile_count_x(d2); t.ny = tile_count_y(d1, kTileRows); t.zc = d0;
    const BatchTileLaunch k = batch_tile_pick(kAxisPacked, variant == 1 ? 1 : 2, true);
    if (batch_tile_prepare(kAxisPacked) != cudaSuccess) return 2;
    if (cudaMemcpy(tiles, &t, sizeof(t), cudaMemcpyHostToDevice) != cudaSuccess) return 3;
    for (int run = 0; run < 3; ++run) {
        CUtensorMap m[4];
        if (!tile_map(m, in, d0, d1, t.V.pitch, 4, kTileRows + 1) ||
            !tile_map(m + 1, in, d0, d1, t.V.pitch, 2, run < 2 ? kTileRows - 1 : kTileRows) ||
            !tile_map(m + 2, in, d0, d1, t.V.pitch, 4, kTileRows) || !tile_map(m + 3, in, d0, d1, t.V.pitch, 2, kTileRows))
            return 3;
        if (cudaMemcpy(maps, m, sizeof(m), cudaMemcpyHostToDevice) != cudaSuccess) return 4;
        if (run == 2 && (cudaMemset(err, 0, 256) != cudaSuccess || cudaMemset(state, 0, 256) != cudaSuccess)) return 4;
        if (cudaMemset(ho, 0x41, np * 16) != cudaSuccess || cudaMemset(uo, 0x41, np * 8) != cudaSuccess) return 4;
        if (!timed([&] { k.kernel<<<t.nx * t.ny, dim3(kTileLanes, kTileNW), k.smem>>>(nullptr, 0, tiles, state, partials, 0); },
                   &out[run].ms))
            return 5;
        if (cudaMemcpy(&out[run].error, err, 4, cudaMemcpyDeviceToHost) != cudaSuccess ||
            cudaMemcpy(&out[run].stop, state, 4, cudaMemcpyDeviceToHost) != cudaSuccess)
            return 6;
        out[run].untouched = all_bytes(ho, np * 16, 0x41) && all_bytes(uo, np * 8, 0x41);
    }
    cudaFree(in); cudaFree(ho); cudaFree(uo); cudaFree(err); cudaFree(state); cudaFree(tiles); cudaFree(maps);
    cudaFree(partials);
    return 0;
}
#endif
