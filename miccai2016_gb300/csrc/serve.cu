// serve.cu -- continuous batching of ATV max-flow requests (m16_server_*).
//
// A request is one volume with its own solve (an instance of the batched
// engine, batch_kernels.cuh).  The server holds one caller workspace: its
// tables (descriptors, control words, work list) at the front and an arena for
// the requests behind them.  Admission allocates a request's inputs, state and
// partial sums in one arena block; the inputs are uploaded on the server's copy
// stream and the set-up kernels run on the compute stream behind an event, so
// uploads overlap the iterations of resident requests; iteration 0 and its
// check follow the set-up.  A step runs the params->update iterations up to the
// next check of every resident request (without a check for a request in its
// last iterations), reads the stop mask, retires requests at the bound or at
// num_iter, and starts their u downloads on the copy stream; poll() hands out
// requests whose download has finished and returns their memory.
//
// Steps are pipelined by one: a step call enqueues the next step first and
// only then waits for the previous step's stop mask, so the device runs while
// the host retires, admits and polls.  A request that stopped in step k is
// still listed (masked, no work) in step k + 1; its slot and memory are
// reused only after the last step that lists it has been processed.
#include <cuda_runtime.h>
#include <math.h>
#include <float.h>

#include <algorithm>
#include <iterator>
#include <map>
#include <utility>
#include <vector>

#include "batch_kernels.cuh"

namespace m16 {
namespace {

constexpr size_t kAlign = 256;

// first-fit allocator over [0, size) in 256-byte granules; adjacent free
// ranges are merged on release
class Arena {
public:
    void init(size_t size) {
        free_.clear();
        used_.clear();
        if (size >= kAlign) free_[0] = size / kAlign * kAlign;
    }
    bool alloc(size_t bytes, size_t *off) {
        bytes = align_up(std::max<size_t>(bytes, 1), kAlign);
        for (auto it = free_.begin(); it != free_.end(); ++it) {
            if (it->second < bytes) continue;
            const size_t o = it->first, sz = it->second;
            free_.erase(it);
            if (sz > bytes) free_[o + bytes] = sz - bytes;
            used_[o] = bytes;
            *off = o;
            return true;
        }
        return false;
    }
    void release(size_t off) {
        auto u = used_.find(off);
        if (u == used_.end()) return;
        const size_t o = u->first;
        size_t sz = u->second;
        used_.erase(u);
        auto nx = free_.lower_bound(o);
        if (nx != free_.end() && o + sz == nx->first) {   // merge with the next range
            sz += nx->second;
            nx = free_.erase(nx);
        }
        if (nx != free_.begin()) {                          // and with the previous one
            auto pv = std::prev(nx);
            if (pv->first + pv->second == o) {
                pv->second += sz;
                return;
            }
        }
        free_[o] = sz;
    }
    size_t free_bytes() const {
        size_t t = 0;
        for (const auto &f : free_) t += f.second;
        return t;
    }
    size_t largest() const {
        size_t m = 0;
        for (const auto &f : free_) m = std::max(m, f.second);
        return m;
    }

private:
    std::map<size_t, size_t> free_, used_;   // offset -> size
};

// Where a request's fields sit in its arena block.  Tile sweeps: 72 bytes a
// voxel, the two state buffers, the directions and the capacities.  The inputs
// are read by the set-up kernels only and share that memory: the image sits
// where the capacities go (the state is written first), the others where the
// second state buffer is, the maximum where the directions go; the result is
// gathered there at the end.  Compact: the inputs stay, one planar state.
struct ReqLayout {
    size_t img, quat3, alpha, cs, ct, maxpart, denom, total;
    size_t h[2], u[2], dir, caps, rad;         // tile sweeps
    size_t q4, state;                          // compact sweeps
    size_t partials;                           // tiles > kSlotPartials
    int tiles, zc;
    bool compact;
    int64_t n, slab;
};

constexpr int kSlotPartials = 1024;   // partial sums kept in the server's tables per slot

inline ReqLayout req_layout(int d0, int d1, int d2, bool compact, bool rad)
{
    ReqLayout R;
    const int64_t n = (int64_t)d0 * d1 * d2;
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off = align_up(off + bytes, kAlign); return o; };
    R.n = n;
    R.compact = compact;
    R.quat3 = take(n * 12);
    R.alpha = take(n * 4);   // |grad I|^2, or the per-voxel alpha
    R.cs = take(n * 4);
    R.ct = take(n * 4);
    R.slab = (int64_t)(align_up(n * 4, kAlign) / 4);
    if (compact) {
        R.img = take(n * 4);
        R.q4 = take(n * 16);
        R.state = take(kFields * R.slab * 4);
        R.zc = compact_zc(d0, d1, d2);
        R.tiles = compact_tiles(d0, d1, d2);
        R.maxpart = take(kSetupBlocks * 4);
        R.denom = take(4);
    } else {
        const size_t np = (size_t)tile_voxels(d0, d1, d2);
        R.h[1] = 0;
        R.u[1] = align_up(np * 16, kAlign);
        off = std::max(off, R.u[1] + align_up(np * 8, kAlign));
        R.h[0] = take(np * 16);
        R.u[0] = take(np * 8);
        R.dir = take(std::max<size_t>(np * 16, kSetupBlocks * 4 + 4));
        R.caps = R.img = take(np * 8);
        R.rad = rad ? take(np * 4) : 0;
        R.maxpart = R.dir;
        R.denom = R.dir + kSetupBlocks * 4;
        // the chunk of z as if four such requests shared the device
        const int nx = tile_count_x(d2), ny = tile_count_y(d1, kTileRows);
        R.zc = tile_zc(d0, 4 * (int64_t)nx * ny);
        R.tiles = (int)(nx * ny * div_up(d0, R.zc));
    }
    R.partials = R.tiles > kSlotPartials ? take((size_t)R.tiles * 4) : 0;
    R.total = off;
    return R;
}

struct Tables {
    size_t vols, tiles, maps, groups, insts, ctrl, state, work, list, partials, err, total;
};

inline Tables tables(int max_slots, int max_work)
{
    Tables T;
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off = align_up(off + bytes, kAlign); return o; };
    T.vols = take(sizeof(VolDev) * max_slots);
    T.tiles = take(sizeof(TileDev) * max_slots);
    T.maps = take(8 * sizeof(CUtensorMap) * max_slots);
    T.groups = take(sizeof(GroupDev) * max_slots);
    T.insts = take(sizeof(InstDev) * max_slots);
    T.ctrl = take(sizeof(InstCtrl) * max_slots);
    T.state = take(sizeof(unsigned) * max_slots);
    T.work = take(sizeof(int2) * (size_t)max_work);
    T.list = take(sizeof(int) * max_slots);
    T.partials = take(sizeof(float) * kSlotPartials * (size_t)max_slots);
    T.err = take(sizeof(int));
    T.total = off;
    return T;
}

enum SlotState { kFree = 0, kResident = 1, kDraining = 2 };

struct Slot {
    int state = kFree;
    int iters_planned = 0;   // iterations enqueued so far (before any stop is known)
    bool done_planning = false;   // its last step is enqueued
    int64_t last_listed = -1;   // the last step whose work list holds the slot
    int64_t tag = 0;
    size_t block = 0;        // arena offset (from the arena's base)
    size_t u_off = 0;        // workspace offset of the contiguous u
    int64_t n = 0;
    int tiles = 0, kind = 0;
    int iters_done = 0;      // iterations run so far
    int iterations = 0;      // at retirement
    double resid = NAN;
    float *u_host = nullptr;
    cudaEvent_t ev = nullptr;   // draining: the u download
};

// pinned host copies of one slot's descriptors, uploaded at admission
struct Staging {
    VolDev vol;
    TileDev tile;
    GroupDev group;
    InstDev inst;
    InstCtrl ctrl;
    unsigned state;
    CUtensorMap maps[8];
};

}  // namespace
}  // namespace m16

using namespace m16;

struct m16_server {
    m16_cut_params params;
    cudaStream_t stream = nullptr, copy = nullptr;
    // per step parity (steps k and k + 1 are in flight together): the end of
    // the step's kernels, its stop-mask copy, and timed events around its kernels
    cudaEvent_t step_end[2] = {nullptr, nullptr}, ctrl_ev[2] = {nullptr, nullptr};
    cudaEvent_t t_start[2] = {nullptr, nullptr}, t_end[2] = {nullptr, nullptr};
    char *ws = nullptr;
    size_t ws_bytes = 0;
    int max_slots = 0, max_work = 0;
    Tables T;
    size_t arena_base = 0;
    Arena arena;
    std::vector<Slot> slots;
    std::vector<int> free_slots;
    bool dirty = true;
    // pinned host buffers
    Staging *stage = nullptr;        // max_slots
    int2 *work_h[2] = {nullptr, nullptr};   // max_work each, by rebuild parity
    int *list_h[2] = {nullptr, nullptr};    // max_slots each, by rebuild parity
    InstCtrl *ctrl_h[2] = {nullptr, nullptr};   // max_slots each, by step parity
    int *err_h = nullptr;            // by step parity: a sweep's copies did not arrive
    // the work list: requests whose step ends with a check, then those in
    // their last iterations; the check list holds the former first
    int seg[2][kKinds + 1] = {};
    int n_full = 0, n_list = 0;      // slots with a check, slots in the current list
    int64_t rebuilds = 0;
    std::vector<int> list_cur;       // the current list (host copy)
    // the list of each step in flight, by step parity: slots and the
    // iterations they have run after it
    std::vector<std::pair<int, int>> step_list[2];
    int64_t steps = 0;               // steps enqueued
    int64_t processed = 0;           // steps whose stop masks have been read (all steps < processed)
    int64_t voxel_iterations = 0;    // iterations that ran, times each request's voxels
    double gpu_ms = 0.0;             // device time of the steps' kernels
    bool failed = false;             // a step's copies did not arrive: no further admission or step
    struct Done {
        int64_t tag;
        int iterations;
        double resid;
    };
    std::vector<Done> done;          // downloaded, not yet polled (by value: the slot may be reused)
};

namespace {

void release_host(m16_server *s)
{
    if (s->stage) cudaFreeHost(s->stage);
    for (int b = 0; b < 2; ++b) {
        if (s->work_h[b]) cudaFreeHost(s->work_h[b]);
        if (s->list_h[b]) cudaFreeHost(s->list_h[b]);
        if (s->ctrl_h[b]) cudaFreeHost(s->ctrl_h[b]);
        if (s->step_end[b]) cudaEventDestroy(s->step_end[b]);
        if (s->ctrl_ev[b]) cudaEventDestroy(s->ctrl_ev[b]);
        if (s->t_start[b]) cudaEventDestroy(s->t_start[b]);
        if (s->t_end[b]) cudaEventDestroy(s->t_end[b]);
    }
    if (s->err_h) cudaFreeHost(s->err_h);
    for (Slot &sl : s->slots)
        if (sl.ev) cudaEventDestroy(sl.ev);
    if (s->copy) cudaStreamDestroy(s->copy);
}

// whether the slot's next step ends with a check: iteration 0 and its check ran
// at admission, a step is the `update` iterations up to the next check, the
// last step those that remain without one
bool full_step(const m16_server *s, const Slot &sl)
{
    return sl.iters_planned - 1 + s->params.update < s->params.num_iter;
}

// rebuild the work list and the check list over the resident slots that
// still have a step to run.  The host sources alternate by rebuild: the
// copy from a buffer is ordered before the step enqueued after it, which has
// been processed (its stop mask read) before the buffer's next rebuild.
int rebuild(m16_server *s)
{
    const int rb = (int)(s->rebuilds & 1);
    int2 *work = s->work_h[rb];
    int *list = s->list_h[rb];
    int nw = 0, nl = 0;
    s->list_cur.clear();
    for (int pass = 0; pass < 2; ++pass) {
        for (int kind = 0; kind < kKinds; ++kind) {
            s->seg[pass][kind] = nw;
            for (int k = 0; k < s->max_slots; ++k) {
                const Slot &sl = s->slots[k];
                if (sl.state != kResident || sl.kind != kind || sl.done_planning) continue;
                if (full_step(s, sl) != (pass == 0)) continue;
                if (nw + sl.tiles > s->max_work) return M16_ERR_TOO_LARGE;
                for (int t = 0; t < sl.tiles; ++t) work[nw++] = make_int2(k, t);
                list[nl++] = k;
                s->list_cur.push_back(k);
            }
        }
        s->seg[pass][kKinds] = nw;
        if (pass == 0) s->n_full = nl;
    }
    s->n_list = nl;
    if (nw > 0)
        M16_CUDA_TRY(cudaMemcpyAsync(s->ws + s->T.work, work, sizeof(int2) * nw, cudaMemcpyHostToDevice, s->stream));
    if (nl > 0)
        M16_CUDA_TRY(cudaMemcpyAsync(s->ws + s->T.list, list, sizeof(int) * nl, cudaMemcpyHostToDevice, s->stream));
    s->rebuilds += 1;
    s->dirty = false;
    return M16_OK;
}

BatchTables server_tables(m16_server *s)
{
    BatchTables B;
    B.work = (const int2 *)(s->ws + s->T.work);
    B.tiles = (const TileDev *)(s->ws + s->T.tiles);
    B.vols = (const VolDev *)(s->ws + s->T.vols);
    B.groups = (const GroupDev *)(s->ws + s->T.groups);
    B.insts = (const InstDev *)(s->ws + s->T.insts);
    B.ctrl = (InstCtrl *)(s->ws + s->T.ctrl);
    B.state = (unsigned *)(s->ws + s->T.state);
    B.partials = (float *)s->ws;   // part_off counts floats from the workspace start
    return B;
}

cudaError_t launch_check(m16_server *s, const BatchTables &B, int count, const int *list, int first, int flip)
{
    return launch_pdl(bt_check_kernel, dim3(count), dim3(256), s->stream, true, B.insts, B.ctrl, B.state,
                      (const float *)B.partials, s->params.error_bound, s->params.update, flip, list, first);
}

// the retired slot's u goes to the host on the copy stream, after the step
// (of parity b) in which it became final; flip: that step ended without the
// check that stores the current buffer, after an odd number of launches
int start_download(m16_server *s, int k, int b, int flip)
{
    Slot &sl = s->slots[k];
    sl.state = kDraining;
    M16_CUDA_TRY(cudaStreamWaitEvent(s->copy, s->step_end[b], 0));
    if (sl.kind < kTileKinds) {
        // the tile sweeps' u is padded and beside p_t: gathered first (steps
        // that still list the slot do not touch it any more)
        const int blocks = (int)std::min<int64_t>(kSetupBlocks, div_up(sl.n, 256));
        const BatchTables B = server_tables(s);
        bt_result_kernel<<<dim3(blocks, 1), 256, 0, s->copy>>>(B.insts, B.state, k, flip);
        M16_CUDA_TRY(cudaGetLastError());
    }
    M16_CUDA_TRY(cudaMemcpyAsync(sl.u_host, s->ws + sl.u_off, sl.n * 4, cudaMemcpyDeviceToHost, s->copy));
    M16_CUDA_TRY(cudaEventRecord(sl.ev, s->copy));
    s->dirty = true;
    return M16_OK;
}

int process_step(m16_server *s, int64_t idx);

// hand out downloaded slots and return their memory: once the download has
// finished and every step that lists the slot has been processed.  Steps
// whose stop masks have arrived are processed first (without waiting), so the
// last requests come back without another step call.
void collect(m16_server *s)
{
    while (!s->failed && s->processed < s->steps && cudaEventQuery(s->ctrl_ev[s->processed & 1]) == cudaSuccess)
        if (process_step(s, s->processed) != M16_OK) break;
    for (int k = 0; k < s->max_slots; ++k) {
        Slot &sl = s->slots[k];
        if (sl.state != kDraining || sl.last_listed >= s->processed) continue;
        if (cudaEventQuery(sl.ev) != cudaSuccess) continue;
        s->arena.release(sl.block);
        sl.state = kFree;
        s->free_slots.push_back(k);
        s->done.push_back({sl.tag, sl.iterations, sl.resid});
    }
}

}  // namespace

extern "C" size_t m16_server_request_bytes(int32_t d0, int32_t d1, int32_t d2, int32_t has_alpha)
{
    (void)has_alpha;   // the alpha field takes the place of |grad I|^2
    if (d0 < 1 || d1 < 1 || d2 < 1 || (int64_t)d0 * d1 * d2 > (int64_t)INT32_MAX) return 0;
    const bool tiled = tile_shape_ok(d0, d1, d2);
    const size_t bytes = req_layout(d0, d1, d2, !tiled, false).total;
    // with few rows the sweeps depend on the eigenvalues
    if (!tiled || tile_rows_ok(kMetricConst, d0, d1, d2, kSmallInstance)) return bytes;
    return std::max(bytes, req_layout(d0, d1, d2, true, false).total);
}

extern "C" size_t m16_server_table_bytes(int32_t max_slots, int32_t max_work_items)
{
    if (max_slots < 1 || max_work_items < 1) return 0;
    return tables(max_slots, max_work_items).total;
}

extern "C" int m16_server_create(const m16_cut_params *params, int32_t max_slots, int32_t max_work_items,
                                 void *workspace, size_t workspace_bytes, void *stream, m16_server **out)
{
    if (!out) return M16_ERR_BAD_ARG;
    *out = nullptr;
    if (!params || params->update < 1 || params->num_iter < 1 || params->num_iter % params->update != 0 ||
        !(params->cc > 0.0) || max_slots < 1 || max_work_items < 1)
        return M16_ERR_BAD_ARG;
    const Tables T = tables(max_slots, max_work_items);
    if (!workspace || ((uintptr_t)workspace & (kAlign - 1)) || workspace_bytes < T.total + kAlign)
        return M16_ERR_WORKSPACE;
    m16_server *s = new m16_server();
    s->params = *params;
    s->stream = (cudaStream_t)stream;
    s->ws = (char *)workspace;
    s->ws_bytes = workspace_bytes;
    s->max_slots = max_slots;
    s->max_work = max_work_items;
    s->T = T;
    s->arena_base = T.total;
    s->arena.init(workspace_bytes - T.total);
    s->slots.resize(max_slots);
    for (int k = max_slots - 1; k >= 0; --k) s->free_slots.push_back(k);
    bool ok = cudaStreamCreateWithFlags(&s->copy, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMallocHost((void **)&s->stage, sizeof(Staging) * max_slots) == cudaSuccess &&
              cudaMallocHost((void **)&s->err_h, 2 * sizeof(int)) == cudaSuccess &&
              cudaMemsetAsync(s->ws + T.err, 0, sizeof(int), s->stream) == cudaSuccess;
    for (int k = 0; ok && k < kTileKinds; ++k) ok = batch_tile_prepare(k) == cudaSuccess;
    for (int b = 0; ok && b < 2; ++b)
        ok = cudaEventCreateWithFlags(&s->step_end[b], cudaEventDisableTiming) == cudaSuccess &&
             cudaEventCreateWithFlags(&s->ctrl_ev[b], cudaEventDisableTiming) == cudaSuccess &&
             cudaEventCreate(&s->t_start[b]) == cudaSuccess && cudaEventCreate(&s->t_end[b]) == cudaSuccess &&
             cudaMallocHost((void **)&s->work_h[b], sizeof(int2) * (size_t)max_work_items) == cudaSuccess &&
             cudaMallocHost((void **)&s->list_h[b], sizeof(int) * max_slots) == cudaSuccess &&
             cudaMallocHost((void **)&s->ctrl_h[b], sizeof(InstCtrl) * max_slots) == cudaSuccess;
    for (int k = 0; ok && k < max_slots; ++k)
        ok = cudaEventCreateWithFlags(&s->slots[k].ev, cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        release_host(s);
        delete s;
        return M16_ERR_CUDA;
    }
    *out = s;
    return M16_OK;
}

extern "C" int m16_server_admit(m16_server *s, const m16_serve_request *req, int32_t *admitted)
{
    if (!s || !req || !admitted) return M16_ERR_BAD_ARG;
    *admitted = 0;
    if (s->failed) return M16_ERR_TIMEOUT;
    if (req->d0 < 1 || req->d1 < 1 || req->d2 < 1) return M16_ERR_BAD_SHAPE;
    if ((int64_t)req->d0 * req->d1 * req->d2 > (int64_t)INT32_MAX) return M16_ERR_BAD_SHAPE;
    if (!req->img || !req->quat3 || !req->cs || !req->ct || !req->u) return M16_ERR_BAD_ARG;
    if (!req->alpha && (!req->grad2 || !(req->decay != 0.0))) return M16_ERR_BAD_ARG;
    for (int k = 0; k < 3; ++k)
        if (!(req->scaling[k] > 0.0) || !(req->sqevals[k] > 0.0)) return M16_ERR_BAD_ARG;
    collect(s);
    if (s->failed) return M16_ERR_TIMEOUT;
    if (s->free_slots.empty()) return M16_OK;
    TileView view = TileView();
    int axis;
    const int metric = tile_metric(req->sqevals, view, &axis);
    tile_view(view, req->d0, req->d1, req->d2, req->scaling, s->params);
    const bool rad = metric == kMetricConst;   // a radius field beside the quaternions
    const bool tiled = tile_shape_ok(req->d0, req->d1, req->d2) &&
                       tile_rows_ok(metric, req->d0, req->d1, req->d2, kSmallInstance);
    ReqLayout R = req_layout(req->d0, req->d1, req->d2, !tiled, rad);
    size_t block;
    if (R.tiles > s->max_work || !s->arena.alloc(R.total, &block)) {
        // A request that the tile sweeps' fields do not fit even alone takes the
        // compact sweeps' (68 bytes a voxel); others wait for room.
        const bool alone = (int)s->free_slots.size() == s->max_slots;
        const ReqLayout C = req_layout(req->d0, req->d1, req->d2, true, false);
        if (R.tiles > s->max_work && C.tiles > s->max_work) return M16_ERR_TOO_LARGE;
        if ((R.tiles <= s->max_work && !alone) || C.tiles > s->max_work || !s->arena.alloc(C.total, &block))
            return M16_OK;
        R = C;
    }
    const int k = s->free_slots.back();
    s->free_slots.pop_back();
    Slot &sl = s->slots[k];
    char *base = s->ws + s->arena_base + block;
    const int64_t n = R.n;
    cudaStream_t cp = s->copy, st = s->stream;

    // inputs on the copy stream
    M16_CUDA_TRY(cudaMemcpyAsync(base + R.img, req->img, n * 4, cudaMemcpyHostToDevice, cp));
    M16_CUDA_TRY(cudaMemcpyAsync(base + R.quat3, req->quat3, n * 12, cudaMemcpyHostToDevice, cp));
    M16_CUDA_TRY(cudaMemcpyAsync(base + R.alpha, req->alpha ? req->alpha : req->grad2, n * 4,
                                 cudaMemcpyHostToDevice, cp));
    M16_CUDA_TRY(cudaMemcpyAsync(base + R.cs, req->cs, n * 4, cudaMemcpyHostToDevice, cp));
    M16_CUDA_TRY(cudaMemcpyAsync(base + R.ct, req->ct, n * 4, cudaMemcpyHostToDevice, cp));

    // descriptors (staged in pinned memory, uploaded on the copy stream too)
    Staging &S = s->stage[k];
    const float *img = (const float *)(base + R.img), *quat3 = (const float *)(base + R.quat3);
    const float *value = (const float *)(base + R.alpha), *cs = (const float *)(base + R.cs),
                *ct = (const float *)(base + R.ct);
    float *denom = (float *)(base + R.denom);
    const float w = (float)req->weighting;
    const float nid2 = req->alpha ? 0.f : (float)(-1.0 / (req->decay * req->decay));
    const int64_t part_off = (int64_t)((R.tiles > kSlotPartials ? s->arena_base + block + R.partials
                                                                 : s->T.partials + sizeof(float) * kSlotPartials * k) / 4);
    S.inst.n = n;
    S.inst.part_off = part_off;
    S.inst.nparts = R.tiles;
    S.inst.d2 = req->d2;
    S.inst.rcc = view.rcc;
    S.inst.u2[0] = S.inst.u2[1] = nullptr;
    S.inst.u1 = nullptr;
    S.inst.u_out = nullptr;
    S.vol = VolDev();
    S.group = GroupDev();
    S.tile = TileDev();
    VolumeFields F = VolumeFields();
    if (R.compact) {
        compact_volume(S.vol, req->d0, req->d1, req->d2, R.zc, view);
        S.vol.q4 = (const float4 *)(base + R.q4);
        S.vol.grad2 = req->alpha ? nullptr : value;
        S.vol.cs = cs; S.vol.ct = ct;
        GroupDev &g = S.group;
        g.vol = k;
        g.part_off = part_off;
        g.w = w;
        g.nid2 = nid2;
        g.sq0 = view.sq0; g.sq1 = view.sq1; g.sq2 = view.sq2;
        g.isq0 = view.isq0; g.isq1 = view.isq1; g.isq2 = view.isq2;
        g.state = (float *)(base + R.state);
        g.slab = R.slab;
        g.alpha = req->alpha ? value : nullptr;
        g.img = img;
        g.denom = denom;
        S.inst.u1 = g.state + 5 * g.slab;
        sl.kind = req->alpha ? kCompactAlpha : kCompactExp;
    } else {
        TileDev &t = S.tile;
        t.V = view;
        t.V.exp_radius = req->alpha ? 0 : 1;
        t.V.w = w;
        t.V.nid2 = nid2;
        t.V.labels = nullptr;
        t.fail = TileFail{(int *)(s->ws + s->T.err), (int *)(s->ws + s->T.state) + k};
        CUtensorMap *dm = (CUtensorMap *)(s->ws + s->T.maps) + 8 * k;
        bool ok = true;
        for (int b = 0; b < 2; ++b) {
            t.h[b] = (float4 *)(base + R.h[b]);
            t.u[b] = (float2 *)(base + R.u[b]);
            ok = ok && tile_map(S.maps + b, t.h[b], req->d0, req->d1, view.pitch, 4, kTileRows + 1) &&
                 tile_map(S.maps + 2 + b, t.u[b], req->d0, req->d1, view.pitch, 2, kTileRows);
            t.mh[b] = dm + b;
            t.mu[b] = dm + 2 + b;
            S.inst.u2[b] = t.u[b];
        }
        F.caps = (float2 *)(base + R.caps);
        ok = ok && tile_map(S.maps + 4, F.caps, req->d0, req->d1, view.pitch, 2, kTileRows);
        t.V.mcaps = dm + 4;
        // the direction with the radius, the radius alone in its place, or the
        // quaternion and a radius field
        if (metric == kMetricAxis) F.dir[axis] = (float4 *)(base + R.dir);
        else if (metric == kMetricConst) F.q4 = (float4 *)(base + R.dir);
        if (metric != kMetricAxis) F.rad = (float *)(base + (metric == kMetricConst ? R.rad : R.dir));
        if (metric != kMetricIso)
            ok = ok && tile_map(S.maps + 5, base + R.dir, req->d0, req->d1, view.pitch, 4, kTileRows);
        if (F.rad) ok = ok && tile_map(S.maps + 6, F.rad, req->d0, req->d1, view.pitch, 1, kTileRows);
        if (!ok) {
            s->arena.release(block);
            s->free_slots.push_back(k);
            return M16_ERR_CUDA;
        }
        t.V.mdir = dm + 5;
        t.V.mrad = dm + 6;
        t.part_off = part_off;
        t.rows = (int64_t)req->d0 * req->d1;
        t.nx = tile_count_x(req->d2);
        t.ny = tile_count_y(req->d1, kTileRows);
        t.zc = R.zc;
        t.img = img; t.cs = cs; t.ct = ct; t.alpha = nullptr; t.denom = denom; t.rad = nullptr;
        S.inst.u_out = (float *)(base + R.dir);
        sl.kind = metric == kMetricAxis ? kAxisPacked : metric == kMetricIso ? kIsoPlanar : kConstPlanar;
        M16_CUDA_TRY(cudaMemcpyAsync(dm, S.maps, sizeof(S.maps), cudaMemcpyHostToDevice, cp));
    }
    S.ctrl = InstCtrl{0, s->params.num_iter, 0, 0, NAN};
    S.state = 0u;
    auto up = [&](size_t table, const void *src, size_t bytes) {
        return cudaMemcpyAsync(s->ws + table + bytes * k, src, bytes, cudaMemcpyHostToDevice, cp);
    };
    M16_CUDA_TRY(up(s->T.vols, &S.vol, sizeof(VolDev)));
    M16_CUDA_TRY(up(s->T.tiles, &S.tile, sizeof(TileDev)));
    M16_CUDA_TRY(up(s->T.groups, &S.group, sizeof(GroupDev)));
    M16_CUDA_TRY(up(s->T.insts, &S.inst, sizeof(InstDev)));
    M16_CUDA_TRY(up(s->T.ctrl, &S.ctrl, sizeof(InstCtrl)));
    M16_CUDA_TRY(up(s->T.state, &S.state, sizeof(unsigned)));
    M16_CUDA_TRY(cudaEventRecord(sl.ev, cp));

    // set-up on the compute stream once the uploads are in, then iteration 0
    // and its check
    M16_CUDA_TRY(cudaStreamWaitEvent(st, sl.ev, 0));
    BatchTables B = server_tables(s);
    const int blocks = (int)std::min<int64_t>(kSetupBlocks, div_up(n, 256));
    float *mp = (float *)(base + R.maxpart);
    bt_max_kernel<<<blocks, 256, 0, st>>>(img, n, mp);
    bt_denom_kernel<<<1, 256, 0, st>>>(mp, blocks, denom);
    if (R.compact) {
        bt_expand_kernel<<<blocks, 256, 0, st>>>(quat3, (float4 *)(base + R.q4), n);
        bt1_state_kernel<<<dim3(blocks, 1), 256, 0, st>>>(B.vols, B.groups, k);
    } else {
        // in this order: the volume's fields overwrite the image and the maximum
        bt_state_kernel<<<dim3(blocks, 1), 256, 0, st>>>(B.tiles, k);
        bt_volume_kernel<<<blocks, 256, 0, st>>>(quat3, value, cs, ct, req->d2, (int64_t)req->d0 * req->d1, F);
    }
    M16_CUDA_TRY(cudaGetLastError());
    B.work = nullptr;
    B.first = k;
    for (int i = sl.kind + 1; i <= kKinds; ++i) B.seg[i] = R.tiles;
    int launches = 0;
    const int sweeps = enqueue_iterations(B, 1, true, st, launches);
    if (sweeps < 0) return M16_ERR_CUDA;
    M16_CUDA_TRY(launch_check(s, B, 1, nullptr, k, sweeps & 1));

    sl.state = kResident;
    sl.tag = req->tag;
    sl.block = block;
    sl.u_off = s->arena_base + block + (R.compact ? R.state + (size_t)5 * R.slab * 4 : R.dir);
    sl.n = n;
    sl.tiles = R.tiles;
    sl.iters_done = 0;
    sl.iters_planned = 1;
    sl.done_planning = false;
    sl.last_listed = -1;
    sl.iterations = 0;
    sl.resid = NAN;
    sl.u_host = req->u;
    s->dirty = true;
    *admitted = 1;
    return M16_OK;
}

namespace {

// read the stop mask of step idx (enqueued, not yet processed) and retire the
// requests that stopped in it or ran their last iteration in it
int process_step(m16_server *s, int64_t idx)
{
    if (idx != s->processed) return M16_ERR_BAD_ARG;   // in order only
    const int b = (int)(idx & 1);
    M16_CUDA_TRY(cudaEventSynchronize(s->ctrl_ev[b]));
    float step_ms = 0.f;
    M16_CUDA_TRY(cudaEventElapsedTime(&step_ms, s->t_start[b], s->t_end[b]));
    s->gpu_ms += step_ms;
    if (s->err_h[b]) s->failed = true;
    if (s->failed) return M16_ERR_TIMEOUT;
    for (const auto &entry : s->step_list[b]) {
        const int k = entry.first, target = entry.second;
        Slot &sl = s->slots[k];
        if (sl.state != kResident) continue;   // retired after an earlier step: masked here
        const InstCtrl &c = s->ctrl_h[b][k];
        sl.resid = c.resid;
        // a request that stopped at this step's check (or at iteration 0's)
        // ran up to it
        const int ran = c.stopped ? c.iterations : target;
        s->voxel_iterations += sl.n * std::max(0, ran - sl.iters_done);
        sl.iters_done = ran;
        if (!c.stopped && ran < s->params.num_iter) continue;
        sl.iterations = c.stopped ? c.iterations : s->params.num_iter;
        // the last iterations end without a check: update / 2 launches
        const int r = start_download(s, k, b, !c.stopped && (s->params.update / 2) & 1);
        if (r != M16_OK) return r;
    }
    s->processed = idx + 1;
    return M16_OK;
}

}  // namespace

extern "C" int m16_server_step(m16_server *s)
{
    if (!s) return M16_ERR_BAD_ARG;
    if (s->failed) return M16_ERR_TIMEOUT;
    collect(s);
    if (s->failed) return M16_ERR_TIMEOUT;
    if (s->dirty) {
        const int r = rebuild(s);
        if (r != M16_OK) return r;
    }
    const bool enqueue = s->n_list > 0;
    if (enqueue) {
        cudaStream_t st = s->stream;
        const int64_t c = s->steps;
        const int b = (int)(c & 1);   // step c - 2 of this parity has been processed
        BatchTables B = server_tables(s);
        M16_CUDA_TRY(cudaEventRecord(s->t_start[b], st));
        // programmatic dependent launch between the sweeps (common.cuh); the
        // first sweep follows an event record and launches in stream order
        int launches = 0;
        std::copy(s->seg[0], s->seg[0] + kKinds + 1, B.seg);
        if (s->n_full > 0) {
            const int sweeps = enqueue_iterations(B, s->params.update, true, st, launches);
            if (sweeps < 0) return M16_ERR_CUDA;
            M16_CUDA_TRY(launch_check(s, B, s->n_full, (const int *)(s->ws + s->T.list), 0, sweeps & 1));
        }
        std::copy(s->seg[1], s->seg[1] + kKinds + 1, B.seg);
        if (s->n_list > s->n_full && enqueue_iterations(B, s->params.update - 1, false, st, launches) < 0)
            return M16_ERR_CUDA;
        M16_CUDA_TRY(cudaGetLastError());
        M16_CUDA_TRY(cudaEventRecord(s->t_end[b], st));
        M16_CUDA_TRY(cudaEventRecord(s->step_end[b], st));
        M16_CUDA_TRY(cudaMemcpyAsync(s->ctrl_h[b], B.ctrl, sizeof(InstCtrl) * s->max_slots, cudaMemcpyDeviceToHost,
                                     st));
        M16_CUDA_TRY(cudaMemcpyAsync(s->err_h + b, s->ws + s->T.err, sizeof(int), cudaMemcpyDeviceToHost, st));
        M16_CUDA_TRY(cudaEventRecord(s->ctrl_ev[b], st));
        s->step_list[b].clear();
        for (int k : s->list_cur) {
            Slot &sl = s->slots[k];
            const bool full = full_step(s, sl);
            sl.iters_planned += full ? s->params.update : s->params.update - 1;
            sl.done_planning = !full;
            sl.last_listed = c;
            if (!full || !full_step(s, sl)) s->dirty = true;   // out of the next list, or in its other part
            s->step_list[b].push_back({k, sl.iters_planned});
        }
        s->steps = c + 1;
    }
    // the steps before the one just enqueued (all of them when none was)
    const int64_t upto = enqueue ? s->steps - 1 : s->steps;
    while (s->processed < upto) {
        const int r = process_step(s, s->processed);
        if (r != M16_OK) return r;
    }
    return M16_OK;
}

extern "C" int m16_server_poll(m16_server *s, int64_t *tags, int32_t *iterations, double *residuals, int32_t cap,
                               int32_t *n)
{
    if (!s || !n || cap < 0 || (cap > 0 && !tags)) return M16_ERR_BAD_ARG;
    collect(s);
    const int cnt = std::min<int>(cap, (int)s->done.size());
    for (int j = 0; j < cnt; ++j) {
        tags[j] = s->done[j].tag;
        if (iterations) iterations[j] = s->done[j].iterations;
        if (residuals) residuals[j] = s->done[j].resid;
    }
    s->done.erase(s->done.begin(), s->done.begin() + cnt);
    *n = cnt;
    return s->failed && cnt == 0 ? M16_ERR_TIMEOUT : M16_OK;
}

extern "C" int m16_server_get_info(const m16_server *s, m16_server_info *info)
{
    if (!s || !info) return M16_ERR_BAD_ARG;
    int res = 0, dr = 0;
    for (const Slot &sl : s->slots) {
        res += sl.state == kResident;
        dr += sl.state == kDraining;
    }
    info->resident = res;
    info->draining = dr;
    info->free_slots = (int32_t)s->free_slots.size();
    info->reserved = 0;
    info->free_bytes = (int64_t)s->arena.free_bytes();
    info->largest_free = (int64_t)s->arena.largest();
    info->steps = s->steps;
    info->voxel_iterations = s->voxel_iterations;
    info->gpu_ms = s->gpu_ms;
    return M16_OK;
}

extern "C" int m16_server_destroy(m16_server *s)
{
    if (!s) return M16_ERR_BAD_ARG;
    cudaError_t e1 = cudaStreamSynchronize(s->stream);
    cudaError_t e2 = s->copy ? cudaStreamSynchronize(s->copy) : cudaSuccess;
    release_host(s);
    delete s;
    return (e1 == cudaSuccess && e2 == cudaSuccess) ? M16_OK : M16_ERR_CUDA;
}
