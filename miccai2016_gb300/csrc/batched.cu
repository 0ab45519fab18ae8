// batched.cu -- m16_batch_solve: a fixed batch of ATV max-flow instances
// run to completion, every launch covering all active instances (device side
// and layout in batch_kernels.cuh).
#include <cuda_runtime.h>
#include <math.h>
#include <float.h>

#include <algorithm>
#include <cstddef>
#include <map>
#include <mutex>
#include <vector>

#include "batch_kernels.cuh"

namespace m16 {
namespace {

// ---- host side --------------------------------------------------------------

// Double-buffered state is asked for up to this many bytes.  In a workspace that
// does not hold the whole batch that way it is solved in cohorts that fit, one
// after the other, an instance that does not even fit alone by the compact
// sweeps; the step interface, which holds every instance at once, takes the
// compact sweeps for all of them.
constexpr size_t kPairBudget = (size_t)128 << 30;

// Tile shapes of the autotuner, named by their target blocks per SM: 16 is the
// chunk of z of batch_chunk's rule, 8 twice and 32 half of it.  The candidates
// are timed on one check interval each of the solve itself and the fastest is
// kept for the rest of it and for later batches of the same shape (a
// process-wide cache).
constexpr int kTuneBps[3] = {8, 16, 32};
constexpr int kDefaultBps = 16;
constexpr int kTuneMinItems = kTileBlocks * kSMs;   // less than a wave of blocks: keep the default

std::mutex g_tune_mu;
std::map<std::vector<int64_t>, int> g_tuned;   // batch shape -> blocks per SM

struct VolumePlan {
    int instances = 0;       // that refer to it
    bool tiles = false;      // padded fields for the tile sweeps
    bool compact = false;    // q4 of the compact sweeps
    bool axis[3] = {false, false, false}, q4 = false, rad = false;
};

struct BatchLayout {
    std::vector<VolumePlan> vol;
    std::vector<int> kind, axis;                      // per instance
    std::vector<size_t> caps, dir[3], vq4, vrad, cq4, maxpart;   // per volume (0 where absent)
    std::vector<size_t> h[2], u[2], rad, cstate;      // per instance
    size_t denom, ctrl, state, insts, tiles, maps, cvols, groups, work, partials, err, total;
    int64_t max_items;
};

// z-chunk of a volume of depth d0 for the batch's chunk zcb: equal chunks
inline int equal_chunk(int d0, int zcb) { return (int)div_up(d0, div_up(d0, std::max(zcb, 1))); }

// The batch's chunk of z: the least waves x marched planes over all instances'
// tiles (tile_zc's rule for one volume)
inline int batch_chunk(const m16_batch_volume *vols, int nvol, const std::vector<int> &instances, int bps)
{
    int dmax = 1;
    for (int v = 0; v < nvol; ++v)
        if (instances[v]) dmax = std::max(dmax, vols[v].d0);
    const int64_t slots = (int64_t)kTileBlocks * kSMs;
    int best = 1;
    int64_t cost = INT64_MAX;
    for (int zcb = 1; zcb <= std::min(dmax, 4096); ++zcb) {
        int64_t blocks = 0;
        for (int v = 0; v < nvol; ++v)
            blocks += (int64_t)instances[v] * tile_count_x(vols[v].d2) * tile_count_y(vols[v].d1, kTileRows) *
                      div_up(vols[v].d0, zcb);
        const int64_t c = div_up(blocks, slots) * (zcb + 4);
        if (c <= cost) {
            cost = c;
            best = zcb;
        }
    }
    return bps < kDefaultBps ? 2 * best : bps > kDefaultBps ? std::max(1, best / 2) : best;
}

inline std::vector<int> tile_instances(const BatchLayout &L)
{
    std::vector<int> n;
    for (const VolumePlan &v : L.vol) n.push_back(v.tiles ? v.instances : 0);
    return n;
}

// inst[first, last); compact: no double buffers
inline BatchLayout batch_layout(const m16_batch_volume *vols, int nvol, const m16_batch_instance *inst, int first,
                                int last, bool compact)
{
    BatchLayout L;
    const int ninst = last - first;
    L.vol.resize(nvol);
    for (int i = 0; i < ninst; ++i) {
        const m16_batch_instance &I = inst[first + i];
        const m16_batch_volume &V = vols[I.volume];
        VolumePlan &P = L.vol[I.volume];
        P.instances += 1;
        TileView view;
        int axis;
        const int metric = tile_metric(I.sqevals, view, &axis);
        L.axis.push_back(axis);
        if (compact || !tile_shape_ok(V.d0, V.d1, V.d2) ||
            !tile_rows_ok(metric, V.d0, V.d1, V.d2, kSmallInstance)) {
            P.compact = true;
            L.kind.push_back(I.alpha ? kCompactAlpha : kCompactExp);
            continue;
        }
        P.tiles = true;
        if (metric == kMetricAxis) {
            P.axis[axis] = true;
            L.kind.push_back(I.alpha ? kAxisPlanar : kAxisPacked);
        } else {
            P.q4 = P.q4 || metric == kMetricConst;
            P.rad = P.rad || !I.alpha;
            L.kind.push_back(metric == kMetricIso ? kIsoPlanar : kConstPlanar);
        }
    }
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off = align_up(off + bytes, 256); return o; };
    std::vector<int64_t> items(nvol, 0);
    int zmin = INT32_MAX;   // the finest candidate's chunk
    for (int c : kTuneBps) zmin = std::min(zmin, batch_chunk(vols, nvol, tile_instances(L), c));
    for (int v = 0; v < nvol; ++v) {
        const VolumePlan &P = L.vol[v];
        const int d0 = vols[v].d0, d1 = vols[v].d1, d2 = vols[v].d2;
        const size_t n = (size_t)d0 * d1 * d2, np = (size_t)tile_voxels(d0, d1, d2);
        L.maxpart.push_back(P.instances ? take(kSetupBlocks * 4) : 0);
        L.caps.push_back(P.tiles ? take(np * 8) : 0);
        for (int k = 0; k < 3; ++k) L.dir[k].push_back(P.axis[k] ? take(np * 16) : 0);
        L.vq4.push_back(P.q4 ? take(np * 16) : 0);
        L.vrad.push_back(P.rad ? take(np * 4) : 0);
        L.cq4.push_back(P.compact ? take(n * 16) : 0);
        const int64_t fine = (int64_t)tile_count_x(d2) * tile_count_y(d1, kTileRows) * div_up(d0, equal_chunk(d0, zmin));
        items[v] = std::max<int64_t>(P.tiles ? fine : 0, P.compact ? compact_tiles(d0, d1, d2) : 0);
    }
    L.max_items = 0;
    for (int i = 0; i < ninst; ++i) {
        const m16_batch_volume &V = vols[inst[first + i].volume];
        const size_t n = (size_t)V.d0 * V.d1 * V.d2, np = (size_t)tile_voxels(V.d0, V.d1, V.d2);
        const bool c = L.kind[i] >= kTileKinds;
        for (int k = 0; k < 2; ++k) {
            L.h[k].push_back(c ? 0 : take(np * 16));
            L.u[k].push_back(c ? 0 : take(np * 8));
        }
        L.rad.push_back(!c && inst[first + i].alpha ? take(np * 4) : 0);
        L.cstate.push_back(c ? take(kFields * align_up(n * 4, 256)) : 0);
        L.max_items += items[inst[first + i].volume];
    }
    L.denom = take(sizeof(float) * nvol);
    L.ctrl = take(sizeof(InstCtrl) * ninst);
    L.state = take(sizeof(unsigned) * ninst);
    L.insts = take(sizeof(InstDev) * ninst);
    L.tiles = take(sizeof(TileDev) * ninst);
    L.maps = take(sizeof(CUtensorMap) * (6 * (size_t)nvol + 5 * (size_t)ninst));
    L.cvols = take(sizeof(VolDev) * nvol);
    L.groups = take(sizeof(GroupDev) * ninst);
    L.work = take(sizeof(int2) * std::max<int64_t>(L.max_items, 1));
    L.partials = take(sizeof(float) * std::max<int64_t>(L.max_items, 1));
    L.err = take(sizeof(int));
    L.total = off;
    return L;
}

bool batch_args_ok(const m16_batch_volume *vols, int nvol, const m16_batch_instance *inst, int ninst)
{
    if (!vols || !inst || nvol < 1 || ninst < 1) return false;
    for (int v = 0; v < nvol; ++v) {
        const m16_batch_volume &V = vols[v];
        if (V.d0 < 1 || V.d1 < 1 || V.d2 < 1 || !V.img || !V.quat3 || !V.cs || !V.ct) return false;
        // the sweeps index a volume with 32-bit voxel offsets
        if ((int64_t)V.d0 * V.d1 * V.d2 > (int64_t)INT32_MAX) return false;
        for (int k = 0; k < 3; ++k)
            if (!(V.scaling[k] > 0.0)) return false;
    }
    for (int i = 0; i < ninst; ++i) {
        const m16_batch_instance &I = inst[i];
        if (I.volume < 0 || I.volume >= nvol || !I.u) return false;
        if (!I.alpha && (!vols[I.volume].grad2 || !(I.decay != 0.0))) return false;
        for (int k = 0; k < 3; ++k)
            if (!(I.sqevals[k] > 0.0)) return false;
    }
    return true;
}

// Workspace bytes of a batch
inline size_t batch_bytes(const m16_batch_volume *vols, int nvol, const m16_batch_instance *inst, int ninst)
{
    const size_t full = batch_layout(vols, nvol, inst, 0, ninst, false).total;
    if (full <= kPairBudget) return full;
    return std::max(kPairBudget, batch_layout(vols, nvol, inst, 0, ninst, true).total);
}

// The least that m16_batch_solve runs in: every instance alone, compact.  Such
// layouts differ in these fields only, so one of them is laid out.
inline size_t batch_bytes_min(const m16_batch_volume *vols, int nvol, const m16_batch_instance *inst, int ninst)
{
    size_t most = 0;
    int which = 0;
    for (int i = 0; i < ninst; ++i) {
        const m16_batch_volume &V = vols[inst[i].volume];
        const size_t n = (size_t)V.d0 * V.d1 * V.d2, items = compact_tiles(V.d0, V.d1, V.d2);
        const size_t bytes = align_up(n * 16, 256) + kFields * align_up(n * 4, 256) +
                             align_up(items * sizeof(int2), 256) + align_up(items * sizeof(float), 256);
        if (bytes > most) {
            most = bytes;
            which = i;
        }
    }
    return batch_layout(vols, nvol, inst, which, which + 1, true).total;
}

// A batch's descriptors on host and device and its work list
struct BatchRun {
    BatchLayout L;
    int nvol = 0, ninst = 0;
    const m16_batch_volume *vols = nullptr;   // valid during set-up only
    const m16_batch_instance *inst = nullptr;
    std::vector<TileDev> ht;
    std::vector<InstDev> hi;
    std::vector<VolDev> hv;
    std::vector<GroupDev> hg;
    std::vector<InstCtrl> hctrl;
    std::vector<unsigned> hstate;
    std::vector<CUtensorMap> hmaps;
    std::vector<int> volume;                  // per instance
    std::vector<int2> work;
    char *ws = nullptr;
    BatchTables T;
};

// Descriptors, uploads and the set-up kernels.  The uploads read the host
// vectors of B until they have run.
int batch_prepare(BatchRun &B, const m16_batch_volume *vols, int nvol, const m16_batch_instance *inst, int ninst,
                  const m16_cut_params *params, char *ws, cudaStream_t st)
{
    const BatchLayout &L = B.L;
    B.nvol = nvol;
    B.ninst = ninst;
    B.ws = ws;
    B.ht.assign(ninst, TileDev());
    B.hi.assign(ninst, InstDev());
    B.hv.assign(nvol, VolDev());
    B.hg.assign(ninst, GroupDev());
    B.hctrl.assign(ninst, InstCtrl());
    B.hstate.assign(ninst, 0u);
    B.hmaps.assign(6 * (size_t)nvol + 5 * (size_t)ninst, CUtensorMap());
    B.volume.resize(ninst);
    CUtensorMap *dmaps = (CUtensorMap *)(ws + L.maps);
    float *denom = (float *)(ws + L.denom);
    auto field = [&](size_t off) -> char * { return ws + off; };
    std::vector<TileView> view(nvol);
    for (int v = 0; v < nvol; ++v) {
        const m16_batch_volume &V = vols[v];
        const VolumePlan &P = L.vol[v];
        tile_view(view[v], V.d0, V.d1, V.d2, V.scaling, *params);
        const int pitch = view[v].pitch;
        CUtensorMap *m = B.hmaps.data() + 6 * v;
        bool ok = true;
        if (P.tiles) ok = ok && tile_map(m, field(L.caps[v]), V.d0, V.d1, pitch, 2, kTileRows);
        for (int k = 0; k < 3; ++k)
            if (P.axis[k]) ok = ok && tile_map(m + 1 + k, field(L.dir[k][v]), V.d0, V.d1, pitch, 4, kTileRows);
        if (P.q4) ok = ok && tile_map(m + 4, field(L.vq4[v]), V.d0, V.d1, pitch, 4, kTileRows);
        if (P.rad) ok = ok && tile_map(m + 5, field(L.vrad[v]), V.d0, V.d1, pitch, 1, kTileRows);
        if (!ok) return M16_ERR_CUDA;
        if (P.compact) {
            VolDev &d = B.hv[v];
            compact_volume(d, V.d0, V.d1, V.d2, compact_zc(V.d0, V.d1, V.d2), view[v]);
            d.q4 = (const float4 *)field(L.cq4[v]);
            d.grad2 = V.grad2; d.cs = V.cs; d.ct = V.ct;
        }
    }
    for (int i = 0; i < ninst; ++i) {
        const m16_batch_instance &I = inst[i];
        const m16_batch_volume &V = vols[I.volume];
        const int v = I.volume;
        B.volume[i] = v;
        InstDev &d = B.hi[i];
        d.n = (int64_t)V.d0 * V.d1 * V.d2;
        d.d2 = V.d2;
        d.rcc = view[v].rcc;
        d.u2[0] = d.u2[1] = nullptr;
        d.u1 = nullptr;
        d.u_out = I.u;
        B.hctrl[i] = InstCtrl{0, params->num_iter, 0, 0, NAN};
        const float w = (float)I.weighting;
        const float nid2 = I.alpha ? 0.f : (float)(-1.0 / (I.decay * I.decay));
        if (L.kind[i] >= kTileKinds) {
            GroupDev &g = B.hg[i];
            g.vol = v;
            g.w = w;
            g.nid2 = nid2;
            g.sq0 = (float)I.sqevals[0]; g.sq1 = (float)I.sqevals[1]; g.sq2 = (float)I.sqevals[2];
            g.isq0 = (float)(1.0 / I.sqevals[0]); g.isq1 = (float)(1.0 / I.sqevals[1]);
            g.isq2 = (float)(1.0 / I.sqevals[2]);
            g.state = (float *)field(L.cstate[i]);
            g.slab = (int64_t)(align_up((size_t)d.n * 4, 256) / 4);
            g.alpha = I.alpha;
            g.img = V.img;
            g.denom = denom + v;
            d.u1 = g.state + 5 * g.slab;
            continue;
        }
        TileDev &t = B.ht[i];
        t.V = view[v];
        int axis;
        tile_metric(I.sqevals, t.V, &axis);
        t.V.exp_radius = I.alpha ? 0 : 1;
        t.V.w = w;
        t.V.nid2 = nid2;
        t.V.labels = nullptr;
        t.fail = TileFail{(int *)field(L.err), (int *)field(L.state) + i};
        CUtensorMap *m = B.hmaps.data() + 6 * nvol + 5 * i;
        CUtensorMap *dm = dmaps + 6 * nvol + 5 * i, *dv = dmaps + 6 * v;
        bool ok = true;
        for (int k = 0; k < 2; ++k) {
            t.h[k] = (float4 *)field(L.h[k][i]);
            t.u[k] = (float2 *)field(L.u[k][i]);
            ok = ok && tile_map(m + k, t.h[k], V.d0, V.d1, t.V.pitch, 4, kTileRows + 1) &&
                 tile_map(m + 2 + k, t.u[k], V.d0, V.d1, t.V.pitch, 2, kTileRows);
            t.mh[k] = dm + k;
            t.mu[k] = dm + 2 + k;
            d.u2[k] = t.u[k];
        }
        t.rad = I.alpha ? (float *)field(L.rad[i]) : nullptr;
        if (I.alpha) ok = ok && tile_map(m + 4, t.rad, V.d0, V.d1, t.V.pitch, 1, kTileRows);
        if (!ok) return M16_ERR_CUDA;
        t.V.mcaps = dv;
        t.V.mdir = L.kind[i] == kConstPlanar ? dv + 4 : dv + 1 + std::max(axis, 0);
        t.V.mrad = I.alpha ? dm + 4 : dv + 5;
        t.rows = (int64_t)V.d0 * V.d1;
        t.nx = tile_count_x(V.d2);
        t.ny = tile_count_y(V.d1, kTileRows);
        t.img = V.img; t.cs = V.cs; t.ct = V.ct; t.alpha = I.alpha; t.denom = denom + v;
    }
    BatchTables &T = B.T;
    T.work = (const int2 *)(ws + L.work);
    T.tiles = (const TileDev *)(ws + L.tiles);
    T.vols = (const VolDev *)(ws + L.cvols);
    T.groups = (const GroupDev *)(ws + L.groups);
    T.insts = (const InstDev *)(ws + L.insts);
    T.ctrl = (InstCtrl *)(ws + L.ctrl);
    T.state = (unsigned *)(ws + L.state);
    T.partials = (float *)(ws + L.partials);
    for (int k = 0; k < kTileKinds; ++k)
        if (std::find(L.kind.begin(), L.kind.end(), k) != L.kind.end()) M16_CUDA_TRY(batch_tile_prepare(k));
    auto up = [&](void *dst, const void *src, size_t bytes) {
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    };
    M16_CUDA_TRY(up(dmaps, B.hmaps.data(), sizeof(CUtensorMap) * B.hmaps.size()));
    M16_CUDA_TRY(up((void *)T.vols, B.hv.data(), sizeof(VolDev) * nvol));
    M16_CUDA_TRY(up(T.ctrl, B.hctrl.data(), sizeof(InstCtrl) * ninst));
    M16_CUDA_TRY(up(T.state, B.hstate.data(), sizeof(unsigned) * ninst));
    M16_CUDA_TRY(cudaMemsetAsync(ws + L.err, 0, sizeof(int), st));
    return M16_OK;
}

// per-volume set-up, then the instances' state (after batch_configure's upload
// of their descriptors)
int batch_setup_kernels(const BatchRun &B, const m16_batch_volume *vols, cudaStream_t st, int &launches)
{
    const BatchLayout &L = B.L;
    char *ws = B.ws;
    float *denom = (float *)(ws + L.denom);
    for (int v = 0; v < B.nvol; ++v) {
        const VolumePlan &P = L.vol[v];
        if (!P.instances) continue;
        const m16_batch_volume &V = vols[v];
        const int64_t n = (int64_t)V.d0 * V.d1 * V.d2;
        const int blocks = (int)std::min<int64_t>(kSetupBlocks, div_up(n, 256));
        float *mp = (float *)(ws + L.maxpart[v]);
        bt_max_kernel<<<blocks, 256, 0, st>>>(V.img, n, mp);
        bt_denom_kernel<<<1, 256, 0, st>>>(mp, blocks, denom + v);
        launches += 2;
        if (P.tiles) {
            VolumeFields F;
            F.caps = (float2 *)(ws + L.caps[v]);
            for (int k = 0; k < 3; ++k) F.dir[k] = P.axis[k] ? (float4 *)(ws + L.dir[k][v]) : nullptr;
            F.q4 = P.q4 ? (float4 *)(ws + L.vq4[v]) : nullptr;
            F.rad = P.rad ? (float *)(ws + L.vrad[v]) : nullptr;
            bt_volume_kernel<<<blocks, 256, 0, st>>>(V.quat3, V.grad2, V.cs, V.ct, V.d2, (int64_t)V.d0 * V.d1, F);
            ++launches;
        }
        if (P.compact) {
            bt_expand_kernel<<<blocks, 256, 0, st>>>(V.quat3, (float4 *)(ws + L.cq4[v]), n);
            ++launches;
        }
    }
    // runs of instances of one mode and volume, so that a launch's grid fits them
    for (int i = 0; i < B.ninst;) {
        const bool c = L.kind[i] >= kTileKinds;
        int j = i + 1;
        while (j < B.ninst && j - i < 65535 && B.volume[j] == B.volume[i] && (L.kind[j] >= kTileKinds) == c) ++j;
        const int blocks = (int)std::min<int64_t>(kSetupBlocks, div_up(B.hi[i].n, 256));
        if (c) bt1_state_kernel<<<dim3(blocks, j - i), 256, 0, st>>>(B.T.vols, B.T.groups, i);
        else bt_state_kernel<<<dim3(blocks, j - i), 256, 0, st>>>(B.T.tiles, i);
        ++launches;
        i = j;
    }
    M16_CUDA_TRY(cudaGetLastError());
    return M16_OK;
}

// The work list: per kind and volume, tile by tile with the volume's active
// instances side by side
void batch_work(BatchRun &B, const std::vector<char> &active)
{
    const BatchLayout &L = B.L;
    B.work.clear();
    for (int k = 0; k < kKinds; ++k) {
        B.T.seg[k] = (int)B.work.size();
        for (int v = 0; v < B.nvol; ++v) {
            std::vector<int> members;
            int tiles = 0;
            if (!L.vol[v].instances) continue;
            for (int i = 0; i < B.ninst; ++i)
                if (active[i] && L.kind[i] == k && B.volume[i] == v) {
                    members.push_back(i);
                    tiles = B.hi[i].nparts;
                }
            for (int t = 0; t < tiles; ++t)
                for (int i : members) B.work.push_back(make_int2(i, t));
        }
    }
    B.T.seg[kKinds] = (int)B.work.size();
}

// The tile shape: z-chunks, the instances' partial sums, their descriptors and
// the work list onto the device.  Uploads read B's vectors until they have run.
int batch_configure(BatchRun &B, const m16_batch_volume *vols, int bps, const std::vector<char> &active,
                    cudaStream_t st)
{
    const BatchLayout &L = B.L;
    const int zcb = batch_chunk(vols, B.nvol, tile_instances(L), bps);
    int64_t off = 0;
    for (int i = 0; i < B.ninst; ++i) {
        const m16_batch_volume &V = vols[B.volume[i]];
        if (L.kind[i] >= kTileKinds) {
            B.hi[i].nparts = compact_tiles(V.d0, V.d1, V.d2);
        } else {
            TileDev &t = B.ht[i];
            t.zc = equal_chunk(V.d0, zcb);
            B.hi[i].nparts = (int)(t.nx * t.ny * div_up(V.d0, t.zc));
        }
        B.hi[i].part_off = B.ht[i].part_off = B.hg[i].part_off = off;
        off += B.hi[i].nparts;
    }
    batch_work(B, active);
    auto up = [&](const void *dst, const void *src, size_t bytes) {
        return cudaMemcpyAsync((void *)dst, src, bytes, cudaMemcpyHostToDevice, st);
    };
    M16_CUDA_TRY(up(B.T.tiles, B.ht.data(), sizeof(TileDev) * B.ninst));
    M16_CUDA_TRY(up(B.T.insts, B.hi.data(), sizeof(InstDev) * B.ninst));
    M16_CUDA_TRY(up(B.T.groups, B.hg.data(), sizeof(GroupDev) * B.ninst));
    if (!B.work.empty()) M16_CUDA_TRY(up(B.T.work, B.work.data(), sizeof(int2) * B.work.size()));
    return M16_OK;
}

// m iterations; with `check` the last one's residuals, else the buffers' state
// is stored by a launch of its own where it changed.  False on a launch error.
bool batch_run(const BatchTables &T, int ninst, const m16_cut_params &p, int m, bool check, cudaStream_t st,
               int &launches, PairTimer *timer = nullptr)
{
    if (m <= 0) return true;
    const int sweeps = enqueue_iterations(T, m, check, st, launches, timer);
    if (sweeps < 0) return false;
    if (check) {
        ++launches;
        return launch_pdl(bt_check_kernel, dim3(ninst), dim3(256), st, true, T.insts, T.ctrl, T.state,
                          (const float *)T.partials, p.error_bound, p.update, sweeps & 1, (const int *)nullptr,
                          0) == cudaSuccess;
    }
    if (sweeps & 1) {
        ++launches;
        return launch_pdl(bt_flip_kernel, dim3((unsigned)div_up(ninst, 256)), dim3(256), st, true, T.state, ninst) ==
               cudaSuccess;
    }
    return true;
}

int batch_results(const BatchRun &B, cudaStream_t st, int &launches)
{
    for (int i = 0; i < B.ninst;) {
        int j = i + 1;
        while (j < B.ninst && j - i < 65535 && B.volume[j] == B.volume[i]) ++j;
        const int blocks = (int)std::min<int64_t>(kSetupBlocks, div_up(B.hi[i].n, 256));
        bt_result_kernel<<<dim3(blocks, j - i), 256, 0, st>>>(B.T.insts, B.T.state, i, 0);
        ++launches;
        i = j;
    }
    M16_CUDA_TRY(cudaGetLastError());
    return M16_OK;
}

// One cohort to completion: inst[0, ninst) over the layout of B.L
int batch_solve_cohort(BatchRun &B, const m16_batch_volume *vols, int nvol, const m16_batch_instance *inst, int ninst,
                       const m16_cut_params *params, int32_t *iterations, double *residuals, char *ws,
                       cudaStream_t st, m16_solve_stats *stats)
{
    int launches = 0;
    {
        const int r = batch_prepare(B, vols, nvol, inst, ninst, params, ws, st);
        if (r != M16_OK) return r;
    }
    const BatchTables &T = B.T;
    const BatchLayout &L = B.L;
    const int num_iter = params->num_iter, update = params->update;
    std::vector<char> active(ninst, 1);
    std::vector<int64_t> tune_key;
    bool shared = false;   // a volume with several instances of one kind
    for (int v = 0; v < nvol; ++v) {
        tune_key.push_back(vols[v].d0); tune_key.push_back(vols[v].d1); tune_key.push_back(vols[v].d2);
        for (int k = 0; k < kKinds; ++k) {
            int64_t c = 0;
            for (int i = 0; i < ninst; ++i) c += B.volume[i] == v && L.kind[i] == k;
            tune_key.push_back(c);
            shared = shared || (k < kTileKinds && c >= 3);
        }
    }
    tune_key.push_back(update);
    int bps = kDefaultBps;
    bool tune = false;
    if (stats && (stats->flags & M16_BATCH_NO_TUNE)) {
        if (stats->blocks_per_sm > 0) bps = stats->blocks_per_sm;   // a fixed tile shape
    } else {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto f = g_tuned.find(tune_key);
        if (f != g_tuned.end()) bps = f->second;
        else tune = true;
    }
    const bool timing = stats && stats->time_kernels;
    // ragged batches keep the rule's shape
    {
        const int r = batch_configure(B, vols, bps, active, st);
        if (r != M16_OK) return r;
    }
    if (timing || !shared || (int64_t)B.work.size() < kTuneMinItems || num_iter < 4 * update) tune = false;
    {
        const int r = batch_setup_kernels(B, vols, st, launches);
        if (r != M16_OK) return r;
    }

    // whole check intervals -- update iterations ending with a check -- are
    // captured several to a CUDA graph per work list and replayed
    const bool use_graph = !timing && !(stats && (stats->flags & M16_BATCH_NO_GRAPH));
    const int per_graph = std::max(1, 64 / update);
    cudaStream_t cap = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t gexec = nullptr;
    int graph_launches = 0;
    cudaEvent_t t0 = nullptr, t1 = nullptr;
    auto drop_graph = [&]() {
        if (gexec) cudaGraphExecDestroy(gexec);
        if (graph) cudaGraphDestroy(graph);
        gexec = nullptr;
        graph = nullptr;
    };
    auto release = [&]() {
        drop_graph();
        if (cap) cudaStreamDestroy(cap);
        if (t0) cudaEventDestroy(t0);
        if (t1) cudaEventDestroy(t1);
    };
#define M16_BT_TRY(expr)                                           \
    do {                                                           \
        cudaError_t e__ = (expr);                                  \
        if (e__ != cudaSuccess) { release(); return M16_ERR_CUDA; } \
    } while (0)
    if (use_graph) M16_BT_TRY(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
    if (timing || tune) {
        M16_BT_TRY(cudaEventCreate(&t0));
        M16_BT_TRY(cudaEventCreate(&t1));
    }
    // m iterations on st; timing: their launches of two iterations are timed;
    // time_it (the tuner): all of them, into last_ms
    double pair_ms = 0.0, last_ms = 0.0;
    int pair_n = 0;
    auto run = [&](int m, bool check, bool time_it = false) -> cudaError_t {
        PairTimer timer;
        timer.begin = t0;
        timer.end = t1;
        cudaError_t e = time_it ? cudaEventRecord(t0, st) : cudaSuccess;
        if (e != cudaSuccess) return e;
        if (!batch_run(T, ninst, *params, m, check, st, launches, timing ? &timer : nullptr))
            return cudaErrorLaunchFailure;
        if (!time_it && !timer.pairs) return cudaGetLastError();
        if (time_it && (e = cudaEventRecord(t1, st)) != cudaSuccess) return e;
        if ((e = cudaEventSynchronize(t1)) != cudaSuccess) return e;
        float ms = 0.f;
        e = cudaEventElapsedTime(&ms, t0, t1);
        last_ms = ms;
        pair_ms += timing ? ms : 0.f;
        pair_n += timer.pairs;
        return e;
    };
    std::vector<unsigned> state(ninst);
    int n_active = ninst, listed = ninst;
    auto read_state = [&]() -> cudaError_t {
        cudaError_t e = cudaMemcpyAsync(state.data(), T.state, sizeof(unsigned) * ninst, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        n_active = 0;
        for (int i = 0; i < ninst; ++i) n_active += active[i] = !(state[i] & kStopped);
        return e;
    };
    // iteration 0 ends the first run of launches (it is a check)
    int it = 0;
    if (num_iter > 0) {
        M16_BT_TRY(run(1, true));
        it = 1;
    }
    int tune_stage = tune ? 0 : -1;
    double tune_ms[3] = {0.0, 0.0, 0.0};
    auto reshape = [&](int next) -> int {
        bps = next;
        const int r = batch_configure(B, vols, bps, active, st);
        if (r != M16_OK) return r;
        drop_graph();
        listed = n_active;
        // the host vectors must stay unchanged until the copies ran
        return cudaStreamSynchronize(st) == cudaSuccess ? M16_OK : M16_ERR_CUDA;
    };
#define M16_BT_OK(expr)                              \
    do {                                             \
        const int r__ = (expr);                      \
        if (r__ != M16_OK) { release(); return r__; } \
    } while (0)
    M16_BT_TRY(read_state());
    while (it < num_iter && n_active > 0) {
        if (it - 1 + (int64_t)update >= num_iter) {   // no check left: the last iterations
            M16_BT_TRY(run(num_iter - it, false));
            it = num_iter;
            break;
        }
        if (tune_stage >= 0) {
            if (bps != kTuneBps[tune_stage]) M16_BT_OK(reshape(kTuneBps[tune_stage]));
            int64_t vox = 0;   // voxels of the active instances: the work this interval does
            for (int i = 0; i < ninst; ++i)
                if (active[i]) vox += B.hi[i].n;
            M16_BT_TRY(run(update, true, true));
            it += update;
            tune_ms[tune_stage] = vox > 0 ? last_ms / (double)vox : 0.0;
            if (++tune_stage == 3) {
                int best = 0;
                for (int k = 1; k < 3; ++k)
                    if (tune_ms[k] < tune_ms[best]) best = k;
                {
                    std::lock_guard<std::mutex> lk(g_tune_mu);
                    g_tuned[tune_key] = kTuneBps[best];
                }
                tune_stage = -1;
                M16_BT_TRY(read_state());
                if (bps != kTuneBps[best] && n_active > 0) M16_BT_OK(reshape(kTuneBps[best]));
            }
        } else if (use_graph && it - 1 + (int64_t)per_graph * update < num_iter) {
            if (!gexec) {
                M16_BT_TRY(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
                graph_launches = 0;
                bool ok = true;
                for (int k = 0; k < per_graph; ++k)
                    ok = ok && batch_run(T, ninst, *params, update, true, cap, graph_launches);
                const cudaError_t ce = cudaStreamEndCapture(cap, &graph);
                if (ce != cudaSuccess || !ok) { release(); return M16_ERR_CUDA; }
                M16_BT_TRY(cudaGraphInstantiate(&gexec, graph, 0));
            }
            M16_BT_TRY(cudaGraphLaunch(gexec, st));
            launches += graph_launches;
            it += per_graph * update;
        } else {
            M16_BT_TRY(run(update, true));
            it += update;
        }
        M16_BT_TRY(read_state());
        // drop stopped instances from the work list once they are a quarter of it
        if (n_active > 0 && n_active * 4 <= listed * 3) {
            batch_work(B, active);
            listed = n_active;
            drop_graph();   // the segments changed: capture again
            M16_BT_TRY(cudaMemcpyAsync((void *)T.work, B.work.data(), sizeof(int2) * B.work.size(),
                                       cudaMemcpyHostToDevice, st));
        }
    }
    release();
#undef M16_BT_TRY
#undef M16_BT_OK
    {
        const int r = batch_results(B, st, launches);
        if (r != M16_OK) return r;
    }
    int err = 0;
    M16_CUDA_TRY(cudaMemcpyAsync(B.hctrl.data(), T.ctrl, sizeof(InstCtrl) * ninst, cudaMemcpyDeviceToHost, st));
    M16_CUDA_TRY(cudaMemcpyAsync(&err, ws + L.err, sizeof(int), cudaMemcpyDeviceToHost, st));
    M16_CUDA_TRY(cudaStreamSynchronize(st));
    if (err) return M16_ERR_TIMEOUT;
    for (int i = 0; i < ninst; ++i) {
        if (iterations) iterations[i] = B.hctrl[i].iterations;
        if (residuals) residuals[i] = B.hctrl[i].resid;
    }
    if (stats) {
        stats->blocks_per_sm = bps;
        stats->launches += launches;
        stats->pair_launches += pair_n;
        stats->pair_ms += pair_ms;
    }
    return M16_OK;
}

}  // namespace
}  // namespace m16

using namespace m16;

extern "C" size_t m16_batch_workspace_bytes(const m16_batch_volume *vols, int32_t nvol,
                                            const m16_batch_instance *inst, int32_t ninst)
{
    if (!batch_args_ok(vols, nvol, inst, ninst)) return 0;
    return batch_bytes(vols, nvol, inst, ninst);
}

extern "C" size_t m16_batch_workspace_bytes_min(const m16_batch_volume *vols, int32_t nvol,
                                                const m16_batch_instance *inst, int32_t ninst)
{
    if (!batch_args_ok(vols, nvol, inst, ninst)) return 0;
    return batch_bytes_min(vols, nvol, inst, ninst);
}

extern "C" size_t m16_batch_steps_bytes_min(const m16_batch_volume *vols, int32_t nvol, const m16_batch_instance *inst,
                                            int32_t ninst)
{
    if (!batch_args_ok(vols, nvol, inst, ninst)) return 0;
    return batch_layout(vols, nvol, inst, 0, ninst, true).total;
}

extern "C" int m16_batch_solve(const m16_batch_volume *vols, int32_t nvol, const m16_batch_instance *inst,
                               int32_t ninst, const m16_cut_params *params, int32_t *iterations, double *residuals,
                               void *workspace, size_t workspace_bytes, void *stream, m16_solve_stats *stats)
{
    if (!params || params->update < 1 || params->num_iter < 0 || !(params->cc > 0.0)) return M16_ERR_BAD_ARG;
    if (!batch_args_ok(vols, nvol, inst, ninst)) return M16_ERR_BAD_ARG;
    if (stats && stats->path != M16_PATH_DEFAULT && stats->path != M16_PATH_TWO_SWEEPS) return M16_ERR_BAD_ARG;
    if (stats && (stats->flags & M16_BATCH_NO_TUNE) && stats->blocks_per_sm > 0) {
        bool known = false;   // one of the tuner's candidates (the workspace is sized for them)
        for (int c : kTuneBps) known = known || c == stats->blocks_per_sm;
        if (!known) return M16_ERR_BAD_ARG;
    }
    if (!workspace || workspace_bytes < batch_bytes_min(vols, nvol, inst, ninst) || ((uintptr_t)workspace & 255))
        return M16_ERR_WORKSPACE;
    if (stats) {
        stats->launches = stats->p_launches = stats->u_launches = stats->pair_launches = 0;
        stats->p_ms = stats->u_ms = stats->pair_ms = 0.0;
    }
    for (int first = 0; first < ninst;) {
        // as many of the instances as the workspace holds at once
        int last = ninst;
        BatchRun B;
        B.L = batch_layout(vols, nvol, inst, first, last, false);
        while (B.L.total > workspace_bytes && last - first > 1) {
            last = first + (last - first + 1) / 2;
            B.L = batch_layout(vols, nvol, inst, first, last, false);
        }
        if (B.L.total > workspace_bytes) B.L = batch_layout(vols, nvol, inst, first, last, true);
        if (B.L.total > workspace_bytes) return M16_ERR_WORKSPACE;
        const int r = batch_solve_cohort(B, vols, nvol, inst + first, last - first, params,
                                         iterations ? iterations + first : nullptr,
                                         residuals ? residuals + first : nullptr, (char *)workspace,
                                         (cudaStream_t)stream, stats);
        if (r != M16_OK) return r;
        first = last;
    }
    return M16_OK;
}

// ---- the batch as a sequence of capture-safe steps ------------------------------
//
// m16_batch_begin prepares a batch on the stream (descriptors, set-up
// kernels, the default tile shape and a work list over every instance) and
// returns a handle; m16_batch_iterate enqueues iterations and does nothing
// else -- no synchronisation, no allocation, no copies -- so a caller may
// capture it into a CUDA graph of its own; m16_batch_end writes every
// instance's u to its output, reads the iteration counts and residuals and
// frees the handle.  Instances stop on the device at their residual bound;
// the work list is not shrunk between steps.

struct m16_batch {
    BatchRun B;
    m16_cut_params params;
    int iterations_run = 0;          // iterations enqueued by m16_batch_iterate
};

// least: the workspace may be too small for the size that m16_batch_workspace_bytes gives
static int batch_begin(const m16_batch_volume *vols, int32_t nvol, const m16_batch_instance *inst, int32_t ninst,
                       const m16_cut_params *params, void *workspace, size_t workspace_bytes, void *stream, bool least,
                       m16_batch **out)
{
    if (!out) return M16_ERR_BAD_ARG;
    *out = nullptr;
    if (!params || params->update < 1 || params->num_iter < 0 || !(params->cc > 0.0)) return M16_ERR_BAD_ARG;
    if (!batch_args_ok(vols, nvol, inst, ninst)) return M16_ERR_BAD_ARG;
    if (!workspace || ((uintptr_t)workspace & 255)) return M16_ERR_WORKSPACE;
    if (!least && workspace_bytes < batch_bytes(vols, nvol, inst, ninst)) return M16_ERR_WORKSPACE;
    BatchLayout layout = batch_layout(vols, nvol, inst, 0, ninst, false);
    if (layout.total > workspace_bytes) layout = batch_layout(vols, nvol, inst, 0, ninst, true);
    if (layout.total > workspace_bytes) return M16_ERR_WORKSPACE;
    m16_batch *b = new m16_batch();
    BatchRun &B = b->B;
    B.L = layout;
    b->params = *params;
    cudaStream_t st = (cudaStream_t)stream;
    int launches = 0;
    int r = batch_prepare(B, vols, nvol, inst, ninst, params, (char *)workspace, st);
    // the handle owns the host sources until the copies have run
    if (r == M16_OK) r = batch_configure(B, vols, kDefaultBps, std::vector<char>(ninst, 1), st);
    if (r == M16_OK) r = batch_setup_kernels(B, vols, st, launches);
    if (r != M16_OK) {
        cudaStreamSynchronize(st);
        delete b;
        return r;
    }
    *out = b;
    return M16_OK;
}

extern "C" int m16_batch_begin(const m16_batch_volume *vols, int32_t nvol, const m16_batch_instance *inst,
                               int32_t ninst, const m16_cut_params *params, void *workspace, size_t workspace_bytes,
                               void *stream, m16_batch **out)
{
    return batch_begin(vols, nvol, inst, ninst, params, workspace, workspace_bytes, stream, false, out);
}

extern "C" int m16_batch_begin_min(const m16_batch_volume *vols, int32_t nvol, const m16_batch_instance *inst,
                                   int32_t ninst, const m16_cut_params *params, void *workspace, size_t workspace_bytes,
                                   void *stream, m16_batch **out)
{
    return batch_begin(vols, nvol, inst, ninst, params, workspace, workspace_bytes, stream, true, out);
}

extern "C" int m16_batch_iterate(m16_batch *b, int32_t count, void *stream)
{
    if (!b || count < 0) return M16_ERR_BAD_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const int update = b->params.update;
    int left = std::min(count, b->params.num_iter - b->iterations_run), launches = 0;
    while (left > 0) {
        // up to the next check, an iteration that is a multiple of update
        const int to_check = (update - b->iterations_run % update) % update + 1;
        const int m = std::min(left, to_check);
        if (!batch_run(b->B.T, b->B.ninst, b->params, m, m == to_check, st, launches)) return M16_ERR_CUDA;
        b->iterations_run += m;
        left -= m;
    }
    M16_CUDA_TRY(cudaGetLastError());
    return M16_OK;
}

extern "C" int m16_batch_end(m16_batch *b, int32_t *iterations, double *residuals, void *stream)
{
    if (!b) return M16_ERR_BAD_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    BatchRun &B = b->B;
    int launches = 0, err = 0;
    int rc = batch_results(B, st, launches);
    if (rc == M16_OK &&
        (cudaMemcpyAsync(B.hctrl.data(), B.T.ctrl, sizeof(InstCtrl) * B.ninst, cudaMemcpyDeviceToHost, st) !=
             cudaSuccess ||
         cudaMemcpyAsync(&err, B.ws + B.L.err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
         cudaStreamSynchronize(st) != cudaSuccess))
        rc = M16_ERR_CUDA;
    if (rc == M16_OK && err) rc = M16_ERR_TIMEOUT;
    if (rc == M16_OK) {
        for (int i = 0; i < B.ninst; ++i) {
            const InstCtrl &c = B.hctrl[i];
            // an instance that never stopped ran every iteration enqueued
            // directly or, replayed from graphs of whole check intervals, one
            // check interval per check
            const int ran = std::min(b->params.num_iter, std::max(b->iterations_run, c.n_checks * b->params.update));
            if (iterations) iterations[i] = c.stopped ? c.iterations : ran;
            if (residuals) residuals[i] = c.resid;
        }
    }
    delete b;
    return rc;
}
