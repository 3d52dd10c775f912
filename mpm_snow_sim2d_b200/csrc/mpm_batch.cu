// Batched 2D scenes: C ABI (include/mpm/mpm.h, mpm_batch_*), the scenes' shared
// arrays, the step sequence and its CUDA graphs. Kernels: mpm_batch.cuh.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <string>
#include <tuple>
#include <vector>

#include <cuda_runtime.h>

#include "mpm/mpm.h"
#include "mpm_batch.cuh"
#include "mpm_host.h"
#include "mpm_readback.h"

using namespace mpm;

namespace {

constexpr int kClusterSizes[4] = {1, 2, 4, 8};
constexpr int kMaxSegment = 64;    // steps of one graph
constexpr size_t kMaxGraphs = 64;  // graphs kept

struct BatchBuffers {
    float *x, *v, *B, *Fe, *Jp, *mass, *vol;
    int* id;  // creation index of the particle within its scene
};

// The grid of the parts of a batch (below).
struct SharedGrid {
    unsigned long long* acc;
    float4* gv;
    int *mark, *mark_list;
};

}  // namespace

struct mpm_batch {
    ReadbackUser readback;
    DeviceArena arena;  // every device array below but those made on demand
    int device = 0;
    int nscenes = 0;
    int sms = 148;
    long long N = 0;
    std::vector<int> counts;
    std::vector<BatchScene> scenes;  // host copy
    BatchBuffers buf[2] = {};
    int parity = 0;                  // which buffer holds the particles
    float* A = nullptr;              // P2G affine matrix of the queued particles
    BatchArrays arr{};
    TileInfo ti{};
    SlowQueue q{};
    ManyScenes many{};
    long long nodes = 0;
    size_t stamps_cap = 0;
    int last_steps = 0;
    int since_sort = 0;              // steps since the last sort
    bool needs_sort = true;
    bool any_fresh = true;           // a scene has no pending grid sums (arr.fresh)
    bool unfinished = false;         // a step call failed on its way (recover)
    bool sorted = false;             // there are items to step
    int captured = -1;               // the buffer that steps captured by the caller work on
    std::vector<unsigned long long*> old_stamps;  // which they write to
    cudaStream_t stream = nullptr, own_stream = nullptr;
    mpm_batch_config cfg{};
    int cap_max = 0;                 // nodes per CTA of the largest scene's cluster (limit on a scene's grid)
    // graphs of [sort +] n steps, by (steps, sort, buffer)
    std::map<std::tuple<int, int, int>, cudaGraphExec_t> graphs;
    bool use_graphs = true;
    std::string err;
    // Scenes whose grids do not fit the device's memory side by side: consecutive scenes
    // in parts, batches of their own that share one grid and are stepped one after the other. A part
    // forms its sums from its particles when its turn comes, which gives the same sums.
    // Empty: all scenes are in this object.
    std::vector<mpm_batch*> parts;
    std::vector<int> part_first;     // first scene of each part
};

namespace {

mpm_status bfail(mpm_batch* b, mpm_status code, const std::string& what) {
    if (b) b->err = what;
    return code;
}

#define BATCH_CUDA(b, call)                                                                                \
    do {                                                                                                   \
        cudaError_t e_ = (call);                                                                           \
        if (e_ != cudaSuccess) {                                                                           \
            cudaGetLastError();                                                                            \
            return bfail((b), e_ == cudaErrorMemoryAllocation ? MPM_ERR_OUT_OF_MEMORY : MPM_ERR_CUDA,      \
                         std::string(#call) + ": " + cudaGetErrorString(e_));                              \
        }                                                                                                  \
    } while (0)

template <typename T> cudaError_t balloc(T** p, size_t count) {
    *p = nullptr;
    return cudaMalloc(reinterpret_cast<void**>(p), (count ? count : 1) * sizeof(T));
}

void drop_graphs(mpm_batch* b) {
    if (b->graphs.empty()) return;
    cudaStreamSynchronize(b->stream);
    for (auto& g : b->graphs)
        if (g.second) cudaGraphExecDestroy(g.second);
    b->graphs.clear();
}

void release(mpm_batch* b) {
    for (mpm_batch* p : b->parts) {
        release(p);
        delete p;
    }
    b->parts.clear();
    b->part_first.clear();
    drop_graphs(b);
    if (b->arr.stamps) cudaFree(b->arr.stamps);
    for (unsigned long long* p : b->old_stamps) cudaFree(p);
    b->arena.release();
    if (b->own_stream) cudaStreamDestroy(b->own_stream);
}

Particles particles(const mpm_batch* b) {
    const BatchBuffers& f = b->buf[b->parity];
    Particles P{};
    P.x = f.x; P.v = f.v; P.B = f.B; P.Fe = f.Fe; P.Jp = f.Jp; P.A = b->A;
    P.mass = f.mass; P.vol = f.vol;
    P.n = (int)b->N;
    return P;
}

// ---- the step sequence ----

// All scenes' particles into the other buffer, by (tile, cell, id); without v and B
// when every scene's sums are pending (the next G2P writes them unread).
cudaError_t enqueue_sort(mpm_batch* b, bool pending) {
    if (b->N == 0) return cudaSuccess;
    const Particles P = particles(b);
    const int threads = 256;
    const int blocks = (int)((b->N + threads - 1) / threads);
    const int scan_blocks = (b->ti.n_tiles + kScanTiles - 1) / kScanTiles;
    cudaError_t e = launch_chained(k_sort_count<2, 4, ManyScenes>, blocks, threads, 0, b->stream, P, b->many, b->ti);
    if (e == cudaSuccess) e = launch_chained(k_sort_block_sums, scan_blocks, kScanTiles, 0, b->stream, b->ti);
    if (e == cudaSuccess) e = launch_chained(k_sort_scan, scan_blocks, kScanTiles, 0, b->stream, b->ti);
    if (e == cudaSuccess) e = launch_chained(k_sort_bucket, blocks, threads, 0, b->stream, (int)b->N, b->ti);
    if (e != cudaSuccess) return e;
    const BatchBuffers& t = b->buf[b->parity ^ 1];
    const SortBuffers dst{t.x, pending ? nullptr : t.v, pending ? nullptr : t.B, t.Fe, t.Jp, nullptr, t.mass, t.vol, t.id};
    e = launch_chained(k_tile_sort<2, 4, ManyScenes>, b->sms * SortGeom<2>::CTAS_PER_SM, 256, 0, b->stream, P,
                       b->buf[b->parity].id, dst, b->many, b->ti);
    if (e == cudaSuccess) {
        b->parity ^= 1;
        b->sorted = true;
    }
    return e;
}

cudaError_t enqueue_step(mpm_batch* b) {
    cudaError_t e = launch_chained(k_batch_grid, b->sms * 8, 256, 0, b->stream, b->arr, b->ti);
    if (e != cudaSuccess || b->N == 0) return e;
    const Particles P = particles(b);
    e = launch_chained(k_batch_step<true>, b->sms * MPM_FUSED_MIN_BLOCKS, FusedGeom<2>::THREADS, 0, b->stream, P, b->arr,
                       b->ti, b->q);
    if (e == cudaSuccess) e = launch_chained(k_batch_plastic, b->sms * 4, 256, 0, b->stream, P, b->arr, b->q);
    if (e == cudaSuccess)
        e = launch_chained(k_batch_windows, b->sms * 8, FusedGeom<2>::THREADS, 0, b->stream, P, b->arr, b->ti, b->q);
    return e;
}

cudaError_t enqueue_segment(mpm_batch* b, int steps, bool sort) {
    cudaError_t e = sort ? enqueue_sort(b, true) : cudaSuccess;
    for (int k = 0; k < steps && e == cudaSuccess; ++k) e = enqueue_step(b);
    return e;
}

// [sort +] steps, from a graph captured on first use on a stream of its own.
mpm_status run_segment(mpm_batch* b, int steps, bool sort) {
    if (!b->use_graphs) {
        BATCH_CUDA(b, enqueue_segment(b, steps, sort));
        return MPM_OK;
    }
    const auto key = std::make_tuple(steps, (int)sort, b->parity);
    auto it = b->graphs.find(key);
    if (it == b->graphs.end()) {
        if (b->graphs.size() >= kMaxGraphs) drop_graphs(b);
        cudaStream_t cap = nullptr;
        cudaGraph_t g = nullptr;
        cudaGraphExec_t ex = nullptr;
        const cudaStream_t saved = b->stream;
        const int parity = b->parity;
        cudaError_t e = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            b->stream = cap;
            const cudaError_t e1 = enqueue_segment(b, steps, sort);
            b->stream = saved;
            const cudaError_t e2 = cudaStreamEndCapture(cap, &g);
            e = e1 != cudaSuccess ? e1 : e2;
        }
        b->parity = parity;  // nothing ran
        if (e == cudaSuccess) e = cudaGraphInstantiate(&ex, g, 0);
        if (g) cudaGraphDestroy(g);
        if (cap) cudaStreamDestroy(cap);
        if (e != cudaSuccess) {  // direct launches for the life of the batch
            cudaGetLastError();
            b->use_graphs = false;
            BATCH_CUDA(b, enqueue_segment(b, steps, sort));
            return MPM_OK;
        }
        it = b->graphs.emplace(key, ex).first;
    }
    BATCH_CUDA(b, cudaGraphLaunch(it->second, b->stream));
    if (sort && b->N > 0) b->parity ^= 1;
    return MPM_OK;
}

int sort_period(const mpm_batch* b) { return b->cfg.sort_period > 0 ? b->cfg.sort_period : 16; }

// A call on a stream that is being captured: direct launches, so that the caller's graph
// can be replayed any number of times, also after uploads. Nothing runs now, so
// the host's account of the batch stays; the sums of uploaded states are formed where
// the device says so (arr.fresh), and sorts, on which no result depends, come in pairs,
// which leave the particles in the buffer they started in (from here on plain calls
// leave them there as well). A short call has none.
mpm_status capture_steps(mpm_batch* b, int steps) {
    if (!b->sorted) return bfail(b, MPM_ERR_CUDA, "a batch is stepped once before its steps are captured");
    if (b->N > 0)
        k_batch_step<false><<<b->sms * MPM_FUSED_MIN_BLOCKS, FusedGeom<2>::THREADS, 0, b->stream>>>(particles(b), b->arr, b->ti,
                                                                                                   b->q);
    BATCH_CUDA(b, cudaGetLastError());
    BATCH_CUDA(b, cudaMemsetAsync(b->arr.fresh, 0, sizeof(int) * (size_t)b->nscenes, b->stream));
    const int period = sort_period(b);
    const int sorts = steps >= period ? 2 * ((steps - 1) / (2 * period) + 1) : 0;
    if (sorts == 0) BATCH_CUDA(b, enqueue_segment(b, steps, false));
    for (int k = 0; k < sorts; ++k) {
        const int n = (int)((long long)steps * (k + 1) / sorts - (long long)steps * k / sorts);
        if (n > 0) BATCH_CUDA(b, enqueue_segment(b, n, true));
    }
    k_batch_end<<<1, 256, 0, b->stream>>>(b->arr);
    BATCH_CUDA(b, cudaGetLastError());
    b->captured = b->parity;
    return MPM_OK;
}

// Memory for one call that waits for the stream before it returns: between sorts the
// other buffer is free, its x, v, B, F_E and J_p one behind the other (a whole state).
float* scratch(const mpm_batch* b) { return b->buf[b->parity ^ 1].x; }

// Every scene's pending sums are void: the next step forms them from the state.
mpm_status forget_sums(mpm_batch* b) {
    BATCH_CUDA(b, cudaMemsetAsync(b->arr.acc, 0, sizeof(unsigned long long) * 4 * (size_t)b->nodes, b->stream));
    BATCH_CUDA(b, cudaMemsetAsync(b->ti.mark, 0, sizeof(int) * (size_t)b->ti.n_blocks, b->stream));
    BATCH_CUDA(b, cudaMemsetAsync(b->ti.n_marked, 0, sizeof(int), b->stream));
    BATCH_CUDA(b, cudaMemsetAsync(b->arr.fresh, 1, sizeof(int) * (size_t)b->nscenes, b->stream));
    b->any_fresh = true;
    b->needs_sort = true;
    return MPM_OK;
}

// After a call that failed on its way: what its kernels hand each other through device
// counters (the call's step, which says where time stamps go, and the tiles' counts of a
// sort) starts over, and the sums are formed anew from the particles as they are.
mpm_status recover(mpm_batch* b) {
    BATCH_CUDA(b, cudaMemsetAsync(b->arr.step, 0, sizeof(int), b->stream));
    BATCH_CUDA(b, cudaMemsetAsync(b->ti.tile_count, 0, sizeof(int) * (size_t)b->ti.n_tiles, b->stream));
    return forget_sums(b);
}

// A configuration is valid when its numbers are and every scene's grid fits the
// largest cluster it allows (the limit on a scene's size that the interface states).
mpm_status configure(mpm_batch* b, const mpm_batch_config& cfg) {
    if (cfg.threads != 256 && cfg.threads != 512 && cfg.threads != 1024)
        return bfail(b, MPM_ERR_INVALID_ARGUMENT, "threads must be 256, 512 or 1024");
    if (cfg.max_cluster != 1 && cfg.max_cluster != 2 && cfg.max_cluster != 4 && cfg.max_cluster != 8)
        return bfail(b, MPM_ERR_INVALID_ARGUMENT, "max_cluster must be 1, 2, 4 or 8");
    if (cfg.particles_per_cta < 0) return bfail(b, MPM_ERR_INVALID_ARGUMENT, "particles_per_cta must be >= 0");
    if (cfg.sort_period < 0) return bfail(b, MPM_ERR_INVALID_ARGUMENT, "sort_period must be >= 0");
    for (int s = 0; s < b->nscenes; ++s) {
        const int nx = b->scenes[s].C.nx, ny = b->scenes[s].C.ny;
        bool fits = false;
        for (int c = 0; c < 4 && kClusterSizes[c] <= cfg.max_cluster; ++c)
            fits = fits || (long long)((ny + kClusterSizes[c] - 1) / kClusterSizes[c]) * nx <= b->cap_max;
        if (!fits)
            return bfail(b, MPM_ERR_CAPACITY,
                         "scene " + std::to_string(s) + ": its grid of " + std::to_string((long long)nx * ny) +
                             " nodes does not fit in the shared memory of a cluster of " +
                             std::to_string(cfg.max_cluster) + " CTAs");
    }
    b->cfg = cfg;
    return MPM_OK;
}

// The part that holds a scene (null: there are no parts), and the scene's number in it.
mpm_batch* part_of(const mpm_batch* b, int32_t& scene) {
    if (b->parts.empty()) return nullptr;
    const size_t k = std::upper_bound(b->part_first.begin(), b->part_first.end(), scene) - b->part_first.begin() - 1;
    scene -= b->part_first[k];
    return b->parts[k];
}

// What a part answered, as the batch's own answer.
mpm_status answer(mpm_batch* b, const mpm_batch* part, mpm_status st) {
    if (st != MPM_OK) b->err = part->err;
    return st;
}

bool valid_scene(const mpm_batch* b, int32_t s) { return b && s >= 0 && s < b->nscenes; }

const int kComps[5] = {2, 2, 4, 4, 1};  // position, velocity, B, F_E, J_p

float* field(const mpm_batch* b, int f) {
    const BatchBuffers& F = b->buf[b->parity];
    float* soa[] = {F.x, F.v, F.B, F.Fe, F.Jp};
    return soa[f];
}

// Fields of a scene in creation order (null: skipped).
mpm_status read_scene(mpm_batch* b, int scene, float* const* host) {
    const int n = b->counts[scene];
    if (n == 0) return MPM_OK;
    size_t floats = 0;
    for (int f = 0; f < 5; ++f) floats += host[f] ? (size_t)n * kComps[f] : 0;
    if (floats == 0) return MPM_OK;
    const long long p0 = b->scenes[scene].p0;
    void* dst[5];
    size_t bytes[5], at = 0;
    for (int f = 0; f < 5; ++f) {
        dst[f] = host[f];
        bytes[f] = host[f] ? sizeof(float) * (size_t)n * kComps[f] : 0;
        if (!host[f]) continue;
        k_batch_export<<<(n + 255) / 256, 256, 0, b->stream>>>(field(b, f), b->N, kComps[f], p0, n, b->buf[b->parity].id,
                                                               scratch(b) + at);
        at += (size_t)n * kComps[f];
    }
    BATCH_CUDA(b, cudaGetLastError());
    BATCH_CUDA(b, ReadbackRing::get().read_parts(b->stream, scratch(b), dst, bytes, 5));
    return MPM_OK;
}

// A batch of all scenes in one; with `grid` a part, whose grid is that.
mpm_status create_whole(const mpm_params* params, const mpm_particles_init* init, int32_t nscenes, int dev,
                        const SharedGrid* grid, mpm_batch** out) {
    long long N = 0;
    for (int s = 0; s < nscenes; ++s) N += init[s].count;
    mpm_batch* b = new mpm_batch();
    auto bail = [&](mpm_status code) { release(b); delete b; return code; };
    b->device = dev;
    b->nscenes = nscenes;
    b->N = N;
    int optin = 0, sms = 0;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return bail(MPM_ERR_CUDA);
    b->sms = sms > 0 ? sms : 148;
    // nodes of 24 bytes in a CTA's shared memory (less 3.7 KB): the size limit of a scene
    const int smem = (optin - 3776) / 256 * 256;
    b->cap_max = smem / 24;

    // Per-scene constants and fixed-point scales, as mpm_create chooses them; the
    // scenes' places in the shared arrays.
    constexpr int T = TileGeom<2>::T;
    b->counts.resize(nscenes);
    b->scenes.resize(nscenes);
    std::vector<float> massv((size_t)N), volv((size_t)N);
    std::vector<int> of_slots((size_t)N), of_tiles, of_blocks;
    long long off = 0;
    for (int s = 0; s < nscenes; ++s) {
        const int n = (int)init[s].count;
        double total_mass = 0.0;
        for (int i = 0; i < n; ++i) {
            const float vol = init[s].volume[i];
            const float m = init[s].mass ? init[s].mass[i] : (vol * params[s].rho) / 100.f;
            if (!std::isfinite(vol) || !std::isfinite(m)) return bail(MPM_ERR_INVALID_ARGUMENT);
            volv[off + i] = vol;
            massv[off + i] = m;
            of_slots[off + i] = s;
            total_mass += m;
        }
        for (long long i = 0; i < 2LL * n; ++i)
            if (!std::isfinite(init[s].position[i]) || (init[s].velocity && !std::isfinite(init[s].velocity[i])))
                return bail(MPM_ERR_INVALID_ARGUMENT);
        BatchScene& S = b->scenes[s];
        S.C = step_consts(params[s], 2);
        int l2[3];
        fixed_point_scales(params[s], total_mass, S.C, l2);
        S.p0 = off;
        S.n = n;
        S.node0 = b->nodes;
        S.view = SceneView{{S.C.W, S.C.H, 0}, {(S.C.W + T - 1) / T, (S.C.H + T - 1) / T, 1}, (int)of_tiles.size()};
        S.nblk[0] = (S.C.nx + T - 1) / T;
        S.nblk[1] = (S.C.ny + T - 1) / T;
        S.blk0 = (int)of_blocks.size();
        of_tiles.insert(of_tiles.end(), (size_t)S.view.tiles[0] * S.view.tiles[1], s);
        of_blocks.insert(of_blocks.end(), (size_t)S.nblk[0] * S.nblk[1], s);
        b->nodes += S.C.nodes;
        b->counts[s] = n;
        off += n;
    }
    mpm_batch_config cfg{};
    cfg.threads = 512;
    cfg.particles_per_cta = 8192;
    cfg.max_cluster = 8;
    cfg.sort_period = 16;
    const mpm_status cs = configure(b, cfg);
    if (cs != MPM_OK) return bail(cs);

    if (cudaStreamCreateWithFlags(&b->own_stream, cudaStreamNonBlocking) != cudaSuccess) return bail(MPM_ERR_CUDA);
    b->stream = b->own_stream;
    const size_t n = (size_t)N, nt = of_tiles.size(), nb = of_blocks.size();
    TileInfo& ti = b->ti;
    ti.n_tiles = (int)nt;
    ti.n_blocks = (int)nb;
    ti.win = FusedGeom<2>::WIN;
    ti.item_win = 1;
    b->q.capacity = n > 0 ? (int)n : 1;
    b->q.win_capacity = b->q.capacity / ti.win + (int)nt + 1;
    DeviceArena& arena = b->arena;
    for (BatchBuffers& f : b->buf) {
        arena.want(&f.x, n * 2).want(&f.v, n * 2).want(&f.B, n * 4).want(&f.Fe, n * 4).want(&f.Jp, n);
        arena.want(&f.mass, n).want(&f.vol, n).want(&f.id, n);
    }
    BatchScene* d_scenes = nullptr;
    int *d_of_slots = nullptr, *d_of_tiles = nullptr, *d_of_blocks = nullptr;
    arena.want(&d_scenes, (size_t)nscenes).want(&d_of_slots, n).want(&d_of_tiles, nt).want(&d_of_blocks, nb);
    arena.want(&b->A, n * 4);
    if (grid) {
        b->arr.acc = grid->acc;
        b->arr.gv = grid->gv;
        ti.mark = grid->mark;
        ti.mark_list = grid->mark_list;
    } else {
        arena.want(&b->arr.acc, (size_t)b->nodes * 4).want(&b->arr.gv, (size_t)b->nodes);
        arena.want(&ti.mark, nb).want(&ti.mark_list, nb);
    }
    arena.want(&b->arr.status, (size_t)nscenes).want(&b->arr.fresh, (size_t)nscenes).want(&b->arr.step, 1);
    arena.want(&ti.key, n).want(&ti.tile_count, nt).want(&ti.tile_cursor, nt).want(&ti.tile_start, nt);
    arena.want(&ti.n_marked, 1).want(&ti.perm, n).want(&ti.tile_list, nt);
    arena.want(&ti.n_tile_list, 1).want(&ti.tile_len, nt).want(&ti.fused_next, 1);
    arena.want(&ti.items, nt + n / (size_t)ti.win).want(&ti.n_items, 1).want(&ti.scan, nt / kScanTiles + 1);
    arena.want(&ti.grid_done, 1).want(&ti.skey, n).want(&ti.sval, n).want(&b->q.list, (size_t)b->q.capacity);
    arena.want(&b->q.count, 2).want(&b->q.fh, (size_t)b->q.capacity * 4).want(&b->q.win, (size_t)b->q.win_capacity);
    if (!arena.allocate()) return bail(MPM_ERR_OUT_OF_MEMORY);
    b->arr.scenes = d_scenes;
    b->arr.of_slots = d_of_slots;
    b->arr.of_blocks = d_of_blocks;
    ti.tile_scene = d_of_tiles;
    b->q.nwin = b->q.count + 1;
    ti.zero[0] = ti.fused_next;
    ti.zero[1] = b->q.count;
    b->arr.nscenes = nscenes;
    b->many = ManyScenes{d_scenes, d_of_slots, d_of_tiles};
    // SoA upload into buffer 0: F_E = I, B = 0, J_p = 1 (Particle ctor,
    // src/cpu/Particles.cpp:7-19); slot order = creation order.
    const BatchBuffers& F = b->buf[0];
    std::vector<float> soa(n * 4, 0.f);
    bool ok = true;
    auto up = [&](void* dst, const void* src, size_t bytes) {
        return bytes == 0 || cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice) == cudaSuccess;
    };
    auto zero = [&](void* dst, size_t bytes) { return cudaMemset(dst, 0, bytes) == cudaSuccess; };
    for (int s = 0; s < nscenes; ++s)
        for (int i = 0; i < b->counts[s]; ++i)
            for (int k = 0; k < 2; ++k) soa[(size_t)k * n + b->scenes[s].p0 + i] = init[s].position[(size_t)i * 2 + k];
    ok = ok && up(F.x, soa.data(), sizeof(float) * n * 2);
    for (int s = 0; s < nscenes; ++s)
        for (int i = 0; i < b->counts[s]; ++i)
            for (int k = 0; k < 2; ++k)
                soa[(size_t)k * n + b->scenes[s].p0 + i] = init[s].velocity ? init[s].velocity[(size_t)i * 2 + k] : 0.f;
    ok = ok && up(F.v, soa.data(), sizeof(float) * n * 2) && zero(F.B, sizeof(float) * n * 4);
    for (int k = 0; k < 4; ++k) std::fill(soa.begin() + k * n, soa.begin() + (k + 1) * n, (k % 3 == 0) ? 1.f : 0.f);
    ok = ok && up(F.Fe, soa.data(), sizeof(float) * n * 4) && up(F.Jp, soa.data(), sizeof(float) * n);
    ok = ok && up(F.mass, massv.data(), sizeof(float) * n) && up(F.vol, volv.data(), sizeof(float) * n);
    std::vector<int> ids(n);
    for (int s = 0; s < nscenes; ++s)
        for (int i = 0; i < b->counts[s]; ++i) ids[b->scenes[s].p0 + i] = i;
    ok = ok && up(F.id, ids.data(), sizeof(int) * n) && up(d_of_slots, of_slots.data(), sizeof(int) * n) &&
         up(d_of_tiles, of_tiles.data(), sizeof(int) * nt) && up(d_of_blocks, of_blocks.data(), sizeof(int) * nb) &&
         up(d_scenes, b->scenes.data(), sizeof(BatchScene) * (size_t)nscenes);
    ok = ok && zero(b->arr.status, sizeof(unsigned) * nscenes) && zero(b->arr.step, sizeof(int)) &&
         zero(b->arr.gv, sizeof(float4) * (size_t)b->nodes) && zero(ti.tile_count, sizeof(int) * nt) &&
         zero(ti.tile_cursor, sizeof(int) * nt) && zero(ti.grid_done, sizeof(int)) && zero(ti.n_items, sizeof(int)) &&
         zero(ti.n_tile_list, sizeof(int)) && zero(ti.fused_next, sizeof(int)) && zero(b->q.count, 2 * sizeof(int));
    if (!ok || cudaDeviceSynchronize() != cudaSuccess) { cudaGetLastError(); return bail(MPM_ERR_CUDA); }
    const mpm_status st = forget_sums(b);
    if (st != MPM_OK) return bail(st);
    *out = b;
    return MPM_OK;
}

// The scenes in `k` parts or a few more, of about as many nodes each.
mpm_status create_parts(const mpm_params* params, const mpm_particles_init* init, int32_t nscenes, int dev, int k,
                        mpm_batch** out) {
    constexpr int T = TileGeom<2>::T;
    auto nodes_of = [&](int s) { return (long long)(params[s].width + 1) * (params[s].height + 1); };
    auto blocks_of = [&](int s) { return (long long)((params[s].width + T) / T) * ((params[s].height + T) / T); };
    mpm_batch* b = new mpm_batch();
    auto bail = [&](mpm_status code) { release(b); delete b; return code; };
    b->device = dev;
    b->nscenes = nscenes;
    long long total = 0, nodes = 0, blocks = 0, most_nodes = 0, most_blocks = 0;
    for (int s = 0; s < nscenes; ++s) {
        total += nodes_of(s);
        b->N += init[s].count;
        b->counts.push_back((int)init[s].count);
    }
    const long long share = (total + k - 1) / k;
    for (int s = 0; s < nscenes; ++s) {
        if (s == 0 || nodes + nodes_of(s) > share) {
            b->part_first.push_back(s);
            nodes = blocks = 0;
        }
        nodes += nodes_of(s);
        blocks += blocks_of(s);
        most_nodes = std::max(most_nodes, nodes);
        most_blocks = std::max(most_blocks, blocks);
    }
    if (cudaStreamCreateWithFlags(&b->own_stream, cudaStreamNonBlocking) != cudaSuccess) return bail(MPM_ERR_CUDA);
    b->stream = b->own_stream;
    SharedGrid grid{};
    b->arena.want(&grid.acc, (size_t)most_nodes * 4).want(&grid.gv, (size_t)most_nodes);
    b->arena.want(&grid.mark, (size_t)most_blocks).want(&grid.mark_list, (size_t)most_blocks);
    if (!b->arena.allocate()) return bail(MPM_ERR_OUT_OF_MEMORY);
    for (size_t p = 0; p < b->part_first.size(); ++p) {
        const int s0 = b->part_first[p], s1 = p + 1 < b->part_first.size() ? b->part_first[p + 1] : nscenes;
        mpm_batch* part = nullptr;
        mpm_status st = create_whole(params + s0, init + s0, s1 - s0, dev, &grid, &part);
        if (st != MPM_OK) return bail(st);
        b->parts.push_back(part);
        if ((st = mpm_batch_set_stream(part, b->own_stream)) != MPM_OK) return bail(st);
    }
    *out = b;
    return MPM_OK;
}

}  // namespace

extern "C" {

mpm_status mpm_batch_create(const mpm_params* params, const mpm_particles_init* init, int32_t nscenes,
                            mpm_batch** out) {
    if (!out) return MPM_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    if (!params || !init || nscenes < 1) return MPM_ERR_INVALID_ARGUMENT;
    long long N = 0;
    for (int s = 0; s < nscenes; ++s) {
        std::string why;
        mpm_status st = validate_params(&params[s], why);
        if (st != MPM_OK) return st;
        if (params[s].dim != 2 || params[s].formulation != MPM_FORMULATION_MLS) return MPM_ERR_UNSUPPORTED;
        if (params[s].height + 1 > kBatchMaxRows) return MPM_ERR_CAPACITY;
        if (init[s].count < 0 || init[s].count > 0x7fffffff) return MPM_ERR_INVALID_ARGUMENT;
        if (init[s].count > 0 && (!init[s].position || !init[s].volume)) return MPM_ERR_INVALID_ARGUMENT;
        N += init[s].count;
    }
    if (N > 0x7fffffffLL) return MPM_ERR_INVALID_ARGUMENT;
    int ndev = 0, dev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return MPM_ERR_NO_DEVICE; }
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return MPM_ERR_NO_DEVICE; }
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, k_batch_step<true>) != cudaSuccess) { cudaGetLastError(); return MPM_ERR_NO_DEVICE; }

    mpm_status st = create_whole(params, init, nscenes, dev, nullptr, out);
    for (long long k = 2; st == MPM_ERR_OUT_OF_MEMORY && k < 2LL * nscenes; k *= 2)
        st = create_parts(params, init, nscenes, dev, (int)std::min<long long>(k, nscenes), out);
    return st;
}

mpm_status mpm_batch_destroy(mpm_batch* b) {
    if (!b) return MPM_ERR_INVALID_ARGUMENT;
    if (b->stream) cudaStreamSynchronize(b->stream);
    release(b);
    delete b;
    return MPM_OK;
}

const char* mpm_batch_last_error(const mpm_batch* b) { return b ? b->err.c_str() : "null batch"; }

mpm_status mpm_batch_info(const mpm_batch* b, int32_t* nscenes, int64_t* total) {
    if (!b) return MPM_ERR_INVALID_ARGUMENT;
    if (nscenes) *nscenes = b->nscenes;
    if (total) *total = b->N;
    return MPM_OK;
}

mpm_status mpm_batch_step(mpm_batch* b, int32_t nsteps) {
    if (!b || nsteps < 0) return MPM_ERR_INVALID_ARGUMENT;
    if (nsteps == 0) return MPM_OK;
    for (mpm_batch* p : b->parts) {
        mpm_status st = forget_sums(p);  // the grid was another part's
        if (st == MPM_OK) st = mpm_batch_step(p, nsteps);
        if (st != MPM_OK) return answer(b, p, st);
    }
    if (!b->parts.empty()) {
        b->last_steps = nsteps;
        return MPM_OK;
    }
    const size_t need = (size_t)b->nscenes * ((size_t)nsteps + 1);
    if (need > b->stamps_cap) {
        drop_graphs(b);
        BATCH_CUDA(b, cudaStreamSynchronize(b->stream));
        if (b->arr.stamps && b->captured >= 0) b->old_stamps.push_back(b->arr.stamps);
        else if (b->arr.stamps) cudaFree(b->arr.stamps);
        b->arr.stamps = nullptr;
        b->stamps_cap = 0;
        BATCH_CUDA(b, balloc(&b->arr.stamps, need));
        b->stamps_cap = need;
    }
    if (b->unfinished) {
        const mpm_status st = recover(b);
        if (st != MPM_OK) return st;
    }
    b->unfinished = true;
    b->last_steps = nsteps;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    BATCH_CUDA(b, cudaStreamIsCapturing(b->stream, &capture));
    if (capture != cudaStreamCaptureStatusNone) {
        const mpm_status st = capture_steps(b, nsteps);
        b->unfinished = st != MPM_OK;
        return st;
    }
    if (b->any_fresh) {
        // sums of the new states: sort, then their P2G
        BATCH_CUDA(b, enqueue_sort(b, false));
        b->needs_sort = false;
        b->since_sort = 0;
        if (b->N > 0)
            k_batch_step<false><<<b->sms * MPM_FUSED_MIN_BLOCKS, FusedGeom<2>::THREADS, 0, b->stream>>>(particles(b), b->arr,
                                                                                                       b->ti, b->q);
        BATCH_CUDA(b, cudaGetLastError());
        BATCH_CUDA(b, cudaMemsetAsync(b->arr.fresh, 0, sizeof(int) * (size_t)b->nscenes, b->stream));
        b->any_fresh = false;
    }
    for (int left = nsteps; left > 0;) {
        const int period = sort_period(b);
        const bool sort = b->needs_sort || b->since_sort >= period;
        const int len = std::min({left, kMaxSegment, sort ? period : period - b->since_sort});
        const mpm_status st = run_segment(b, len, sort);
        if (st != MPM_OK) return st;
        b->since_sort = (sort ? 0 : b->since_sort) + len;
        b->needs_sort = false;
        left -= len;
    }
    if (b->captured >= 0 && b->parity != b->captured && b->N > 0) {
        BATCH_CUDA(b, enqueue_sort(b, false));
        b->since_sort = 0;
    }
    k_batch_end<<<1, 256, 0, b->stream>>>(b->arr);
    BATCH_CUDA(b, cudaGetLastError());
    b->unfinished = false;
    return MPM_OK;
}

mpm_status mpm_batch_set_stream(mpm_batch* b, void* stream) {
    if (!b) return MPM_ERR_INVALID_ARGUMENT;
    BATCH_CUDA(b, cudaStreamSynchronize(b->stream));
    b->stream = stream ? (cudaStream_t)stream : b->own_stream;
    for (mpm_batch* p : b->parts) {
        const mpm_status st = mpm_batch_set_stream(p, b->stream);
        if (st != MPM_OK) return answer(b, p, st);
    }
    return MPM_OK;
}

mpm_status mpm_batch_get_state(mpm_batch* b, int32_t scene, mpm_state_host* st) {
    if (!valid_scene(b, scene) || !st || st->count != b->counts[scene]) return MPM_ERR_INVALID_ARGUMENT;
    if (mpm_batch* p = part_of(b, scene)) return answer(b, p, mpm_batch_get_state(p, scene, st));
    float* const host[5] = {st->position, st->velocity, st->affine_b, st->elastic_f, st->plastic_det};
    return read_scene(b, scene, host);
}

// Fields left NULL keep their values. The scene's pending grid sums are void; it is
// sorted and its sums formed anew at the next step.
mpm_status mpm_batch_set_state(mpm_batch* b, int32_t scene, const mpm_state_host* st) {
    if (!valid_scene(b, scene) || !st || st->count != b->counts[scene]) return MPM_ERR_INVALID_ARGUMENT;
    if (mpm_batch* p = part_of(b, scene)) return answer(b, p, mpm_batch_set_state(p, scene, st));
    const int n = b->counts[scene];
    const float* given[5] = {st->position, st->velocity, st->affine_b, st->elastic_f, st->plastic_det};
    for (int f = 0; f < 5; ++f)
        for (size_t i = 0; given[f] && i < (size_t)n * kComps[f]; ++i)
            if (!std::isfinite(given[f][i])) return bfail(b, MPM_ERR_INVALID_ARGUMENT, "state holds non-finite values");
    if (n == 0) return MPM_OK;
    const BatchScene& S = b->scenes[scene];
    for (int f = 0; f < 5; ++f) {
        if (!given[f]) continue;
        BATCH_CUDA(b, cudaMemcpyAsync(scratch(b), given[f], sizeof(float) * (size_t)n * kComps[f], cudaMemcpyHostToDevice,
                                      b->stream));
        k_batch_import<<<(n + 255) / 256, 256, 0, b->stream>>>(field(b, f), b->N, kComps[f], S.p0, n, b->buf[b->parity].id,
                                                               scratch(b));
        BATCH_CUDA(b, cudaGetLastError());
        BATCH_CUDA(b, cudaStreamSynchronize(b->stream));
    }
    BATCH_CUDA(b, cudaMemsetAsync(b->arr.acc + S.node0 * 4, 0, sizeof(unsigned long long) * 4 * (size_t)S.C.nodes, b->stream));
    BATCH_CUDA(b, cudaMemsetAsync(b->arr.fresh + scene, 1, sizeof(int), b->stream));
    BATCH_CUDA(b, cudaStreamSynchronize(b->stream));
    b->any_fresh = true;
    b->needs_sort = true;
    return MPM_OK;
}

mpm_status mpm_batch_get_positions(mpm_batch* b, int32_t scene, float* out, size_t cap_floats) {
    if (!valid_scene(b, scene) || (!out && b->counts[scene] > 0)) return MPM_ERR_INVALID_ARGUMENT;
    if (cap_floats < (size_t)b->counts[scene] * 2) return bfail(b, MPM_ERR_CAPACITY, "output buffer too small");
    if (mpm_batch* p = part_of(b, scene)) return answer(b, p, mpm_batch_get_positions(p, scene, out, cap_floats));
    float* const host[5] = {out, nullptr, nullptr, nullptr, nullptr};
    return read_scene(b, scene, host);
}

mpm_status mpm_batch_get_status(mpm_batch* b, int32_t scene, uint32_t* flags) {
    if (!valid_scene(b, scene) || !flags) return MPM_ERR_INVALID_ARGUMENT;
    if (mpm_batch* p = part_of(b, scene)) return answer(b, p, mpm_batch_get_status(p, scene, flags));
    unsigned f = 0;
    BATCH_CUDA(b, cudaMemcpyAsync(&f, b->arr.status + scene, sizeof(f), cudaMemcpyDeviceToHost, b->stream));
    BATCH_CUDA(b, cudaStreamSynchronize(b->stream));
    *flags = f;
    return MPM_OK;
}

mpm_status mpm_batch_step_times(mpm_batch* b, uint64_t* out, size_t cap, int32_t* nsteps) {
    if (!b || !nsteps) return MPM_ERR_INVALID_ARGUMENT;
    *nsteps = b->last_steps;
    const size_t steps = (size_t)b->last_steps + 1, k = (size_t)b->nscenes;
    if (b->last_steps == 0) return MPM_OK;
    if (!out || cap < steps * k) return bfail(b, MPM_ERR_CAPACITY, "output buffer too small");
    for (size_t p = 0; p < b->parts.size(); ++p) {
        int32_t ns = 0;
        const size_t at = steps * (size_t)b->part_first[p];
        const mpm_status st = mpm_batch_step_times(b->parts[p], out + at, cap - at, &ns);
        if (st != MPM_OK) return answer(b, b->parts[p], st);
    }
    if (!b->parts.empty()) return MPM_OK;
    std::vector<unsigned long long> t(steps * k);  // [step][scene] on the device
    BATCH_CUDA(b, cudaMemcpyAsync(t.data(), b->arr.stamps, sizeof(uint64_t) * t.size(), cudaMemcpyDeviceToHost, b->stream));
    BATCH_CUDA(b, cudaStreamSynchronize(b->stream));
    for (size_t s = 0; s < k; ++s)
        for (size_t j = 0; j < steps; ++j) out[s * steps + j] = t[j * k + s];
    return MPM_OK;
}

mpm_status mpm_batch_get_config(const mpm_batch* b, mpm_batch_config* cfg) {
    if (!b || !cfg) return MPM_ERR_INVALID_ARGUMENT;
    *cfg = b->parts.empty() ? b->cfg : b->parts[0]->cfg;
    return MPM_OK;
}

mpm_status mpm_batch_set_config(mpm_batch* b, const mpm_batch_config* cfg) {
    if (!b || !cfg) return MPM_ERR_INVALID_ARGUMENT;
    if (b->parts.empty()) return configure(b, *cfg);
    const mpm_batch_config old = b->parts[0]->cfg;
    for (mpm_batch* p : b->parts) {
        const mpm_status st = configure(p, *cfg);
        if (st == MPM_OK) continue;
        answer(b, p, st);
        for (mpm_batch* q : b->parts) configure(q, old);
        return st;
    }
    return MPM_OK;
}

mpm_status mpm_batch_tune(mpm_batch* b, int32_t trial_steps, mpm_batch_config* chosen, double* best_ms) {
    if (!b || trial_steps < 1) return MPM_ERR_INVALID_ARGUMENT;
    if (!b->parts.empty()) {
        double sum = 0.0;
        for (mpm_batch* p : b->parts) {
            double ms = 0.0;
            mpm_status st = forget_sums(p);
            if (st == MPM_OK) st = mpm_batch_tune(p, trial_steps, chosen, &ms);
            if (st != MPM_OK) return answer(b, p, st);
            sum += ms;
        }
        if (best_ms) *best_ms = sum;
        return MPM_OK;
    }
    BATCH_CUDA(b, cudaStreamSynchronize(b->stream));
    const size_t n = (size_t)b->N;
    // Snapshot of the particles and flags; the sums are formed anew from them.
    const BatchBuffers F = b->buf[b->parity];
    struct Span { void* p; size_t bytes; };
    const Span spans[] = {{F.x, 8 * n}, {F.v, 8 * n}, {F.B, 16 * n}, {F.Fe, 16 * n}, {F.Jp, 4 * n}, {F.mass, 4 * n},
                          {F.vol, 4 * n}, {F.id, 4 * n}, {b->arr.status, sizeof(unsigned) * (size_t)b->nscenes}};
    size_t total = 0;
    for (const Span& sp : spans) total += (sp.bytes + 255) / 256 * 256;
    unsigned char* snap = nullptr;
    BATCH_CUDA(b, balloc(&snap, total));
    const int parity = b->parity, last = b->last_steps;
    auto copy_all = [&](bool save) {
        size_t o = 0;
        cudaError_t e = cudaSuccess;
        for (const Span& sp : spans) {
            if (e == cudaSuccess && sp.bytes)
                e = cudaMemcpyAsync(save ? snap + o : sp.p, save ? sp.p : snap + o, sp.bytes, cudaMemcpyDeviceToDevice,
                                    b->stream);
            o += (sp.bytes + 255) / 256 * 256;
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
        return e;
    };
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    float ms = 0.f;
    mpm_status st = MPM_OK;
    cudaError_t ce = copy_all(true);
    if (ce == cudaSuccess) ce = cudaEventCreate(&e0);
    if (ce == cudaSuccess) ce = cudaEventCreate(&e1);
    // one untimed call (graph capture, sort, sums), then the timed one
    if (ce == cudaSuccess) st = mpm_batch_step(b, trial_steps);
    if (ce == cudaSuccess && st == MPM_OK) ce = cudaEventRecord(e0, b->stream);
    if (ce == cudaSuccess && st == MPM_OK) st = mpm_batch_step(b, trial_steps);
    if (ce == cudaSuccess && st == MPM_OK) ce = cudaEventRecord(e1, b->stream);
    if (ce == cudaSuccess && st == MPM_OK) ce = cudaEventSynchronize(e1);
    if (ce == cudaSuccess && st == MPM_OK) ce = cudaEventElapsedTime(&ms, e0, e1);
    // put the batch back as it was, whatever happened above
    cudaStreamSynchronize(b->stream);
    b->parity = parity;
    b->last_steps = last;
    const cudaError_t cr = copy_all(false);
    if (ce == cudaSuccess) ce = cr;
    const mpm_status sf = forget_sums(b);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(snap);
    if (ce != cudaSuccess) {
        cudaGetLastError();
        return bfail(b, MPM_ERR_CUDA, std::string("tuner: ") + cudaGetErrorString(ce));
    }
    if (st != MPM_OK) return st;
    if (sf != MPM_OK) return sf;
    if (chosen) *chosen = b->cfg;
    if (best_ms) *best_ms = ms;
    return MPM_OK;
}

}  // extern "C"
