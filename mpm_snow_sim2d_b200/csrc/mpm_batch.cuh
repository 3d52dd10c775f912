// Batched 2D scenes: many independent MLS scenes of uneven size stepped together
// by the kernels of the single-scene solver.
//
// The scenes lie side by side: one particle array (scene after scene), one grid
// (each scene's nodes after the last scene's), one list of cell tiles and of node
// blocks. A step is the single solver's: grid update over the marked node blocks,
// G2P and the next P2G by one warp per window of 32 slots (fused_window), the
// queued particles' return map, their P2G. A window lies in one tile of one scene,
// whose constants its warp reads from shared memory. Every sort_period steps all
// scenes are sorted by (tile, cell, id).
//
// A scene's result depends neither on the other scenes, nor on the order of its
// particles, nor on when it was sorted: each particle's contribution to a node is
// rounded to int64 fixed point by itself (the EXACT scatter; integer sums), and
// all else is per particle or per node.
//
// Bound: as k_g2p2g_direct (memory pipe and issue). The former kernel held each
// scene's grid in the shared memory of a thread-block cluster and added 48 int64
// values per particle and step there (red.shared::cluster, 68% of their wavefronts
// bank conflicts); one persistent cluster per scene left the GPU waiting for the
// largest ones. 256 scenes, 2.81M particles, 100 steps: 0.83 ms a step, now 0.34.
#pragma once

#include "mpm_fused.cuh"

namespace mpm {

constexpr int kBatchMaxRows = 512;  // node rows of one scene

struct BatchScene {
    StepConsts C;
    SceneView view;    // extents, tiles per axis, first tile
    long long p0;      // first particle slot
    long long node0;   // first node
    int n;             // particles
    int blk0;          // first node block
    int nblk[2];       // node blocks per axis
};

struct ManyScenes {
    const BatchScene* scenes;
    const int* of_slots;  // scene of each slot
    const int* of_tiles;  // scene of each tile
    __device__ __forceinline__ const SceneView& of_slot(int i) const { return scenes[of_slots[i]].view; }
    __device__ __forceinline__ const SceneView& of_tile(int t) const { return scenes[of_tiles[t]].view; }
};

struct BatchArrays {
    const BatchScene* scenes;
    const int* of_slots;
    const int* of_blocks;        // scene of each node block
    unsigned long long* acc;     // [nodes][4]
    float4* gv;                  // [nodes]
    unsigned* status;            // per scene: MPM_FLAG_* bits
    int* fresh;                  // per scene: the pending sums are missing (new or uploaded state)
    unsigned long long* stamps;  // [step of the call][scene] device timestamps (ns)
    int* step;                   // device scalar: steps of the call done so far
    int nscenes;
};

__device__ __forceinline__ unsigned long long device_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// A scene's own view of the tiles and node blocks.
__device__ __forceinline__ TileInfo scene_tiles(const TileInfo& TI, const BatchScene& S) {
    TileInfo V = TI;
    V.tiles[0] = S.view.tiles[0];
    V.tiles[1] = S.view.tiles[1];
    V.nblk[0] = S.nblk[0];
    V.nblk[1] = S.nblk[1];
    V.blk0 = S.blk0;
    return V;
}

// The scene's record into the warp's shared memory.
__device__ __forceinline__ const BatchScene& stage_scene(const BatchScene* scenes, int s, BatchScene* mine) {
    constexpr int W = sizeof(BatchScene) / 4;
    __syncwarp();
    for (int k = threadIdx.x & 31; k < W; k += 32)
        reinterpret_cast<int*>(mine)[k] = reinterpret_cast<const int*>(scenes + s)[k];
    __syncwarp();
    return *mine;
}

// Grid update of the marked node blocks of all scenes (k_grid_marked per scene);
// records the time at which a step begins.
__global__ void __launch_bounds__(256) k_batch_grid(BatchArrays B, TileInfo TI) {
    using G = TileGeom<2>;
    chain_wait();
    const int nb = *TI.n_marked;
    const long long total = (long long)nb * G::BN;
    if (blockIdx.x == 0) {
        const int step = *B.step;
        const unsigned long long t = device_ns();
        for (int s = threadIdx.x; s < B.nscenes; s += blockDim.x) B.stamps[(long long)step * B.nscenes + s] = t;
    }
    for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < total;
         w += (long long)gridDim.x * blockDim.x) {
        const int blk = TI.mark_list[w / G::BN], loc = int(w % G::BN);
        const int sc = B.of_blocks[blk];
        const BatchScene& S = B.scenes[sc];
        const int rb = blk - S.blk0;
        const int gx = rb % S.nblk[0] * G::T + loc % G::T, gy = rb / S.nblk[0] * G::T + loc / G::T;
        if (loc == 0) TI.mark[blk] = 0;
        if (gx >= S.C.nx || gy >= S.C.ny) continue;
        grid_node_at<2, kMLS>(S.C, B.acc + S.node0 * 4, B.gv + S.node0, B.status + sc, (long long)gy * S.C.nx + gx, gx, gy, 0);
    }
    grid_finish(TI, B.step);
}

// The fused step of one window per warp (k_g2p2g_direct), or with G2P = false the
// P2G of the stored state of the scenes that have no pending sums.
template <bool G2P>
__global__ void __launch_bounds__(FusedGeom<2>::THREADS, MPM_FUSED_MIN_BLOCKS)
    k_batch_step(Particles P, BatchArrays B, TileInfo TI, SlowQueue Q) {
    using G = FusedGeom<2>;
    __shared__ float4 pay_s[G::WARPS][G::PAY / 4];
    __shared__ BatchScene scene_s[G::WARPS];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float* pay = reinterpret_cast<float*>(pay_s[wid]);
    chain_wait();
    const int nitems = *TI.n_items;
    for (int e = wid * gridDim.x + blockIdx.x; e < nitems; e += G::WARPS * gridDim.x) {
        const int4 item = TI.items[e];
        if (!G2P && !B.fresh[item.w]) continue;
        const BatchScene& S = stage_scene(B.scenes, item.w, &scene_s[wid]);
        const TileInfo V = scene_tiles(TI, S);
        SlowQueue QS = Q;
        QS.scene = item.w;
        int tc[3] = {0, 0, 0}, bo[3] = {0, 0, 0};
        tile_origin<2>(V, item.x - S.view.tile0, tc, bo);
        const unsigned bits = __reduce_or_sync(
            0xffffffffu, fused_window<2, 4, G2P, true, true>(P, S.C, V, B.gv + S.node0, B.acc + S.node0 * 4, QS,
                                                             B.status + item.w, nullptr, nullptr, bo, item.y, item.z, TI.win, 0, pay));
        if (lane < 9 && (bits >> lane) & 1u)
            mark_block_once(V, (tc[1] - 1 + lane / 3) * V.nblk[0] + tc[0] - 1 + lane % 3);
    }
}

__global__ void __launch_bounds__(256) k_batch_plastic(Particles P, BatchArrays B, SlowQueue Q) {
    chain_wait();
    const int m = *Q.count;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m; e += gridDim.x * blockDim.x) {
        const int entry = Q.list[e], sc = B.of_slots[entry >= 0 ? entry : -1 - entry];
        const BatchScene& S = B.scenes[sc];
        g2p_queued_exact<2, 4>(P, S.C, B.gv + S.node0, Q, e, B.status + sc);
    }
}

// P2G of the queued particles (k_p2g_windows).
__global__ void __launch_bounds__(FusedGeom<2>::THREADS) k_batch_windows(Particles P, BatchArrays B, TileInfo TI, SlowQueue Q) {
    using G = FusedGeom<2>;
    __shared__ float4 pay_s[G::WARPS][G::PAY / 4];
    __shared__ BatchScene scene_s[G::WARPS];
    const int wid = threadIdx.x >> 5;
    chain_wait();
    const int nw = min(*Q.nwin, Q.win_capacity);
    for (int r = blockIdx.x * G::WARPS + wid; r < nw; r += gridDim.x * G::WARPS) {
        const int4 rec = Q.win[r];
        const BatchScene& S = stage_scene(B.scenes, rec.w, &scene_s[wid]);
        queued_window<2, 4, true>(P, S.C, scene_tiles(TI, S), rec, B.acc + S.node0 * 4, B.status + rec.w,
                                  reinterpret_cast<float*>(pay_s[wid]));
    }
}

// End of a call, one CTA: the last time stamp; the step count starts over.
__global__ void __launch_bounds__(256) k_batch_end(BatchArrays B) {
    const unsigned long long t = device_ns();
    const int step = *B.step;
    for (int s = threadIdx.x; s < B.nscenes; s += blockDim.x) B.stamps[(long long)step * B.nscenes + s] = t;
    __syncthreads();
    if (threadIdx.x == 0) *B.step = 0;
}

// One field of a scene, creation order, and back (slots of the scene hold particles
// id[slot]; an upload keeps the slot order, the next sort restores locality).
__global__ void __launch_bounds__(256) k_batch_export(const float* __restrict__ soa, long long stride, int comps, long long p0,
                                                      int n, const int* __restrict__ id, float* __restrict__ aos) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int p = id[p0 + s];
    for (int c = 0; c < comps; ++c) aos[(long long)p * comps + c] = soa[c * stride + p0 + s];
}

__global__ void __launch_bounds__(256) k_batch_import(float* __restrict__ soa, long long stride, int comps, long long p0, int n,
                                                      const int* __restrict__ id, const float* __restrict__ aos) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int p = id[p0 + s];
    for (int c = 0; c < comps; ++c) soa[c * stride + p0 + s] = aos[(long long)p * comps + c];
}

}  // namespace mpm
