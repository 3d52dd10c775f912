// Seeded Poisson-disk sampling of snow shapes on the device: the reference's
// PoissonDiskCircle / PoissonDiskSphere (src/shared/Shapes.h:17-117,143-234,
// Bridson's sequential algorithm seeded from std::random_device) replaced by a
// parallel, reproducible grid-phase dart thrower.
//
// Background grid of cells of side min_dist / sqrt(dim): a cell holds at most
// one sample. Cells whose indices agree modulo 3 on every axis form a phase;
// two cells of one phase are at least 2 cell sides = 2 min_dist / sqrt(dim) >=
// min_dist apart, so every cell of a phase can try a candidate at once without
// two new samples conflicting. Each round visits the 3^dim phases in order;
// in each, every empty cell that overlaps a shape draws one candidate
// uniformly in the cell from a counter-based hash of (seed, cell, round, axis)
// and keeps it when it lies in a shape and no sample in the 5^dim surrounding
// cells is closer than min_dist. The result depends on the seed alone.
#include <algorithm>
#include <cmath>

#include <cuda_runtime.h>

#include "mpm/mpm.h"

namespace {

constexpr int kMaxShapes = 64;

struct SampleShapes {
    int n;
    int kind[kMaxShapes];
    float c[kMaxShapes][3], r[kMaxShapes], h[kMaxShapes][3];
};

struct SampleGrid {
    int dim;
    int nc[3];          // cells per axis
    float origin[3];
    float cell, min_dist;
    unsigned long long seed;
};

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    // splitmix64 finaliser (Steele, Lea, Flood 2014)
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ float uniform01(unsigned long long seed, long long cell, int round, int axis) {
    const unsigned long long h =
        mix64(seed ^ mix64((unsigned long long)cell * 4 + (unsigned long long)axis + ((unsigned long long)round << 40)));
    return float(h >> 40) * (1.0f / 16777216.0f);  // 24 bits: exactly representable in [0, 1)
}

// Every floating-point step below is an explicitly rounded operation (no
// fused multiply-add), so that a float32 restatement on the CPU reproduces
// the samples bit for bit.
__device__ __forceinline__ bool inside(const SampleShapes& S, int dim, const float* p) {
    for (int s = 0; s < S.n; ++s) {
        if (S.kind[s] == MPM_SHAPE_BALL) {
            float d2 = 0.f;
            for (int k = 0; k < dim; ++k) {
                const float d = __fsub_rn(p[k], S.c[s][k]);
                d2 = __fadd_rn(d2, __fmul_rn(d, d));
            }
            if (d2 <= __fmul_rn(S.r[s], S.r[s])) return true;
        } else {
            bool in = true;
            for (int k = 0; k < dim; ++k) in = in && fabsf(__fsub_rn(p[k], S.c[s][k])) <= S.h[s][k];
            if (in) return true;
        }
    }
    return false;
}

// One phase of one round: cells (3a + px, 3b + py, 3c + pz), LANES lanes each.
// Small grids are bound by latency: a phase of a reference snowball has 8k cells, and
// the phases run one after the other (30 rounds x 27 of them). Eight lanes share the
// cell's candidate and split its 5^(dim-1) rows of five neighbours, so that all of a
// cell's are in flight at once: 5.8 us a phase, 12 with one lane, 28 with one lane that
// reads one neighbour after the other. Large grids are bound by issue, and most of
// their cells are filled, or have a sample too near among the first neighbours: one lane
// reads row by row and stops. Whole calls (3D, 30 rounds; 8 lanes, 1): 524k cells 8.7, 10.6 ms; 1.0M 14.5,
// 11.9; 4.1M 51, 25; 64M 939, 150 (a neighbour at a time: 536). 2D: 81k 1.66, 1.75; 321k 4.2, 2.5;
// 8.0M 93, 11 (90).
// The launch of the next phase overlaps this one up to griddepcontrol.wait: the
// candidate depends on nothing. A cell found filled before the wait stays filled; one
// found free may have been filled since, by its own phase of the round before, which
// need not be complete while phases overlap: the test after the wait includes the cell
// itself. Reads of `cells` go to L2, since lines read before the wait may hold
// neighbours of earlier phases.
constexpr long long kManyLanes2 = 10240, kManyLanes3 = 24576;  // cells of a phase up to which eight lanes are faster

template <int LANES>
__global__ void __launch_bounds__(256, LANES > 1 ? 2 : 6) k_sample_phase(SampleGrid G, const SampleShapes* __restrict__ shapes,
                                                      const unsigned char* __restrict__ live, int round, int px, int py,
                                                      int pz, float4* cells) {
    const int mx = (G.nc[0] - px + 2) / 3, my = (G.nc[1] - py + 2) / 3, mz = G.dim == 3 ? (G.nc[2] - pz + 2) / 3 : 1;
    const long long total = (long long)mx * my * mz;
    const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LANES;
    const int sub = threadIdx.x % LANES;
    const int ix = 3 * int(t % mx) + px, iy = 3 * int((t / mx) % my) + py, iz = G.dim == 3 ? 3 * int(t / ((long long)mx * my)) + pz : 0;
    const long long id = ((long long)iz * G.nc[1] + iy) * G.nc[0] + ix;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    bool ok = t < total && ix < G.nc[0] && iy < G.nc[1] && (G.dim != 3 || iz < G.nc[2]);
    ok = ok && live[id] && __ldcg(&cells[id]).w == 0.f;
    float p[3] = {0.f, 0.f, 0.f};
    if (ok) {
        const int ic[3] = {ix, iy, iz};
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (k < G.dim)
                p[k] = __fadd_rn(G.origin[k], __fmul_rn(__fadd_rn(float(ic[k]), uniform01(G.seed, id, round, k)), G.cell));
        ok = inside(*shapes, G.dim, p);
    }
    // (the pointer passes through the wait, so that no later load can move ahead of it)
    asm volatile("griddepcontrol.wait;" : "+l"(cells) : : "memory");
    // the cell's lanes agree on `ok`; all lanes of the warp stay for the vote
    bool clash = false;
    if (ok) {
        const float r2 = __fmul_rn(G.min_dist, G.min_dist);
        const int rows = G.dim == 3 ? 25 : 5;
        // eight lanes: all neighbours in flight at once; one: row by row until a sample is too near
#pragma unroll(LANES > 1 ? 4 : 1)
        for (int q = 0; LANES > 1 ? q < 4 : q < rows && !clash; ++q) {
            const int r = sub + q * LANES;
            const int jy = iy + r % 5 - 2, jz = G.dim == 3 ? iz + r / 5 - 2 : 0;
            const bool in = r < rows && jy >= 0 && jy < G.nc[1] && jz >= 0 && jz < G.nc[2];
            const long long row = ((long long)jz * G.nc[1] + jy) * G.nc[0];
            float4 n[5];
#pragma unroll
            for (int dx = 0; dx < 5; ++dx) {
                const int jx = ix + dx - 2;
                n[dx] = in && jx >= 0 && jx < G.nc[0] ? __ldcg(&cells[row + jx]) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int dx = 0; dx < 5; ++dx) {
                const float ddx = __fsub_rn(n[dx].x, p[0]), ddy = __fsub_rn(n[dx].y, p[1]), ddz = __fsub_rn(n[dx].z, p[2]);
                clash = clash || (n[dx].w != 0.f && r == rows / 2 && dx == 2);  // the cell itself
                clash = clash || (n[dx].w != 0.f &&
                                  __fadd_rn(__fadd_rn(__fmul_rn(ddx, ddx), __fmul_rn(ddy, ddy)), __fmul_rn(ddz, ddz)) < r2);
            }
        }
    }
    const unsigned any = __ballot_sync(0xffffffffu, clash);
    const int first = (threadIdx.x & 31) / LANES * LANES;
    if (ok && sub == 0 && ((any >> first) & ((1u << LANES) - 1)) == 0u) cells[id] = make_float4(p[0], p[1], p[2], 1.f);
}

// Cells that can hold a sample: those overlapping a shape's bounding box.
__global__ void k_sample_live(SampleGrid G, const SampleShapes* __restrict__ shapes, long long ncells,
                              unsigned char* __restrict__ live) {
    const SampleShapes& S = *shapes;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= ncells) return;
    const int ic[3] = {int(id % G.nc[0]), int((id / G.nc[0]) % G.nc[1]), int(id / ((long long)G.nc[0] * G.nc[1]))};
    bool any = false;
    for (int s = 0; s < S.n && !any; ++s) {
        bool in = true;
        for (int k = 0; k < G.dim; ++k) {
            const float lo = __fadd_rn(G.origin[k], __fmul_rn(float(ic[k]), G.cell)), hi = __fadd_rn(lo, G.cell);
            const float e = S.kind[s] == MPM_SHAPE_BALL ? S.r[s] : S.h[s][k];
            in = in && hi >= __fsub_rn(S.c[s][k], e) && lo <= __fadd_rn(S.c[s][k], e);
        }
        any = in;
    }
    live[id] = any ? 1 : 0;
}

// Which shape a sample belongs to (the first that contains it).
__device__ __forceinline__ int shape_index(const SampleShapes& S, int dim, const float* p) {
    for (int s = 0; s < S.n; ++s) {
        if (S.kind[s] == MPM_SHAPE_BALL) {
            float d2 = 0.f;
            for (int k = 0; k < dim; ++k) {
                const float d = __fsub_rn(p[k], S.c[s][k]);
                d2 = __fadd_rn(d2, __fmul_rn(d, d));
            }
            if (d2 <= __fmul_rn(S.r[s], S.r[s])) return s;
        } else {
            bool in = true;
            for (int k = 0; k < dim; ++k) in = in && fabsf(__fsub_rn(p[k], S.c[s][k])) <= S.h[s][k];
            if (in) return s;
        }
    }
    return -1;
}

// The samples in cell order (deterministic): how many in each block of
// kCompact cells, then each block's to its place in the output (the first
// `capacity` of them; `total` gets the number of all). The host used to scan the
// whole cell array, 1.1 ms of its copy and scan for a reference snowball.
constexpr int kCompact = 1024;

__global__ void __launch_bounds__(kCompact) k_sample_count(const float4* __restrict__ cells, long long ncells,
                                                           int* __restrict__ count) {
    const long long i = (long long)blockIdx.x * kCompact + threadIdx.x;
    const int n = __syncthreads_count(i < ncells && cells[i].w != 0.f);
    if (threadIdx.x == 0) count[blockIdx.x] = n;
}

__global__ void __launch_bounds__(kCompact) k_sample_compact(const SampleShapes* __restrict__ shapes, int dim,
                                                             const float4* __restrict__ cells, long long ncells,
                                                             const int* __restrict__ count, long long capacity,
                                                             float* __restrict__ pos, int* __restrict__ owner,
                                                             unsigned long long* __restrict__ total) {
    __shared__ unsigned long long s_before;
    __shared__ int s_warp[kCompact / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_before = 0ull;
    __syncthreads();
    unsigned long long b = 0ull;
    for (int k = tid; k < (int)blockIdx.x; k += kCompact) b += (unsigned)count[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
    if (lane == 0 && b) atomicAdd(&s_before, b);
    const long long i = (long long)blockIdx.x * kCompact + tid;
    const float4 q = i < ncells ? cells[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const unsigned mine = __ballot_sync(0xffffffffu, q.w != 0.f);
    if (lane == 0) s_warp[warp] = __popc(mine);
    __syncthreads();
    unsigned long long at = s_before + __popc(mine & ((1u << lane) - 1));
    for (int w = 0; w < warp; ++w) at += s_warp[w];
    if (q.w != 0.f && (long long)at < capacity) {
        const float p[3] = {q.x, q.y, q.z};
        for (int k = 0; k < dim; ++k) pos[at * dim + k] = p[k];
        if (owner) owner[at] = shape_index(*shapes, dim, p);
    }
    if (blockIdx.x == gridDim.x - 1 && tid == kCompact - 1) *total = at + (q.w != 0.f);
}

}  // namespace

extern "C" {

mpm_status mpm_sample_shapes(int32_t dim, const mpm_shape* shapes, int32_t nshapes, float min_dist, uint64_t seed,
                             int32_t rounds, float* positions, int32_t* shape_of, int64_t capacity, int64_t* count) {
    if ((dim != 2 && dim != 3) || !shapes || nshapes < 1 || nshapes > kMaxShapes || !(min_dist > 0.f) ||
        !std::isfinite(min_dist) || rounds < 1 || rounds > 1000 || !count || capacity < 0 ||
        (capacity > 0 && !positions))
        return MPM_ERR_INVALID_ARGUMENT;
    *count = 0;
    SampleShapes S{};
    S.n = nshapes;
    float lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
    for (int s = 0; s < nshapes; ++s) {
        const mpm_shape& sh = shapes[s];
        if (sh.kind != MPM_SHAPE_BALL && sh.kind != MPM_SHAPE_BOX) return MPM_ERR_INVALID_ARGUMENT;
        S.kind[s] = sh.kind;
        S.r[s] = sh.radius;
        for (int k = 0; k < 3; ++k) { S.c[s][k] = sh.center[k]; S.h[s][k] = sh.half[k]; }
        for (int k = 0; k < dim; ++k) {
            const float e = sh.kind == MPM_SHAPE_BALL ? sh.radius : sh.half[k];
            if (!(e >= 0.f) || !std::isfinite(e) || !std::isfinite(sh.center[k])) return MPM_ERR_INVALID_ARGUMENT;
            lo[k] = s == 0 ? sh.center[k] - e : std::min(lo[k], sh.center[k] - e);
            hi[k] = s == 0 ? sh.center[k] + e : std::max(hi[k], sh.center[k] + e);
        }
    }
    SampleGrid G{};
    G.dim = dim;
    G.min_dist = min_dist;
    G.cell = min_dist / std::sqrt((float)dim);
    G.seed = seed;
    double ncd = 1.0;
    for (int k = 0; k < 3; ++k) {
        G.origin[k] = k < dim ? lo[k] : 0.f;
        G.nc[k] = k < dim ? std::max(1, (int)std::ceil((hi[k] - lo[k]) / G.cell) + 1) : 1;
        ncd *= G.nc[k];
    }
    if (ncd > 4.0e8) return MPM_ERR_CAPACITY;  // 6.4 GB of cells: refuse rather than exhaust the device
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return MPM_ERR_NO_DEVICE; }
    const long long ncells = (long long)ncd;
    // one allocation: the cells, the shapes, the output, which cells can hold a sample
    const long long room = std::min<long long>(capacity, ncells), blocks = (ncells + kCompact - 1) / kCompact;
    size_t bytes = 0;
    auto take = [&](size_t n) { const size_t at = bytes; bytes += (n + 255) / 256 * 256; return at; };
    const size_t cell_bytes = sizeof(float4) * (size_t)ncells;
    const size_t o_cells = take(cell_bytes), o_shapes = take(sizeof(SampleShapes)), o_total = take(sizeof(unsigned long long)),
                 o_count = take(sizeof(int) * (size_t)blocks), o_pos = take(sizeof(float) * (size_t)(room * dim)),
                 o_owner = take(shape_of ? sizeof(int) * (size_t)room : 0), o_live = take((size_t)ncells);
    unsigned char* base = nullptr;
    if (cudaMalloc(&base, bytes) != cudaSuccess) {
        cudaGetLastError();
        return MPM_ERR_OUT_OF_MEMORY;
    }
    float4* cells = reinterpret_cast<float4*>(base + o_cells);
    SampleShapes* dshapes = reinterpret_cast<SampleShapes*>(base + o_shapes);
    unsigned long long* dtotal = reinterpret_cast<unsigned long long*>(base + o_total);
    int *dcount = reinterpret_cast<int*>(base + o_count), *downer = shape_of ? reinterpret_cast<int*>(base + o_owner) : nullptr;
    float* dpos = reinterpret_cast<float*>(base + o_pos);
    unsigned char* live = base + o_live;
    if (cudaMemset(cells, 0, cell_bytes) != cudaSuccess ||
        cudaMemcpy(dshapes, &S, sizeof(S), cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(base);
        return MPM_ERR_CUDA;
    }
    const int threads = 256;
    k_sample_live<<<(unsigned)((ncells + threads - 1) / threads), threads>>>(G, dshapes, ncells, live);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc = {};
    lc.blockDim = dim3(threads);
    lc.attrs = attr;
    lc.numAttrs = 0;  // the first phase waits for all of k_sample_live
    cudaError_t le = cudaGetLastError();
    const int pz_n = dim == 3 ? 3 : 1;
    for (int r = 0; r < rounds && le == cudaSuccess; ++r)
        for (int pz = 0; pz < pz_n; ++pz)
            for (int py = 0; py < 3; ++py)
                for (int px = 0; px < 3; ++px) {
                    const long long mx = (G.nc[0] - px + 2) / 3, my = (G.nc[1] - py + 2) / 3,
                                    mz = dim == 3 ? (G.nc[2] - pz + 2) / 3 : 1;
                    const long long phase = mx * my * mz;
                    if (phase == 0 || le != cudaSuccess) continue;
                    const int lanes = phase <= (dim == 3 ? kManyLanes3 : kManyLanes2) ? 8 : 1;
                    lc.gridDim = dim3((unsigned)((phase * lanes + threads - 1) / threads));
                    le = cudaLaunchKernelEx(&lc, lanes == 8 ? k_sample_phase<8> : k_sample_phase<1>, G, (const SampleShapes*)dshapes,
                                            (const unsigned char*)live, r, px, py, pz, cells);
                    lc.numAttrs = 1;
                }
    unsigned long long total = 0;
    if (le == cudaSuccess) {
        k_sample_count<<<(unsigned)blocks, kCompact>>>(cells, ncells, dcount);
        k_sample_compact<<<(unsigned)blocks, kCompact>>>(dshapes, dim, cells, ncells, dcount, room, dpos, downer, dtotal);
        le = cudaGetLastError();
    }
    if (le == cudaSuccess) le = cudaMemcpy(&total, dtotal, sizeof(total), cudaMemcpyDeviceToHost);
    const size_t n = (size_t)std::min<unsigned long long>(total, (unsigned long long)room);
    if (le == cudaSuccess && n > 0) le = cudaMemcpy(positions, dpos, sizeof(float) * n * dim, cudaMemcpyDeviceToHost);
    if (le == cudaSuccess && n > 0 && shape_of) le = cudaMemcpy(shape_of, downer, sizeof(int) * n, cudaMemcpyDeviceToHost);
    cudaFree(base);
    if (le != cudaSuccess) {
        cudaGetLastError();
        return MPM_ERR_CUDA;
    }
    *count = (int64_t)total;
    return (int64_t)total > capacity ? MPM_ERR_CAPACITY : MPM_OK;
}

}  // extern "C"
