// Fused transfer for the tiled MLS path: G2P of step n and P2G of step n+1 in
// one kernel per step (the G2P2G scheme of Wang et al., "A Massively Parallel
// and Scalable Multi-GPU Material Point Method", ACM TOG 39(4), 2020).
//
// Work is handed out as items. In k_g2p2g_pipe an item is up to 32 windows of a cell
// tile of the last sort (nearly always all of it): a CTA has the node velocities of a fixed
// box of BE^D nodes around the tile in shared memory (the stencils of every particle sorted
// into the tile that has since moved less than a cell), loaded one item ahead by TMA tensor
// loads (cp.async.bulk.tensor, out-of-grid nodes zero-filled); its warps meet at
// mbarriers only. In k_g2p2g_direct an item is one window and nothing is staged.
// Each warp, on its own, takes windows of up to 32 consecutive slots of a tile
// and for its window
//   1. per particle (one lane each): gathers the grid
//      (src/gpu/shaders/3d/g2p.glsl:28-71), updates x, v, B and the trial F_E,
//      and when the return map is provably the identity (elastic band)
//      computes the next step's P2G affine matrix A = 3 m B - 3 dt V sigma in
//      registers (3d/p2g.glsl:44-90); the rest are queued for the exact (or
//      learned) return map with their trial F;
//   2. writes each in-band particle's P2G payload (stencil weights at the new
//      position, m v, A) to the warp's shared memory, ordered by stencil, and sums
//      them over the node columns its lanes own, in FP32 registers; what leaves
//      the registers goes to the grid as int64 fixed point (red.global, no
//      return value): scatter_rows.
// Particles whose stencil leaves the box (drifted more than a cell since the
// sort) gather from global memory. Queued particles (out of the elastic band, or
// a stencil clipped by the grid edge) are scattered after their return map: the
// warp records its window (first slot, mask of the lanes to scatter: the queued
// ones, or with them all the others) for k_p2g_windows.
//
// Determinism: every sum beyond one window is an integer add, and the FP32 sums
// in it are a function of the slot order, the window boundaries (fixed offsets
// inside a tile) and which particles were queued -- all functions of the state. After
// creation or a state upload a P2G-only pass of the same kernel (reading the
// stored state) forms the first sums. A checkpoint stores the pending sums
// themselves, so a resumed run never recomputes them.
#pragma once

#include <type_traits>

#include <cuda.h>

#include "mpm_tiled.cuh"

namespace mpm {

#ifndef MPM_FUSED_THREADS
#define MPM_FUSED_THREADS 128
#endif
template <int D> struct FusedGeom {
    static constexpr int T = TileGeom<D>::T;            // cells per tile edge: 4 (3D), 8 (2D)
    static constexpr int BE = T + 5;                    // box edge in nodes: tile nodes - 2 .. tile + T + 2
    static constexpr int BN = D == 3 ? BE * BE * BE : BE * BE;  // 729 (3D), 169 (2D)
    static constexpr int BNP = (BN + 7) / 8 * 8;        // box rows padded to 128 bytes (TMA destinations)
    static constexpr int THREADS = MPM_FUSED_THREADS;
    static constexpr int WARPS = THREADS / 32;
    static constexpr int WIN = 32;                      // slots per warp window (one per lane)
    static constexpr int PS = D == 3 ? 36 : 44;         // payload floats per particle (layout: Scatter)
    static constexpr int PAY = WIN * (PS + 2);          // floats of a warp's window: rows, then stencils
    static_assert(THREADS % 32 == 0, "whole warps");
};

// CTAs per SM the register budget is sized for: 20 warps per SM, 96
// registers (measured on the 128^3 snowball scene: 6 % faster than 24 warps at
// 80 registers, which spill)
#ifndef MPM_FUSED_MIN_BLOCKS
#define MPM_FUSED_MIN_BLOCKS (640 / MPM_FUSED_THREADS)
#endif

// ---------------------------------------------------------------------------
// Interior gather from a node array with strides (sy, sz): the box in shared
// memory (SMEM) or the global grid. Same sums and order as gather_interior.
// `gc0`, `gsy`, `gsz`: the global node id of the first stencil node and the
// global strides, for the wall-velocity pass (3D vc of nodes a wall moved is
// only kept in global memory). That pass reads it for the flagged nodes alone,
// a whole x plane of them in flight at once: the 128^3 snowball scene, whose
// slab rests on the floor, took 56 of 332 us for it with four loads in flight.
template <int D, int S, bool SMEM, typename I>
__device__ __forceinline__ void gather_nodes(const StepConsts& C, const float4* nodes, I c0, I sy, I sz,
                                             const float4* __restrict__ gv, const float4* walls, long long gc0,
                                             long long gsy, long long gsz, const float (*wk)[S], const float (*off)[S], float* nv, float* nB,
                                             float* nx) {
    float wd[3][S];
#pragma unroll
    for (int k = 0; k < D; ++k)
#pragma unroll
        for (int o = 0; o < S; ++o) wd[k][o] = wk[k][o] * off[k][o];
    float vc[D];
    bool wall = false;
    // x and y components in packed FP32, z in scalar (3D). Whole steps: 1.65M particles
    // 324 -> 309 us, 3.8M 785 -> 766, quadratic 1.65M 271 -> 265, 2D 627k 62.0 -> 61.3
    const float2 zero = make_float2(0.f, 0.f);
    float2 v2 = zero, b2[3] = {zero, zero, zero}, c2 = zero;  // v; B's columns; 2D: vc
    float v1 = 0.f, b1[3] = {0.f, 0.f, 0.f};
#pragma unroll 1
    for (int a = 0; a < S; ++a) {
        float2 q2 = zero, qy2 = zero, qz2 = zero, qc2 = zero;
        float q1 = 0.f, qy1 = 0.f, qz1 = 0.f;
#pragma unroll
        for (int b = 0; b < S; ++b) {
            const float y1 = wk[1][b], yd1 = wd[1][b];
            const float2 y = make_float2(y1, y1), yd = make_float2(yd1, yd1);
            if constexpr (D == 3) {
                float2 p2 = zero, d2 = zero;
                float p1 = 0.f, d1 = 0.f;
#pragma unroll
                for (int c = 0; c < S; ++c) {
                    const I cid = c0 + a + b * sy + c * sz;
                    const float4 g = SMEM ? nodes[cid] : __ldg(&nodes[cid]);
                    wall = wall || g.w != 0.f;
                    const float z = wk[2][c], zd = wd[2][c];
                    p2 = __ffma2_rn(make_float2(z, z), make_float2(g.x, g.y), p2);
                    d2 = __ffma2_rn(make_float2(zd, zd), make_float2(g.x, g.y), d2);
                    p1 += z * g.z;
                    d1 += zd * g.z;
                }
                q2 = __ffma2_rn(y, p2, q2);
                qy2 = __ffma2_rn(yd, p2, qy2);
                qz2 = __ffma2_rn(y, d2, qz2);
                q1 += y1 * p1;
                qy1 += yd1 * p1;
                qz1 += y1 * d1;
            } else {
                const I cid = c0 + a + b * sy;
                const float4 g = SMEM ? nodes[cid] : __ldg(&nodes[cid]);
                q2 = __ffma2_rn(y, make_float2(g.x, g.y), q2);
                qy2 = __ffma2_rn(yd, make_float2(g.x, g.y), qy2);
                qc2 = __ffma2_rn(y, make_float2(g.z, g.w), qc2);
            }
        }
        const float x1 = pick<S>(wk[0], a), xd1 = pick<S>(wd[0], a);
        const float2 x = make_float2(x1, x1), xd = make_float2(xd1, xd1);
        v2 = __ffma2_rn(x, q2, v2);
        b2[0] = __ffma2_rn(xd, q2, b2[0]);
        b2[1] = __ffma2_rn(x, qy2, b2[1]);
        if constexpr (D == 3) {
            b2[2] = __ffma2_rn(x, qz2, b2[2]);
            v1 += x1 * q1;
            b1[0] += xd1 * q1;
            b1[1] += x1 * qy1;
            b1[2] += x1 * qz1;
        } else {
            c2 = __ffma2_rn(x, qc2, c2);
        }
    }
    nv[0] = v2.x;
    nv[1] = v2.y;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        nB[k] = b2[k].x;
        nB[D + k] = b2[k].y;
        if (D == 3) nB[2 * D + k] = b1[k];
    }
    vc[0] = c2.x;
    vc[1] = c2.y;
    if constexpr (D == 3) {
        nv[2] = v1;
        vc[2] = 0.f;
    }
    if constexpr (D == 3) {
        if (!wall) {
#pragma unroll
            for (int r = 0; r < 3; ++r) vc[r] = nv[r];
        } else {
#pragma unroll 1
            for (int a = 0; a < S; ++a) {
                float Qc[3] = {0.f, 0.f, 0.f};
#pragma unroll
                for (int b = 0; b < S; ++b) {
                    float Pc[3] = {0.f, 0.f, 0.f};
#pragma unroll
                    for (int c = 0; c < S; ++c) {
                        const I cid = c0 + a + b * sy + c * sz;
                        float4 g = SMEM ? nodes[cid] : __ldg(&nodes[cid]);
                        if (g.w != 0.f) {
                            if (SMEM && walls) g = walls[cid];
                            else g = __ldg(&gv[C.nodes + gc0 + a + b * gsy + c * gsz]);
                        }
                        const float z = wk[2][c];
                        Pc[0] += z * g.x; Pc[1] += z * g.y; Pc[2] += z * g.z;
                    }
                    const float y = wk[1][b];
#pragma unroll
                    for (int r = 0; r < 3; ++r) Qc[r] += y * Pc[r];
                }
                const float x = pick<S>(wk[0], a);
#pragma unroll
                for (int r = 0; r < 3; ++r) vc[r] += x * Qc[r];
            }
        }
    }
    float sw[3], swd[3];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        sw[k] = sum_s<S>(wk[k]);
        swd[k] = sum_s<S>(wd[k]);
    }
#pragma unroll
    for (int r = 0; r < D; ++r) {
        float t = swd[r];
#pragma unroll
        for (int l = 0; l < D; ++l)
            if (l != r) t *= sw[l];
        nx[r] = t + C.dt * vc[r];
    }
}

// ---------------------------------------------------------------------------
// P2G of one warp's window of 32 slots.
//
// The window's particles are ordered by stencil (lowest node id first) in the
// warp's shared memory; the warp then walks that order as a whole. Every lane
// owns one node column of the stencil (3D: offsets (b, c) in y and z; 2D: offset
// b in y and one channel pair) and holds the column's S nodes in x in registers;
// the warp sums G particles at a time. Cells are sorted x fastest, so the next
// stencil is mostly one node further in x: then only the node plane that falls
// out of the stencil is added to the grid, and the others go on accumulating.
//
// Bound: the shared-memory and reduction pipe (a 16-byte shared load costs 2.7
// cycles whether its lanes read one row or four, a red.global 20 to 26) and
// instruction issue. The former layout (SPLIT lanes per run of one stencil, each
// holding 8 nodes x 4 channels, every run adding all S^D nodes) sent 2.5 times
// the int64 adds and let lanes wait for the longest run.
//
// Payload of one particle (floats):
//   wx[4] | per b: wy yd | 3D, per c: wz zd | 3D: s0 s1 m s2, A00 A10 0 A20,
//   A01 A11 0 A21, A02 A12 0 A22; 2D: s0 s1 A00 A10, m 0 0 0, A01 A11, 0 0
// and after the rows, for the first row of each stencil: key, particles sharing it;
// with yd = wy (b - 1 - fy), zd = wz (c - 1 - fz), s_r = m v_r - fx A_r0 and
// f = x - (base + 1). The rows are 36 (2D 44) floats apart: 16-byte accesses of eight
// neighbouring rows then fall into distinct banks.
template <int D, int S> struct Scatter {
    static constexpr int PS = FusedGeom<D>::PS;            // floats per row
    static constexpr int Y = 4, Z = 12, M = D == 3 ? 20 : 12;
    static constexpr int INFO = FusedGeom<D>::WIN * PS;    // the stencils: key, count of each row
    // particles at a time (lanes of one: 3D 16, its 4 x 4 node columns, of which
    // the quadratic stencil uses 3 x 3; 2D 8, four columns times two channel
    // pairs) and channel pairs per lane
    static constexpr int G = D == 3 ? 2 : 4, PAIRS = D == 3 ? 2 : 1;
};

// Stencil keys: the node id of the stencil's first node (node ids stay below
// 2e9, validate_params); kClipped when part of the stencil is outside the grid
// (scatter_clipped does those); kNoKey for a lane with no row.
constexpr int kNoKey = -1, kClipped = 0x7fffffff;

template <int D, int S>
__device__ __forceinline__ int stencil_key(const StepConsts& C, const float* x, int* base) {
    bool interior = true;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const int ext = k == 0 ? C.W : (k == 1 ? C.H : C.Dp);
        base[k] = Stencil<S>::base(x[k], ext);
        interior = interior && base[k] >= 0 && base[k] + (S - 1) <= ext;
    }
    if (!interior) return kClipped;
    return ((D == 3 ? base[2] * C.ny : 0) + base[1]) * C.nx + base[0];
}

// Row of this lane's particle in the window's order, and the number of
// particles sharing its stencil; `total` gets the window's particle count.
// Whole warp.
__device__ __forceinline__ int window_row(int key, int* count, bool* first, int* total) {
    const int lane = threadIdx.x & 31;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const unsigned before = peers & ((1u << lane) - 1);
    *first = key != kNoKey && before == 0u;
    *count = __popc(peers);
    *total = __popc(__ballot_sync(0xffffffffu, key != kNoKey));
    int row = __popc(before);
    for (unsigned m = __ballot_sync(0xffffffffu, *first); m; m &= m - 1) {
        const int l = __ffs(m) - 1;
        const int kl = __shfl_sync(0xffffffffu, key, l), cl = __shfl_sync(0xffffffffu, *count, l);
        row += kl < key ? cl : 0;
    }
    return row;
}

template <int D, int S>
__device__ __forceinline__ void write_payload(const StepConsts& C, const float* x, const int* base, const float* v,
                                              const float* A, float mass, int key, int count, bool first, float* pay, int row, bool every = false) {
    using L = Scatter<D, S>;
    float f[3], w[3][4];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        w[k][3] = 0.f;
        Stencil<S>::weights(x[k], base[k], w[k]);
        f[k] = x[k] - float(base[k] + 1);
    }
    float4* q4 = reinterpret_cast<float4*>(pay + row * L::PS);
    q4[0] = make_float4(w[0][0], w[0][1], w[0][2], w[0][3]);
#pragma unroll
    for (int o = 0; o < S; o += 2) {
        q4[(L::Y + 2 * o) / 4] = make_float4(w[1][o], w[1][o] * (float(o - 1) - f[1]), w[1][o + 1],
                                             w[1][o + 1] * (float(o) - f[1]));
        if constexpr (D == 3)
            q4[(L::Z + 2 * o) / 4] = make_float4(w[2][o], w[2][o] * (float(o - 1) - f[2]), w[2][o + 1],
                                                 w[2][o + 1] * (float(o) - f[2]));
    }
    const float s0 = mass * v[0] - f[0] * A[0], s1 = mass * v[1] - f[0] * A[D];
    if constexpr (D == 3) {
        q4[L::M / 4] = make_float4(s0, s1, mass, mass * v[2] - f[0] * A[6]);
        q4[L::M / 4 + 1] = make_float4(A[0], A[3], 0.f, A[6]);
        q4[L::M / 4 + 2] = make_float4(A[1], A[4], 0.f, A[7]);
        q4[L::M / 4 + 3] = make_float4(A[2], A[5], 0.f, A[8]);
    } else {
        q4[L::M / 4] = make_float4(s0, s1, A[0], A[2]);
        q4[L::M / 4 + 1] = make_float4(mass, 0.f, 0.f, 0.f);
        q4[L::M / 4 + 2] = make_float4(A[1], A[3], 0.f, 0.f);
    }
    if (first || every) *reinterpret_cast<int2*>(pay + L::INFO + 2 * row) = make_int2(key, count);
}

// One lane's share of a window: the S node planes of its column as channel
// pairs (momentum x, y; mass, momentum z), the largest scaled sum so far (range
// check) and where and how it adds to the grid.
// EXACT (batched scenes): every particle's contribution becomes int64 fixed point
// before it is summed, so that a node's sum depends neither on the order nor on
// the grouping of the particles. Each is checked by itself (as to_fixed does): one that
// is not a number raises MPM_FLAG_NAN_STATE and counts as 0. (100 steps of 256 scenes:
// 50.1 ms with the check, 48.9 with one for the range alone; comparing every value, 51.3.)
struct Fixed2 {
    long long x, y;
};

template <int D, int S, bool EXACT = false> struct ScatterLane {
    std::conditional_t<EXACT, Fixed2, float2> a[S][Scatter<D, S>::PAIRS];
    float top;               // EXACT: unused
    unsigned* status;        // EXACT
    unsigned long long* at;  // first node column and channel the lane adds to, at node 0
    int at2;                 // its second add, relative to the first
    float scale0, scale1;
    int b, c, h, g;          // column, channel pair (2D), particle group
    bool on, both;           // adds anything; its second sum too
};

// The lane's two sums of one node plane at `node` to the grid.
template <int D, int S, bool EXACT>
__device__ __forceinline__ void add_sums(ScatterLane<D, S, EXACT>& T, long long node, float2 v) {
    unsigned long long* p = T.at + node * 4;
    const float t0 = v.x * T.scale0, t1 = v.y * T.scale1;
    T.top = fmaxf(T.top, fmaxf(fabsf(t0), fabsf(t1)));
    red_scaled(p, t0);
    if (T.both) red_scaled(p + T.at2, t1);
}

template <int D, int S>
__device__ __forceinline__ void add_sums(ScatterLane<D, S, true>& T, long long node, Fixed2 v) {
    unsigned long long* p = T.at + node * 4;
    red_int(p, v.x);
    if (T.both) red_int(p + T.at2, v.y);
}

__device__ __forceinline__ Fixed2 shfl_xor2(Fixed2 v, int m) {
    return Fixed2{__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m)};
}
__device__ __forceinline__ float2 shfl_xor2(float2 v, int m) {
    return make_float2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}

// One node plane `v` (x = node's) to the grid.
template <int D, int S, bool EXACT, typename V>
__device__ __forceinline__ void add_plane(ScatterLane<D, S, EXACT>& T, long long node, const V* v) {
    if constexpr (D == 3) {
        // the two groups' sums, one channel pair left to each; then neighbouring
        // columns (b, b ^ 1) swap so that a lane holds one channel of both: each
        // add then covers whole 32-byte nodes (four lanes a node), which the memory
        // pipe takes in 19.7 cycles a warp against 25.7 for half nodes
        float2 keep = T.g ? v[1] : v[0];
        const float2 got = shfl_xor2(T.g ? v[0] : v[1], 16);
        keep.x += got.x;
        keep.y += got.y;
        const float other = __shfl_xor_sync(0xffffffffu, T.b & 1 ? keep.x : keep.y, 1);
        if (T.on) add_sums(T, node, T.b & 1 ? make_float2(other, keep.y) : make_float2(keep.x, other));
    } else {
        // the four groups' sums of one node
        V u = v[0];
        V got = shfl_xor2(u, 16);
        u.x += got.x;
        u.y += got.y;
        got = shfl_xor2(u, 8);
        u.x += got.x;
        u.y += got.y;
        if (T.on && T.g == 0) add_sums(T, node, u);
    }
}

// A stencil that starts `ahead` (1 .. S) nodes further in x: the planes before
// it go to the grid, the others move up.
template <int D, int S, bool EXACT>
__device__ __forceinline__ void move_planes(ScatterLane<D, S, EXACT>& T, long long node, int ahead) {
#pragma unroll 1
    for (int n = 0; n < ahead; ++n) {
        add_plane(T, node + n, T.a[0]);
#pragma unroll
        for (int p = 0; p < Scatter<D, S>::PAIRS; ++p) {
#pragma unroll
            for (int a = 0; a + 1 < S; ++a) T.a[a][p] = T.a[a + 1][p];
            T.a[S - 1][p] = {};
        }
    }
}

// 2D: all S planes to the grid; clears them. The four groups sum each others'
// planes and are left with one each. (3D adds them with move_planes: unrolled
// they cost more in instruction fetch than the register moves they save, 320
// -> 332 us on the 128^3 snowball scene.)
template <int D, int S, bool EXACT>
__device__ __forceinline__ void add_planes(ScatterLane<D, S, EXACT>& T, long long node) {
    if constexpr (D == 2) {
        using V = std::remove_reference_t<decltype(T.a[0][0])>;
        V v[4] = {}, k[2];
#pragma unroll
        for (int a = 0; a < S; ++a) v[a] = T.a[a][0];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            k[i] = T.g & 2 ? v[2 + i] : v[i];
            const V got = shfl_xor2(T.g & 2 ? v[i] : v[2 + i], 16);
            k[i].x += got.x;
            k[i].y += got.y;
        }
        V u = T.g & 1 ? k[1] : k[0];
        const V got = shfl_xor2(T.g & 1 ? k[0] : k[1], 8);
        u.x += got.x;
        u.y += got.y;
        if (T.on && T.g < S) add_sums(T, node + T.g, u);
#pragma unroll
        for (int a = 0; a < S; ++a) T.a[a][0] = {};
    }
}

// Adds one particle's plane values  wx_a (P + (a - 1) Q)  of a channel pair.
template <int D, int S>
__device__ __forceinline__ void sum_pair(ScatterLane<D, S, false>& T, int p, const float2* x, float2 P, float2 Q) {
    T.a[0][p] = __ffma2_rn(x[0], __fadd2_rn(P, make_float2(-Q.x, -Q.y)), T.a[0][p]);
    T.a[1][p] = __ffma2_rn(x[1], P, T.a[1][p]);
    P = __fadd2_rn(P, Q);
    T.a[2][p] = __ffma2_rn(x[2], P, T.a[2][p]);
    if constexpr (S == 4) T.a[3][p] = __ffma2_rn(x[3], __fadd2_rn(P, Q), T.a[3][p]);
}

// max(a, |b|, |c|), NaN if one of them is (fmaxf drops a NaN).
__device__ __forceinline__ float max_abs_nan(float a, float b, float c) {
    float d;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

template <int D, int S>
__device__ __forceinline__ void sum_pair(ScatterLane<D, S, true>& T, int p, const float2* x, float2 P, float2 Q) {
    const float2 scale = make_float2(T.scale0, T.scale1);
    P = __fmul2_rn(P, scale);  // powers of two: exact
    Q = __fmul2_rn(Q, scale);
    P = __fadd2_rn(P, make_float2(-Q.x, -Q.y));
    const float2 first = P;
    float top = 0.f;
#pragma unroll
    for (int a = 0; a < S; ++a) {
        const float2 t = __fmul2_rn(x[a], P);
        top = max_abs_nan(top, t.x, t.y);
        T.a[a][p].x += __float2ll_rn(t.x);
        T.a[a][p].y += __float2ll_rn(t.y);
        P = __fadd2_rn(P, Q);
    }
    if (__builtin_expect(!(top < kFixedLimit), 0)) {  // rare: to_fixed in place of the plain conversions
        P = first;
#pragma unroll
        for (int a = 0; a < S; ++a) {
            const float2 t = __fmul2_rn(x[a], P);
            T.a[a][p].x += to_fixed(t.x, 1.f, T.status) - __float2ll_rn(t.x);
            T.a[a][p].y += to_fixed(t.y, 1.f, T.status) - __float2ll_rn(t.y);
            P = __fadd2_rn(P, Q);
        }
    }
}

// The particle rows [0, count) at q, all of one stencil, into the planes.
// (row j = T.g, T.g + G, ... of them per lane.)
template <int D, int S, bool EXACT>
__device__ __forceinline__ void sum_rows(ScatterLane<D, S, EXACT>& T, const float* q, int count) {
    using L = Scatter<D, S>;
    constexpr int G = L::G;
    q += T.g * L::PS;
    for (int j = T.g; j < count; j += G, q += G * L::PS) {
        const float4* q4 = reinterpret_cast<const float4*>(q);
        const float4 w = q4[0];
        const float2 x[4] = {make_float2(w.x, w.x), make_float2(w.y, w.y), make_float2(w.z, w.z), make_float2(w.w, w.w)};
        const float2 wy = *reinterpret_cast<const float2*>(q + L::Y + 2 * T.b);
        if constexpr (D == 3) {
            const float2 wz = *reinterpret_cast<const float2*>(q + L::Z + 2 * T.c);
            const float yz_ = wy.x * wz.x, ydz_ = wy.y * wz.x, yzd_ = wy.x * wz.y;
            const float2 yz = make_float2(yz_, yz_), ydz = make_float2(ydz_, ydz_), yzd = make_float2(yzd_, yzd_);
            const float4 s = q4[L::M / 4], a0 = q4[L::M / 4 + 1], a1 = q4[L::M / 4 + 2], a2 = q4[L::M / 4 + 3];
            sum_pair(T, 0, x,
                           __ffma2_rn(yzd, make_float2(a2.x, a2.y),
                                      __ffma2_rn(ydz, make_float2(a1.x, a1.y), __fmul2_rn(yz, make_float2(s.x, s.y)))),
                           __fmul2_rn(yz, make_float2(a0.x, a0.y)));
            sum_pair(T, 1, x,
                           __ffma2_rn(yzd, make_float2(a2.z, a2.w),
                                      __ffma2_rn(ydz, make_float2(a1.z, a1.w), __fmul2_rn(yz, make_float2(s.z, s.w)))),
                           __fmul2_rn(yz, make_float2(a0.z, a0.w)));
        } else {
            const float4 sa = q4[L::M / 4 + T.h];
            const float2 a1 = *reinterpret_cast<const float2*>(q + L::M + 8 + 2 * T.h);
            const float2 y = make_float2(wy.x, wy.x), yd = make_float2(wy.y, wy.y);
            sum_pair(T, 0, x, __ffma2_rn(yd, a1, __fmul2_rn(y, make_float2(sa.x, sa.y))),
                               __fmul2_rn(y, make_float2(sa.z, sa.w)));
        }
    }
}

// P2G of a particle part of whose stencil is outside the grid, by one lane: its
// nodes inside the grid one by one, and their blocks.
template <int D, int S, bool EXACT>
__device__ __forceinline__ void scatter_clipped(const StepConsts& C, const TileInfo& TI, const float* x, const int* base,
                                                const float* v, const float* A, float mass,
                                                unsigned long long* __restrict__ acc, unsigned* __restrict__ status) {
    constexpr int TE = TileGeom<D>::T;
    float top = 0.f;
    auto add = [&](unsigned long long* p, float t) {
        if constexpr (EXACT) {
            red_int(p, to_fixed(t, 1.f, status));
        } else {
            red_scaled(p, t);
            top = fmaxf(top, fabsf(t));
        }
    };
#pragma unroll 1
    for (int j = 0; j < (D == 3 ? S * S * S : S * S); ++j) {
        const int gx = base[0] + j % S, gy = base[1] + (j / S) % S, gz = D == 3 ? base[2] + j / (S * S) : 0;
        if (gx < 0 || gx > C.W || gy < 0 || gy > C.H || (D == 3 && (gz < 0 || gz > C.Dp))) continue;
        const float d[3] = {float(gx) - x[0], float(gy) - x[1], D == 3 ? float(gz) - x[D - 1] : 0.f};
        float w = Stencil<S>::w(d[0]) * Stencil<S>::w(d[1]);
        if (D == 3) w *= Stencil<S>::w(d[2]);
        unsigned long long* n = acc + (((long long)gz * C.ny + gy) * C.nx + gx) * 4;
        add(n + 2, w * mass * C.sm);
#pragma unroll
        for (int r = 0; r < D; ++r) {
            float s = mass * v[r];
#pragma unroll
            for (int k = 0; k < D; ++k) s += A[r * D + k] * d[k];
            s *= w * C.sp;
            add(n + (r < 2 ? r : 3), s);
        }
        mark_block_once(TI, ((D == 3 ? gz / TE : 0) * TI.nblk[1] + gy / TE) * TI.nblk[0] + gx / TE);
    }
    raise_flag(status, top < kFixedLimit ? 4u : 4u | 2u);
}

// One lane's planes on the way to a stencil `ahead` nodes further (any other value: to
// another row): those it leaves go to the grid as they are, without the other groups'.
template <int S>
__device__ __forceinline__ void leave_planes(ScatterLane<2, S, true>& T, int node, int ahead) {
    const int n = ahead > 0 && ahead < S ? ahead : S;
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        if (T.on) add_sums(T, (long long)node + k, T.a[0][0]);
#pragma unroll
        for (int a = 0; a + 1 < S; ++a) T.a[a][0] = T.a[a + 1][0];
        T.a[S - 1][0] = {};
    }
}
// Particles a stencil from which the whole warp walks an EXACT window (scatter_rows):
// it adds each plane once, but takes 250 instructions a stencil, of which one with fewer
// than four particles leaves groups idle. Below, each group walks a quarter of the
// rows by itself, with the same sums. Whole steps, never and always by groups: 1 a cell, 105k
// particles in 256 scenes 58, 44 us; 4 a cell, 7.4M 1376, 1062; 8 a cell, 1.5M 220, 203; 64 a cell, 8.1M 936, 997.
constexpr int kSharedStencil = 16;

// The ordered rows of a window (`total` of them, of so many stencils) into the grid. Whole
// warp.
template <int D, int S, bool EXACT = false>
__device__ __forceinline__ void scatter_rows(const StepConsts& C, const float* pay, int total, [[maybe_unused]] int stencils,
                                             unsigned long long* __restrict__ acc, unsigned* __restrict__ status) {
    using L = Scatter<D, S>;
    const int lane = threadIdx.x & 31;
    ScatterLane<D, S, EXACT> T;
    int col = 0, ch = 0;  // of the lane's first add
    T.b = lane & 3;
    if constexpr (D == 3) {
        T.c = (lane >> 2) & 3;
        T.g = lane >> 4;
        T.h = 0;
        T.on = T.c < S;
        // one channel of columns b & ~1 and b | 1 (add_plane)
        ch = 2 * T.g + (T.b & 1);
        col = T.c * C.ny + (T.b & 2);
        T.at2 = 4 * C.nx;
        T.both = (T.b | 1) < S;
        T.scale0 = T.scale1 = ch == 2 ? C.sm : C.sp;
    } else {
        T.c = 0;
        T.h = (lane >> 2) & 1;
        T.g = lane >> 3;
        T.on = T.b < S;
        ch = 2 * T.h;
        col = T.b;
        T.at2 = 1;
        T.both = T.h == 0;
        T.scale0 = T.h == 0 ? C.sp : C.sm;
        T.scale1 = C.sp;
    }
    T.top = 0.f;
    T.status = status;
    T.at = acc + (long long)col * C.nx * 4 + ch;
#pragma unroll
    for (int a = 0; a < S; ++a)
#pragma unroll
        for (int p = 0; p < L::PAIRS; ++p) T.a[a][p] = {};
    int at = kNoKey;  // first node of the planes
    if constexpr (D == 2 && EXACT) {
        if (total < kSharedStencil * stencils) {
            // few particles share a stencil: each group walks a quarter of the rows by itself
            const int end = total * (T.g + 1) / 4;
            const int own = T.g;
            T.g = 0;
            for (int j = total * own / 4; j < end; ++j) {
                const int key = *reinterpret_cast<const int*>(pay + L::INFO + 2 * j);
                if (key != at) {
                    if (at != kNoKey) leave_planes(T, at, key - at);
                    at = key;
                }
                sum_rows(T, pay + j * L::PS, 1);
            }
            if (at != kNoKey) leave_planes(T, at, S);
            __syncwarp();  // the rows are reused by the next window
            return;
        }
    }
    for (int j = 0; j <= total;) {
        const int2 info = j < total ? *reinterpret_cast<const int2*>(pay + L::INFO + 2 * j) : make_int2(kNoKey, 1);
        // stencils in the grid whose node ids differ by less than S are in one row
        const int ahead = info.x - at;
        if (at != kNoKey) {
            if constexpr (D == 3) {
                move_planes(T, at, ahead > 0 ? min(ahead, S) : S);
            } else {
                if (ahead > 0 && ahead < S) move_planes(T, at, ahead);
                else add_planes(T, at);
            }
        }
        at = info.x;
        if (j < total) {
            sum_rows(T, pay + j * L::PS, info.y);
            __syncwarp();
        }
        j += info.y;
    }
    if (!(T.top < kFixedLimit)) raise_flag(status, 2u);
    __syncwarp();  // the rows are reused by the next window
}

// Marks the node blocks of a stencil (all of it in the grid).
template <int D, int S>
__device__ __forceinline__ void mark_stencil(const TileInfo& TI, const int* base) {
    constexpr int TE = TileGeom<D>::T;
    const int x0 = base[0] / TE, x1 = (base[0] + S - 1) / TE, y0 = base[1] / TE, y1 = (base[1] + S - 1) / TE;
    const int z0 = D == 3 ? base[2] / TE : 0, z1 = D == 3 ? (base[2] + S - 1) / TE : 0;
    for (int bz = z0; bz <= z1; ++bz)
        for (int by = y0; by <= y1; ++by)
            for (int bx = x0; bx <= x1; ++bx) mark_block_once(TI, (bz * TI.nblk[1] + by) * TI.nblk[0] + bx);
}

// The same of a stencil partly outside the grid: the blocks of its nodes in the grid.
template <int D, int S>
__device__ __forceinline__ void mark_clipped(const StepConsts& C, const TileInfo& TI, const int* base) {
    constexpr int TE = TileGeom<D>::T;
    int b0[3] = {0, 0, 0}, b1[3] = {0, 0, 0};
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const int ext = k == 0 ? C.W : (k == 1 ? C.H : C.Dp);
        const int lo = max(base[k], 0), hi = min(base[k] + S - 1, ext);
        if (lo > hi) return;
        b0[k] = lo / TE;
        b1[k] = hi / TE;
    }
    for (int bz = b0[2]; bz <= b1[2]; ++bz)
        for (int by = b0[1]; by <= b1[1]; ++by)
            for (int bx = b0[0]; bx <= b1[0]; ++bx) mark_block_once(TI, (bz * TI.nblk[1] + by) * TI.nblk[0] + bx);
}

// The node blocks of a stencil as bits of the 3^D blocks around the tile whose
// node box starts at bo (2 nodes before the tile); the stencil lies in the box.
template <int D, int S>
__device__ __forceinline__ unsigned stencil_block_bits(const int* base, const int* bo) {
    constexpr int TE = TileGeom<D>::T;
    unsigned m[3] = {1u, 1u, 1u};
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const int r = base[k] - bo[k] + TE - 2;  // from the first node of the block before the tile
        m[k] = (1u << (r / TE)) | (1u << ((r + S - 1) / TE));
    }
    unsigned bits = m[0] * ((m[1] & 1u) | (m[1] & 2u) << 2 | (m[1] & 4u) << 4);
    if constexpr (D == 3) bits *= (m[2] & 1u) | (m[2] & 2u) << 8 | (m[2] & 4u) << 16;
    return bits;
}

// P2G of the particles left over of one recorded window (rec: first slot, mask of
// the lanes, mask of those whose node blocks are not marked yet) after the return
// map, by one warp: x, v, A as the G2P and return-map kernels left them,
// scattered as in the fused kernel. The order inside a window is a function of its
// queued particles, so the int64 sums do not depend on the order in which windows
// were recorded. The fused kernel has marked the node blocks of every queued
// particle whose new position it knew; the others are marked here.
template <int D, int S, bool EXACT>
__device__ __forceinline__ void queued_window(const Particles& P, const StepConsts& C, const TileInfo& TI, int4 rec,
                                              unsigned long long* __restrict__ acc, unsigned* __restrict__ status,
                                              float* pay) {
    using L = Scatter<D, S>;
    const int lane = threadIdx.x & 31;
    const long long n = P.n;
    const bool queued = ((unsigned)rec.y >> lane) & 1u, unmarked = ((unsigned)rec.z >> lane) & 1u;
    int key = kNoKey, base[3] = {0, 0, 0};
    float mass = 0.f, x[D], v[D], A[D * D];
    if (queued) {
        const int i = rec.x + lane;
        mass = P.mass ? P.mass[i] : P.mass_u;
#pragma unroll
        for (int k = 0; k < D; ++k) { x[k] = P.x[k * n + i]; v[k] = P.v[k * n + i]; }
#pragma unroll
        for (int k = 0; k < D * D; ++k) A[k] = P.A[k * n + i];
        key = stencil_key<D, S>(C, x, base);
        if (key == kClipped) {
            scatter_clipped<D, S, EXACT>(C, TI, x, base, v, A, mass, acc, status);
            key = kNoKey;
        } else if (unmarked) {
            mark_stencil<D, S>(TI, base);
        }
    }
    if constexpr (EXACT) {
        if (unmarked && !queued) {  // no volume: reads the grid next step, adds nothing
#pragma unroll
            for (int k = 0; k < D; ++k) x[k] = P.x[k * n + rec.x + lane];
            if (stencil_key<D, S>(C, x, base) == kClipped) mark_clipped<D, S>(C, TI, base);
            else mark_stencil<D, S>(TI, base);
        }
    }
    int count, total;
    bool first;
    const int row = window_row(key, &count, &first, &total);
    if (key != kNoKey) write_payload<D, S>(C, x, base, v, A, mass, key, count, first, pay, row, EXACT);
    __syncwarp();
    const int stencils = EXACT ? __popc(__ballot_sync(0xffffffffu, first)) : 0;
    scatter_rows<D, S, EXACT>(C, pay, total, stencils, acc, status);
}

template <int D, int S>
__global__ void __launch_bounds__(FusedGeom<D>::THREADS) k_p2g_windows(Particles P, StepConsts C, TileInfo TI,
                                                                      SlowQueue Q,
                                                                      unsigned long long* __restrict__ acc,
                                                                      unsigned* __restrict__ status) {
    using G = FusedGeom<D>;
    extern __shared__ __align__(128) unsigned char fused_smem[];
    const int wid = threadIdx.x >> 5;
    float* pay = reinterpret_cast<float*>(fused_smem) + wid * G::PAY;
    chain_wait();
    const int nw = min(*Q.nwin, Q.win_capacity);
    for (int r = blockIdx.x * G::WARPS + wid; r < nw; r += gridDim.x * G::WARPS)
        queued_window<D, S, false>(P, C, TI, Q.win[r], acc, status, pay);
}

// ---------------------------------------------------------------------------
// TMA load of a tile's node box and its mbarrier (sm_90+ PTX): each CTA loads
// its own boxes from this GPU's memory.
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Orders this thread's earlier generic-proxy accesses of shared memory before
// later async-proxy (TMA) writes to it.
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Waits for the phase `parity` of the mbarrier to complete; false after
// `limit` polls (each poll may suspend the thread for a short while).
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, int limit) {
    const uint32_t a = smem_u32(bar);
    for (int it = 0; it < limit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
constexpr int kBoxWaitPolls = 1 << 20;

// One arrival on the mbarrier (release at CTA scope).
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_expect(unsigned long long* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// The node box with origin node bo into `dst`: one tensor load of the node
// velocities viewed as [2][nz][ny][nx][4] floats (3D; `half` 1: the wall velocities)
// or [ny][nx][4]; nodes outside the grid read as zero.
template <int D>
__device__ __forceinline__ void box_load(const CUtensorMap& map, const int* bo, int half, float4* dst,
                                         unsigned long long* bar) {
    const uint32_t b = smem_u32(bar), d = smem_u32(dst);
    if constexpr (D == 3) {
        asm volatile(
            "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], "
            "[%7];" ::"r"(d), "l"(reinterpret_cast<uint64_t>(&map)), "r"(0), "r"(bo[0]), "r"(bo[1]), "r"(bo[2]), "r"(half),
            "r"(b)
            : "memory");
    } else {
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
            ::"r"(d), "l"(reinterpret_cast<uint64_t>(&map)), "r"(0), "r"(bo[0]), "r"(bo[1]), "r"(b)
            : "memory");
    }
}

// Tile coordinates and box origin node of tile t.
template <int D>
__device__ __forceinline__ void tile_origin(const TileInfo& TI, int t, int* tc, int* bo) {
#pragma unroll
    for (int k = 0; k < D; ++k) { tc[k] = t % TI.tiles[k]; t /= TI.tiles[k]; bo[k] = tc[k] * FusedGeom<D>::T - 2; }
}

// Marks the node blocks given by the warp's bits (stencil_block_bits) around a tile.
template <int D>
__device__ __forceinline__ void mark_tile_blocks(const TileInfo& TI, const int* tc, unsigned bits) {
    const int lane = threadIdx.x & 31;
    if (lane < (D == 3 ? 27 : 9) && (bits >> lane) & 1u) {
        const int bx = tc[0] - 1 + lane % 3, by = tc[1] - 1 + (lane / 3) % 3, bz = D == 3 ? tc[2] - 1 + lane / 9 : 0;
        mark_block_once(TI, (bz * TI.nblk[1] + by) * TI.nblk[0] + bx);
    }
}

// ---------------------------------------------------------------------------
// Window w (slots start + win w ...) of an item of m slots, by one warp: G2P of
// each slot's particle against the tile's node box (G2P = true) or the stored
// state (G2P = false), then the scatter of the in-band particles' payloads.
// Returns this lane's node-block bits around the tile (box origin bo). DIRECT:
// there is no staged box, every particle gathers from the global grid. EXACT: blocks
// are also marked for particles without volume, which add nothing but read them next
// step; a block that the grid update does not come to keeps old velocities.
template <int D, int S, bool G2P, bool DIRECT = false, bool EXACT = false>
__device__ __forceinline__ unsigned fused_window(const Particles& P, const StepConsts& C, const TileInfo& TI,
                                                 const float4* __restrict__ gv, unsigned long long* __restrict__ acc,
                                                 const SlowQueue& Q, unsigned* __restrict__ status, const float4* box,
                                                 const float4* walls, const int* bo, int start, int m, int win, int w, float* pay) {
    using G = FusedGeom<D>;
    using L = Scatter<D, S>;
    using St = Stencil<S>;
    const int lane = threadIdx.x & 31;
    const long long n = P.n;
    const long long gsy = C.nx, gsz = (long long)C.nx * C.ny;
    const int cnt = min(win, m - w * win);
    const bool valid = lane < cnt;
    const int i = start + w * win + lane;
    int key = kNoKey, nbase[3] = {0, 0, 0};
    bool deferred = false;   // queued: scattered after the return map (k_p2g_windows)
    bool unmarked = false;   // queued with its whole G2P: new position not known here (EXACT: also without volume)
    unsigned bits = 0u;
    float mass = 0.f, x[D], v[D], A[D * D];
    if (valid) {
        const float vol = P.vol ? P.vol[i] : P.vol_u;
        mass = P.mass ? P.mass[i] : P.mass_u;
        bool scatter = vol != 0.f;  // p2g.glsl:42
        if constexpr (G2P) {
            float xo[D];
#pragma unroll
            for (int k = 0; k < D; ++k) xo[k] = P.x[k * n + i];
            int base[3] = {0, 0, 0};
            float wk[3][S], off[3][S];
            bool interior = true, boxed = true;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const int ext = k == 0 ? C.W : (k == 1 ? C.H : C.Dp);
                base[k] = St::base(xo[k], ext);
                interior = interior && base[k] >= 0 && base[k] + (S - 1) <= ext;
                boxed = boxed && base[k] - bo[k] >= 0 && base[k] + (S - 1) - bo[k] <= G::BE - 1;
                St::weights(xo[k], base[k], wk[k]);
#pragma unroll
                for (int o = 0; o < S; ++o) off[k][o] = float(base[k] + o) - xo[k];
            }
            if (!interior) {
                // stencil partly outside the grid: the general kernel does the whole G2P
                Q.list[queue_slot(Q)] = -1 - i;
                deferred = scatter;
                unmarked = EXACT || scatter;
                scatter = false;
            } else {
                float nv[D], nx[D], nB[D * D];
                const long long gc0 = (D == 3 ? base[2] * gsz : 0) + base[1] * gsy + base[0];
                if (!DIRECT && boxed) {
                    const int l0 = (D == 3 ? (base[2] - bo[2]) * G::BE * G::BE : 0) + (base[1] - bo[1]) * G::BE +
                                   (base[0] - bo[0]);
                    gather_nodes<D, S, true, int>(C, box, l0, G::BE, G::BE * G::BE, gv, walls, gc0, gsy, gsz, wk, off,
                                                  nv, nB, nx);
                } else {
                    gather_nodes<D, S, false, long long>(C, gv, gc0, gsy, gsz, gv, nullptr, gc0, gsy, gsz, wk, off, nv, nB,
                                                         nx);
                }
                bool finite = true;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    x[k] = xo[k] + nx[k];
                    v[k] = nv[k];
                    P.v[k * n + i] = nv[k];
                    P.x[k * n + i] = x[k];
                    finite = finite && isfinite(x[k]);
                }
                if (!finite) raise_flag(status, 1u);
#pragma unroll
                for (int k = 0; k < D * D; ++k) P.B[k * n + i] = nB[k];
                float Fe[D * D], Fh[D * D];
#pragma unroll
                for (int k = 0; k < D * D; ++k) Fe[k] = P.Fe[k * n + i];
#pragma unroll
                for (int r = 0; r < D; ++r)
#pragma unroll
                    for (int c = 0; c < D; ++c) {
                        float s = Fe[r * D + c];
#pragma unroll
                        for (int k = 0; k < D; ++k) s += (C.dt * St::DINV * nB[r * D + k]) * Fe[k * D + c];
                        Fh[r * D + c] = s;
                    }
                const float Jp = P.Jp[i];
                bool band = det<D>(Fh) > 0.f && band_gershgorin<D>(Fh, 1.f - C.theta_c, 1.f + C.theta_s);
                if constexpr (D == 2) {
                    band = band && affine2<S>(C, Fh, Jp, nB, mass, vol, A);
                } else {
                    float sig[D * D];
                    band = band && hardened_stress_series<D>(Fh, Jp, C.mu0, C.la0, C.xi, sig);
                    if (band)
#pragma unroll
                        for (int k = 0; k < D * D; ++k)
                            A[k] = St::DINV * mass * nB[k] - St::DINV * C.dt * vol * sig[k];
                }
                if (band) {
#pragma unroll
                    for (int k = 0; k < D * D; ++k) P.Fe[k * n + i] = Fh[k];
                } else {
                    const int slot = queue_slot(Q);
                    Q.list[slot] = i;
#pragma unroll
                    for (int k = 0; k < D * D; ++k) Q.fh[k * Q.capacity + slot] = Fh[k];
                    deferred = scatter;
                    scatter = false;
                }
            }
        } else {
            float B[D * D], Fe[D * D];
#pragma unroll
            for (int k = 0; k < D; ++k) { x[k] = P.x[k * n + i]; v[k] = P.v[k * n + i]; }
#pragma unroll
            for (int k = 0; k < D * D; ++k) { B[k] = P.B[k * n + i]; Fe[k] = P.Fe[k * n + i]; }
            mls_affine<D, S>(C, B, Fe, P.Jp[i], mass, vol, A);
        }
        // the new stencil, and its node blocks (of queued particles too: their
        // return map leaves the position alone)
        if (EXACT ? !unmarked : scatter || (deferred && !unmarked)) {
            const int k = stencil_key<D, S>(C, x, nbase);
            if (k != kClipped) {
                bool boxed = true;
#pragma unroll
                for (int d = 0; d < D; ++d)
                    boxed = boxed && nbase[d] - bo[d] >= 0 && nbase[d] + (S - 1) - bo[d] <= G::BE - 1;
                if (boxed) bits = stencil_block_bits<D, S>(nbase, bo);
                else mark_stencil<D, S>(TI, nbase);
                if (scatter) key = k;
            } else if (scatter) {
                scatter_clipped<D, S, EXACT>(C, TI, x, nbase, v, A, mass, acc, status);
            } else if (EXACT && !deferred) {
                mark_clipped<D, S>(C, TI, nbase);
            }
        }
    }
    if constexpr (G2P) {
        // A window some of whose particles wait for the return map is recorded. In 3D
        // and in batches it is put off as a whole: scattered twice, it would add its
        // node planes twice, which costs more than handing the other particles' A on
        // through memory (3.8M particles in collision, a third of them queued: 462 us
        // here and 327 in k_p2g_windows, put off 302 and 334; 2.8M in 256 2D scenes
        // 331 + 19.3, 327 + 18.5). A single 2D scene queues a few windows and waits
        // for the longest of them: 22.3 + 3.4 us at 186k particles, put off 21.9 + 6.0.
        constexpr bool PUT_OFF = D == 3 || EXACT;
        if (__builtin_expect(__any_sync(0xffffffffu, deferred || unmarked), 0)) {
            const unsigned rows = __ballot_sync(0xffffffffu, deferred || (PUT_OFF && key != kNoKey));
            const unsigned um = __ballot_sync(0xffffffffu, unmarked);
            if (PUT_OFF && key != kNoKey) {
#pragma unroll
                for (int k = 0; k < D * D; ++k) P.A[k * n + i] = A[k];
            }
            if (lane == 0) {
                const int r = atomicAdd(Q.nwin, 1);
                if (r < Q.win_capacity) Q.win[r] = make_int4(start + w * win, (int)rows, (int)um, Q.scene);
            }
            if (PUT_OFF) return bits;
        }
    }
    int count, total;
    bool first;
    const int row = window_row(key, &count, &first, &total);
    if (key != kNoKey) write_payload<D, S>(C, x, nbase, v, A, mass, key, count, first, pay, row, EXACT);
    __syncwarp();
    const int stencils = EXACT ? __popc(__ballot_sync(0xffffffffu, first)) : 0;
    scatter_rows<D, S, EXACT>(C, pay, total, stencils, acc, status);
    return bits;
}

// ---------------------------------------------------------------------------
// The fused step without staged boxes: an item is one window, every warp takes
// windows on its own and gathers from the global grid. A staged box is worth its round
// trip to L2 only where many windows read it and there are tiles enough for every CTA
// (the dispatch's rule: windows per warp of the GPU, particles per cell). Whole steps in
// us, direct and staged:
//   3D cubic, 8 a cell, windows per warp 2.0: 73, 70;  5.0: 125, 113;  17: 384, 309
//     3 a cell, 3.7: 123, 124;  23: 639, 568;   2 a cell, 4.3: 159, 176;  72: 2080, 2250
//     1 a cell, 5.0: 237, 328;  70: 2710, 4080;  0.6 a cell, 17.6k particles (fused kernel): 17.5, 23.0
//   3D quadratic, 8 a cell, 9.8: 164, 165;  17: 273, 266;  60: 853, 784
//     4 to 6 a cell, 13: 219, 234;  45: 694, 662;  73: 1251, 1252;   1 a cell, 18: 593, 1166
//   2D, 4 to 8 a cell, windows per warp 7.8: 83, 84;  16: 182, 176;  34: 376, 350
//     27 a cell, 6.6: 62, 69;  64 a cell, 16: 233, 228;  63: 764, 686
//     2 a cell, 7.8: 128, 158;  31: 461, 574
//
// G2P = false: the P2G of the stored state only (after creation or a state upload),
// reading B, F_E, J_p and forming A as every other path does (mls_affine), for items
// of any length.
template <int D, int S, bool G2P>
__global__ void __launch_bounds__(FusedGeom<D>::THREADS, MPM_FUSED_MIN_BLOCKS)
    k_g2p2g_direct(Particles P, StepConsts C, TileInfo TI, const float4* __restrict__ gv,
                   unsigned long long* __restrict__ acc, SlowQueue Q, unsigned* __restrict__ status) {
    using G = FusedGeom<D>;
    extern __shared__ __align__(128) unsigned char fused_smem[];
    const int wid = threadIdx.x >> 5;
    float* pay = reinterpret_cast<float*>(fused_smem) + wid * G::PAY;
    chain_wait();
    const int nitems = *TI.n_items;
    for (int e = wid * gridDim.x + blockIdx.x; e < nitems; e += G::WARPS * gridDim.x) {
        const int4 item = TI.items[e];  // tile, first slot, slots
        int tc[3] = {0, 0, 0}, bo[3] = {0, 0, 0};
        tile_origin<D>(TI, item.x, tc, bo);
        const int nwin = G2P ? 1 : (item.z + TI.win - 1) / TI.win;
        unsigned bits = 0u;
        for (int w = 0; w < nwin; ++w)
            bits |= fused_window<D, S, G2P, true>(P, C, TI, gv, acc, Q, status, nullptr, nullptr, bo, item.y, item.z,
                                                  TI.win, w, pay);
        mark_tile_blocks<D>(TI, tc, __reduce_or_sync(0xffffffffu, bits));
    }
}

// ---------------------------------------------------------------------------
// The fused step with staged node boxes: persistent CTAs, each a pipeline of
// items. Stage k (item k of the CTA) lives in buffer k % STAGES: its item, its
// box of node velocities and, where the tile is near the domain's walls, the box of
// wall velocities (TMA tensor loads, whose mbarrier `full` completes when the bytes
// have landed), a window counter, a count of the warps that have left it, and its
// node-block bits. Each warp waits for the stage's box, takes windows of the item
// until none are left, and moves on to stage k + 1, which is already loaded; the
// last warp to leave stage k marks the tile's node blocks and refills the buffer
// with stage k + STAGES (the next item from the global counter, or an empty stage
// that ends the CTA). A warp is thus held up only by a box that has not arrived,
// never by the other warps' windows. Stages are refilled in order (a warp that
// refills stage k has not left stage k + 1 yet), so item numbers grow with the stage
// and the first empty stage ends the work for every warp. Every wait is bounded: a
// box that does not arrive raises MPM_FLAG_TIMEOUT.
//
// Bound: instruction issue and the shared-memory pipe at 20 warps per SM (96
// registers). 1.65M particles, snowball above a slab on the floor: 308 us with one
// buffer per CTA of 4 warps, filled by the CTA between two barriers (the kernel this
// one replaces), 300 with this one (286 since the gather is in packed FP32), of which the wall boxes give 13 (particles near a wall
// otherwise read vc from L2 node by node); 3.8M in collision: 537 and 502. One CTA
// of 20 warps and 4 stages: 303 and 518 (all warps of an SM then add to the same
// nodes); 4 CTAs of 5 warps, which leave no room for wall boxes: 318 and 490.
template <int D> struct PipeGeom {
    static constexpr int STAGES = 2, WARPS = 10, CTAS = 2, THREADS = 32 * WARPS;
};

template <int D> struct PipeSmem {
    using G = FusedGeom<D>;
    using R = PipeGeom<D>;
    alignas(128) float4 box[R::STAGES][G::BNP];                             // 3D: (vf, wall flag); 2D: (vf, vc)
    alignas(128) float4 wall[D == 3 ? R::STAGES : 1][D == 3 ? G::BNP : 8];  // 3D: vc of the flagged nodes
    unsigned long long full[R::STAGES];                                     // the stage's boxes arrived (or it is empty)
    int4 item[R::STAGES];                                                   // tile, first slot, slots (0: empty), near a wall
    int next_win[R::STAGES];
    int left[R::STAGES];                                                    // warps done with the stage
    unsigned bmask[R::STAGES];
    float4 pay[R::WARPS][G::PAY / 4];
};

// Stage for buffer b: item e, its box loads and its particles' G2P inputs (x, F_E,
// J_p) towards L2, or an empty stage. One warp.
template <int D>
__device__ __forceinline__ void pipe_refill(PipeSmem<D>& SM, int b, int e, int nitems, const Particles& P,
                                            const StepConsts& C, const TileInfo& TI, const CUtensorMap& map) {
    using G = FusedGeom<D>;
    const int lane = threadIdx.x & 31;
    if (e >= nitems) {
        if (lane == 0) {
            SM.item[b] = make_int4(0, 0, 0, 0);
            mbar_arrive(&SM.full[b]);
        }
        return;
    }
    int4 item = TI.items[e];
    if (lane == 0) {
        int tc[3] = {0, 0, 0}, bo[3] = {0, 0, 0};
        tile_origin<D>(TI, item.x, tc, bo);
        bool near = false;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const int ext = k == 0 ? C.W : (k == 1 ? C.H : C.Dp);
            near = near || bo[k] <= C.margin || bo[k] + G::BE - 1 >= ext - C.margin;
        }
        item.w = D == 3 && near;
        SM.item[b] = item;
        fence_proxy_async_smem();
        mbar_expect(&SM.full[b], (item.w ? 2 : 1) * G::BN * (uint32_t)sizeof(float4));
        box_load<D>(map, bo, 0, SM.box[b], &SM.full[b]);
        if (item.w) box_load<D>(map, bo, 1, SM.wall[b], &SM.full[b]);
    }
    if (lane < D + D * D + 1) {
        const long long n = P.n;
        const float* a = lane < D ? P.x + lane * n : (lane < D + D * D ? P.Fe + (lane - D) * n : P.Jp);
        // whole 16-byte words inside the tile's slots
        const uint64_t lo = (reinterpret_cast<uint64_t>(a + item.y) + 15) & ~15ull;
        const uint64_t hi = reinterpret_cast<uint64_t>(a + item.y + item.z) & ~15ull;
        if (hi > lo)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lo), "r"((uint32_t)(hi - lo)) : "memory");
    }
}

template <int D, int S>
__global__ void __launch_bounds__(PipeGeom<D>::THREADS, PipeGeom<D>::CTAS)
    k_g2p2g_pipe(Particles P, StepConsts C, TileInfo TI, const float4* __restrict__ gv,
                 unsigned long long* __restrict__ acc, SlowQueue Q, unsigned* __restrict__ status,
                 const __grid_constant__ CUtensorMap gv_map) {
    using R = PipeGeom<D>;
    extern __shared__ __align__(128) unsigned char fused_smem[];
    PipeSmem<D>& SM = *reinterpret_cast<PipeSmem<D>*>(fused_smem);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    chain_wait();
    const int nitems = *TI.n_items;
    if (wid == 0) {
        if (lane < R::STAGES) {
            mbar_init(&SM.full[lane], 1);
            SM.next_win[lane] = 0;
            SM.left[lane] = 0;
            SM.bmask[lane] = 0u;
        }
        mbar_init_fence();
        __syncwarp();
        int e = 0;
        if (lane == 0) e = atomicAdd(TI.fused_next, R::STAGES);
        e = __shfl_sync(0xffffffffu, e, 0);
        for (int b = 0; b < R::STAGES; ++b) pipe_refill<D>(SM, b, e + b, nitems, P, C, TI, gv_map);
    }
    __syncthreads();
    int b = 0;
    unsigned par = 0u;
    for (;;) {
        if (!__all_sync(0xffffffffu, mbar_wait(&SM.full[b], par, kBoxWaitPolls))) {
            // the box never arrived (flagged); let the other buffers' loads land first
            if (lane == 0) {
                raise_flag(status, 16u);
                for (int j = 1; j < R::STAGES; ++j)
                    mbar_wait(&SM.full[(b + j) % R::STAGES], b + j < R::STAGES ? par : par ^ 1u, kBoxWaitPolls);
            }
            return;
        }
        const int4 item = SM.item[b];
        const int start = item.y, m = item.z;
        if (m == 0) break;
        int tc[3] = {0, 0, 0}, bo[3] = {0, 0, 0};
        tile_origin<D>(TI, item.x, tc, bo);
        const int nwin = (m + TI.win - 1) / TI.win;
        unsigned bits = 0u;
        for (;;) {
            int w = 0;
            if (lane == 0) w = atomicAdd(&SM.next_win[b], 1);
            w = __shfl_sync(0xffffffffu, w, 0);
            if (w >= nwin) break;
            bits |= fused_window<D, S, true>(P, C, TI, gv, acc, Q, status, SM.box[b],
                                             D == 3 && item.w ? SM.wall[b] : nullptr, bo, start, m, TI.win, w,
                                             reinterpret_cast<float*>(SM.pay[wid]));
        }
        bits = __reduce_or_sync(0xffffffffu, bits);
        int last = 0;
        if (lane == 0) {
            if (bits) atomicOr(&SM.bmask[b], bits);
            __threadfence_block();  // the bits and this warp's reads of the box before the count
            last = atomicAdd(&SM.left[b], 1) == R::WARPS - 1;
        }
        if (__shfl_sync(0xffffffffu, last, 0)) {
            // last warp out: mark the tile's node blocks, then stage k + STAGES into this buffer
            __threadfence_block();
            unsigned bm = 0u;
            int e = 0;
            if (lane == 0) {
                bm = atomicOr(&SM.bmask[b], 0u);
                SM.bmask[b] = 0u;
                SM.next_win[b] = 0;
                SM.left[b] = 0;
                e = atomicAdd(TI.fused_next, 1);
            }
            mark_tile_blocks<D>(TI, tc, __shfl_sync(0xffffffffu, bm, 0));
            pipe_refill<D>(SM, b, __shfl_sync(0xffffffffu, e, 0), nitems, P, C, TI, gv_map);
            __syncwarp();
        }
        if (++b == R::STAGES) {
            b = 0;
            par ^= 1u;
        }
    }
}

}  // namespace mpm
