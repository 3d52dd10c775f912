// Learned plasticity surrogate: a 10 -> 64 -> 64 -> 64 -> 10 MLP with GELU,
// BF16 weights and activations, FP32 accumulation on the tensor cores
// (mma.sync m16n8k16 bf16), FP32 master weights trained with AdamW.
//
// It maps the trial elastic gradient and the plastic volume ratio of a particle
// whose trial F lies outside the elastic band (inputs: F_hat - I, log J_p) to
// the return map's correction (outputs: F_E' - F_hat, log J_p' - log J_p), both
// normalised per feature. Training pairs come from the exact return map of the
// plain solver (k_g2p_plastic with the pair log enabled).
#pragma once

#include <cuda_bf16.h>

#include "mpm_kernels.cuh"

namespace mpm {

constexpr int kMlpIn = 10, kMlpHid = 64, kMlpOut = 10, kMlpInPad = 16, kMlpOutPad = 16;
// Parameter block (row-major W[out][in]): W1[64][16] b1[64] W2[64][64] b2[64]
// W3[64][64] b3[64] W4[16][64] b4[16]; padded rows/columns are kept at zero.
struct MlpOff {
    static constexpr int W1 = 0, b1 = W1 + kMlpHid * kMlpInPad, W2 = b1 + kMlpHid, b2 = W2 + kMlpHid * kMlpHid,
                         W3 = b2 + kMlpHid, b3 = W3 + kMlpHid * kMlpHid, W4 = b3 + kMlpHid,
                         b4 = W4 + kMlpOutPad * kMlpHid, total = b4 + kMlpOutPad;
};

struct MlpNorm {
    float in_mean[kMlpIn], in_std[kMlpIn], out_mean[kMlpOut], out_std[kMlpOut];
};

// ---------------------------------------------------------------------------
// Tensor-core fragments, m16n8k16 layouts (PTX ISA): with g = lane / 4, t = lane % 4,
//   A regs: (g, 2t..2t+1), (g+8, 2t..), (g, 2t+8..), (g+8, 2t+8..)
//   B regs: (k = 2t..2t+1, n = g), (k = 2t+8.., n = g)
//   C/D   : (g, 2t), (g, 2t+1), (g+8, 2t), (g+8, 2t+1)
__device__ __forceinline__ void mma_bf16(float* d, const uint32_t* a, const uint32_t* b) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// GELU in its tanh form (Hendrycks & Gimpel 2016):
//   gelu(x) = x/2 (1 + tanh(c (x + 0.044715 x^3))),  c = sqrt(2/pi),
// with the hardware tanh (PTX tanh.approx.f32, relative error ~2^-11, below the
// bf16 rounding of the stored activations). Training and inference share it.
__device__ __forceinline__ float tanh_hw(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
constexpr float kGeluC = 0.7978845608028654f, kGeluA = 0.044715f;
__device__ __forceinline__ float gelu(float x) {
    const float th = tanh_hw(kGeluC * x * fmaf(kGeluA, x * x, 1.f));
    return 0.5f * x * (1.f + th);
}
// Of two values, in packed FP32 (8 instructions for what takes 14 one by one).
__device__ __forceinline__ float2 gelu2(float2 x) {
    const float2 u = __fmul2_rn(x, __ffma2_rn(__fmul2_rn(x, x), make_float2(kGeluC * kGeluA, kGeluC * kGeluA),
                                              make_float2(kGeluC, kGeluC)));
    const float2 h = __fmul2_rn(x, make_float2(0.5f, 0.5f));
    return __ffma2_rn(h, make_float2(tanh_hw(u.x), tanh_hw(u.y)), h);
}
__device__ __forceinline__ float gelu_grad(float x) {
    const float x2 = x * x;
    const float th = tanh_hw(kGeluC * x * fmaf(kGeluA, x2, 1.f));
    return 0.5f * (1.f + th) + 0.5f * x * (1.f - th * th) * kGeluC * fmaf(3.f * kGeluA, x2, 1.f);
}

// Raw pair -> normalised network input (row of kMlpInPad bf16) and target.
// Pair layout (20 floats): F_hat[9] J_p[1] F_E'[9] J_p'[1].
__device__ __forceinline__ void mlp_features(const float* Fh, float Jp, const MlpNorm& N, float* in) {
#pragma unroll
    for (int k = 0; k < 9; ++k) in[k] = ((Fh[k] - (k % 4 == 0 ? 1.f : 0.f)) - N.in_mean[k]) * (1.f / N.in_std[k]);
    in[9] = (logf(Jp) - N.in_mean[9]) * (1.f / N.in_std[9]);
}
__device__ __forceinline__ void mlp_targets(const float* pair, const MlpNorm& N, float* tg) {
#pragma unroll
    for (int k = 0; k < 9; ++k) tg[k] = ((pair[10 + k] - pair[k]) - N.out_mean[k]) / N.out_std[k];
    tg[9] = ((logf(pair[19]) - logf(pair[9])) - N.out_mean[9]) / N.out_std[9];
}

// ---------------------------------------------------------------------------
// Residual check of a predicted return map (3D). The exact map is
//   F_hat = U S_hat V^T,  F_E' = U S V^T,  S = clamp(S_hat, t0, t1),
// so with M = F_hat F_E'^-1 = U diag(S_hat / S) U^T and Q = F_E' F_E'^T =
// U S^2 U^T: M is symmetric and commutes with Q, every eigenvalue of Q lies in
// [t0^2, t1^2], and in each common eigendirection either m = 1 (unclamped) or
// q is at a band edge with m on the right side of 1:
//   (M - I)(Q - t0^2 I)(Q - t1^2 I) = 0,  (M - I)(Q - t0^2 I) >= 0,  (M - I)(Q - t1^2 I) >= 0.
// These conditions characterise the map (with M > 0, so that S_hat = M S keeps
// the sign of S). `tol` bounds the relative error of the predicted F_E': an
// error E in F_E' moves M and Q by O(|E|), so each condition is tested to the
// slack that |E| = tol |F_E'| can produce (asymmetry and commutator relative
// to |M| and |M||Q|; Q's eigenvalues to 2 tol outside the band; the sign
// conditions to -tol (w + 2|M - I|), w = t1^2 - t0^2). Semidefiniteness is
// tested by Gershgorin first and, when that is inconclusive, by Sylvester's
// criterion in FP64 on the shifted matrix. Any failure sends the particle to
// the exact SVD.
__device__ __forceinline__ bool gersh_min_ge(const float* S, float bound) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        float r = 0.f;
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (j != i) r += fabsf(S[i * 3 + j]);
        if (S[i * 4] - r < bound) return false;
    }
    return true;
}

// A symmetric 3x3 S satisfies S >= bound I (bound <= 0): Gershgorin, else
// Sylvester's criterion on S - 1.0001 bound I in FP64.
__device__ __forceinline__ bool sym_min_ge(const float* S, float bound) {
    if (gersh_min_ge(S, bound)) return true;
    double D[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) D[k] = double(S[k]) - (k % 4 == 0 ? 1.0001 * double(bound) : 0.0);
    return D[0] > 0.0 && D[0] * D[4] - D[1] * D[3] > 0.0 && det<3>(D) > 0.0;
}

__device__ __forceinline__ bool mlp_residual_ok(const float* Fh, const float* Fe, float t0, float t1, float tol) {
    const float dE = det<3>(Fe);
    if (!(dE > 0.f) || !(det<3>(Fh) > 0.f)) return false;
    float inv[9];
    const float r = 1.f / dE;
    inv[0] = (Fe[4] * Fe[8] - Fe[5] * Fe[7]) * r;
    inv[1] = (Fe[2] * Fe[7] - Fe[1] * Fe[8]) * r;
    inv[2] = (Fe[1] * Fe[5] - Fe[2] * Fe[4]) * r;
    inv[3] = (Fe[5] * Fe[6] - Fe[3] * Fe[8]) * r;
    inv[4] = (Fe[0] * Fe[8] - Fe[2] * Fe[6]) * r;
    inv[5] = (Fe[2] * Fe[3] - Fe[0] * Fe[5]) * r;
    inv[6] = (Fe[3] * Fe[7] - Fe[4] * Fe[6]) * r;
    inv[7] = (Fe[1] * Fe[6] - Fe[0] * Fe[7]) * r;
    inv[8] = (Fe[0] * Fe[4] - Fe[1] * Fe[3]) * r;
    float M[9], Q[9];
    matmul<3>(Fh, inv, M);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) Q[i * 3 + j] = Fe[i * 3] * Fe[j * 3] + Fe[i * 3 + 1] * Fe[j * 3 + 1] + Fe[i * 3 + 2] * Fe[j * 3 + 2];
    float asym = 0.f, nm = 0.f;
    float Ms[9], G[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const float a = M[i * 3 + j] - M[j * 3 + i];
            asym += a * a;
            nm += M[i * 3 + j] * M[i * 3 + j];
            Ms[i * 3 + j] = 0.5f * (M[i * 3 + j] + M[j * 3 + i]);
            G[i * 3 + j] = Ms[i * 3 + j] - (i == j ? 1.f : 0.f);
        }
    if (asym > tol * tol * nm) return false;
    // commutation
    float MQ[9], QM[9];
    matmul<3>(Ms, Q, MQ);
    matmul<3>(Q, Ms, QM);
    float comm = 0.f, nq = 0.f;
#pragma unroll
    for (int k = 0; k < 9; ++k) { comm += (MQ[k] - QM[k]) * (MQ[k] - QM[k]); nq += Q[k] * Q[k]; }
    if (comm > tol * tol * nm * nq) return false;
    // band of Q
    const float a0 = t0 * t0, a1 = t1 * t1, w = a1 - a0;
    float Ql[9], Qh[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) { Ql[k] = Q[k] - (k % 4 == 0 ? a0 : 0.f); Qh[k] = (k % 4 == 0 ? a1 : 0.f) - Q[k]; }
    if (!sym_min_ge(Ql, -2.f * tol) || !sym_min_ge(Qh, -2.f * tol)) return false;
    if (!gersh_min_ge(Ms, 0.5f)) return false;
    // (M - I)(Q - t0^2)(Q - t1^2) = 0 and the sign conditions
    float GL[9], GH[9], P[9];
    float Qh_neg[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) Qh_neg[k] = -Qh[k];  // Q - t1^2 I
    matmul<3>(G, Ql, GL);
    matmul<3>(G, Qh_neg, GH);
    matmul<3>(GL, Qh_neg, P);
    float np = 0.f, ng = 0.f;
#pragma unroll
    for (int k = 0; k < 9; ++k) { np += P[k] * P[k]; ng += G[k] * G[k]; }
    if (np > tol * tol * (1.f + ng) * w * w * w * w) return false;
    float GLs[9], GHs[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            GLs[i * 3 + j] = 0.5f * (GL[i * 3 + j] + GL[j * 3 + i]);
            GHs[i * 3 + j] = 0.5f * (GH[i * 3 + j] + GH[j * 3 + i]);
        }
    const float sg = -tol * (w + 2.f * sqrtf(ng));
    if (!sym_min_ge(GLs, sg) || !sym_min_ge(GHs, sg)) return false;
    return true;
}

struct MlpParams {
    const __nv_bfloat16* wbf;
    const float* wf32;
    MlpNorm norm;
    float tol;
    unsigned long long* counters;  // [0] accepted, [1] rejected (fell back to the SVD)
};

// ---------------------------------------------------------------------------
// Warp-tiled inference for the solver. Each warp takes 32 queued particles
// (lane = particle) and runs the network on them as two 16-row tiles whose
// activations never leave registers: the m16n8 accumulators of one layer,
// after bias + GELU, are packed to bf16 pairs that are exactly the m16k16 A
// fragments of the next layer (accumulator n-tiles 2kb, 2kb+1 = A k-block kb).
// Weights sit in shared memory with rows padded by 8 bf16 so that the eight rows
// of a B fragment (ldmatrix) fall into distinct banks.
//
// Bound: instruction issue (GELU half of it) at 16 warps per SM. The three hidden
// layers run through one copy of the code: with a copy each, the kernel outgrew
// the instruction cache. 474k particles in collision, most of them queued: 119 us a
// step with scalar GELU, 4-byte fragment loads and unrolled layers, now 86.
constexpr int kMwIn = kMlpInPad + 8;  // row stride (bf16) of W1 and of the input tile
constexpr int kMwHid = kMlpHid + 8;   // row stride (bf16) of W2, W3, W4
constexpr int kMwOut = kMlpOutPad + 2;  // row stride (fp32) of the output tile
constexpr int kMlpWarps = 8;

struct MlpWarpSmem {
    alignas(16) __nv_bfloat16 W1[kMlpHid * kMwIn];
    __nv_bfloat16 W23[2][kMlpHid * kMwHid];
    __nv_bfloat16 W4[kMlpOutPad * kMwHid];
    float b[3][kMlpHid], b4[kMlpOutPad];
    alignas(16) __nv_bfloat16 x[kMlpWarps][32 * kMwIn];
    float out[kMlpWarps][32 * kMwOut];
};

__device__ __forceinline__ void mlp_stage_matrix(__nv_bfloat16* dst, int ld_dst, const __nv_bfloat16* src, int rows,
                                                 int cols) {
    const int vpr = cols / 8;  // 16-byte vectors per row
    for (int v = threadIdx.x; v < rows * vpr; v += blockDim.x) {
        const int r = v / vpr, c = (v % vpr) * 8;
        *reinterpret_cast<uint4*>(dst + r * ld_dst + c) = *reinterpret_cast<const uint4*>(src + r * cols + c);
    }
}

__device__ __forceinline__ void mlp_stage_weights(MlpWarpSmem& S, const __nv_bfloat16* wbf, const float* wf32) {
    mlp_stage_matrix(S.W1, kMwIn, wbf + MlpOff::W1, kMlpHid, kMlpInPad);
    mlp_stage_matrix(S.W23[0], kMwHid, wbf + MlpOff::W2, kMlpHid, kMlpHid);
    mlp_stage_matrix(S.W23[1], kMwHid, wbf + MlpOff::W3, kMlpHid, kMlpHid);
    mlp_stage_matrix(S.W4, kMwHid, wbf + MlpOff::W4, kMlpOutPad, kMlpHid);
    for (int i = threadIdx.x; i < kMlpHid; i += blockDim.x) {
        S.b[0][i] = wf32[MlpOff::b1 + i];
        S.b[1][i] = wf32[MlpOff::b2 + i];
        S.b[2][i] = wf32[MlpOff::b3 + i];
    }
    for (int i = threadIdx.x; i < kMlpOutPad; i += blockDim.x) S.b4[i] = wf32[MlpOff::b4 + i];
}

__device__ __forceinline__ uint32_t pack_f2_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t* r, const __nv_bfloat16* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a)
                 : "memory");
}

// acc[j] (n-tile j of a 16 x 8*NT output) = A (16 x 16*KB, fragments a[kb]) * W^T,
// W row-major [out][in] in shared memory with row stride ld. An ldmatrix brings two
// B fragments: of two k-blocks, or (KB = 1) of two n-tiles.
template <int KB, int NT>
__device__ __forceinline__ void mlp_warp_layer(const uint32_t (*a)[4], const __nv_bfloat16* W, int ld, float (*acc)[4]) {
    static_assert(KB == 1 || KB % 2 == 0, "fragments come in pairs");
    const int lane = threadIdx.x & 31, row = lane & 7, mat = lane >> 3;
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    if constexpr (KB == 1) {
        const __nv_bfloat16* w = W + ((mat >> 1) * 8 + row) * ld + (mat & 1) * 8;
#pragma unroll
        for (int j = 0; j < NT; j += 2) {
            uint32_t b[4];
            ldmatrix_x4(b, w + j * 8 * ld);
            mma_bf16(acc[j], a[0], b);
            mma_bf16(acc[j + 1], a[0], b + 2);
        }
    } else {
        const __nv_bfloat16* w = W + row * ld + mat * 8;
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int kb = 0; kb < KB; kb += 2) {
                uint32_t b[4];
                ldmatrix_x4(b, w + j * 8 * ld + kb * 16);
                mma_bf16(acc[j], a[kb], b);
                mma_bf16(acc[j], a[kb + 1], b + 2);
            }
    }
}

// bias + GELU on a 16 x 64 accumulator, packed into the A fragments of the next layer.
__device__ __forceinline__ void mlp_warp_activate(float (*acc)[4], const float* bias, uint32_t (*a)[4]) {
    const int t = threadIdx.x & 3;
#pragma unroll
    for (int kb = 0; kb < kMlpHid / 16; ++kb)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = 2 * kb + h;
            const float2 b = *reinterpret_cast<const float2*>(bias + j * 8 + 2 * t);
            const float2 u = gelu2(__fadd2_rn(make_float2(acc[j][0], acc[j][1]), b));
            const float2 v = gelu2(__fadd2_rn(make_float2(acc[j][2], acc[j][3]), b));
            a[kb][2 * h] = pack_f2_bf16(u.x, u.y);
            a[kb][2 * h + 1] = pack_f2_bf16(v.x, v.y);
        }
}

// Network on the warp's 32-row input tile X (bf16, row stride kMwIn) -> O
// (fp32, normalised outputs, row stride kMwOut).
__device__ __forceinline__ void mlp_warp_forward(const MlpWarpSmem& S, const __nv_bfloat16* X, float* O) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll 1
    for (int mt = 0; mt < 2; ++mt) {
        const int r0 = mt * 16 + g;
        uint32_t a[kMlpHid / 16][4];
        ldmatrix_x4(a[0], X + (mt * 16 + (lane & 15)) * kMwIn + (lane >> 4) * 8);
        float acc[kMlpHid / 8][4];
        mlp_warp_layer<1, kMlpHid / 8>(a, S.W1, kMwIn, acc);
#pragma unroll 1
        for (int l = 0; l < 2; ++l) {
            mlp_warp_activate(acc, S.b[l], a);
            mlp_warp_layer<kMlpHid / 16, kMlpHid / 8>(a, S.W23[l], kMwHid, acc);
        }
        mlp_warp_activate(acc, S.b[2], a);
        float o[kMlpOutPad / 8][4];
        mlp_warp_layer<kMlpHid / 16, kMlpOutPad / 8>(a, S.W4, kMwHid, o);
#pragma unroll
        for (int j = 0; j < kMlpOutPad / 8; ++j) {
            const int c = j * 8 + 2 * t;
            *reinterpret_cast<float2*>(O + r0 * kMwOut + c) = make_float2(o[j][0] + S.b4[c], o[j][1] + S.b4[c + 1]);
            *reinterpret_cast<float2*>(O + (r0 + 8) * kMwOut + c) =
                make_float2(o[j][2] + S.b4[c], o[j][3] + S.b4[c + 1]);
        }
    }
}

// Learned return map of the queued particles (3D tiled MLS path). Accepted
// predictions write F_E', J_p' and the next step's affine matrix and mark
// their queue entry kQueueDone; the rest (rejected by the residual check or
// by the stress series, and grid-clipped stencils) stay queued for
// k_g2p_plastic's exact return map, which runs next.
__global__ void __launch_bounds__(kMlpWarps * 32) k_return_map_mlp(Particles P, StepConsts C, SlowQueue Q,
                                                                   MlpParams ML) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MlpWarpSmem& S = *reinterpret_cast<MlpWarpSmem*>(smem_raw);
    chain_wait();
    const int m = *Q.count;
    // CTAs past the queue's end leave before staging the weights (the grid is
    // sized for the largest queue; most steps queue far fewer particles)
    if ((long long)blockIdx.x * kMlpWarps * 32 >= m) return;
    mlp_stage_weights(S, ML.wbf, ML.wf32);
    __syncthreads();
    const long long n = P.n;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __nv_bfloat16* X = S.x[wid];
    float* O = S.out[wid];
    const float t0 = 1.f - C.theta_c, t1 = 1.f + C.theta_s;
    unsigned n_ok = 0, n_bad = 0;
    const int warps = gridDim.x * kMlpWarps;
    for (int base = (blockIdx.x * kMlpWarps + wid) * 32; base < m; base += warps * 32) {
        const int e = base + lane;
        const int entry = e < m ? Q.list[e] : -1;
        const bool valid = entry >= 0;
        float Fh[9], Jp0 = 1.f, B[9], mass = 0.f, vol = 0.f;
        float in[kMlpIn];
        if (valid) {
#pragma unroll
            for (int k = 0; k < 9; ++k) Fh[k] = Q.fh[k * Q.capacity + e];
            Jp0 = P.Jp[entry];
            mlp_features(Fh, Jp0, ML.norm, in);
        }
        uint32_t* xr = reinterpret_cast<uint32_t*>(X + lane * kMwIn);
#pragma unroll
        for (int k = 0; k < kMlpInPad / 2; ++k) {
            const float lo = valid && 2 * k < kMlpIn ? in[2 * k] : 0.f;
            const float hi = valid && 2 * k + 1 < kMlpIn ? in[2 * k + 1] : 0.f;
            xr[k] = pack_f2_bf16(lo, hi);
        }
        __syncwarp();
        if (__any_sync(0xffffffffu, valid)) mlp_warp_forward(S, X, O);
        __syncwarp();
        if (valid) {
#pragma unroll
            for (int k = 0; k < 9; ++k) B[k] = P.B[k * n + entry];
            mass = P.mass ? P.mass[entry] : P.mass_u;
            vol = P.vol ? P.vol[entry] : P.vol_u;
            const float* o = O + lane * kMwOut;
            float Fp[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) Fp[k] = Fh[k] + (o[k] * ML.norm.out_std[k] + ML.norm.out_mean[k]);
            const float dlj = o[9] * ML.norm.out_std[9] + ML.norm.out_mean[9];
            bool ok = mlp_residual_ok(Fh, Fp, t0, t1, ML.tol);
            float ratio = 1.f;
            if (ok) {
                // J_p' = J_p det(F_hat) / det(F_E') (= J_p prod(S_hat / S)); the
                // network's log J_p' output must agree with it within the tolerance.
                ratio = det<3>(Fh) / det<3>(Fp);
                ok = fabsf(logf(ratio) - dlj) <= ML.tol * (1.f + fabsf(dlj));
            }
            float sig[9];
            const float Jp = Jp0 * ratio;
            if (ok) ok = hardened_stress_series<3>(Fp, Jp, C.mu0, C.la0, C.xi, sig);
            if (ok) {
#pragma unroll
                for (int k = 0; k < 9; ++k) {
                    P.Fe[k * n + entry] = Fp[k];
                    P.A[k * n + entry] = 3.f * mass * B[k] - 3.f * C.dt * vol * sig[k];
                }
                P.Jp[entry] = Jp;
                Q.list[e] = kQueueDone;
                ++n_ok;
            } else {
                ++n_bad;
            }
        }
        __syncwarp();
    }
    if (ML.counters) {
        n_ok = __reduce_add_sync(0xffffffffu, n_ok);
        n_bad = __reduce_add_sync(0xffffffffu, n_bad);
        if (lane == 0) {
            if (n_ok) atomicAdd(&ML.counters[0], (unsigned long long)n_ok);
            if (n_bad) atomicAdd(&ML.counters[1], (unsigned long long)n_bad);
        }
    }
}

// Batched inference on raw pairs' inputs (evaluation and tests), through the
// same warp-tiled path as the solver: out[n][10] = denormalised
// (F_E' - F_hat, log J_p' - log J_p). Rows: input + stride * i, F_hat[9], J_p.
__global__ void __launch_bounds__(kMlpWarps * 32) k_mlp_forward(const float* __restrict__ inputs, int stride, int n,
                                                                const __nv_bfloat16* __restrict__ wbf,
                                                                const float* __restrict__ wf32, MlpNorm N,
                                                                float* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MlpWarpSmem& S = *reinterpret_cast<MlpWarpSmem*>(smem_raw);
    mlp_stage_weights(S, wbf, wf32);
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __nv_bfloat16* X = S.x[wid];
    float* O = S.out[wid];
    const int row = (blockIdx.x * kMlpWarps + wid) * 32 + lane;
    const bool valid = row < n;
    float in[kMlpIn];
    if (valid) mlp_features(inputs + (long long)row * stride, inputs[(long long)row * stride + 9], N, in);
    uint32_t* xr = reinterpret_cast<uint32_t*>(X + lane * kMwIn);
#pragma unroll
    for (int k = 0; k < kMlpInPad / 2; ++k)
        xr[k] = pack_f2_bf16(valid && 2 * k < kMlpIn ? in[2 * k] : 0.f, valid && 2 * k + 1 < kMlpIn ? in[2 * k + 1] : 0.f);
    __syncwarp();
    mlp_warp_forward(S, X, O);
    __syncwarp();
    if (valid)
#pragma unroll
        for (int c = 0; c < kMlpOut; ++c) out[(long long)row * kMlpOut + c] = O[lane * kMwOut + c] * N.out_std[c] + N.out_mean[c];
}

// ---------------------------------------------------------------------------
// Training step: forward, MSE loss, backward on tiles of kMlpTrainRows samples
// (8 warps x 16 rows); a CTA takes tiles until none are left and writes its
// weight gradients and loss once, to its own row of `part` (summed by
// k_mlp_adam / k_mlp_grad_sum in FP64). Samples: row = pair (seed 0 and
// `in_order`) or a hash of (seed, global row) modulo n_pairs.
//
// Every gradient is a sum over blocks of kMlpSumRows rows: a block's weight
// gradients are one chain of mma, its bias gradients are added row by row, and
// blocks are added to each other in plain FP32. A block's part thus rounds alike
// however the rows are split over tiles and CTAs: the same 64-row parts that
// training has always added up, so a run follows earlier ones as closely as they
// follow each other (AdamW and the bf16 copy of the weights amplify the last bits
// of a gradient: 32 steps at a batch of 16384 apart by 1.6e-5 in the median, when
// the same parts were added by atomics in two orders).
//
// A warp keeps its 16 rows in registers through the layers: the m16n8
// accumulators of one layer, after bias + GELU, are the m16k16 A fragments of the
// next (as in the inference kernel), backward as well (dX = dY W with W transposed
// in shared memory), and GELU' stays in registers from the forward pass. Only the
// bf16 activations and dY go to shared memory, from which every warp takes
// transposed fragments (ldmatrix.trans) for its share of dW = dY^T X.
// Bound: latency (8 warps per SM, one tile per CTA at the usual batch of 16384,
// about 600 dependent mma and tanh a warp). The former kernel (64-row tiles,
// every fragment from 2-byte shared loads, an fp32 atomic per weight and CTA)
// took 107 us at that batch, this one about 17 us, 2.3 of them for the parts of 64
// rows and their bias sums (16 steps with their updates: 420 us).
constexpr int kMlpTrainRows = 128;
constexpr int kMlpSumRows = 64;
constexpr int kMlpTrainCtas = 148;              // most CTAs (rows of `part`)
constexpr int kMlpPart = MlpOff::total + 16;    // floats per row: gradients, then the loss

struct MlpTrainSmem {
    __nv_bfloat16 W1[kMlpHid * kMwIn], W2[kMlpHid * kMwHid], W3[kMlpHid * kMwHid], W4[kMlpOutPad * kMwHid];
    __nv_bfloat16 W2t[kMlpHid * kMwHid], W3t[kMlpHid * kMwHid], W4t[kMlpHid * kMwIn];  // [in][out]
    float b1[kMlpHid], b2[kMlpHid], b3[kMlpHid], b4[kMlpOutPad];
    __nv_bfloat16 x0[kMlpTrainRows * kMwIn];
    __nv_bfloat16 h[3][kMlpTrainRows * kMwHid];
    __nv_bfloat16 dy[kMlpTrainRows * kMwHid];    // gradient wrt the current layer's pre-activation
    __nv_bfloat16 dy4[kMlpTrainRows * kMwIn];
    float tgt[kMlpTrainRows * kMlpOutPad];      // targets, then gradient wrt the output
    float red[8];                               // per warp: loss
    float db[kMlpTrainRows / kMlpSumRows][3 * kMlpHid + kMlpOutPad];
};

__device__ __forceinline__ unsigned hash_u32(unsigned x) {
    x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
    return x;
}

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t* r, const __nv_bfloat16* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a)
                 : "memory");
}

// bias + GELU on a warp's 16 x 64 accumulator: A fragments of the next layer and
// their copy in shared memory (rows r0 .. r0 + 15), GELU' kept in fp32.
__device__ __forceinline__ void mlp_train_activate(float (*acc)[4], const float* bias, uint32_t (*a)[4], float (*gp)[4],
                                                   __nv_bfloat16* h, int r0) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int j = 0; j < kMlpHid / 8; ++j) {
        const int c = j * 8 + 2 * t;
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float x = acc[j][q] + bias[c + (q & 1)];
            v[q] = gelu(x);
            gp[j][q] = gelu_grad(x);
        }
        const uint32_t lo = pack_f2_bf16(v[0], v[1]), hi = pack_f2_bf16(v[2], v[3]);
        a[j / 2][2 * (j & 1)] = lo;
        a[j / 2][2 * (j & 1) + 1] = hi;
        *reinterpret_cast<uint32_t*>(h + (r0 + g) * kMwHid + c) = lo;
        *reinterpret_cast<uint32_t*>(h + (r0 + g + 8) * kMwHid + c) = hi;
    }
}

// dY of a hidden layer from dX (accumulator) and GELU': bf16 A fragments and
// their copy in shared memory.
__device__ __forceinline__ void mlp_train_back(float (*acc)[4], float (*gp)[4], uint32_t (*a)[4], __nv_bfloat16* dy, int r0) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int j = 0; j < kMlpHid / 8; ++j) {
        const uint32_t lo = pack_f2_bf16(acc[j][0] * gp[j][0], acc[j][1] * gp[j][1]);
        const uint32_t hi = pack_f2_bf16(acc[j][2] * gp[j][2], acc[j][3] * gp[j][3]);
        a[j / 2][2 * (j & 1)] = lo;
        a[j / 2][2 * (j & 1) + 1] = hi;
        *reinterpret_cast<uint32_t*>(dy + (r0 + g) * kMwHid + j * 8 + 2 * t) = lo;
        *reinterpret_cast<uint32_t*>(dy + (r0 + g + 8) * kMwHid + j * 8 + 2 * t) = hi;
    }
}

// The warp's share of dW[n][k] += sum_r dY[r][n] X[r][k] over the tile's blocks of
// rows: output rows n0 .. n0 + 15, NT column tiles of 8 from k0 on.
template <int NT>
__device__ __forceinline__ void mlp_train_dw(const __nv_bfloat16* dY, int ldd, const __nv_bfloat16* X, int ldx, int n0,
                                             int k0, float (*dw)[4]) {
    const int lane = threadIdx.x & 31, mi = lane >> 3, row = lane & 7;
#pragma unroll
    for (int blk = 0; blk < kMlpTrainRows; blk += kMlpSumRows) {
        float s[NT][4] = {};
#pragma unroll
        for (int r0 = blk; r0 < blk + kMlpSumRows; r0 += 16) {
            uint32_t a[4];
            ldmatrix_x4_trans(a, dY + (r0 + (mi >> 1) * 8 + row) * ldd + n0 + (mi & 1) * 8);
#pragma unroll
            for (int j = 0; j < NT; j += 2) {
                uint32_t b[4];
                // matrices: (r0, k), (r0 + 8, k), (r0, k + 8), (r0 + 8, k + 8); with one tile the second pair repeats the first
                const int kc = k0 + j * 8 + (NT > 1 ? (mi >> 1) * 8 : 0);
                ldmatrix_x4_trans(b, X + (r0 + (mi & 1) * 8 + row) * ldx + kc);
                mma_bf16(s[j], a, b);
                if constexpr (NT > 1) mma_bf16(s[j + 1], a, b + 2);
            }
        }
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) dw[j][q] += s[j][q];
    }
}

// db[n] of one block of rows, by one thread: column n of dY (row stride ld), row by row.
template <typename T> __device__ __forceinline__ float mlp_train_db(const T* dY, int ld) {
    float s = 0.f;
#pragma unroll 32
    for (int r = 0; r < kMlpSumRows; ++r) s += float(dY[r * ld]);
    return s;
}

// The transpose of a row-major [rows][cols] matrix.
__device__ __forceinline__ void mlp_stage_transposed(__nv_bfloat16* dst, int ld_dst, const __nv_bfloat16* src, int rows,
                                                     int cols) {
    for (int v = threadIdx.x; v < rows * cols; v += blockDim.x) dst[(v % cols) * ld_dst + v / cols] = src[v];
}

__global__ void __launch_bounds__(256, 1) k_mlp_train(const float* __restrict__ pairs, long long n_pairs, bool in_order,
                                                      int n_rows, unsigned seed, const __nv_bfloat16* __restrict__ wbf,
                                                      const float* __restrict__ wf32, MlpNorm N,
                                                      float* __restrict__ part) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MlpTrainSmem& S = *reinterpret_cast<MlpTrainSmem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    mlp_stage_matrix(S.W1, kMwIn, wbf + MlpOff::W1, kMlpHid, kMlpInPad);
    mlp_stage_matrix(S.W2, kMwHid, wbf + MlpOff::W2, kMlpHid, kMlpHid);
    mlp_stage_matrix(S.W3, kMwHid, wbf + MlpOff::W3, kMlpHid, kMlpHid);
    mlp_stage_matrix(S.W4, kMwHid, wbf + MlpOff::W4, kMlpOutPad, kMlpHid);
    mlp_stage_transposed(S.W2t, kMwHid, wbf + MlpOff::W2, kMlpHid, kMlpHid);
    mlp_stage_transposed(S.W3t, kMwHid, wbf + MlpOff::W3, kMlpHid, kMlpHid);
    mlp_stage_transposed(S.W4t, kMwIn, wbf + MlpOff::W4, kMlpOutPad, kMlpHid);
    if (tid < kMlpHid) {
        S.b1[tid] = wf32[MlpOff::b1 + tid];
        S.b2[tid] = wf32[MlpOff::b2 + tid];
        S.b3[tid] = wf32[MlpOff::b3 + tid];
    }
    if (tid < kMlpOutPad) S.b4[tid] = wf32[MlpOff::b4 + tid];
    // the warp's share of dW: rows n0.. of W2 and W3 and half of their columns,
    // one tile each of W1 and W4
    const int n0 = (warp & 3) * 16, kh = (warp >> 2) * 32;
    float dw2[4][4] = {}, dw3[4][4] = {}, dw1[1][4] = {}, dw4[1][4] = {}, lsum = 0.f;
    const int r0 = warp * 16;
    // bias gradients: one thread per column and block of rows; warps 0-3 those of the
    // hidden layers, warp 4 the output's
    static_assert(kMlpTrainRows / kMlpSumRows == 2 && kMlpHid == 64 && kMlpOutPad == 16, "threads of the bias gradients");
    float db1 = 0.f, db2 = 0.f, db3 = 0.f, db4 = 0.f;
    const bool sums_h = tid < 2 * kMlpHid, sums_o = warp == 4;
    const int hid = (tid >> 6 & 1) * kMlpSumRows * kMwHid + (tid & 63);
    const int outp = (tid >> 4 & 1) * kMlpSumRows * kMlpOutPad + (tid & 15);
    for (long long row0 = (long long)blockIdx.x * kMlpTrainRows; row0 < n_rows; row0 += (long long)gridDim.x * kMlpTrainRows) {
        __syncthreads();  // the last tile's fragments have been read (first tile: nothing)
        if (tid < kMlpTrainRows) {
            const long long gr = row0 + tid;
            float in[kMlpIn], tg[kMlpOut];
            const bool valid = gr < n_rows;
            if (valid) {
                const unsigned u = (unsigned)gr;
                const long long p = in_order ? gr
                                             : (long long)((((unsigned long long)hash_u32(seed ^ hash_u32(u)) << 20) ^
                                                            hash_u32(u * 2654435761u + seed)) % (unsigned long long)n_pairs);
                float pr[20];
#pragma unroll
                for (int q = 0; q < 5; ++q) {  // rows of 80 bytes, 16-byte aligned
                    const float4 f = reinterpret_cast<const float4*>(pairs + p * 20)[q];
                    pr[4 * q] = f.x; pr[4 * q + 1] = f.y; pr[4 * q + 2] = f.z; pr[4 * q + 3] = f.w;
                }
                mlp_features(pr, pr[9], N, in);
                mlp_targets(pr, N, tg);
            }
#pragma unroll
            for (int k = 0; k < kMlpInPad; k += 2)
                *reinterpret_cast<uint32_t*>(S.x0 + tid * kMwIn + k) =
                    pack_f2_bf16(valid && k < kMlpIn ? in[k < kMlpIn ? k : 0] : 0.f,
                                 valid && k + 1 < kMlpIn ? in[k + 1 < kMlpIn ? k + 1 : 0] : 0.f);
#pragma unroll
            for (int k = 0; k < kMlpOutPad; ++k) S.tgt[tid * kMlpOutPad + k] = valid && k < kMlpOut ? tg[k < kMlpOut ? k : 0] : 0.f;
        }
        __syncthreads();
        uint32_t a[kMlpHid / 16][4];
        float acc[kMlpHid / 8][4], gp1[kMlpHid / 8][4], gp2[kMlpHid / 8][4], gp3[kMlpHid / 8][4];
        const __nv_bfloat16* X = S.x0 + r0 * kMwIn;
        a[0][0] = *reinterpret_cast<const uint32_t*>(X + g * kMwIn + 2 * t);
        a[0][1] = *reinterpret_cast<const uint32_t*>(X + (g + 8) * kMwIn + 2 * t);
        a[0][2] = *reinterpret_cast<const uint32_t*>(X + g * kMwIn + 2 * t + 8);
        a[0][3] = *reinterpret_cast<const uint32_t*>(X + (g + 8) * kMwIn + 2 * t + 8);
        mlp_warp_layer<1, kMlpHid / 8>(a, S.W1, kMwIn, acc);
        mlp_train_activate(acc, S.b1, a, gp1, S.h[0], r0);
        mlp_warp_layer<kMlpHid / 16, kMlpHid / 8>(a, S.W2, kMwHid, acc);
        mlp_train_activate(acc, S.b2, a, gp2, S.h[1], r0);
        mlp_warp_layer<kMlpHid / 16, kMlpHid / 8>(a, S.W3, kMwHid, acc);
        mlp_train_activate(acc, S.b3, a, gp3, S.h[2], r0);
        float o[kMlpOutPad / 8][4];
        mlp_warp_layer<kMlpHid / 16, kMlpOutPad / 8>(a, S.W4, kMwHid, o);
        // loss and dL/dY4 (mean over all rows of the launch)
#pragma unroll
        for (int j = 0; j < kMlpOutPad / 8; ++j) {
            const int c = j * 8 + 2 * t;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = r0 + g + (q & 2 ? 8 : 0), cc = c + (q & 1);
                const bool valid = row0 + r < n_rows && cc < kMlpOut;
                const float diff = valid ? o[j][q] + S.b4[cc] - S.tgt[r * kMlpOutPad + cc] : 0.f;
                lsum += diff * diff;
                o[j][q] = 2.f * diff / float(n_rows);
                S.tgt[r * kMlpOutPad + cc] = o[j][q];
            }
            const uint32_t lo = pack_f2_bf16(o[j][0], o[j][1]), hi = pack_f2_bf16(o[j][2], o[j][3]);
            a[0][2 * j] = lo;
            a[0][2 * j + 1] = hi;
            *reinterpret_cast<uint32_t*>(S.dy4 + (r0 + g) * kMwIn + c) = lo;
            *reinterpret_cast<uint32_t*>(S.dy4 + (r0 + g + 8) * kMwIn + c) = hi;
        }
        mlp_warp_layer<1, kMlpHid / 8>(a, S.W4t, kMwIn, acc);  // dX = dY4 W4
        mlp_train_back(acc, gp3, a, S.dy, r0);
        __syncthreads();
        mlp_train_dw<1>(S.dy4, kMwIn, S.h[2], kMwHid, 0, warp * 8, dw4);
        mlp_train_dw<4>(S.dy, kMwHid, S.h[1], kMwHid, n0, kh, dw3);
        if (sums_h) db3 += mlp_train_db(S.dy + hid, kMwHid);
        if (sums_o) db4 += mlp_train_db(S.tgt + outp, kMlpOutPad);
        mlp_warp_layer<kMlpHid / 16, kMlpHid / 8>(a, S.W3t, kMwHid, acc);
        __syncthreads();  // dY3 has been read
        mlp_train_back(acc, gp2, a, S.dy, r0);
        __syncthreads();
        mlp_train_dw<4>(S.dy, kMwHid, S.h[0], kMwHid, n0, kh, dw2);
        if (sums_h) db2 += mlp_train_db(S.dy + hid, kMwHid);
        mlp_warp_layer<kMlpHid / 16, kMlpHid / 8>(a, S.W2t, kMwHid, acc);
        __syncthreads();
        mlp_train_back(acc, gp1, a, S.dy, r0);
        __syncthreads();
        mlp_train_dw<1>(S.dy, kMwHid, S.x0, kMwIn, n0, (warp >> 2) * 8, dw1);
        if (sums_h) db1 += mlp_train_db(S.dy + hid, kMwHid);
    }
    // this CTA's row of `part` (every entry written)
    float* P = part + (long long)blockIdx.x * kMlpPart;
    auto put = [&](float* dst, int ld, const float* v) {  // an m16n8 tile
        *reinterpret_cast<float2*>(dst + g * ld + 2 * t) = make_float2(v[0], v[1]);
        *reinterpret_cast<float2*>(dst + (g + 8) * ld + 2 * t) = make_float2(v[2], v[3]);
    };
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        put(P + MlpOff::W2 + n0 * kMlpHid + kh + j * 8, kMlpHid, dw2[j]);
        put(P + MlpOff::W3 + n0 * kMlpHid + kh + j * 8, kMlpHid, dw3[j]);
    }
    put(P + MlpOff::W1 + n0 * kMlpInPad + (warp >> 2) * 8, kMlpInPad, dw1[0]);
    put(P + MlpOff::W4 + warp * 8, kMlpHid, dw4[0]);
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, m);
    if (lane == 0) S.red[warp] = lsum;
    if (sums_h) {
        float* d = S.db[tid >> 6] + (tid & 63);
        d[0] = db1;
        d[kMlpHid] = db2;
        d[2 * kMlpHid] = db3;
    }
    if (sums_o) S.db[tid >> 4 & 1][3 * kMlpHid + (tid & 15)] = db4;
    __syncthreads();
    if (tid < 3 * kMlpHid + kMlpOutPad) {
        const int l = tid >> 6;  // layer: 0-2 hidden, 3 output
        P[(l == 0 ? MlpOff::b1 : l == 1 ? MlpOff::b2 : l == 2 ? MlpOff::b3 : MlpOff::b4) + (tid & 63)] = S.db[0][tid] + S.db[1][tid];
    }
    if (tid == 0) {
        float s = 0.f;
        for (int w = 0; w < 8; ++w) s += S.red[w];
        P[MlpOff::total] = s;
    }
}

// Sum of entry i over the CTAs' rows of `part` in FP64, by the four threads q =
// 0..3 of a quad group 64 threads apart in the block: rows q, q + 4, ... each, then
// the four. `s` holds 256 doubles.
__device__ __forceinline__ float mlp_part_sum(const float* __restrict__ part, int ctas, int i, double* s) {
    const int q = threadIdx.x >> 6;
    double v = 0.0;
    if (i < kMlpPart) {
#pragma unroll 8
        for (int c = q; c < ctas; c += 4) v += part[(long long)c * kMlpPart + i];
    }
    s[threadIdx.x] = v;
    __syncthreads();
    return q == 0 ? float(((v + s[threadIdx.x + 64]) + s[threadIdx.x + 128]) + s[threadIdx.x + 192]) : 0.f;
}

// The summed gradient (and loss) of a training launch, without an update.
__global__ void __launch_bounds__(256) k_mlp_grad_sum(const float* __restrict__ part, int ctas, float* __restrict__ grad,
                                                      float* __restrict__ loss) {
    __shared__ double s[256];
    const int i = blockIdx.x * 64 + (threadIdx.x & 63);
    const float v = mlp_part_sum(part, ctas, i, s);
    if (threadIdx.x >= 64) return;
    if (i < MlpOff::total) grad[i] = v;
    else if (i == MlpOff::total) *loss = v;
}

// AdamW on the fp32 master weights from the summed gradients of the step's
// CTAs; refreshes the bf16 copy, stores the step's loss. Padded entries (input
// columns >= 10 of W1, output rows >= 10 of W4 and b4) stay zero. 64 parameters a
// block, four threads each.
__global__ void __launch_bounds__(256) k_mlp_adam(float* __restrict__ w, __nv_bfloat16* __restrict__ wbf,
                                                  const float* __restrict__ part, int ctas, float* __restrict__ m1,
                                                  float* __restrict__ m2, float* __restrict__ loss, float lr, float beta1,
                                                  float beta2, float eps, float wd, float bc1, float bc2) {
    __shared__ double s[256];
    const int i = blockIdx.x * 64 + (threadIdx.x & 63);
    const float gr = mlp_part_sum(part, ctas, i, s);
    if (threadIdx.x >= 64) return;
    if (i >= MlpOff::total) {
        if (i == MlpOff::total) *loss = gr;
        return;
    }
    bool pad = false;
    if (i < MlpOff::b1) pad = (i % kMlpInPad) >= kMlpIn;
    else if (i >= MlpOff::W4 && i < MlpOff::b4) pad = (i - MlpOff::W4) / kMlpHid >= kMlpOut;
    else if (i >= MlpOff::b4) pad = (i - MlpOff::b4) >= kMlpOut;
    if (pad) { w[i] = 0.f; wbf[i] = __float2bfloat16_rn(0.f); return; }
    const bool is_bias = (i >= MlpOff::b1 && i < MlpOff::W2) || (i >= MlpOff::b2 && i < MlpOff::W3) ||
                         (i >= MlpOff::b3 && i < MlpOff::W4) || i >= MlpOff::b4;
    const float a = beta1 * m1[i] + (1.f - beta1) * gr;
    const float b = beta2 * m2[i] + (1.f - beta2) * gr * gr;
    m1[i] = a;
    m2[i] = b;
    float x = w[i];
    if (!is_bias) x -= lr * wd * x;
    x -= lr * (a / bc1) / (sqrtf(b / bc2) + eps);
    w[i] = x;
    wbf[i] = __float2bfloat16_rn(x);
}

}  // namespace mpm
