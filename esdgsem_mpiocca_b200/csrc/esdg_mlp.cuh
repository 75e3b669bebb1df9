// Learned troubled-cell indicator: an MLP (F -> 32 -> 32 -> 1, ReLU) on
// per-element features, BF16 weights and activations on the tensor cores
// (warp-level bf16 MMA with FP32 accumulation), FP32 master weights and
// Adam.  It predicts the modal shock sensor's sigma = log10(energy ratio)
// (okl/ShockCapturing/ShockCapturing.okl:131-204).  No counterpart in the
// reference.
//
// Features of one element (row of X, bf16, KP columns, zero padded), for
// the fields f = eta (= h + b, what the sensor sees), hu, hv over the n^2
// nodes:
//   x[f*n^2 + p] = (v_fp - mean_f) / rms_f        (0 when rms_f <= 1e-12 |mean_f|)
//   x[3 n^2 + f] = s_f / 4,  s_f = log10(rms_f^2 / (mean_f^2 + rms_f^2))
//                  clamped to [-12, 0]
// (rms_f is the RMS of the deviation from the mean).  The network output y
// is the scale-free part: sigma_hat = y + s_eta.  Training targets are
// t = clamp(sigma, -12, 0) - s_eta.
//
// The GEMMs are 16-row tiles per warp (K = KP, N = 32): the network's work
// is a few thousand MACs per element, well below the cost of reading the
// element's state, so warp-level MMA suffices; no tile is large enough for
// a CTA-wide tensor-memory pipeline to pay.
#pragma once

#include <cuda_bf16.h>
#include <mma.h>

#include "esdg_pdl.cuh"

namespace esdg {

constexpr int MLP_H = 32;
constexpr double MLP_S_MIN = -12.0;
constexpr double MLP_REL_FLAT = 1e-12;  // rms / |mean| below this: no shape features

__host__ __device__ constexpr int mlp_nin(int ngl) { return 3 * ngl * ngl + 3; }
__host__ __device__ constexpr int mlp_kp(int ngl) { return (mlp_nin(ngl) + 15) / 16 * 16; }

// Parameter block (floats): W1[32][KP] (padding columns unused, kept 0),
// b1[32], W2[32][32], b2[32], w3[32], b3, pad to a multiple of 4.
struct MlpLayout {
    int kp, w1, b1, w2, b2, w3, b3, total;
};
__host__ __device__ inline MlpLayout mlp_layout(int ngl) {
    MlpLayout L;
    L.kp = mlp_kp(ngl);
    L.w1 = 0;
    L.b1 = L.w1 + MLP_H * L.kp;
    L.w2 = L.b1 + MLP_H;
    L.b2 = L.w2 + MLP_H * MLP_H;
    L.w3 = L.b2 + MLP_H;
    L.b3 = L.w3 + MLP_H;
    L.total = (L.b3 + 1 + 3) / 4 * 4;
    return L;
}

// Modal sensor value sigma of one element: log10 of the larger of the two
// energy ratios (okl/ShockCapturing/ShockCapturing.okl:131-204), -inf when
// the modal energy n1 is below ZeroTOL (then *tiny is set).  By a warp: m =
// nodal (h + b) [eta][xi], V, and room for the two products in shared memory;
// an entry per lane, and the four order-dependent sums on a lane each, in the
// reference's order.  Valid on lane 0.
template <int NGL>
__device__ __forceinline__ double sensor_sigma(double ZeroTOL, const double* m, const double* V, double* M1, double* w,
                                               bool* tiny) {
    constexpr int N = NGL - 1, N2 = NGL * NGL;
    const int lane = threadIdx.x & 31;
    for (int p = lane; p < N2; p += 32) {
        const int i = p / NGL, j = p % NGL;
        double acc = 0.0;
        for (int l = 0; l < NGL; ++l) acc += V[i * NGL + l] * m[j * NGL + l];
        M1[p] = acc;
    }
    __syncwarp();
    for (int p = lane; p < N2; p += 32) {
        const int i = p / NGL, j = p % NGL;
        double acc = 0.0;
        for (int l = 0; l < NGL; ++l) acc += M1[i * NGL + l] * V[j * NGL + l];
        w[p] = acc;
    }
    __syncwarp();
    double s = 0.0;
    if (lane < 2) {  // z1 and z2: the two highest modes' rows and columns
        const int n = N - lane;
        for (int i = 0; i < n; ++i) s += w[i * NGL + n] * w[i * NGL + n] + w[n * NGL + i] * w[n * NGL + i];
        s += w[n * NGL + n] * w[n * NGL + n];
    } else if (lane < 4) {  // n1 and n2: all modes, without the highest
        const int n = lane == 2 ? NGL : N;
        for (int i = 0; i < n; ++i)
            for (int j = 0; j < n; ++j) s += w[i * NGL + j] * w[i * NGL + j];
    }
    const double z1 = s, z2 = __shfl_sync(0xffffffffu, s, 1);
    const double n1 = __shfl_sync(0xffffffffu, s, 2), n2s = __shfl_sync(0xffffffffu, s, 3);
    const double t1 = (n1 < ZeroTOL) ? 0.0 : z1 / n1;
    const double t2 = (n1 < ZeroTOL) ? 0.0 : z2 / n2s;
    *tiny = n1 < ZeroTOL;
    return log10((t1 < t2) ? t2 : t1);
}

// Writes one element's feature row (bf16, KP columns) from the warp's
// register copy of the element (node p = lane + 32 k): mean, RMS of the
// deviation and s of the three fields, their butterflies side by side, and
// one log10 pass (lanes 0, 1, 2: a field each).  Returns s_eta on lane 0.
template <int NGL>
__device__ __forceinline__ double mlp_feature_row(const double (&v)[3][(NGL * NGL + 31) / 32],
                                                  __nv_bfloat16* __restrict__ xr) {
    constexpr int N2 = NGL * NGL, R = (N2 + 31) / 32, KP = mlp_kp(NGL);
    const int lane = threadIdx.x & 31;
    double mean[3], rms[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        mean[f] = 0.0;
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (lane + 32 * k < N2) mean[f] += v[f][k];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int f = 0; f < 3; ++f) mean[f] += __shfl_xor_sync(0xffffffffu, mean[f], off);
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        mean[f] = mean[f] / N2;
        rms[f] = 0.0;
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (lane + 32 * k < N2) rms[f] += (v[f][k] - mean[f]) * (v[f][k] - mean[f]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int f = 0; f < 3; ++f) rms[f] += __shfl_xor_sync(0xffffffffu, rms[f], off);
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        rms[f] = sqrt(rms[f] / N2);
        // a deviation at rounding level (constant field) is not a shape
        const double inv = (rms[f] > MLP_REL_FLAT * fabs(mean[f]) && rms[f] > 0.0) ? 1.0 / rms[f] : 0.0;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int p = lane + 32 * k;
            if (p < N2) xr[f * N2 + p] = __float2bfloat16((float)((v[f][k] - mean[f]) * inv));
        }
    }
    double s = MLP_S_MIN;
    if (lane < 3) {
        const double m = lane == 0 ? mean[0] : (lane == 1 ? mean[1] : mean[2]);
        const double r = lane == 0 ? rms[0] : (lane == 1 ? rms[1] : rms[2]);
        const double tot = m * m + r * r;
        if (tot > 0.0 && r > 0.0) s = fmax(log10(r * r / tot), MLP_S_MIN);
        xr[3 * N2 + lane] = __float2bfloat16((float)(0.25 * s));
    }
    for (int p = 3 * N2 + 3 + lane; p < KP; p += 32) xr[p] = __float2bfloat16(0.0f);
    return s;
}

// Feature rows of every element, and optionally the training target
// t = clamp(sigma, -12, 0) - s_eta (NaN where the modal energy is below
// ZeroTOL: sigma is then set by an absolute threshold that scale-free
// features cannot see) and s_eta.  One warp per element.
template <int NGL>
__global__ void __launch_bounds__(256) k_mlp_features(int K, const double* __restrict__ q, const double* __restrict__ B,
                                                      const double* __restrict__ Vinv, double ZeroTOL,
                                                      __nv_bfloat16* __restrict__ X, float* __restrict__ tgt,
                                                      float* __restrict__ seta) {
    constexpr int N2 = NGL * NGL, R = (N2 + 31) / 32, KP = mlp_kp(NGL);
    __shared__ double sV[N2];
    __shared__ double se[8][N2], sM1[8][N2], sW[8][N2];
    const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
    if (threadIdx.x < N2) sV[threadIdx.x] = Vinv[threadIdx.x];
    __syncthreads();
    const int e = blockIdx.x * 8 + w;
    if (e >= K) return;
    const double* qe = q + (long)e * 3 * N2;
    double v[3][R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int p = lane + 32 * k;
        v[0][k] = v[1][k] = v[2][k] = 0.0;
        if (p < N2) {
            v[0][k] = qe[p] + B[(long)e * N2 + p];
            v[1][k] = qe[p + N2];
            v[2][k] = qe[p + 2 * N2];
            se[w][p] = B[(long)e * N2 + p] + qe[p];
        }
    }
    const double s_eta = mlp_feature_row<NGL>(v, X + (long)e * KP);
    if (tgt) {
        __syncwarp();
        bool tiny = false;
        const double sg = sensor_sigma<NGL>(ZeroTOL, se[w], sV, sM1[w], sW[w], &tiny);
        if (lane == 0) {
            const double c = fmin(fmax(sg, MLP_S_MIN), 0.0);  // -inf -> -12
            tgt[e] = tiny ? __int_as_float(0x7fc00000) : (float)(c - s_eta);
            if (seta) seta[e] = (float)s_eta;
        }
    } else if (seta && lane == 0) {
        seta[e] = (float)s_eta;
    }
}

using namespace nvcuda;

// Row strides of the backward kernel's shared matrices (bf16 rows of KP and
// 32 columns, float rows of 32): eight bf16 or four floats past the row, so
// that the fragment loads of eight rows and the row walks of sixteen lanes
// fall on different banks.
template <int KP>
struct MlpPad {
    static constexpr int X = KP + 8, B = MLP_H + 8, Z = MLP_H + 4;
};

// One warp's forward pass on 16 rows held in shared memory (strides MlpPad):
// Z1 = X W1^T + b1, A1 = relu(Z1) (bf16), Z2 = A1 W2^T + b2 (float, left
// in z), y = relu(Z2) . w3 + b3 into y16[0..15].  b1, b2: the lane's entries.
template <int KP>
__device__ __forceinline__ void mlp_warp_forward(const __nv_bfloat16* Xrows, const __nv_bfloat16* W1b,
                                                 const __nv_bfloat16* W2b, const float* __restrict__ sw3, float b1,
                                                 float b2, float b3, __nv_bfloat16* a1b, float* z, float* y16) {
    using S = MlpPad<KP>;
    const int lane = threadIdx.x & 31;
    wmma::fragment<wmma::accumulator, 16, 16, 16, float> acc[2];
    wmma::fragment<wmma::matrix_a, 16, 16, 16, __nv_bfloat16, wmma::row_major> fa;
    wmma::fragment<wmma::matrix_b, 16, 16, 16, __nv_bfloat16, wmma::col_major> fb;
#pragma unroll
    for (int n = 0; n < 2; ++n) wmma::fill_fragment(acc[n], 0.0f);
#pragma unroll
    for (int k = 0; k < KP / 16; ++k) {
        wmma::load_matrix_sync(fa, Xrows + k * 16, S::X);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            wmma::load_matrix_sync(fb, W1b + n * 16 * S::X + k * 16, S::X);  // B(k, n) = W1[n][k]
            wmma::mma_sync(acc[n], fa, fb, acc[n]);
        }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) wmma::store_matrix_sync(z + n * 16, acc[n], S::Z, wmma::mem_row_major);
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 16; ++r) a1b[r * S::B + lane] = __float2bfloat16(fmaxf(z[r * S::Z + lane] + b1, 0.0f));
    __syncwarp();
#pragma unroll
    for (int n = 0; n < 2; ++n) wmma::fill_fragment(acc[n], 0.0f);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        wmma::load_matrix_sync(fa, a1b + k * 16, S::B);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            wmma::load_matrix_sync(fb, W2b + n * 16 * S::B + k * 16, S::B);
            wmma::mma_sync(acc[n], fa, fb, acc[n]);
        }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) wmma::store_matrix_sync(z + n * 16, acc[n], S::Z, wmma::mem_row_major);
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 16; ++r) z[r * S::Z + lane] += b2;
    __syncwarp();
    if (lane < 16) {
        float s = b3;
#pragma unroll
        for (int j = 0; j < 32; ++j) s += fmaxf(z[lane * S::Z + j], 0.0f) * sw3[j];
        y16[lane] = s;
    }
    __syncwarp();
}

// ---------------------------------------------------------------------------
// Forward pass on registers: mma.sync.m16n8k16 (BF16 in, FP32 accumulate)
// with the PTX ISA fragment layouts -- lane = 4 g + t; A (16x16, row):
// a0 (g, 2t..2t+1), a1 (g+8, 2t..), a2 (g, 2t+8..), a3 (g+8, 2t+8..);
// B (16x8, col): b0 (k 2t..2t+1, n g), b1 (k 2t+8..2t+9, n g);
// C (16x8): c0,c1 (g, 2t..2t+1), c2,c3 (g+8, 2t..2t+1).  Layer-1 outputs
// of two adjacent n8 tiles form the layer-2 A fragment of one k16 block, so
// bias, ReLU and the BF16 packing stay in registers; the 32 -> 1 layer is a
// per-lane partial dot product reduced over the four lanes of a quad.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned mlp_pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);  // .x = lo (low half)
    return *reinterpret_cast<const unsigned*>(&v);
}

__device__ __forceinline__ void mlp_mma16816(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                             unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The FP32 vectors a lane needs (biases and w3 at its fragment columns
// 8 j + 2 t, 8 j + 2 t + 1), loaded once per warp.
struct MlpLaneParams {
    float b1[8], b2[8], w3[8], b3;
};

__device__ __forceinline__ MlpLaneParams mlp_lane_params(const float* __restrict__ P, const MlpLayout& L) {
    MlpLaneParams r;
    const int t = threadIdx.x & 3;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            r.b1[2 * j + k] = P[L.b1 + 8 * j + 2 * t + k];
            r.b2[2 * j + k] = P[L.b2 + 8 * j + 2 * t + k];
            r.w3[2 * j + k] = P[L.w3 + 8 * j + 2 * t + k];
        }
    r.b3 = P[L.b3];
    return r;
}

// y for the 16 rows of X (bf16, shared, ld KP): lanes with t == 0 hold
// y[g] in y_lo and y[g + 8] in y_hi (every lane of the quad has them).
// W1 [32][KP], W2 [32][32] bf16 in shared memory.
template <int KP>
__device__ __forceinline__ void mlp_warp_forward_regs(const __nv_bfloat16* X, const __nv_bfloat16* W1,
                                                      const __nv_bfloat16* W2, const MlpLaneParams& R,
                                                      float& y_lo, float& y_hi) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const unsigned* Xu = reinterpret_cast<const unsigned*>(X);    // pairs of bf16
    const unsigned* W1u = reinterpret_cast<const unsigned*>(W1);
    const unsigned* W2u = reinterpret_cast<const unsigned*>(W2);
    float acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float b0 = R.b1[2 * j], b1v = R.b1[2 * j + 1];
        acc[j][0] = b0; acc[j][1] = b1v; acc[j][2] = b0; acc[j][3] = b1v;
    }
#pragma unroll
    for (int kb = 0; kb < KP / 16; ++kb) {
        const int c = kb * 8 + t;  // column pair index (2 bf16 per unsigned)
        const unsigned a0 = Xu[g * (KP / 2) + c], a1 = Xu[(g + 8) * (KP / 2) + c];
        const unsigned a2 = Xu[g * (KP / 2) + c + 4], a3 = Xu[(g + 8) * (KP / 2) + c + 4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = 8 * j + g;  // B(k, n) = W1[n][k]
            mlp_mma16816(acc[j], a0, a1, a2, a3, W1u[n * (KP / 2) + c], W1u[n * (KP / 2) + c + 4]);
        }
    }
    float acc2[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float b0 = R.b2[2 * j], b1v = R.b2[2 * j + 1];
        acc2[j][0] = b0; acc2[j][1] = b1v; acc2[j][2] = b0; acc2[j][3] = b1v;
    }
#pragma unroll
    for (int kb = 0; kb < 2; ++kb) {
        // A1 k16 block kb = layer-1 n8 tiles 2 kb and 2 kb + 1, after ReLU
        const int j0 = 2 * kb, j1 = 2 * kb + 1;
        const unsigned a0 = mlp_pack_bf16(fmaxf(acc[j0][0], 0.f), fmaxf(acc[j0][1], 0.f));
        const unsigned a1 = mlp_pack_bf16(fmaxf(acc[j0][2], 0.f), fmaxf(acc[j0][3], 0.f));
        const unsigned a2 = mlp_pack_bf16(fmaxf(acc[j1][0], 0.f), fmaxf(acc[j1][1], 0.f));
        const unsigned a3 = mlp_pack_bf16(fmaxf(acc[j1][2], 0.f), fmaxf(acc[j1][3], 0.f));
        const int c = kb * 8 + t;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = 8 * j + g;  // B(k, n) = W2[n][k]
            mlp_mma16816(acc2[j], a0, a1, a2, a3, W2u[n * 16 + c], W2u[n * 16 + c + 4]);
        }
    }
    float lo = 0.f, hi = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float w0 = R.w3[2 * j], w1 = R.w3[2 * j + 1];
        lo += fmaxf(acc2[j][0], 0.f) * w0 + fmaxf(acc2[j][1], 0.f) * w1;
        hi += fmaxf(acc2[j][2], 0.f) * w0 + fmaxf(acc2[j][3], 0.f) * w1;
    }
    lo += __shfl_xor_sync(0xffffffffu, lo, 1);
    lo += __shfl_xor_sync(0xffffffffu, lo, 2);
    hi += __shfl_xor_sync(0xffffffffu, hi, 1);
    hi += __shfl_xor_sync(0xffffffffu, hi, 2);
    y_lo = lo + R.b3;
    y_hi = hi + R.b3;
}

// The same forward pass for a warp that holds only R rows (R divides 8):
// row r of the 16-row MMA tile is row r % R of X, so a0 = a1 and a2 = a3,
// and every row's dot products are those mlp_warp_forward_regs forms for it
// in a full tile (the same operands, MMAs and FP32 additions, in the same
// order).  Biases and w3 come from shared memory (P32: b1, b2, w3 [32 each],
// b3), so a warp keeps no network parameters in registers between tiles.
// Lane 4 r holds y of row r (r < R).
// Row strides (bf16 elements): XS of X, W1S of W1 [32][W1S], W2S of W2
// [32][W2S]; strides of KP + 8 and 40 keep the fragment loads of a warp free
// of shared-memory bank conflicts.
template <int KP, int R, int XS = KP, int W1S = KP, int W2S = MLP_H>
__device__ __forceinline__ float mlp_warp_forward_rows(const __nv_bfloat16* X, const __nv_bfloat16* W1,
                                                       const __nv_bfloat16* W2, const float* P32) {
    static_assert(8 % R == 0, "rows per warp divide 8");
    static_assert(XS % 8 == 0 && W1S % 8 == 0 && W2S % 8 == 0, "16-byte rows");
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int row = g % R;
    const unsigned* Xu = reinterpret_cast<const unsigned*>(X);
    const unsigned* W1u = reinterpret_cast<const unsigned*>(W1);
    const unsigned* W2u = reinterpret_cast<const unsigned*>(W2);
    const float2* b1 = reinterpret_cast<const float2*>(P32);
    const float2* b2 = reinterpret_cast<const float2*>(P32 + MLP_H);
    const float2* w3 = reinterpret_cast<const float2*>(P32 + 2 * MLP_H);
    float acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 b = b1[4 * j + t];
        acc[j][0] = b.x; acc[j][1] = b.y; acc[j][2] = b.x; acc[j][3] = b.y;
    }
#pragma unroll
    for (int kb = 0; kb < KP / 16; ++kb) {
        const int c = kb * 8 + t;
        const unsigned a0 = Xu[row * (XS / 2) + c], a2 = Xu[row * (XS / 2) + c + 4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = 8 * j + g;
            mlp_mma16816(acc[j], a0, a0, a2, a2, W1u[n * (W1S / 2) + c], W1u[n * (W1S / 2) + c + 4]);
        }
    }
    float acc2[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 b = b2[4 * j + t];
        acc2[j][0] = b.x; acc2[j][1] = b.y; acc2[j][2] = b.x; acc2[j][3] = b.y;
    }
#pragma unroll
    for (int kb = 0; kb < 2; ++kb) {
        const int j0 = 2 * kb, j1 = 2 * kb + 1;
        const unsigned a0 = mlp_pack_bf16(fmaxf(acc[j0][0], 0.f), fmaxf(acc[j0][1], 0.f));
        const unsigned a2 = mlp_pack_bf16(fmaxf(acc[j1][0], 0.f), fmaxf(acc[j1][1], 0.f));
        const int c = kb * 8 + t;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = 8 * j + g;
            mlp_mma16816(acc2[j], a0, a0, a2, a2, W2u[n * (W2S / 2) + c], W2u[n * (W2S / 2) + c + 4]);
        }
    }
    float lo = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 w = w3[4 * j + t];
        lo += fmaxf(acc2[j][0], 0.f) * w.x + fmaxf(acc2[j][1], 0.f) * w.y;
    }
    lo += __shfl_xor_sync(0xffffffffu, lo, 1);
    lo += __shfl_xor_sync(0xffffffffu, lo, 2);
    return lo + P32[3 * MLP_H];
}

// Shared-memory carve-up of the MLP kernels (bytes).  Forward: the BF16
// weights once per block and an X tile per warp.  Backward: the weights and
// w3 once per block, then per warp X tile, A1 (bf16), Z (float), dZ2 and dZ1
// (bf16), scratch (float), y, in the strides of MlpPad.
template <int KP>
struct MlpSmem {
    using P = MlpPad<KP>;
    static constexpr int W1 = MLP_H * KP * 2, W2 = MLP_H * MLP_H * 2;
    static constexpr int XW = 16 * KP * 2;
    static constexpr int BW1 = MLP_H * P::X * 2, BW2 = MLP_H * P::B * 2, BW3 = MLP_H * 4;
    static constexpr int BX = 16 * P::X * 2, A1 = 16 * P::B * 2, Z = 16 * P::Z * 4, G = 16 * P::B * 2, Y = 16 * 4;
    static constexpr int PER_WARP = BX + A1 + Z + 2 * G + Z + Y;
    static constexpr int bytes(int warps) { return BW1 + BW2 + BW3 + warps * PER_WARP; }
    static constexpr int fwd_bytes(int warps) { return W1 + W2 + warps * XW; }
};

__global__ void k_mlp_cast(int n, const float* __restrict__ P, __nv_bfloat16* __restrict__ Pb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) Pb[i] = __float2bfloat16(P[i]);
}

__device__ __forceinline__ void mlp_stage_weights(int KP, const __nv_bfloat16* __restrict__ Pb, const MlpLayout& L,
                                                  __nv_bfloat16* sW1, __nv_bfloat16* sW2) {
    for (int i = threadIdx.x; i < MLP_H * KP; i += blockDim.x) sW1[i] = Pb[L.w1 + i];
    for (int i = threadIdx.x; i < MLP_H * MLP_H; i += blockDim.x) sW2[i] = Pb[L.w2 + i];
}

// Network output y for M rows.  4 warps per block, grid-stride over 16-row
// tiles; each warp holds its next tile in registers while it evaluates the
// current one.  Dynamic shared memory MlpSmem<KP>::fwd_bytes(4).
template <int KP>
__global__ void __launch_bounds__(128) k_mlp_forward(int M, const __nv_bfloat16* __restrict__ X,
                                                     const float* __restrict__ P,
                                                     const __nv_bfloat16* __restrict__ Pb, float* __restrict__ y,
                                                     MlpLayout L, const int* __restrict__ Mlive = nullptr) {
    pdl_wait();
    if (Mlive) M = min(M, *Mlive);  // rows past a live extent are skipped
    using S = MlpSmem<KP>;
    constexpr int VPR = KP / 8;        // 16-byte vectors per row
    constexpr int NV = 16 * VPR / 32;  // vectors per lane per tile
    extern __shared__ __align__(128) unsigned char mlp_smem[];
    __nv_bfloat16* sW1 = reinterpret_cast<__nv_bfloat16*>(mlp_smem);
    __nv_bfloat16* sW2 = reinterpret_cast<__nv_bfloat16*>(mlp_smem + S::W1);
    const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
    __nv_bfloat16* sX = reinterpret_cast<__nv_bfloat16*>(mlp_smem + S::W1 + S::W2 + w * S::XW);
    mlp_stage_weights(KP, Pb, L, sW1, sW2);
    __syncthreads();
    if (M <= 0) return;
    const int tiles = (M + 15) / 16;
    const int stride = gridDim.x * 4;
    auto fetch = [&](int t, uint4 (&buf)[NV]) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const int i = lane + 32 * k;
            const int r = min(t * 16 + i / VPR, M - 1);
            buf[k] = reinterpret_cast<const uint4*>(X + (long)r * KP)[i % VPR];
        }
    };
    const MlpLaneParams R = mlp_lane_params(P, L);
    uint4 buf[NV];
    int t = blockIdx.x * 4 + w;
    if (t < tiles) fetch(t, buf);
    for (; t < tiles; t += stride) {
#pragma unroll
        for (int k = 0; k < NV; ++k) reinterpret_cast<uint4*>(sX)[lane + 32 * k] = buf[k];
        __syncwarp();
        if (t + stride < tiles) fetch(t + stride, buf);  // in flight during this tile
        float ylo, yhi;
        mlp_warp_forward_regs<KP>(sX, sW1, sW2, R, ylo, yhi);
        const int g = lane >> 2, r0 = t * 16;
        if ((lane & 3) == 0) {
            if (r0 + g < M) y[r0 + g] = ylo;
            if (r0 + g + 8 < M) y[r0 + g + 8] = yhi;
        }
        __syncwarp();  // sX is rewritten next iteration
    }
}

// Gradient of the loss (1/M) sum (y - t)^2 over M rows.  Each warp
// accumulates over its tiles and writes one partial row of L.total floats
// to partial[(blockIdx.x * 4 + warp) * L.total]; slot b3 + 1 of the row
// holds the warp's sum of squared errors.  k_mlp_adam sums the rows in a
// fixed order, so training is deterministic.
template <int KP>
__global__ void __launch_bounds__(128) k_mlp_backward(int M, const __nv_bfloat16* __restrict__ X,
                                                      const float* __restrict__ tgt, const float* __restrict__ P,
                                                      const __nv_bfloat16* __restrict__ Pb,
                                                      float* __restrict__ partial, MlpLayout L) {
    using S = MlpSmem<KP>;
    extern __shared__ __align__(128) unsigned char mlp_smem[];
    __nv_bfloat16* sW1 = reinterpret_cast<__nv_bfloat16*>(mlp_smem);
    __nv_bfloat16* sW2 = reinterpret_cast<__nv_bfloat16*>(mlp_smem + S::BW1);
    float* sw3 = reinterpret_cast<float*>(mlp_smem + S::BW1 + S::BW2);
    const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
    unsigned char* mine = mlp_smem + S::BW1 + S::BW2 + S::BW3 + w * S::PER_WARP;
    __nv_bfloat16* sX = reinterpret_cast<__nv_bfloat16*>(mine);
    __nv_bfloat16* a1b = reinterpret_cast<__nv_bfloat16*>(mine + S::BX);
    float* z = reinterpret_cast<float*>(mine + S::BX + S::A1);
    __nv_bfloat16* g2b = reinterpret_cast<__nv_bfloat16*>(mine + S::BX + S::A1 + S::Z);
    __nv_bfloat16* g1b = reinterpret_cast<__nv_bfloat16*>(mine + S::BX + S::A1 + S::Z + S::G);
    float* scr = reinterpret_cast<float*>(mine + S::BX + S::A1 + S::Z + 2 * S::G);
    float* y16 = reinterpret_cast<float*>(mine + S::BX + S::A1 + S::Z + 2 * S::G + S::Z);
    constexpr int XS = MlpPad<KP>::X, BS = MlpPad<KP>::B, ZS = MlpPad<KP>::Z;
    for (int i = threadIdx.x; i < MLP_H * KP; i += blockDim.x) sW1[(i / KP) * XS + i % KP] = Pb[L.w1 + i];
    for (int i = threadIdx.x; i < MLP_H * MLP_H; i += blockDim.x) sW2[(i / MLP_H) * BS + i % MLP_H] = Pb[L.w2 + i];
    if (threadIdx.x < MLP_H) sw3[threadIdx.x] = P[L.w3 + threadIdx.x];
    __syncthreads();
    const float b1 = P[L.b1 + lane], b2 = P[L.b2 + lane], b3 = P[L.b3];
    // the next tile's rows and targets in registers while a tile is processed
    constexpr int VPR = KP / 8, NV = 16 * VPR / 32;
    uint4 buf[NV];
    float tnext = 0.f;
    auto fetch = [&](int t) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const int i = lane + 32 * k;
            const int r = min(t * 16 + i / VPR, M - 1);  // rows past M - 1 repeat the last one
            buf[k] = reinterpret_cast<const uint4*>(X + (long)r * KP)[i % VPR];
        }
        tnext = (lane < 16 && t * 16 + lane < M) ? tgt[t * 16 + lane] : 0.f;
    };
    const int tiles = (M + 15) / 16;
    const float scale = 2.0f / (float)M;
    wmma::fragment<wmma::accumulator, 16, 16, 16, float> gW2[2][2];
    wmma::fragment<wmma::accumulator, 16, 16, 16, float> gW1[2][KP / 16];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
#pragma unroll
        for (int b = 0; b < 2; ++b) wmma::fill_fragment(gW2[a][b], 0.0f);
#pragma unroll
        for (int b = 0; b < KP / 16; ++b) wmma::fill_fragment(gW1[a][b], 0.0f);
    }
    float gb1 = 0.f, gb2 = 0.f, gw3 = 0.f, gb3 = 0.f, l2 = 0.f;  // lane j: column j
    const float w3j = P[L.w3 + lane];
    if ((int)blockIdx.x * 4 + w < tiles) fetch(blockIdx.x * 4 + w);
    for (int t = blockIdx.x * 4 + w; t < tiles; t += gridDim.x * 4) {
        const int r0 = t * 16;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const int i = lane + 32 * k;
            *reinterpret_cast<uint4*>(sX + (i / VPR) * XS + (i % VPR) * 8) = buf[k];
        }
        const float tcur = tnext;
        __syncwarp();
        if (t + (int)gridDim.x * 4 < tiles) fetch(t + gridDim.x * 4);
        mlp_warp_forward<KP>(sX, sW1, sW2, sw3, b1, b2, b3, a1b, z, y16);  // z = Z2
        float dy = 0.f;
        if (lane < 16 && r0 + lane < M) {
            const float e = y16[lane] - tcur;
            dy = scale * e;
            l2 += e * e;
        }
        // dZ2 = dy w3 where Z2 > 0; column sums for b2, w3, b3
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const float dyr = __shfl_sync(0xffffffffu, dy, r);
            const float zz = z[r * ZS + lane];
            gw3 += dyr * fmaxf(zz, 0.f);
            const float g = (zz > 0.f) ? dyr * w3j : 0.f;
            gb2 += g;
            g2b[r * BS + lane] = __float2bfloat16(g);
            gb3 += (lane == 0) ? dyr : 0.f;
        }
        __syncwarp();
        // gW2 += dZ2^T A1: A(m=j, k=r) = dZ2[r][j] (col-major), B(k=r, n=i) = A1[r][i] (row-major)
        {
            wmma::fragment<wmma::matrix_a, 16, 16, 16, __nv_bfloat16, wmma::col_major> fa;
            wmma::fragment<wmma::matrix_b, 16, 16, 16, __nv_bfloat16, wmma::row_major> fb;
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                wmma::load_matrix_sync(fa, g2b + a * 16, BS);
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    wmma::load_matrix_sync(fb, a1b + b * 16, BS);
                    wmma::mma_sync(gW2[a][b], fa, fb, gW2[a][b]);
                }
            }
        }
        // dA1 = dZ2 W2: A = dZ2 (row-major), B(k=j, n=i) = W2[j][i] (row-major)
        {
            wmma::fragment<wmma::matrix_a, 16, 16, 16, __nv_bfloat16, wmma::row_major> fa;
            wmma::fragment<wmma::matrix_b, 16, 16, 16, __nv_bfloat16, wmma::row_major> fb;
            wmma::fragment<wmma::accumulator, 16, 16, 16, float> acc[2];
#pragma unroll
            for (int n = 0; n < 2; ++n) wmma::fill_fragment(acc[n], 0.f);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                wmma::load_matrix_sync(fa, g2b + k * 16, BS);
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    wmma::load_matrix_sync(fb, sW2 + k * 16 * BS + n * 16, BS);
                    wmma::mma_sync(acc[n], fa, fb, acc[n]);
                }
            }
#pragma unroll
            for (int n = 0; n < 2; ++n) wmma::store_matrix_sync(scr + n * 16, acc[n], ZS, wmma::mem_row_major);
        }
        __syncwarp();
        // dZ1 = dA1 where A1 > 0
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const float g = (__bfloat162float(a1b[r * BS + lane]) > 0.f) ? scr[r * ZS + lane] : 0.f;
            gb1 += g;
            g1b[r * BS + lane] = __float2bfloat16(g);
        }
        __syncwarp();
        // gW1 += dZ1^T X: A(m=j, k=r) = dZ1[r][j] (col-major), B(k=r, n=c) = X[r][c] (row-major)
        {
            wmma::fragment<wmma::matrix_a, 16, 16, 16, __nv_bfloat16, wmma::col_major> fa;
            wmma::fragment<wmma::matrix_b, 16, 16, 16, __nv_bfloat16, wmma::row_major> fb;
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                wmma::load_matrix_sync(fa, g1b + a * 16, BS);
#pragma unroll
                for (int b = 0; b < KP / 16; ++b) {
                    wmma::load_matrix_sync(fb, sX + b * 16, XS);
                    wmma::mma_sync(gW1[a][b], fa, fb, gW1[a][b]);
                }
            }
        }
        __syncwarp();
    }
    float* out = partial + (long)(blockIdx.x * 4 + w) * L.total;
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            wmma::store_matrix_sync(scr, gW2[a][b], 16, wmma::mem_row_major);
            __syncwarp();
            for (int i = lane; i < 256; i += 32) out[L.w2 + (a * 16 + i / 16) * 32 + b * 16 + i % 16] = scr[i];
            __syncwarp();
        }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < KP / 16; ++b) {
            wmma::store_matrix_sync(scr, gW1[a][b], 16, wmma::mem_row_major);
            __syncwarp();
            for (int i = lane; i < 256; i += 32) out[L.w1 + (a * 16 + i / 16) * KP + b * 16 + i % 16] = scr[i];
            __syncwarp();
        }
    out[L.b1 + lane] = gb1;
    out[L.b2 + lane] = gb2;
    out[L.w3 + lane] = gw3;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        l2 += __shfl_xor_sync(0xffffffffu, l2, off);
        gb3 += __shfl_xor_sync(0xffffffffu, gb3, off);
    }
    if (lane == 0) {
        out[L.b3] = gb3;
        out[L.b3 + 1] = l2;
        if (L.b3 + 2 < L.total) out[L.b3 + 2] = 0.f;
        if (L.b3 + 3 < L.total) out[L.b3 + 3] = 0.f;
    }
}

// Sums the R partial rows (fixed order) into G and applies one Adam step
// (Kingma & Ba 2015) to the FP32 master weights, refreshing the BF16 copy;
// c1 = 1 - b1^step, c2 = 1 - b2^step.  Padding columns of W1 and the slots
// past b3 are not updated (slot b3 + 1 of G is the summed squared error).
// A block takes ADAM_COLS columns and stages ADAM_ROWS of their rows at a
// time with all its threads, so the loads of a stage are in flight together
// and the additions, in row order, read shared memory (one thread a column
// walking the rows in global memory waited on 256 of them: 11.5 us at 256
// rows).
constexpr int ADAM_COLS = 32, ADAM_ROWS = 128;

__global__ void __launch_bounds__(256) k_mlp_adam(MlpLayout L, int nin, int R, const float* __restrict__ partial,
                                                  float* __restrict__ G, float* P, __nv_bfloat16* Pb, float* m,
                                                  float* v, float lr, float b1, float b2, float eps, float c1,
                                                  float c2) {
    __shared__ float sP[ADAM_ROWS][ADAM_COLS];
    const int c0 = blockIdx.x * ADAM_COLS, tid = threadIdx.x;
    const int col = tid % ADAM_COLS, row = tid / ADAM_COLS;
    float g = 0.f;
    for (int r0 = 0; r0 < R; r0 += ADAM_ROWS) {
        float x[ADAM_ROWS * ADAM_COLS / 256];
#pragma unroll
        for (int k = 0; k < ADAM_ROWS * ADAM_COLS / 256; ++k) {
            const int r = r0 + row + k * (256 / ADAM_COLS);
            x[k] = (r < R && c0 + col < L.total) ? partial[(long)r * L.total + c0 + col] : 0.f;
        }
#pragma unroll
        for (int k = 0; k < ADAM_ROWS * ADAM_COLS / 256; ++k) sP[row + k * (256 / ADAM_COLS)][col] = x[k];
        __syncthreads();
        if (tid < ADAM_COLS) {
            const int n = min(ADAM_ROWS, R - r0);
            if (n == ADAM_ROWS) {
#pragma unroll 32
                for (int r = 0; r < ADAM_ROWS; ++r) g += sP[r][tid];
            } else {
                for (int r = 0; r < n; ++r) g += sP[r][tid];
            }
        }
        __syncthreads();
    }
    const int i = c0 + tid;
    if (tid >= ADAM_COLS || i >= L.total) return;
    G[i] = g;
    const bool pad = (i < L.b1 && (i % L.kp) >= nin) || i > L.b3;
    if (pad) return;
    const float mi = b1 * m[i] + (1.f - b1) * g;
    const float vi = b2 * v[i] + (1.f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float p = P[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    P[i] = p;
    Pb[i] = __float2bfloat16(p);
}

}  // namespace esdg
