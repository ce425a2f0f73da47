// The learned eddy-viscosity closure (a project extension; the reference has none).
//
//   * training data: the "nCon" velocities of a (fine) context, 3 x 3 x 3 box-filtered on the
//     device, give per sampled cell 10 features of the filtered velocity gradient and the
//     least-squares eddy viscosity of the filtered-out stress as the target;
//   * network: 10 -> 32 (GELU) -> 32 (GELU) -> 1 (softplus) = nu_t / nu, BF16 weights, FP32
//     accumulation; trained by the kernels here (the layers' products over a tile of samples as
//     BF16 tensor-core multiplies with two-term BF16 operands, tile-wise fixed-order gradient
//     sums, Adam on FP32 master weights);
//   * inference: nu_t of every cell of a (coarse) FP32 context before its stress, which then
//     uses nu + nu_t averaged to each face.
// Definitions (filter, features, target, network) are restated in numpy in oracle/closure.py.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/ark_gpu.h"
#include "ark_check.cuh"
#include "ark_kernels.cuh" // qdiv
#include "ark_state.h"

namespace ark {
namespace cl {

constexpr int NIN = 10, NH = 32;
constexpr int NPARAM = NH * NIN + NH + NH * NH + NH + NH + 1; // 1441
constexpr int O_W1 = 0, O_B1 = O_W1 + NH * NIN, O_W2 = O_B1 + NH, O_B2 = O_W2 + NH * NH, O_W3 = O_B2 + NH,
              O_B3 = O_W3 + NH;
static_assert(O_B3 + 1 == NPARAM, "parameter layout");

// ---- network ------------------------------------------------------------------------------

// GELU in its tanh form, z (1 + tanh(k0 (z + k1 z^3))) / 2 (accurate tanhf; with its derivative, for
// training: gelu_both)
constexpr float GK0 = 0.79788456080286536f, GK1 = 0.044715f;
__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + tanhf(GK0 * (z + GK1 * z * z * z))); }
// inference: the same form with the hardware tanh approximation (relative error below 2^-10)
__device__ __forceinline__ float tanh_approx(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float gelu_fast(float z) { return 0.5f * z * (1.0f + tanh_approx(GK0 * (z + GK1 * z * z * z))); }
__device__ __forceinline__ float softplus(float z) { return fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z))); }
__device__ __forceinline__ float sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }

// Network constants as the kernels read them: weights (BF16 values held as float), input
// normalisation.
struct Net {
    float w[NPARAM];
    float mu[NIN], rsd[NIN];
};

// nu_t / nu of one normalised input (w: the parameters, in shared memory)
__device__ __forceinline__ float mlp_forward(const float *w, const float xn[NIN]) {
    float h1[NH];
#pragma unroll 4
    for (int k = 0; k < NH; ++k) {
        float z = w[O_B1 + k];
#pragma unroll
        for (int i = 0; i < NIN; ++i) z += w[O_W1 + k * NIN + i] * xn[i];
        h1[k] = gelu(z);
    }
    float z3 = w[O_B3];
#pragma unroll 2
    for (int k = 0; k < NH; ++k) {
        float z = w[O_B2 + k];
#pragma unroll
        for (int m = 0; m < NH; ++m) z += w[O_W2 + k * NH + m] * h1[m];
        z3 += w[O_W3 + k] * gelu(z);
    }
    return softplus(z3);
}

// ---- tensor-core inference ----------------------------------------------------------------
// A warp evaluates 32 inputs at once with warp-level BF16 matrix multiply-accumulate
// (m16n8k16, FP32 accumulation): layer 1 is [16 x 16] x [16 x 32] per half-warp tile (inputs
// padded from 10 to 16), layer 2 [16 x 32] x [32 x 32]; the FP32 accumulator fragment of a
// layer, after bias and GELU, is in exactly the register layout of the next layer's A fragment
// (rows = inputs, columns = units), packed to BF16 pairs.  Layer 3 (32 -> 1) is a dot product
// reduced over the four threads of a quad.  Activations enter the multiplies as BF16.

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned *>(&v);
}
__device__ __forceinline__ void mma_bf16(float c[4], const unsigned a[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The B fragments of a thread (lane = 4 g + t): layer 1 n-tile j: W1 rows 8j+g, inputs 2t, 2t+1
// and 2t+8, 2t+9 (inputs >= 10 are zero); layer 2 n-tile j, k-step s: W2 row 8j+g, inputs
// 16s+2t(+1), 16s+2t+8(+9).
struct TcWeights {
    unsigned b1[4][2], b2[4][2][2];
};
__device__ __forceinline__ TcWeights tc_weights(const float *w, int lane) {
    const int g = lane >> 2, t = lane & 3;
    TcWeights r;
    auto w1 = [&](int n, int k) { return k < NIN ? w[O_W1 + n * NIN + k] : 0.f; };
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int n = 8 * j + g;
        r.b1[j][0] = pack_bf16(w1(n, 2 * t), w1(n, 2 * t + 1));
        r.b1[j][1] = pack_bf16(w1(n, 2 * t + 8), w1(n, 2 * t + 9));
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            r.b2[j][s][0] = pack_bf16(w[O_W2 + n * NH + 16 * s + 2 * t], w[O_W2 + n * NH + 16 * s + 2 * t + 1]);
            r.b2[j][s][1] = pack_bf16(w[O_W2 + n * NH + 16 * s + 2 * t + 8], w[O_W2 + n * NH + 16 * s + 2 * t + 9]);
        }
    }
    return r;
}

// nu_t / nu of the 16 inputs of one m16 tile, whose normalised features (BF16, 16 per row, the
// last 6 zero) are rows X[0..15] in shared memory; out[0] gets row g, out[1] row g + 8 (every
// thread of the quad holds both).
__device__ __forceinline__ void tc_tile(const float *w, const TcWeights &B, const __nv_bfloat16 *X, int lane, float out[2]) {
    const int g = lane >> 2, t = lane & 3;
    const unsigned *Xw = reinterpret_cast<const unsigned *>(X); // 8 words per row
    unsigned a[4];
    a[0] = Xw[g * 8 + t];
    a[1] = Xw[(g + 8) * 8 + t];
    a[2] = Xw[g * 8 + 4 + t];
    a[3] = Xw[(g + 8) * 8 + 4 + t];
    float h[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        mma_bf16(c, a, B.b1[j][0], B.b1[j][1]);
        const float bl = w[O_B1 + 8 * j + 2 * t], bh = w[O_B1 + 8 * j + 2 * t + 1];
        h[j][0] = gelu_fast(c[0] + bl);
        h[j][1] = gelu_fast(c[1] + bh);
        h[j][2] = gelu_fast(c[2] + bl);
        h[j][3] = gelu_fast(c[3] + bh);
    }
    unsigned a2[2][4];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        a2[s][0] = pack_bf16(h[2 * s][0], h[2 * s][1]);
        a2[s][1] = pack_bf16(h[2 * s][2], h[2 * s][3]);
        a2[s][2] = pack_bf16(h[2 * s + 1][0], h[2 * s + 1][1]);
        a2[s][3] = pack_bf16(h[2 * s + 1][2], h[2 * s + 1][3]);
    }
    float z_lo = 0.f, z_hi = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        mma_bf16(c, a2[0], B.b2[j][0][0], B.b2[j][0][1]);
        mma_bf16(c, a2[1], B.b2[j][1][0], B.b2[j][1][1]);
        const int n = 8 * j + 2 * t;
        const float bl = w[O_B2 + n], bh = w[O_B2 + n + 1], wl = w[O_W3 + n], wh = w[O_W3 + n + 1];
        z_lo += gelu_fast(c[0] + bl) * wl + gelu_fast(c[1] + bh) * wh;
        z_hi += gelu_fast(c[2] + bl) * wl + gelu_fast(c[3] + bh) * wh;
    }
    z_lo += __shfl_xor_sync(0xffffffffu, z_lo, 1);
    z_lo += __shfl_xor_sync(0xffffffffu, z_lo, 2);
    z_hi += __shfl_xor_sync(0xffffffffu, z_hi, 1);
    z_hi += __shfl_xor_sync(0xffffffffu, z_hi, 2);
    out[0] = softplus(z_lo + w[O_B3]);
    out[1] = softplus(z_hi + w[O_B3]);
}

// A warp's 32 inputs: this lane's normalised features x into row `lane` of the warp's X (32
// rows of 16 BF16), then both m16 tiles; returns nu_t / nu of this lane's input.
__device__ __forceinline__ float tc_warp(const float *w, const TcWeights &B, __nv_bfloat16 *X, const float x[NIN], int lane) {
    unsigned *row = reinterpret_cast<unsigned *>(X + lane * 16);
#pragma unroll
    for (int q = 0; q < 5; ++q) row[q] = pack_bf16(x[2 * q], x[2 * q + 1]);
    row[5] = row[6] = row[7] = 0u;
    __syncwarp();
    float o0[2], o1[2];
    tc_tile(w, B, X, lane, o0);
    tc_tile(w, B, X + 16 * 16, lane, o1);
    __syncwarp();
    // row r of tile m: held by every thread of quad (r mod 8); hand each lane its own row
    const int src = (lane & 7) * 4;
    const float a0 = __shfl_sync(0xffffffffu, o0[0], src), a1 = __shfl_sync(0xffffffffu, o0[1], src);
    const float b0 = __shfl_sync(0xffffffffu, o1[0], src), b1 = __shfl_sync(0xffffffffu, o1[1], src);
    return lane < 8 ? a0 : lane < 16 ? a1 : lane < 24 ? b0 : b1;
}

// ---- features -----------------------------------------------------------------------------

// signed roots x^(1/3), x^(1/4), x^(1/6) of |x| with the sign of x
__device__ __forceinline__ float sroot3(float x) { return cbrtf(x); }
__device__ __forceinline__ float sroot4(float x) { return copysignf(sqrtf(sqrtf(fabsf(x))), x); }
__device__ __forceinline__ float sroot6(float x) { return copysignf(cbrtf(sqrtf(fabsf(x))), x); }

// The 10 raw features from the velocity gradient A[m][d] = d u_m / d x_d of a cell at height y, for
// inference (training data: features_fp64).
__device__ __forceinline__ void features_of(const float A[3][3], float y, float ly, float yplus_scale, float f[NIN]) {
    float S[3][3], W[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            S[a][b] = 0.5f * (A[a][b] + A[b][a]);
            W[a][b] = 0.5f * (A[a][b] - A[b][a]);
        }
    float S2[3][3], W2[3][3], W2S[3][3], W2S2[3][3], WS2[3][3];
    auto mul = [](const float X[3][3], const float Y[3][3], float Z[3][3]) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) Z[a][b] = X[a][0] * Y[0][b] + X[a][1] * Y[1][b] + X[a][2] * Y[2][b];
    };
    auto tr_of = [](const float X[3][3], const float Y[3][3]) {
        float t = 0.f;
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) t += X[a][b] * Y[b][a];
        return t;
    };
    mul(S, S, S2);
    mul(W, W, W2);
    mul(W2, S, W2S);
    mul(W2S, S, W2S2);
    mul(W, S2, WS2);
    const float trS = S[0][0] + S[1][1] + S[2][2];
    const float trS2 = S2[0][0] + S2[1][1] + S2[2][2];
    const float trW2 = W2[0][0] + W2[1][1] + W2[2][2];
    f[0] = trS;
    f[1] = sqrtf(trS2 > 0 ? trS2 : 0.f);
    f[2] = sqrtf(-trW2 > 0 ? -trW2 : 0.f);
    f[3] = sroot3(tr_of(S2, S));
    f[4] = sroot3(W2S[0][0] + W2S[1][1] + W2S[2][2]);
    f[5] = sroot4(W2S2[0][0] + W2S2[1][1] + W2S2[2][2]);
    f[6] = sroot6(tr_of(W2S, WS2));
    const float sg = y > 0 ? -1.f : (y < 0 ? 1.f : 0.f);
    f[7] = sg * S[0][1];
    f[8] = sg * W[0][1];
    f[9] = (0.5f * ly - fabsf(y)) * yplus_scale;
}

// x^(1/2) and x^(1/3) of x >= 0 for the training data: the FP32 root of x (truncated to 24 bits by
// integer instructions) and two Newton steps in FP64 with the FP32 slope.  The first leaves an error
// near 2^-46, the second the rounding of its last operation (root3: and a third of an ulp for the cube's
// square): the square root within 0.501 ulp, the cube root within 1 ulp, the bounds of the FP64 sqrt and
// cbrt (k_selftest_closure compares).  Values outside FP32's comfortable range take those, as a call.
static __device__ __noinline__ double sqrt_call(double x) { return sqrt(x); }
static __device__ __noinline__ double cbrt_call(double x) { return cbrt(x); }
__device__ __forceinline__ float to_float24(double x) { // x in [2^-100, 2^100)
    return __uint_as_float((((unsigned)__double2hiint(x) - 0x38000000u) << 3) | ((unsigned)__double2loint(x) >> 29));
}
__device__ __forceinline__ bool float_range(double x) { return ((unsigned)__double2hiint(x) >> 20) - 923u < 200u; }
// x rounded to FP32 (nearest, ties to even) with integer instructions; results outside FP32's normal
// range take the conversion
static __device__ __noinline__ float narrow_call(double x) { return (float)x; }
__device__ __forceinline__ float narrow(double x) {
    const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
    if (((h >> 20) & 0x7FFu) - 897u >= 253u) return ((h << 1) | l) == 0u ? __uint_as_float(h) : narrow_call(x);
    const unsigned m = (((h & 0x7FFFFFFFu) - 0x38000000u) << 3) | (l >> 29), rest = l << 3;
    return __uint_as_float((h & 0x80000000u) | (m + (rest > 0x80000000u || (rest == 0x80000000u && (m & 1u)) ? 1u : 0u)));
}
// A zero and a NaN come back as they are.
__device__ __forceinline__ double root2(double x) {
    if (!float_range(x)) return x > 0 ? sqrt_call(x) : x;
    const float r = sqrtf(to_float24(x));
    const double h = widen(0.5f / r);
    double y = widen(r);
    y = __fma_rn(__fma_rn(-y, y, x), h, y);
    return __fma_rn(__fma_rn(-y, y, x), h, y);
}
__device__ __forceinline__ double root3(double x) {
    if (!float_range(x)) return x > 0 ? cbrt_call(x) : x;
    const float r = cbrtf(to_float24(x));
    const double h = widen(1.0f / (3.0f * r * r));
    double y = widen(r);
    y = __fma_rn(__fma_rn(-y * y, y, x), h, y);
    return __fma_rn(__fma_rn(-y * y, y, x), h, y);
}
// By their bits (a comparison of doubles is an FP64 operation): whether x is finite; x, or 0 for a NaN.
__device__ __forceinline__ bool finite_bits(double x) { return ((unsigned)__double2hiint(x) & 0x7FF00000u) != 0x7FF00000u; }
__device__ __forceinline__ double or_zero(double x) {
    const unsigned h = (unsigned)__double2hiint(x) & 0x7FFFFFFFu;
    return h > 0x7FF00000u || (h == 0x7FF00000u && __double2loint(x) != 0) ? 0.0 : x;
}
// features_of for the training data, in FP64 with the fewest operations: with W x = w cross x (the
// antisymmetric part), W^2 = w w^T - |w|^2 I, so the mixed invariants are dot products of w, S w and
// S S w (A's off-diagonal entries come halved): tr W^2 S = w.Sw - |w|^2 tr S, tr W^2 S^2 = |Sw|^2 - |w|^2 tr S^2, tr W^2 S W S^2 = Sw.(w x SSw).
__device__ __forceinline__ void features_fp64(const double A[3][3], double y, double ly, double yplus_scale, double f[NIN]) {
    const double s00 = A[0][0], s11 = A[1][1], s22 = A[2][2];
    const double s01 = A[0][1] + A[1][0], s02 = A[0][2] + A[2][0], s12 = A[1][2] + A[2][1];
    const double w[3] = {A[2][1] - A[1][2], A[0][2] - A[2][0], A[1][0] - A[0][1]};
    auto mul = [&](const double x[3], double r[3]) { // S x
        r[0] = s00 * x[0] + s01 * x[1] + s02 * x[2];
        r[1] = s01 * x[0] + s11 * x[1] + s12 * x[2];
        r[2] = s02 * x[0] + s12 * x[1] + s22 * x[2];
    };
    auto dot = [](const double x[3], const double z[3]) { return x[0] * z[0] + x[1] * z[1] + x[2] * z[2]; };
    const double off = s01 * s01 + s02 * s02 + s12 * s12;
    const double trS = s00 + s11 + s22, trS2 = s00 * s00 + s11 * s11 + s22 * s22 + 2.0 * off, ww = dot(w, w);
    // S^2 : S from the rows of S (each off-diagonal of S^2 twice)
    const double q00 = s00 * s00 + s01 * s01 + s02 * s02, q11 = s01 * s01 + s11 * s11 + s12 * s12,
                 q22 = s02 * s02 + s12 * s12 + s22 * s22;
    const double q01 = s00 * s01 + s01 * s11 + s02 * s12, q02 = s00 * s02 + s01 * s12 + s02 * s22,
                 q12 = s01 * s02 + s11 * s12 + s12 * s22;
    const double trS3 = q00 * s00 + q11 * s11 + q22 * s22 + 2.0 * (q01 * s01 + q02 * s02 + q12 * s12);
    double v[3], z[3];
    mul(w, v);
    mul(v, z);
    const double c[3] = {w[1] * z[2] - w[2] * z[1], w[2] * z[0] - w[0] * z[2], w[0] * z[1] - w[1] * z[0]};
    const double i4 = dot(w, v) - ww * trS, i5 = dot(v, v) - ww * trS2, i6 = dot(v, c);
    f[0] = trS;
    // of a NaN invariant features 1 and 2 are 0 (the root of its positive part), 3 to 6 NaN; a diagonal
    // that is not finite makes W's diagonal, and so W^2's trace, a NaN
    f[1] = or_zero(root2(trS2));
    f[2] = finite_bits(trS) ? or_zero(root2(2.0 * ww)) : 0.0;
    f[3] = copysign(root3(fabs(trS3)), trS3);
    f[4] = copysign(root3(fabs(i4)), i4);
    f[5] = copysign(root2(root2(fabs(i5))), i5);
    f[6] = copysign(root3(root2(fabs(i6))), i6);
    const double sg = y > 0 ? -1.0 : (y < 0 ? 1.0 : 0.0);
    f[7] = sg * s01;
    f[8] = sg * -w[2];
    f[9] = (0.5 * ly - fabs(y)) * yplus_scale;
}

// ---- dataset kernels ----------------------------------------------------------------------
// All bound by the FP64 pipe (1/64 of the FP32 rate): sums of widened values, one quotient by 27
// per box on the integer pipes instead of a division per pass, FP32 starting values for the roots.

// The mean x / 27 of a box from its sum, one rounding where three means of three had three each (the
// product with RN(1/27), half an ulp from 1/27, was the less precise by a tenth on FP64 fields), as the
// quotient on the integer pipes (by a product and its correction on the FP64 pipe the filter takes 60 us
// more at 256x128x128).
__device__ __forceinline__ double box_mean(double x, const QRecip &q27) { return qdiv(x, 27.0, 1.0 / 27.0, q27); }

// The velocities of level lvl of a channel (periodic x and z, solid walls in y: a neighbour beyond a
// wall counts as minus the cell), box-filtered 3 x 3 x 3, into three compact interior arrays
// ub + m * cells ([k][j][i], FP64).  A block takes 32 x FY cells of a plane and marches up kch planes:
// the sums along x of FY + 2 rows go through shared memory (two planes' buffers in turn, one barrier
// per plane), the sums over x and y of the last three planes stay in registers.  Seven FP64 sums
// per value and a quotient on the integer pipes (box_mean), against six and three divisions in three
// passes over memory: 700 us (and 32 for a gathered FP64 copy) -> 215 at 256x128x128, the FP64 pipe 69%
// busy (16 rows per block and three blocks per SM, with spills, the same).
constexpr int FY = 8;
template <class T>
__global__ void __launch_bounds__(32 * (FY + 2), 4) k_filter_velocity(const __grid_constant__ DevState<T> S, int lvl, double *ub, int kch,
                                                                      const __grid_constant__ QRecip q27) {
    __shared__ double xs[2][3][FY + 2][32];
    const Geom g = S.g;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int by = (int)blockIdx.x / ((g.C1 + 31) / 32), bx = (int)blockIdx.x - by * ((g.C1 + 31) / 32);
    const int i = bx * 32 + tx + 1, j = by * FY + ty; // j: rows j0 - 1 .. j0 + FY
    const int k0 = (int)blockIdx.y * kch + 1, k1 = k0 + kch - 1 < g.C3 ? k0 + kch - 1 : g.C3;
    const bool live = i <= g.C1 && j >= 1 && j <= g.C2;  // a cell whose x sum is taken
    const bool mine = live && ty >= 1 && ty <= FY;       // and whose box is this thread's
    const int im = i == 1 ? g.C1 : i - 1, ip = i == g.C1 ? 1 : i + 1;
    const T *const u[3] = {S.lv[lvl].u1, S.lv[lvl].u2, S.lv[lvl].u3};
    const size_t cells = (size_t)g.C1 * g.C2 * g.C3;
    double z0[3] = {0, 0, 0}, z1[3] = {0, 0, 0};
    for (int p = k0 - 1; p <= k1 + 1; ++p) {
        const int k = p < 1 ? g.C3 : p > g.C3 ? 1 : p, buf = (p - k0) & 1;
        double x[3] = {0, 0, 0};
        if (live) {
            const int64_t row = g.cell(0, j, k);
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                x[m] = (widen(u[m][row + im]) + widen(u[m][row + i])) + widen(u[m][row + ip]);
                xs[buf][m][ty][tx] = x[m];
            }
        }
        __syncthreads();
        if (mine) {
            const size_t out = ((size_t)(p - 2) * g.C2 + (j - 1)) * g.C1 + (i - 1); // plane p - 1
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                // (the sign flipped as an integer: a negation of its own is an FP64 operation)
                const double neg = __hiloint2double(__double2hiint(x[m]) ^ (int)0x80000000, __double2loint(x[m]));
                const double lo = j == 1 ? neg : xs[buf][m][ty - 1][tx], hi = j == g.C2 ? neg : xs[buf][m][ty + 1][tx];
                const double xy = (lo + x[m]) + hi;
                if (p > k0) ub[m * cells + out] = box_mean((z0[m] + z1[m]) + xy, q27);
                z0[m] = z1[m];
                z1[m] = xy;
            }
        }
    }
}

// gradient of compact arrays at (i, j, k): x, z periodic, y walls (solid neighbour = -u_c)
// (the off-diagonal entries halved: S and W are then plain sums and differences)
__device__ __forceinline__ void grad_compact(const double *const u[3], int i, int j, int k, int C1, int C2, int C3,
                                             const double rdx2[3], double A[3][3]) {
    const int pl = C1 * C2, t = (k * C2 + j) * C1 + i;
    const int im = t - i + (i == 0 ? C1 - 1 : i - 1), ip = t - i + (i == C1 - 1 ? 0 : i + 1);
    const int km = t + ((k == 0 ? C3 - 1 : k - 1) - k) * pl, kp = t + ((k == C3 - 1 ? 0 : k + 1) - k) * pl;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        const double c = u[m][t];
        const double jl = j == 0 ? -c : u[m][t - C1], jh = j == C2 - 1 ? -c : u[m][t + C1];
        A[m][0] = mulq(u[m][ip] - u[m][im], m == 0 ? rdx2[0] : 0.5 * rdx2[0]);
        A[m][1] = mulq(jh - jl, m == 1 ? rdx2[1] : 0.5 * rdx2[1]);
        A[m][2] = mulq(u[m][kp] - u[m][km], m == 2 ? rdx2[2] : 0.5 * rdx2[2]);
    }
}

struct SampleArgs {
    const double *ub[3]; // filtered velocities
    float *feat, *targ;  // dataset rows written from `at`
    long long at;
    int sx, sz, ox, oz, nx, nz, jc;
    double rdx2[3], ly, dy, yplus_scale, rnu27; // rnu27: 1 / (27 nu)
};

// Features of the filtered field and the least-squares target at the sampled cells (i = ox +
// sx*a, k = oz + sz*b, every j); sample (a, j, b) goes to row at + (b*C2 + j)*nx + a.  The filtered
// products u_m u_n are needed at the samples only: a thread marches along jc rows of one (a, b), with
// the nine cells' products of a row summed in x and z, and the sums of three rows in registers
// (a row beyond a wall counts as the row itself).  Every product filtered everywhere took 18 passes
// (1400 us) and 55 us of products; the samples of a 4 x 4 lattice take 169 us with the products in them, the
// FP64 pipe 83% busy (before, 180 without them; the gradients' products on the integer pipes save 4).
template <class T> __global__ void __launch_bounds__(128) k_samples(const __grid_constant__ DevState<T> S, int lvl, SampleArgs s) {
    const Geom g = S.g;
    const int C1 = g.C1, C2 = g.C2, C3 = g.C3;
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x), njc = (C2 + s.jc - 1) / s.jc;
    const int a = t % s.nx, r = t / s.nx, b = r / njc, j0 = (r - b * njc) * s.jc;
    if (b >= s.nz) return;
    const int i = s.ox + s.sx * a, k = s.oz + s.sz * b; // zero-based
    const int j1 = j0 + s.jc < C2 ? j0 + s.jc : C2;
    const int ci[3] = {(i == 0 ? C1 - 1 : i - 1) + 1, i + 1, (i == C1 - 1 ? 0 : i + 1) + 1};
    const int ck[3] = {(k == 0 ? C3 - 1 : k - 1) + 1, k + 1, (k == C3 - 1 ? 0 : k + 1) + 1};
    const T *const u[3] = {S.lv[lvl].u1, S.lv[lvl].u2, S.lv[lvl].u3};
    // the products 11 12 13 22 23 33 of row j (zero-based), summed over the nine cells
    auto row_sum = [&](int j, double q[6]) {
#pragma unroll
        for (int n = 0; n < 6; ++n) q[n] = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int64_t row = g.cell(0, j + 1, ck[c]);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double x = widen(u[0][row + ci[d]]), y = widen(u[1][row + ci[d]]), z = widen(u[2][row + ci[d]]);
                q[0] = __fma_rn(x, x, q[0]);
                q[1] = __fma_rn(x, y, q[1]);
                q[2] = __fma_rn(x, z, q[2]);
                q[3] = __fma_rn(y, y, q[3]);
                q[4] = __fma_rn(y, z, q[4]);
                q[5] = __fma_rn(z, z, q[5]);
            }
        }
    };
    double lo[6], mid[6], hi[6];
    row_sum(j0, mid);
    if (j0 > 0) row_sum(j0 - 1, lo);
    else
        for (int n = 0; n < 6; ++n) lo[n] = mid[n];
    for (int j = j0; j < j1; ++j) {
        if (j < C2 - 1) row_sum(j + 1, hi);
        else
            for (int n = 0; n < 6; ++n) hi[n] = mid[n];
        double A[3][3];
        grad_compact(s.ub, i, j, k, C1, C2, C3, s.rdx2, A);
        const double y = -0.5 * s.ly + ((double)j + 0.5) * s.dy;
        double f[NIN];
        features_fp64(A, y, s.ly, s.yplus_scale, f);
        const size_t c = ((size_t)k * C2 + j) * C1 + i;
        const double v[3] = {s.ub[0][c], s.ub[1][c], s.ub[2][c]};
        // 27 tau, of the products' sums as they are: the target's last factor holds the 1/27 (as precise as
        // six rounded means, 1.79 against 1.84 of 2^-53 u^2 on FP64 fields, by nine FP64 operations for 24)
        const double v27[3] = {27.0 * v[0], 27.0 * v[1], 27.0 * v[2]};
        double tau[6];
#pragma unroll
        for (int n = 0; n < 6; ++n) {
            constexpr int p[6] = {0, 0, 0, 1, 1, 2}, q[6] = {0, 1, 2, 1, 2, 2};
            tau[n] = __fma_rn(-v27[p[n]], v[q[n]], (lo[n] + mid[n]) + hi[n]);
            lo[n] = mid[n];
            mid[n] = hi[n];
        }
        // -tau^d : S^d / (2 S^d : S^d), the off-diagonals twice
        const double ts = (A[0][0] + A[1][1] + A[2][2]) * (1.0 / 3.0), tt = (tau[0] + tau[3] + tau[5]) * (1.0 / 3.0);
        const double s00 = A[0][0] - ts, s11 = A[1][1] - ts, s22 = A[2][2] - ts;
        const double s01 = A[0][1] + A[1][0], s02 = A[0][2] + A[2][0], s12 = A[1][2] + A[2][1];
        const double num = -((tau[0] - tt) * s00 + (tau[3] - tt) * s11 + (tau[5] - tt) * s22 +
                             2.0 * (tau[1] * s01 + tau[2] * s02 + tau[4] * s12));
        const double den = 2.0 * (s00 * s00 + s11 * s11 + s22 * s22 + 2.0 * (s01 * s01 + s02 * s02 + s12 * s12));
        const double nut = den > 1e-30 ? fmax(num / den, 0.0) : 0.0;
        const long long row = s.at + ((long long)b * C2 + j) * s.nx + a;
#pragma unroll
        for (int q = 0; q < NIN; ++q) s.feat[row * NIN + q] = narrow(f[q]);
        s.targ[row] = narrow(nut * s.rnu27);
    }
}

// Plane statistics of the filtered velocities (compact FP64 arrays): block j, the same nine
// means as the context's plane statistics, fixed-order sums.
__global__ void __launch_bounds__(256) k_plane_stats_compact(const double *u0, const double *u1, const double *u2, int C1,
                                                             int C2, int C3, double *out) {
    __shared__ double red[9][256];
    const int j = blockIdx.x;
    double a[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int n = C1 * C3;
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        const int i = t % C1, k = t / C1;
        const size_t c = ((size_t)k * C2 + j) * C1 + i;
        const double v1 = u0[c], v2 = u1[c], v3 = u2[c];
        a[0] += v1;
        a[1] += v2;
        a[2] += v3;
        a[3] += v1 * v1;
        a[4] += v2 * v2;
        a[5] += v3 * v3;
        a[6] += v1 * v2;
        a[7] += v1 * v3;
        a[8] += v2 * v3;
    }
    for (int q = 0; q < 9; ++q) red[q][threadIdx.x] = a[q];
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h)
            for (int q = 0; q < 9; ++q) red[q][threadIdx.x] += red[q][threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x < 9) out[9 * j + threadIdx.x] = red[threadIdx.x][0] / (double)n;
}

// Self-check of root2 and root3 on n values (random significands, exponents beyond the range that they
// take themselves on both sides; exact squares and cubes), their errors from FP64 residuals: x - y^2 is
// one exact FMA, x - y^3 comes from the two-term cube.  Counts square roots off by more than 0.501 ulp,
// cube roots by more than 1 ulp (the bounds of sqrt and cbrt), and zeros, infinities and NaN that do not
// come back as they are.  Also narrow against the conversion: any bits, and values about FP32's range
// with halves of the last place and their neighbours (results that are subnormal or overflow included).
__global__ void k_selftest_closure(long long n, unsigned long long seed, unsigned long long *bad) {
    unsigned long long local = 0;
    auto ulp = [](double y) { return __longlong_as_double((__double_as_longlong(y) & 0x7FF0000000000000ll) - (52ll << 52)); };
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(t + 1);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        const long long e = 1023 - 110 + (long long)((z >> 52) % 221); // [2^-110, 2^111)
        double x = __longlong_as_double((e << 52) | (long long)(z & 0x000FFFFFFFFFFFFFull));
        const double m = (double)(long long)(z & 0xFFFFull) + 1.0;
        if ((t & 15) == 7) x = m * m;
        if ((t & 15) == 11) x = m * m * m;
        const double y = root2(x), r2 = __fma_rn(-y, y, x);
        if (!(fabs(r2) <= 0.501 * ulp(y) * (2.0 * y)) || ((t & 15) == 7 && y != m)) ++local;
        const double w = root3(x), s = __dmul_rn(w, w), ds = __fma_rn(w, w, -s), c = __dmul_rn(s, w);
        const double dc = __dadd_rn(__fma_rn(s, w, -c), __dmul_rn(ds, w)), r3 = __dadd_rn(__dadd_rn(x, -c), -dc);
        if (!(fabs(r3) <= ulp(w) * (3.0 * s)) || ((t & 15) == 11 && w != m)) ++local;
        unsigned long long v = z * 0xD1342543DE82EF95ull + 1;
        v ^= v >> 29;
        if (t & 1) {
            v = (v & 0x800FFFFFFFFFFFFFull) | ((unsigned long long)(870 + (z >> 40) % 284) << 52);
            if (t & 2) v = (v & ~0x1FFFFFFFull) | (0x10000000ull + (z >> 20) % 3 - 1);
        }
        const double d = __longlong_as_double((long long)v);
        const float want = (float)d, got = narrow(d);
        if (__float_as_uint(want) != __float_as_uint(got) && (want == want || got == got)) ++local;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const double inf = __longlong_as_double(0x7FF0000000000000ll), nan = __longlong_as_double(0x7FF8000000000000ll);
        if (root2(0.0) != 0.0 || root3(0.0) != 0.0 || root2(inf) != inf || root3(inf) != inf) ++local;
        if (root2(nan) == root2(nan) || root3(nan) == root3(nan)) ++local;
    }
    if (local) atomicAdd(bad, local);
}

// ---- training on the tensor cores ---------------------------------------------------------
// The layers' products over a tile of TS samples are warp-level BF16 matrix multiply-accumulates
// (m16n8k16, FP32 accumulation): the forward layers Z1 = X W1^T, Z2 = H1 W2^T, the backward
// product D2 W2, and the weight gradients D1^T X and D2^T H1 summed over the tile.  The weights
// are BF16 values already (the working weights), so they enter the multiplies exactly; every
// activation or derivative a enters as a two-term BF16 expansion a = hi + lo (hi = bf16(a),
// lo = bf16(a - hi)), and a product of two such operands as hi*hi + hi*lo + lo*hi, which keeps
// about 16 significand bits (relative error near 2^-16 per product) where one BF16 product
// keeps 8.  The elementwise parts (normalisation, GELU and its derivative, the softplus output,
// the loss) stay in FP32 per sample.  All sums run in a fixed order, so the gradient is
// deterministic.
//
// A warp takes 16 of the tile's samples through the whole network in registers: the accumulator
// fragment of a product (row = sample, column = unit) is the A fragment of the next one, tanh is taken
// once per unit for GELU and its derivative, the weights' fragments are packed once per block.  Only
// the sums over samples meet in shared memory (X, H1, H2, D2, D1 as FP32; one barrier before and
// after): eight warps take an m16n8 tile of D2^T H1 each, four of them one of D1^T X, the other four
// the bias sums.  With every layer's operands staged and split again for each product, a barrier
// after each phase and tanh taken four times per unit pair, 65536 samples took 45.8 us, this 19.
constexpr int TS = 128, GW = TS / 16;  // samples per tile, warps per block
constexpr int LDX = 20;                // floats per staged input row (10 inputs padded to 16, + 4 against bank conflicts)
constexpr int LDH = NH + 4;            // floats per staged hidden row
constexpr int FR1 = 8, FR2 = 16;       // B fragments of W1^T (4 n-tiles x 2), of W2^T and of W2 (4 x 2 x 2)

// a two-term BF16 expansion of a pair of values, packed as the pair registers of a fragment
struct Pair2 {
    unsigned hi, lo;
};
__device__ __forceinline__ Pair2 split_pair(float a, float b) {
    const __nv_bfloat16 ah = __float2bfloat16_rn(a), bh = __float2bfloat16_rn(b);
    Pair2 r;
    __nv_bfloat162 h;
    h.x = ah;
    h.y = bh;
    r.hi = *reinterpret_cast<unsigned *>(&h);
    r.lo = pack_bf16(a - __bfloat162float(ah), b - __bfloat162float(bh));
    return r;
}
// C[16 x 8] += A[16 x TS] B[TS x 8] for operands given by element reads a(row, sample), b(sample,
// column), both split.  Thread lane = 4 g + t holds C[g][2t], C[g][2t+1], C[g+8][2t], C[g+8][2t+1].
template <class FA, class FB> __device__ __forceinline__ void mma_samples(float c[4], int g, int t, FA a, FB b) {
#pragma unroll
    for (int k0 = 0; k0 < TS; k0 += 16) {
        const Pair2 a0 = split_pair(a(g, k0 + 2 * t), a(g, k0 + 2 * t + 1));
        const Pair2 a1 = split_pair(a(g + 8, k0 + 2 * t), a(g + 8, k0 + 2 * t + 1));
        const Pair2 a2 = split_pair(a(g, k0 + 2 * t + 8), a(g, k0 + 2 * t + 9));
        const Pair2 a3 = split_pair(a(g + 8, k0 + 2 * t + 8), a(g + 8, k0 + 2 * t + 9));
        const unsigned ahi[4] = {a0.hi, a1.hi, a2.hi, a3.hi}, alo[4] = {a0.lo, a1.lo, a2.lo, a3.lo};
        const Pair2 b0 = split_pair(b(k0 + 2 * t, g), b(k0 + 2 * t + 1, g));
        const Pair2 b1 = split_pair(b(k0 + 2 * t + 8, g), b(k0 + 2 * t + 9, g));
        mma_bf16(c, ahi, b0.hi, b1.hi);
        mma_bf16(c, ahi, b0.lo, b1.lo);
        mma_bf16(c, alo, b0.hi, b1.hi);
    }
}
// GELU and its derivative from one tanh
__device__ __forceinline__ void gelu_both(float z, float &h, float &d) {
    const float th = tanhf(GK0 * (z + GK1 * z * z * z));
    h = 0.5f * z * (1.0f + th);
    d = 0.5f * (1.0f + th) + 0.5f * z * (1.0f - th * th) * GK0 * (1.0f + 3.0f * GK1 * z * z);
}

// Training alternates two short kernels, each launched while the one before still runs (launch_early).
// Before grid_wait a kernel reads only the samples.  What the other one writes (the weights, the
// partials) is written while this one is resident, so it is no constant of the kernel: no parameter is
// const __restrict__, which would allow read-only loads, and those arrays are read from L2 (__ldcg).
constexpr int kMaxRows = 608; // rows of block partials, so also the most blocks: two waves of two per SM

struct GradSmem {
    unsigned f1[FR1][32], f2[FR2][32], f2t[FR2][32]; // the weights' B fragments, per lane
    float b1[NH], b2[NH], w3[NH], mu[16], rsd[16];
    float D3[TS], R2[TS];                            // dL/dz3, squared errors
    float X[TS * LDX], H1[TS * LDH], H2[TS * LDH], D2[TS * LDH], D1[TS * LDH];
};

// Gradient of the mean squared error over samples [first, first + count) of the batch map
// (sample index = (first + q) * stride + offset), into block partials part[block][NPARAM + 1]
// (the last entry: the block's sum of squared errors).  scale = 2 / (samples of the batch).
__global__ void __launch_bounds__(32 * GW, 2) k_mlp_grad(const float *feat, const float *targ,
                                                         long long first, long long count, long long stride, long long offset,
                                                         const Net *net, float scale, float *part) {
    extern __shared__ __align__(16) unsigned char grad_raw[];
    GradSmem &sm = *reinterpret_cast<GradSmem *>(grad_raw);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = lane >> 2, t = lane & 3;
    static_assert(NPARAM <= TS * LDH, "the weights pass through H1's rows");
    float *const w = sm.H1;
    const int s0 = 16 * wid; // this warp's rows of a tile
    // a tile's inputs: this lane's columns of samples g and g + 8 of the warp's, and (lanes 0 .. 15) the
    // target of sample `lane`
    float2 xlo[2], xhi[2];
    float target = 0.f;
    auto fetch = [&](long long tile) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const long long q = tile * TS + s0 + g + 8 * r, smp = q < count ? (first + q) * stride + offset : 0;
            xlo[r] = *reinterpret_cast<const float2 *>(feat + smp * NIN + 2 * t);
            xhi[r] = t == 0 ? *reinterpret_cast<const float2 *>(feat + smp * NIN + 8) : make_float2(0.f, 0.f);
        }
        const long long q = tile * TS + s0 + lane;
        target = lane < 16 && q < count ? targ[(first + q) * stride + offset] : 0.f;
    };
    fetch(blockIdx.x);
    grid_wait();
#pragma unroll
    for (int q = 0; q < (NPARAM + 32 * GW - 1) / (32 * GW); ++q)
        if (tid + q * 32 * GW < NPARAM) w[tid + q * 32 * GW] = __ldcg(net->w + tid + q * 32 * GW);
    if (tid < 16) {
        sm.mu[tid] = tid < NIN ? __ldcg(net->mu + tid) : 0.f;
        sm.rsd[tid] = tid < NIN ? __ldcg(net->rsd + tid) : 0.f;
    }
    __syncthreads();
    for (int f = wid; f < FR1 + 2 * FR2; f += GW) {
        if (f < FR1) { // n-tile f / 2, register f % 2: W1 rows 8 nt + g, inputs 2t (+ 8)
            const int n = 8 * (f >> 1) + g, k = 2 * t + 8 * (f & 1);
            sm.f1[f][lane] = pack_bf16(k < NIN ? w[O_W1 + n * NIN + k] : 0.f, k + 1 < NIN ? w[O_W1 + n * NIN + k + 1] : 0.f);
        } else { // n-tile q / 4, k-step (q / 2) % 2, register q % 2
            const int q = (f - FR1) % FR2, n = 8 * (q >> 2) + g, k = 16 * ((q >> 1) & 1) + 2 * t + 8 * (q & 1);
            if (f - FR1 < FR2) sm.f2[q][lane] = pack_bf16(w[O_W2 + n * NH + k], w[O_W2 + n * NH + k + 1]);
            else sm.f2t[q][lane] = pack_bf16(w[O_W2 + k * NH + n], w[O_W2 + (k + 1) * NH + n]);
        }
    }
    if (tid < NH) {
        sm.b1[tid] = w[O_B1 + tid];
        sm.b2[tid] = w[O_B2 + tid];
        sm.w3[tid] = w[O_W3 + tid];
    }
    const float b3 = w[O_B3];
    __syncthreads();

    // the block's sums: this warp's fragment of D2^T H1, D1^T X, and (warps 4 ..) a lane's bias sum
    float gw2[4] = {0.f, 0.f, 0.f, 0.f}, gw1[4] = {0.f, 0.f, 0.f, 0.f}, gb = 0.f;
    const long long ntiles = (count + TS - 1) / TS;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        // this lane's rows: samples g and g + 8 of the warp's (a sample past the end enters as zeros;
        // its error and derivatives are zero)
        unsigned ahi[2][4], alo[2][4]; // A fragments (two k-steps of 16)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const long long q = tile * TS + s0 + g + 8 * r;
            const bool live = q < count;
            const float2 lo = xlo[r], hi = xhi[r];
            const float x[4] = {live ? (lo.x - sm.mu[2 * t]) * sm.rsd[2 * t] : 0.f,
                                live ? (lo.y - sm.mu[2 * t + 1]) * sm.rsd[2 * t + 1] : 0.f,
                                live ? (hi.x - sm.mu[2 * t + 8]) * sm.rsd[2 * t + 8] : 0.f,
                                live ? (hi.y - sm.mu[2 * t + 9]) * sm.rsd[2 * t + 9] : 0.f};
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const Pair2 p = split_pair(x[2 * c], x[2 * c + 1]);
                ahi[0][r + 2 * c] = p.hi;
                alo[0][r + 2 * c] = p.lo;
                *reinterpret_cast<float2 *>(&sm.X[(s0 + g + 8 * r) * LDX + 2 * t + 8 * c]) = make_float2(x[2 * c], x[2 * c + 1]);
            }
        }
        const long long mine = tile * TS + s0 + lane; // lanes 0 .. 15: the sample whose output they take
        const bool live = lane < 16 && mine < count;
        // Z1 = X W1^T + b1; H1 = gelu(Z1) (the next A fragments), d1 = gelu'(Z1)
        float d1[4][4];
        unsigned hhi[2][4], hlo[2][4];
        auto put = [&](float *m, int r, int n, float a, float b) { // columns n, n + 1 of row g + 8 r
            *reinterpret_cast<float2 *>(&m[(s0 + g + 8 * r) * LDH + n]) = make_float2(a, b);
        };
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            float c[4] = {0.f, 0.f, 0.f, 0.f}, h[4];
            const unsigned w0 = sm.f1[2 * nt][lane], w1 = sm.f1[2 * nt + 1][lane];
            mma_bf16(c, ahi[0], w0, w1);
            mma_bf16(c, alo[0], w0, w1);
            const int n = 8 * nt + 2 * t;
            const float2 bias = *reinterpret_cast<const float2 *>(&sm.b1[n]);
            gelu_both(c[0] + bias.x, h[0], d1[nt][0]);
            gelu_both(c[1] + bias.y, h[1], d1[nt][1]);
            gelu_both(c[2] + bias.x, h[2], d1[nt][2]);
            gelu_both(c[3] + bias.y, h[3], d1[nt][3]);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const Pair2 p = split_pair(h[2 * r], h[2 * r + 1]);
                hhi[nt >> 1][r + 2 * (nt & 1)] = p.hi;
                hlo[nt >> 1][r + 2 * (nt & 1)] = p.lo;
                put(sm.H1, r, n, h[2 * r], h[2 * r + 1]);
            }
        }
        // Z2 = H1 W2^T + b2, H2 = gelu(Z2), d2 = gelu'(Z2)
        float d2[4][4];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            float c[4] = {0.f, 0.f, 0.f, 0.f}, h[4];
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                const unsigned w0 = sm.f2[4 * nt + 2 * ks][lane], w1 = sm.f2[4 * nt + 2 * ks + 1][lane];
                mma_bf16(c, hhi[ks], w0, w1);
                mma_bf16(c, hlo[ks], w0, w1);
            }
            const int n = 8 * nt + 2 * t;
            const float2 bias = *reinterpret_cast<const float2 *>(&sm.b2[n]);
            gelu_both(c[0] + bias.x, h[0], d2[nt][0]);
            gelu_both(c[1] + bias.y, h[1], d2[nt][1]);
            gelu_both(c[2] + bias.x, h[2], d2[nt][2]);
            gelu_both(c[3] + bias.y, h[3], d2[nt][3]);
            put(sm.H2, 0, n, h[0], h[1]);
            put(sm.H2, 1, n, h[2], h[3]);
        }
        __syncwarp();
        // per sample (lanes 0 .. 15): the output z3 = w3 . H2 + b3 summed in order, the error and dL/dz3
        float d3 = 0.f, r2 = 0.f;
        if (lane < 16) {
            float z3 = b3;
            const float *h = &sm.H2[(s0 + lane) * LDH];
#pragma unroll
            for (int k = 0; k < NH; k += 4) {
                const float4 v = *reinterpret_cast<const float4 *>(h + k), q = *reinterpret_cast<const float4 *>(&sm.w3[k]);
                z3 += q.x * v.x;
                z3 += q.y * v.y;
                z3 += q.z * v.z;
                z3 += q.w * v.w;
            }
            if (live) {
                const float y = softplus(z3), r = y - target;
                r2 = r * r;
                d3 = scale * r * sigmoid(z3);
            }
            sm.D3[s0 + lane] = d3;
            sm.R2[s0 + lane] = r2;
        }
        const float d3r[2] = {__shfl_sync(0xffffffffu, d3, g), __shfl_sync(0xffffffffu, d3, g + 8)};
        // D2 = d3 w3 gelu'(Z2)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            const int n = 8 * nt + 2 * t;
            const float2 w3 = *reinterpret_cast<const float2 *>(&sm.w3[n]);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float a = d3r[r] * w3.x * d2[nt][2 * r], b = d3r[r] * w3.y * d2[nt][2 * r + 1];
                const Pair2 p = split_pair(a, b);
                ahi[nt >> 1][r + 2 * (nt & 1)] = p.hi;
                alo[nt >> 1][r + 2 * (nt & 1)] = p.lo;
                put(sm.D2, r, n, a, b);
            }
        }
        // D1 = (D2 W2) gelu'(Z1)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                const unsigned w0 = sm.f2t[4 * nt + 2 * ks][lane], w1 = sm.f2t[4 * nt + 2 * ks + 1][lane];
                mma_bf16(c, ahi[ks], w0, w1);
                mma_bf16(c, alo[ks], w0, w1);
            }
            put(sm.D1, 0, 8 * nt + 2 * t, c[0] * d1[nt][0], c[1] * d1[nt][1]);
            put(sm.D1, 1, 8 * nt + 2 * t, c[2] * d1[nt][2], c[3] * d1[nt][3]);
        }
        __syncthreads();
        // weight gradients over the tile: gW2 = D2^T H1, warp w units 16 (w & 1) .. +15 by columns
        // 8 (w >> 1) .. +7; gW1 = D1^T X, warps 0 .. 3 units 16 (w & 1) by inputs 8 (w >> 1)
        {
            const int k0 = 16 * (wid & 1), n0 = 8 * (wid >> 1);
            float c[4] = {0.f, 0.f, 0.f, 0.f};
            mma_samples(c, g, t, [&](int r, int s) { return sm.D2[s * LDH + k0 + r]; },
                        [&](int s, int n) { return sm.H1[s * LDH + n0 + n]; });
#pragma unroll
            for (int q = 0; q < 4; ++q) gw2[q] += c[q];
            if (wid < 4) {
                float e[4] = {0.f, 0.f, 0.f, 0.f};
                mma_samples(e, g, t, [&](int r, int s) { return sm.D1[s * LDH + k0 + r]; },
                            [&](int s, int n) { return sm.X[s * LDX + n0 + n]; });
#pragma unroll
                for (int q = 0; q < 4; ++q) gw1[q] += e[q];
            } else { // the bias gradients, the last layer's and the squared errors: sums over the tile in order
                float sum = 0.f;
                if (wid == 4) {
#pragma unroll 16
                    for (int s = 0; s < TS; ++s) sum += sm.D1[s * LDH + lane];
                } else if (wid == 5) {
#pragma unroll 16
                    for (int s = 0; s < TS; ++s) sum += sm.D2[s * LDH + lane];
                } else if (wid == 6) {
#pragma unroll 16
                    for (int s = 0; s < TS; ++s) sum += sm.D3[s] * sm.H2[s * LDH + lane];
                } else if (lane < 2) {
                    const float *v = lane ? sm.R2 : sm.D3;
#pragma unroll 16
                    for (int s = 0; s < TS; ++s) sum += v[s];
                }
                gb += sum;
            }
        }
        if (tile + gridDim.x < ntiles) fetch(tile + gridDim.x);
        __syncthreads();
    }
    grid_release();
    float *const out = part + (size_t)blockIdx.x * (NPARAM + 1);
    const int k0 = 16 * (wid & 1) + g, n0 = 8 * (wid >> 1) + 2 * t;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int k = k0 + 8 * (q >> 1), n = n0 + (q & 1);
        out[O_W2 + k * NH + n] = gw2[q];
        if (wid < 4 && n < NIN) out[O_W1 + k * NIN + n] = gw1[q];
    }
    if (wid == 4) out[O_B1 + lane] = gb;
    else if (wid == 5) out[O_B2 + lane] = gb;
    else if (wid == 6) out[O_W3 + lane] = gb;
    else if (wid == 7 && lane < 2) out[lane ? NPARAM : O_B3] = gb;
}

// One Adam step: the FP32 master weights and moments, and the step's constants.
struct Adam {
    float *master, *m, *v, *loss;
    Net *net;
    float lr, beta1, beta2, eps, loss_scale;
    int step; // 1-based count for the bias corrections
};

// The block partials summed in block order (deterministic) into grad[p], p <= NPARAM, 32 parameters
// per block: all threads bring the partials in, their loads in flight together (at most kMaxRows rows
// of 32), one warp adds them from shared memory.  Then, with A.master set, the Adam step of each parameter
// (the network's working weights are the BF16 roundings of its masters) and the batch's error added
// to *A.loss.  One thread per parameter loading as it added 512 partials, and two more launches for
// the step and the loss, took 22.7 + 3.7 + 2.8 us, this 7 (a batch of 65536: 68 -> 26.6 us in all).
__global__ void __launch_bounds__(512) k_mlp_update(const float *part, int nblocks, float *grad, const Adam A) {
    extern __shared__ float rows[]; // [nblocks][32]
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, p = blockIdx.x * 32 + lane;
    const bool step = wid == 0 && p < NPARAM && A.master;
    const float c1 = 1.f - powf(A.beta1, (float)A.step), c2 = 1.f - powf(A.beta2, (float)A.step);
    grid_wait();
    const float m0 = step ? __ldcg(A.m + p) : 0.f, v0 = step ? __ldcg(A.v + p) : 0.f, x0 = step ? __ldcg(A.master + p) : 0.f;
    if (p <= NPARAM) {
#pragma unroll
        for (int q = 0; q < kMaxRows / 16; ++q) {
            const int b = wid + 16 * q;
            if (b < nblocks) rows[32 * b + lane] = __ldcg(part + (size_t)b * (NPARAM + 1) + p);
        }
    }
    grid_release();
    __syncthreads();
    float s = 0.f;
    if (wid == 0) {
#pragma unroll 16
        for (int b = 0; b < nblocks; ++b) s += rows[32 * b + lane];
    }
    if (wid || p > NPARAM) return;
    grad[p] = s;
    if (!A.master) return;
    if (p == NPARAM) {
        *A.loss += s * A.loss_scale;
        return;
    }
    const float g = s;
    const float mm = A.beta1 * m0 + (1.f - A.beta1) * g;
    const float vv = A.beta2 * v0 + (1.f - A.beta2) * g * g;
    A.m[p] = mm;
    A.v[p] = vv;
    const float mh = mm / c1;
    const float vh = vv / c2;
    const float x = x0 - A.lr * mh / (sqrtf(vh) + A.eps);
    A.master[p] = x;
    A.net->w[p] = __bfloat162float(__float2bfloat16_rn(x));
}

__global__ void k_set_working(const float *master, Net *net) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < NPARAM) net->w[p] = __bfloat162float(__float2bfloat16_rn(master[p]));
}

// nu_t / nu of samples [0, n) (prediction for tests and evaluation)
__global__ void k_mlp_predict(const float *feat, long long n, const Net *net, float *out) {
    __shared__ float w[NPARAM];
    __shared__ float mu[NIN], rsd[NIN];
    for (int q = threadIdx.x; q < NPARAM; q += blockDim.x) w[q] = net->w[q];
    if (threadIdx.x < NIN) {
        mu[threadIdx.x] = net->mu[threadIdx.x];
        rsd[threadIdx.x] = net->rsd[threadIdx.x];
    }
    __syncthreads();
    for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x) {
        float xn[NIN];
#pragma unroll
        for (int i = 0; i < NIN; ++i) xn[i] = (feat[s * NIN + i] - mu[i]) * rsd[i];
        out[s] = mlp_forward(w, xn);
    }
}

// per-feature sums (sum, sum of squares) of samples [0, n), for the input normalisation
__global__ void k_feature_moments(const float *feat, long long n, double *mom) {
    __shared__ double red[2 * NIN][8];
    double s[NIN], s2[NIN];
#pragma unroll
    for (int i = 0; i < NIN; ++i) s[i] = s2[i] = 0.0;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
#pragma unroll
        for (int i = 0; i < NIN; ++i) {
            const double x = feat[q * NIN + i];
            s[i] += x;
            s2[i] += x * x;
        }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < NIN; ++i) {
        for (int o = 16; o > 0; o >>= 1) {
            s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
            s2[i] += __shfl_xor_sync(0xffffffffu, s2[i], o);
        }
        if (lane == 0) {
            red[i][wid] = s[i];
            red[NIN + i][wid] = s2[i];
        }
    }
    __syncthreads();
    if (threadIdx.x < 2 * NIN) {
        double z = 0.0;
        for (int v = 0; v < (int)(blockDim.x >> 5); ++v) z += red[threadIdx.x][v];
        atomicAdd(&mom[threadIdx.x], z);
    }
}

// ---- inference in a context ---------------------------------------------------------------

// nu_t of every interior cell of level lvl, and of the ghost cells of periodic x and z (their
// images); solid cells 0.  Reads interior cells and flags only.
// The network staged in shared memory (coalesced loads; the fragments then read it with
// per-lane addresses, which shared memory serves without serialising).
struct NetSmem {
    float w[NPARAM];
    float mu[NIN], rsd[NIN];
};
__device__ __forceinline__ void stage_net(NetSmem &sm, const Net *__restrict__ net) {
    for (int q = threadIdx.x; q < NPARAM; q += blockDim.x) sm.w[q] = net->w[q];
    if (threadIdx.x < NIN) {
        sm.mu[threadIdx.x] = net->mu[threadIdx.x];
        sm.rsd[threadIdx.x] = net->rsd[threadIdx.x];
    }
    __syncthreads();
}

// Run constants of the inference in FP32, computed once on the host (no FP64 per cell).
struct NutConst {
    float rdx2[3];   // 1 / (2 dx_d)
    float ly, dy;    // channel height, cell height
    float vis;       // nu
    float yplus;     // u_tau / nu
};

template <class T> __global__ void __launch_bounds__(128)
    k_nut(const __grid_constant__ DevState<T> S, int lvl, const Net *__restrict__ netd, const NutConst K) {
    __shared__ __align__(16) __nv_bfloat16 X[4][32 * 16];
    __shared__ NetSmem net;
    stage_net(net, netd);
    const float *w = net.w;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const TcWeights B = tc_weights(w, lane);
    const Geom g = S.g;
    const Level<T> L = S.lv[lvl];
    const int nx = g.C1 + 2, nz = g.C3 + 2;
    const int n = nx * g.C2 * nz;
    const int nwarps = gridDim.x * 4;
    // warp-uniform loop: every lane of a warp takes part in each multiply
    for (int base = (blockIdx.x * 4 + wid) * 32; base < n; base += nwarps * 32) {
        const int t = base + lane;
        const bool live = t < n;
        const int tt = live ? t : n - 1;
        const int ig = tt % nx, r = tt / nx, j = r % g.C2 + 1, kg = r / g.C2;
        // the interior cell whose value this position takes (periodic image, else nearest)
        const int i = ig == 0 ? (S.k.periodic_x ? g.C1 : 1) : (ig == g.C1 + 1 ? (S.k.periodic_x ? 1 : g.C1) : ig);
        const int k = kg == 0 ? (S.k.periodic_z ? g.C3 : 1) : (kg == g.C3 + 1 ? (S.k.periodic_z ? 1 : g.C3) : kg);
        const int64_t ncell = g.ncell();
        const int64_t c = ARK_CK(g.cell(i, j, k), ncell);
        const bool fluid = (S.flags[c] & FL_EQ0) != 0;
        float f[NIN];
        {
            float A[3][3];
            // neighbours in x and z by index (periodic image or the zero-gradient copy), so the
            // level's ghost cells are not needed: this runs beside the step's ghost fill
            const int im = i > 1 ? i - 1 : (S.k.periodic_x ? g.C1 : 1), ip = i < g.C1 ? i + 1 : (S.k.periodic_x ? 1 : g.C1);
            const int km = k > 1 ? k - 1 : (S.k.periodic_z ? g.C3 : 1), kp = k < g.C3 ? k + 1 : (S.k.periodic_z ? 1 : g.C3);
            int64_t nb[6] = {g.cell(im, j, k), g.cell(ip, j, k), c - g.cs1, c + g.cs1, g.cell(i, j, km), g.cell(i, j, kp)};
#pragma unroll
            for (int q = 0; q < 6; ++q) nb[q] = ARK_CK(nb[q], ncell);
            const T *u[3] = {L.u1, L.u2, L.u3};
            bool solid[6];
#pragma unroll
            for (int q = 0; q < 6; ++q) solid[q] = (S.flags[nb[q]] & FL_GT) != 0;
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const float uc = (float)u[m][c];
                float v[6];
#pragma unroll
                for (int q = 0; q < 6; ++q) v[q] = solid[q] ? -uc : (float)u[m][nb[q]];
                A[m][0] = (v[1] - v[0]) * K.rdx2[0];
                A[m][1] = (v[3] - v[2]) * K.rdx2[1];
                A[m][2] = (v[5] - v[4]) * K.rdx2[2];
            }
            const float y = -0.5f * K.ly + ((float)j - 0.5f) * K.dy;
            features_of(A, y, K.ly, K.yplus, f);
#pragma unroll
            for (int q = 0; q < NIN; ++q) f[q] = (f[q] - net.mu[q]) * net.rsd[q];
        }
        const float y_nu = tc_warp(w, B, X[wid], f, lane);
        if (live) S.nut[ARK_CK(g.cell(ig, j, kg), ncell)] = fluid ? (T)(y_nu * K.vis) : (T)0;
    }
}

// nu_t / nu of dataset rows through the tensor-core inference of the step (tests)
__global__ void __launch_bounds__(128) k_mlp_predict_tc(const float *feat, long long n, const Net *__restrict__ netd,
                                                        float *out) {
    __shared__ __align__(16) __nv_bfloat16 X[4][32 * 16];
    __shared__ NetSmem net;
    stage_net(net, netd);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const TcWeights B = tc_weights(net.w, lane);
    const long long nwarps = (long long)gridDim.x * 4;
    for (long long base = ((long long)blockIdx.x * 4 + wid) * 32; base < n; base += nwarps * 32) {
        const long long s = base + lane < n ? base + lane : n - 1;
        float x[NIN];
#pragma unroll
        for (int i = 0; i < NIN; ++i) x[i] = (feat[s * NIN + i] - net.mu[i]) * net.rsd[i];
        const float y = tc_warp(net.w, B, X[wid], x, lane);
        if (base + lane < n) out[base + lane] = y;
    }
}

int grid_for(long long n, int threads = 256) {
    const long long b = (n + threads - 1) / threads;
    return (int)(b < 152 * 16 ? (b < 1 ? 1 : b) : 152 * 16);
}

} // namespace cl

template <class T> void closure_nut(const DevState<T> &S, int lvl, const void *net, float yplus_scale, cudaStream_t st) {
    const long long n = (long long)(S.g.C1 + 2) * S.g.C2 * (S.g.C3 + 2);
    cl::NutConst K;
    for (int d = 0; d < 3; ++d) K.rdx2[d] = (float)(0.5 / S.k.dx[d]);
    K.ly = (float)(S.k.dx[1] * S.g.C2);
    K.dy = (float)S.k.dx[1];
    K.vis = (float)S.k.vis;
    K.yplus = yplus_scale;
    // the blocks that fit the SMs at once (five each), which stage the weights once and pass over the cells
    // in whole rounds: 64x48x48 33.8 -> 32.3 us per step against a block per 128 cells (1.6 waves),
    // 96x64x64 69.1 -> 67.3; from eight rounds on more blocks level out better (256x128x128 592, 600 so)
    const long long need = (n + 127) / 128, once = 5 * 152;
    const int grid = need <= 8 * once ? (int)std::min(need, once) : cl::grid_for(n, 128);
    cl::k_nut<T><<<grid, 128, 0, st>>>(S, lvl, (const cl::Net *)net, K);
}
template void closure_nut<float>(const DevState<float> &, int, const void *, float, cudaStream_t);
template void closure_nut<double>(const DevState<double> &, int, const void *, float, cudaStream_t);

} // namespace ark

// ---- C ABI --------------------------------------------------------------------------------

using namespace ark;

namespace {
thread_local std::string g_cl_error;
int cfail(int code, const std::string &m) {
    g_cl_error = m;
    return code;
}
#define CL_CUDA(x)                                                                                    \
    do {                                                                                              \
        cudaError_t e_ = (x);                                                                         \
        if (e_ != cudaSuccess) return cfail(ARK_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_)); \
    } while (0)
} // namespace

struct ark_closure_data {
    int device = 0;
    cudaStream_t st = nullptr;
    long long cap = 0, n = 0;
    float *feat = nullptr, *targ = nullptr;
    // the filtered velocities of the grid last sampled (3 compact FP64 arrays)
    double *scratch = nullptr;
    long long scratch_cells = 0;
    int last[3] = {0, 0, 0}; // grid of the last filtered field (in the scratch)
};

struct ark_mlp {
    int device = 0;
    cudaStream_t st = nullptr;
    cl::Net *net = nullptr; // device: working weights and normalisation
    // masters and Adam moments; the gradient and squared error, the block partials, an epoch's error
    float *master = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr, *part = nullptr, *loss = nullptr;
    int nblocks = 0;
    int step = 0;
};

extern "C" {

const char *ark_closure_last_error(void) { return g_cl_error.c_str(); }

ark_closure_data *ark_closure_data_create(long long capacity, int device, int *status) {
    int dummy;
    if (!status) status = &dummy;
    if (capacity < 1) {
        *status = cfail(ARK_ERR_PARAM, "capacity < 1");
        return nullptr;
    }
    if (cudaSetDevice(device) != cudaSuccess) {
        *status = cfail(ARK_ERR_CUDA, "cudaSetDevice failed");
        return nullptr;
    }
    ark_closure_data *d = new ark_closure_data();
    d->device = device;
    d->cap = capacity;
    if (cudaStreamCreateWithFlags(&d->st, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMalloc(&d->feat, sizeof(float) * cl::NIN * capacity) != cudaSuccess ||
        cudaMalloc(&d->targ, sizeof(float) * capacity) != cudaSuccess) {
        *status = cfail(ARK_ERR_NOMEM, "dataset allocation failed");
        ark_closure_data_destroy(d);
        return nullptr;
    }
    *status = ARK_OK;
    return d;
}

int ark_closure_data_destroy(ark_closure_data *d) {
    if (!d) return ARK_OK;
    if (d->st) cudaStreamSynchronize(d->st);
    cudaFree(d->feat);
    cudaFree(d->targ);
    cudaFree(d->scratch);
    if (d->st) cudaStreamDestroy(d->st);
    delete d;
    return ARK_OK;
}

long long ark_closure_data_size(const ark_closure_data *d) { return d ? d->n : -1; }

int ark_closure_data_clear(ark_closure_data *d) {
    if (!d) return cfail(ARK_ERR_PARAM, "dataset is NULL");
    d->n = 0;
    return ARK_OK;
}

int ark_closure_data_get(ark_closure_data *d, long long first, long long count, float *features, float *targets) {
    if (!d || first < 0 || count < 0 || first + count > d->n) return cfail(ARK_ERR_PARAM, "bad range");
    CL_CUDA(cudaStreamSynchronize(d->st));
    if (features) CL_CUDA(cudaMemcpy(features, d->feat + first * cl::NIN, sizeof(float) * cl::NIN * count, cudaMemcpyDeviceToHost));
    if (targets) CL_CUDA(cudaMemcpy(targets, d->targ + first, sizeof(float) * count, cudaMemcpyDeviceToHost));
    return ARK_OK;
}

int ark_closure_data_filtered_stats(ark_closure_data *d, double *out) {
    if (!d || !out) return cfail(ARK_ERR_PARAM, "NULL argument");
    const int C1 = d->last[0], C2 = d->last[1], C3 = d->last[2];
    if (C1 < 1) return cfail(ARK_ERR_STATE, "no field has been sampled");
    const long long cells = (long long)C1 * C2 * C3;
    const double *ub = d->scratch;
    double *o = nullptr;
    CL_CUDA(cudaMalloc(&o, sizeof(double) * 9 * C2));
    cl::k_plane_stats_compact<<<C2, 256, 0, d->st>>>(ub, ub + cells, ub + 2 * cells, C1, C2, C3, o);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(d->st);
    if (e == cudaSuccess) e = cudaMemcpy(out, o, sizeof(double) * 9 * C2, cudaMemcpyDeviceToHost);
    cudaFree(o);
    if (e != cudaSuccess) return cfail(ARK_ERR_CUDA, std::string("filtered statistics: ") + cudaGetErrorString(e));
    return ARK_OK;
}

int ark_closure_data_append(ark_closure_data *d, long long count, const float *features, const float *targets) {
    if (!d || count < 0 || !features || !targets) return cfail(ARK_ERR_PARAM, "bad arguments");
    if (d->n + count > d->cap) return cfail(ARK_ERR_PARAM, "dataset full");
    CL_CUDA(cudaStreamSynchronize(d->st));
    CL_CUDA(cudaMemcpy(d->feat + d->n * cl::NIN, features, sizeof(float) * cl::NIN * count, cudaMemcpyHostToDevice));
    CL_CUDA(cudaMemcpy(d->targ + d->n, targets, sizeof(float) * count, cudaMemcpyHostToDevice));
    d->n += count;
    return ARK_OK;
}

} // extern "C"

// Used by ark_api.cu (needs the context's internals).
namespace ark {
long long closure_count(int C1, int C2, int C3, int sx, int sz, int ox, int oz) {
    if (sx < 1 || sz < 1 || ox < 0 || oz < 0 || ox >= sx || oz >= sz || ox >= C1 || oz >= C3) return -1;
    return (long long)((C1 - ox + sx - 1) / sx) * C2 * ((C3 - oz + sz - 1) / sz);
}

long long closure_room(const ark_closure_data *d) { return d->cap - d->n; }

// The samples of level lvl of a context, on its stream (waited for).
template <class T>
int closure_sample(const DevState<T> &S, int lvl, ark_closure_data *d, double lx, double ly, double lz, double vis, int sx,
                   int sz, int ox, int oz, double u_tau, cudaStream_t st) {
    const int C1 = S.g.C1, C2 = S.g.C2, C3 = S.g.C3;
    const int nx = (C1 - ox + sx - 1) / sx, nz = (C3 - oz + sz - 1) / sz;
    const long long cells = (long long)C1 * C2 * C3;
    if (d->scratch_cells != cells) {
        cudaFree(d->scratch);
        d->scratch = nullptr;
        d->scratch_cells = 0;
        d->last[0] = 0;
        if (cudaMalloc(&d->scratch, sizeof(double) * 3 * (size_t)cells) != cudaSuccess)
            return cfail(ARK_ERR_NOMEM, "filter scratch allocation failed");
        d->scratch_cells = cells;
    }
    CL_CUDA(cudaStreamSynchronize(d->st));
    // planes per block, two more starting each chunk: the least planes on the SM with the most blocks
    // (256x128x128: 19 planes)
    const int bx = (C1 + 31) / 32, by = (C2 + cl::FY - 1) / cl::FY;
    int kch = C3;
    long long least = 1ll << 60;
    for (int n = 1; n <= std::min(C3, 65535); ++n) { // (a grid's y extent)
        const int c = (C3 + n - 1) / n;
        const long long per = ((long long)bx * by * ((C3 + c - 1) / c) + 151) / 152, load = std::max(2ll, per) * (c + 2);
        if (load < least) {
            least = load;
            kch = c;
        }
    }
    cl::k_filter_velocity<T><<<dim3((unsigned)bx * by, (C3 + kch - 1) / kch), dim3(32, cl::FY + 2), 0, st>>>(S, lvl, d->scratch, kch, make_qrecip(27.0));
    cl::SampleArgs s;
    for (int m = 0; m < 3; ++m) s.ub[m] = d->scratch + m * cells;
    s.feat = d->feat;
    s.targ = d->targ;
    s.at = d->n;
    s.sx = sx;
    s.sz = sz;
    s.ox = ox;
    s.oz = oz;
    s.nx = nx;
    s.nz = nz;
    // rows per thread: two more start each march; two warps per sub-partition first
    s.jc = 16;
    while (s.jc > 2 && (long long)nx * nz * ((C2 + s.jc - 1) / s.jc) < 152 * 4 * 2 * 32) s.jc /= 2;
    const double dx[3] = {lx / C1, ly / C2, lz / C3};
    for (int q = 0; q < 3; ++q) s.rdx2[q] = 0.5 / dx[q];
    s.ly = ly;
    s.dy = dx[1];
    s.yplus_scale = u_tau / vis;
    s.rnu27 = 1.0 / (27.0 * vis);
    const long long threads = (long long)nx * nz * ((C2 + s.jc - 1) / s.jc);
    cl::k_samples<T><<<(unsigned)((threads + 127) / 128), 128, 0, st>>>(S, lvl, s);
    CL_CUDA(cudaGetLastError());
    CL_CUDA(cudaStreamSynchronize(st));
    d->n += (long long)nx * C2 * nz;
    d->last[0] = C1;
    d->last[1] = C2;
    d->last[2] = C3;
    return ARK_OK;
}
template int closure_sample<float>(const DevState<float> &, int, ark_closure_data *, double, double, double, double, int, int, int,
                                   int, double, cudaStream_t);
template int closure_sample<double>(const DevState<double> &, int, ark_closure_data *, double, double, double, double, int, int, int,
                                    int, double, cudaStream_t);
} // namespace ark

extern "C" {

ark_mlp *ark_mlp_create(unsigned long long seed, int device, int *status) {
    int dummy;
    if (!status) status = &dummy;
    if (cudaSetDevice(device) != cudaSuccess) {
        *status = cfail(ARK_ERR_CUDA, "cudaSetDevice failed");
        return nullptr;
    }
    ark_mlp *M = new ark_mlp();
    M->device = device;
    M->nblocks = cl::kMaxRows;
    bool ok = cudaStreamCreateWithFlags(&M->st, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMalloc(&M->net, sizeof(cl::Net)) == cudaSuccess &&
              cudaMalloc(&M->master, sizeof(float) * cl::NPARAM) == cudaSuccess &&
              cudaMalloc(&M->m, sizeof(float) * cl::NPARAM) == cudaSuccess &&
              cudaMalloc(&M->v, sizeof(float) * cl::NPARAM) == cudaSuccess &&
              cudaMalloc(&M->grad, sizeof(float) * (cl::NPARAM + 1)) == cudaSuccess &&
              cudaMalloc(&M->loss, sizeof(float)) == cudaSuccess &&
              cudaMalloc(&M->part, sizeof(float) * (cl::NPARAM + 1) * M->nblocks) == cudaSuccess;
    if (!ok) {
        *status = cfail(ARK_ERR_NOMEM, "network allocation failed");
        ark_mlp_destroy(M);
        return nullptr;
    }
    // initial weights: uniform(-1, 1) * sqrt(3 / fan_in) (splitmix64), zero biases; identity
    // normalisation
    std::vector<float> w(cl::NPARAM, 0.f);
    unsigned long long x = seed;
    auto next = [&]() {
        unsigned long long z = (x += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0);
    };
    for (int q = 0; q < cl::NH * cl::NIN; ++q) w[cl::O_W1 + q] = (float)((2 * next() - 1) * std::sqrt(3.0 / cl::NIN));
    for (int q = 0; q < cl::NH * cl::NH; ++q) w[cl::O_W2 + q] = (float)((2 * next() - 1) * std::sqrt(3.0 / cl::NH));
    for (int q = 0; q < cl::NH; ++q) w[cl::O_W3 + q] = (float)((2 * next() - 1) * std::sqrt(3.0 / cl::NH));
    std::vector<double> mu(cl::NIN, 0.0), sd(cl::NIN, 1.0);
    std::vector<double> wd(w.begin(), w.end());
    *status = ark_mlp_set(M, wd.data(), mu.data(), sd.data());
    if (*status) {
        ark_mlp_destroy(M);
        return nullptr;
    }
    return M;
}

int ark_mlp_destroy(ark_mlp *M) {
    if (!M) return ARK_OK;
    if (M->st) cudaStreamSynchronize(M->st);
    cudaFree(M->net);
    cudaFree(M->master);
    cudaFree(M->m);
    cudaFree(M->v);
    cudaFree(M->grad);
    cudaFree(M->part);
    cudaFree(M->loss);
    if (M->st) cudaStreamDestroy(M->st);
    delete M;
    return ARK_OK;
}

int ark_mlp_set(ark_mlp *M, const double *params, const double *mu, const double *sd) {
    if (!M || !params || !mu || !sd) return cfail(ARK_ERR_PARAM, "NULL argument");
    std::vector<float> w(cl::NPARAM);
    for (int q = 0; q < cl::NPARAM; ++q) w[q] = (float)params[q];
    cl::Net h;
    std::memset(&h, 0, sizeof h);
    for (int q = 0; q < cl::NIN; ++q) {
        if (!(sd[q] > 0)) return cfail(ARK_ERR_PARAM, "sd must be > 0");
        h.mu[q] = (float)mu[q];
        h.rsd[q] = (float)(1.0 / sd[q]);
    }
    CL_CUDA(cudaStreamSynchronize(M->st));
    CL_CUDA(cudaMemcpy(M->master, w.data(), sizeof(float) * cl::NPARAM, cudaMemcpyHostToDevice));
    CL_CUDA(cudaMemset(M->m, 0, sizeof(float) * cl::NPARAM));
    CL_CUDA(cudaMemset(M->v, 0, sizeof(float) * cl::NPARAM));
    CL_CUDA(cudaMemcpy(M->net, &h, sizeof h, cudaMemcpyHostToDevice));
    cl::k_set_working<<<(cl::NPARAM + 255) / 256, 256, 0, M->st>>>(M->master, M->net);
    CL_CUDA(cudaGetLastError());
    CL_CUDA(cudaStreamSynchronize(M->st));
    M->step = 0;
    return ARK_OK;
}

int ark_mlp_get(ark_mlp *M, double *params, double *mu, double *sd) {
    if (!M) return cfail(ARK_ERR_PARAM, "network is NULL");
    CL_CUDA(cudaStreamSynchronize(M->st));
    if (params) {
        std::vector<float> w(cl::NPARAM);
        CL_CUDA(cudaMemcpy(w.data(), M->master, sizeof(float) * cl::NPARAM, cudaMemcpyDeviceToHost));
        for (int q = 0; q < cl::NPARAM; ++q) params[q] = w[q];
    }
    if (mu || sd) {
        cl::Net h;
        CL_CUDA(cudaMemcpy(&h, M->net, sizeof h, cudaMemcpyDeviceToHost));
        for (int q = 0; q < cl::NIN; ++q) {
            if (mu) mu[q] = h.mu[q];
            if (sd) sd[q] = 1.0 / (double)h.rsd[q];
        }
    }
    return ARK_OK;
}

int ark_mlp_fit_normalization(ark_mlp *M, ark_closure_data *d) {
    if (!M || !d || d->n < 2) return cfail(ARK_ERR_PARAM, "need a network and at least two samples");
    double *mom = nullptr;
    CL_CUDA(cudaMalloc(&mom, sizeof(double) * 2 * cl::NIN));
    CL_CUDA(cudaMemsetAsync(mom, 0, sizeof(double) * 2 * cl::NIN, d->st));
    cl::k_feature_moments<<<cl::grid_for(d->n), 256, 0, d->st>>>(d->feat, d->n, mom);
    double h[2 * cl::NIN];
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(d->st);
    if (e == cudaSuccess) e = cudaMemcpy(h, mom, sizeof h, cudaMemcpyDeviceToHost);
    cudaFree(mom);
    if (e != cudaSuccess) return cfail(ARK_ERR_CUDA, std::string("moments: ") + cudaGetErrorString(e));
    cl::Net net;
    CL_CUDA(cudaStreamSynchronize(M->st));
    CL_CUDA(cudaMemcpy(&net, M->net, sizeof net, cudaMemcpyDeviceToHost));
    for (int q = 0; q < cl::NIN; ++q) {
        const double mean = h[q] / d->n;
        const double var = std::max(h[cl::NIN + q] / d->n - mean * mean, 0.0);
        const double sd = std::sqrt(var);
        net.mu[q] = (float)mean;
        net.rsd[q] = (float)(sd > 1e-20 ? 1.0 / sd : 1.0);
    }
    CL_CUDA(cudaMemcpy(M->net, &net, sizeof net, cudaMemcpyHostToDevice));
    return ARK_OK;
}

} // extern "C"

namespace {

// gradient (and summed squared error) of samples (first + q) * stride + offset, q < count,
// with scale 2 / count, into M->grad on M->st; with A.master set, then one Adam step
void launch_grad(ark_mlp *M, const ark_closure_data *d, long long first, long long count, long long stride,
                 long long offset, const cl::Adam &A) {
    const int nb = (int)std::min<long long>(M->nblocks, (count + cl::TS - 1) / cl::TS);
    launch_early(true, cl::k_mlp_grad, dim3(nb), dim3(32 * cl::GW), sizeof(cl::GradSmem), M->st, d->feat, d->targ, first, count, stride,
                 offset, M->net, (float)(2.0 / (double)count), M->part);
    launch_early(true, cl::k_mlp_update, dim3((cl::NPARAM + 1 + 31) / 32), dim3(512), sizeof(float) * 32 * nb, M->st, M->part, nb, M->grad, A);
}

int prepare_grad() {
    static std::once_flag once;
    static cudaError_t err = cudaSuccess;
    std::call_once(once, [] {
        err = cudaFuncSetAttribute(cl::k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(cl::GradSmem));
        if (err == cudaSuccess)
            err = cudaFuncSetAttribute(cl::k_mlp_update, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * 32 * cl::kMaxRows);
    });
    return err == cudaSuccess ? ARK_OK : cfail(ARK_ERR_CUDA, "k_mlp_grad shared memory attribute");
}

} // namespace

extern "C" {

int ark_mlp_gradient(ark_mlp *M, ark_closure_data *d, long long first, long long count, double *grad, double *loss) {
    if (!M || !d || first < 0 || count < 1 || first + count > d->n) return cfail(ARK_ERR_PARAM, "bad range");
    if (int rc = prepare_grad()) return rc;
    CL_CUDA(cudaStreamSynchronize(d->st));
    launch_grad(M, d, first, count, 1, 0, cl::Adam{});
    CL_CUDA(cudaGetLastError());
    std::vector<float> h(cl::NPARAM + 1);
    CL_CUDA(cudaStreamSynchronize(M->st));
    CL_CUDA(cudaMemcpy(h.data(), M->grad, sizeof(float) * (cl::NPARAM + 1), cudaMemcpyDeviceToHost));
    if (grad)
        for (int q = 0; q < cl::NPARAM; ++q) grad[q] = h[q];
    if (loss) *loss = (double)h[cl::NPARAM] / (double)count;
    return ARK_OK;
}

// Mini-batch Adam: epochs over the dataset in batches of `batch` samples; batch b of nb takes
// samples b, b + nb, b + 2 nb, ... (every batch spans the whole dataset).  loss (may be NULL):
// mean squared error of the last epoch's batches (each taken before its step).
int ark_mlp_train(ark_mlp *M, ark_closure_data *d, int epochs, long long batch, double lr, double *loss) {
    if (!M || !d || epochs < 0 || batch < 1 || !(lr > 0)) return cfail(ARK_ERR_PARAM, "bad arguments");
    const long long nb = d->n / batch;
    if (nb < 1) return cfail(ARK_ERR_PARAM, "fewer samples than one batch");
    if (int rc = prepare_grad()) return rc;
    CL_CUDA(cudaStreamSynchronize(d->st));
    cl::Adam a = {M->master, M->m, M->v, M->loss, M->net, (float)lr, 0.9f, 0.999f, 1e-8f,
                  (float)(1.0 / ((double)batch * (double)nb)), 0};
    int rc = ARK_OK;
    for (int ep = 0; ep < epochs && rc == ARK_OK; ++ep) {
        cudaMemsetAsync(M->loss, 0, sizeof(float), M->st);
        for (long long b = 0; b < nb; ++b) {
            M->step += 1;
            a.step = M->step;
            launch_grad(M, d, 0, batch, nb, b, a);
            if (cudaGetLastError() != cudaSuccess) {
                rc = cfail(ARK_ERR_CUDA, "training launch failed");
                break;
            }
        }
    }
    float h = 0.f;
    if (rc == ARK_OK) {
        cudaError_t e = cudaStreamSynchronize(M->st);
        if (e == cudaSuccess) e = cudaMemcpy(&h, M->loss, sizeof(float), cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) rc = cfail(ARK_ERR_CUDA, std::string("training: ") + cudaGetErrorString(e));
    }
    if (rc) return rc;
    if (loss) *loss = epochs > 0 ? (double)h : 0.0;
    return ARK_OK;
}

int ark_mlp_predict_tc(ark_mlp *M, ark_closure_data *d, long long first, long long count, float *out) {
    if (!M || !d || !out || first < 0 || count < 0 || first + count > d->n) return cfail(ARK_ERR_PARAM, "bad range");
    if (count == 0) return ARK_OK;
    float *o = nullptr;
    CL_CUDA(cudaStreamSynchronize(d->st));
    CL_CUDA(cudaMalloc(&o, sizeof(float) * count));
    cl::k_mlp_predict_tc<<<cl::grid_for(count, 128), 128, 0, M->st>>>(d->feat + first * cl::NIN, count, M->net, o);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(M->st);
    if (e == cudaSuccess) e = cudaMemcpy(out, o, sizeof(float) * count, cudaMemcpyDeviceToHost);
    cudaFree(o);
    if (e != cudaSuccess) return cfail(ARK_ERR_CUDA, std::string("predict: ") + cudaGetErrorString(e));
    return ARK_OK;
}

int ark_mlp_predict(ark_mlp *M, ark_closure_data *d, long long first, long long count, float *out) {
    if (!M || !d || !out || first < 0 || count < 0 || first + count > d->n) return cfail(ARK_ERR_PARAM, "bad range");
    if (count == 0) return ARK_OK;
    float *o = nullptr;
    CL_CUDA(cudaStreamSynchronize(d->st));
    CL_CUDA(cudaMalloc(&o, sizeof(float) * count));
    cl::k_mlp_predict<<<cl::grid_for(count), 256, 0, M->st>>>(d->feat + first * cl::NIN, count, M->net, o);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(M->st);
    if (e == cudaSuccess) e = cudaMemcpy(out, o, sizeof(float) * count, cudaMemcpyDeviceToHost);
    cudaFree(o);
    if (e != cudaSuccess) return cfail(ARK_ERR_CUDA, std::string("predict: ") + cudaGetErrorString(e));
    return ARK_OK;
}

} // extern "C"

// the network constants, for ark_api.cu's closure step
namespace ark {
const void *mlp_device_net(const ark_mlp *M) { return M ? (const void *)M->net : nullptr; }
void selftest_closure(long long n, unsigned long long seed, unsigned long long *bad, cudaStream_t st) {
    cl::k_selftest_closure<<<152 * 4, 256, 0, st>>>(n, seed, bad);
}

size_t mlp_bytes() { return sizeof(cl::Net); }
int mlp_snapshot_device(const ark_mlp *M, void *dev_out) {
    if (!M || !dev_out) return ARK_ERR_PARAM;
    if (cudaStreamSynchronize(M->st) != cudaSuccess) return ARK_ERR_CUDA;
    if (cudaMemcpy(dev_out, M->net, sizeof(cl::Net), cudaMemcpyDeviceToDevice) != cudaSuccess) return ARK_ERR_CUDA;
    return ARK_OK;
}
} // namespace ark
