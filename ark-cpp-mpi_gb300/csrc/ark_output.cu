// Output and statistics on the device: the cell data of the reference's VTK writers
// (WriteDataParaView main.cpp:2577-2745, WriteAverageValues main.cpp:2747-2849) packed in file
// order and byte order, the time averages of AverageValues (main.cpp:2878-2891), and the
// kinetic energy of WriteEnergy (main.cpp:2851-2876).  Both precisions; results in double.
#include "ark_state.h"

namespace ark {
namespace {

// IEEE double in big-endian byte order (the reference writes with needSwap = true,
// main.cpp:120, swap8 main.cpp:2975-2989): reverse the 8 bytes.
__device__ __forceinline__ double be64(double v, int swap) {
    if (!swap) return v;
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const unsigned lo = (unsigned)b, hi = (unsigned)(b >> 32);
    const unsigned long long r = ((unsigned long long)__byte_perm(lo, 0, 0x0123) << 32) | __byte_perm(hi, 0, 0x0123);
    return __longlong_as_double((long long)r);
}

template <class T> __device__ __forceinline__ double cell_density(const DevState<T> &S, T v) {
    return Storage<T>::deviation ? S.k.ro0 + (double)v : (double)v;
}

// One thread per interior cell of planes [k0, k1), numbered in file order (i fastest).
template <class T> __global__ void k_pack(const __grid_constant__ DevState<T> S, int ncon, int fcur, CellPack a) {
    const Geom g = S.g;
    const int plane = g.C1 * g.C2;
    const int n = (a.k1 - a.k0) * plane;
    const Level<T> L = S.lv[ncon];
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int kk = t / plane, rem = t - kk * plane;
        const int j = rem / g.C1 + 1, i = rem - (j - 1) * g.C1 + 1, k = a.k0 + kk;
        const int64_t c = g.cell(i, j, k);
        if (a.u) { // U: u1nCon, u2nCon, u3nCon (main.cpp:2653-2667)
            a.u[3 * (int64_t)t + 0] = be64((double)L.u1[c], a.swap);
            a.u[3 * (int64_t)t + 1] = be64((double)L.u2[c], a.swap);
            a.u[3 * (int64_t)t + 2] = be64((double)L.u3[c], a.swap);
        }
        if (a.pc) a.pc[t] = be64(cell_density(S, L.ro[c]), a.swap); // PC: ronCon (main.cpp:2686-2690)
        if (a.r) {
            // R: the curl from face differences (main.cpp:2716-2733), in double
            const FaceSet<T> &F1 = S.fc[fcur][0], &F2 = S.fc[fcur][1], &F3 = S.fc[fcur][2];
            const int64_t f = g.face(i, j, k);
            const double d2u3 = ((double)F2.u[2][f + g.fs1] - (double)F2.u[2][f]) / S.k.dx[1];
            const double d3u2 = ((double)F3.u[1][f + g.fs2] - (double)F3.u[1][f]) / S.k.dx[2];
            const double d3u1 = ((double)F3.u[0][f + g.fs2] - (double)F3.u[0][f]) / S.k.dx[2];
            const double d1u3 = ((double)F1.u[2][f + 1] - (double)F1.u[2][f]) / S.k.dx[0];
            const double d1u2 = ((double)F1.u[1][f + 1] - (double)F1.u[1][f]) / S.k.dx[0];
            const double d2u1 = ((double)F2.u[0][f + g.fs1] - (double)F2.u[0][f]) / S.k.dx[1];
            a.r[3 * (int64_t)t + 0] = be64(d2u3 - d3u2, a.swap);
            a.r[3 * (int64_t)t + 1] = be64(d3u1 - d1u3, a.swap);
            a.r[3 * (int64_t)t + 2] = be64(d1u2 - d2u1, a.swap);
        }
        if (a.avg_out) { // averageU / (TIME - start) (main.cpp:2826-2838)
            const int64_t q = avg_index(g, i, j, k);
            for (int m = 0; m < 3; ++m) a.avg_out[3 * (int64_t)t + m] = be64(a.avg[m][q] / a.avg_div, a.swap);
        }
    }
}

// averageU_m += u_m nCon * dt over interior cells, dt of the step just taken.
template <class T> __global__ void k_average_add(const __grid_constant__ DevState<T> S, int ncon, AvgArrays A) {
    const Geom g = S.g;
    const int plane = g.C1 * g.C2;
    const int n = plane * g.C3;
    const Level<T> L = S.lv[ncon];
    const double dt = S.sc->dt;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int k = t / plane + 1, rem = t - (k - 1) * plane;
        const int j = rem / g.C1 + 1, i = rem - (j - 1) * g.C1 + 1;
        const int64_t c = g.cell(i, j, k), q = avg_index(g, i, j, k);
        A.a[0][q] += (double)L.u1[c] * dt;
        A.a[1][q] += (double)L.u2[c] * dt;
        A.a[2][q] += (double)L.u3[c] * dt;
    }
}

// Moments of a level over the planes, pass 1: each block sums its rows of one y plane (stat_splits
// blocks to a plane), per thread in order, then by a fixed shared-memory tree; pass 2 adds a plane's
// blocks in order.  Deterministic.  ENERGY: u1^2 + u2^2 + u3^2 alone; else u1, u2, u3, u1^2, u2^2, u3^2,
// u1 u2, u1 u3, u2 u3.  Each product goes into its sum as one FMA (the product of two widened FP32
// values is exact, so those sums round as with a separate multiply).  Bound by the FP64 pipe: nine
// FP64 operations per cell (three for the energy).  One block of 256 threads per plane, with separate
// multiplies and converted values, took 187 us at 256x128x128 FP32 (energy 102), this 89 (33).
template <class T, bool ENERGY>
__global__ void __launch_bounds__(32 * kStatWarps) k_moments(const __grid_constant__ DevState<T> S, int ncon, double *part) {
    constexpr int NQ = ENERGY ? 3 : 9; // the energy in three sums, one per component, added at the end
    __shared__ double red[NQ][32 * kStatWarps];
    const Geom g = S.g;
    const Level<T> L = S.lv[ncon];
    const int j = blockIdx.x + 1, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double a[NQ] = {};
    for (int k = (int)blockIdx.y * kStatWarps + w + 1; k <= g.C3; k += kStatWarps * gridDim.y) {
        const int64_t row = g.cell(0, j, k);
        const T *__restrict__ p1 = L.u1 + row, *__restrict__ p2 = L.u2 + row, *__restrict__ p3 = L.u3 + row;
#pragma unroll 2
        for (int i = lane + 1; i <= g.C1; i += 32) {
            const double u1 = widen(p1[i]), u2 = widen(p2[i]), u3 = widen(p3[i]);
            if constexpr (ENERGY) {
                a[0] = __fma_rn(u1, u1, a[0]);
                a[1] = __fma_rn(u2, u2, a[1]);
                a[2] = __fma_rn(u3, u3, a[2]);
            } else {
                a[0] += u1;
                a[1] += u2;
                a[2] += u3;
                a[3] = __fma_rn(u1, u1, a[3]);
                a[4] = __fma_rn(u2, u2, a[4]);
                a[5] = __fma_rn(u3, u3, a[5]);
                a[6] = __fma_rn(u1, u2, a[6]);
                a[7] = __fma_rn(u1, u3, a[7]);
                a[8] = __fma_rn(u2, u3, a[8]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) red[q][threadIdx.x] = a[q];
    __syncthreads();
    // warp w of the tree sums value q = w (and w + 8): its 256 partials by eight per lane, then shuffles
    for (int q = w; q < NQ; q += kStatWarps) {
        double s = 0.0;
        for (int v = 0; v < kStatWarps; ++v) s += red[q][32 * v + lane];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) part[((size_t)q * g.C2 + blockIdx.x) * gridDim.y + blockIdx.y] = s;
    }
}
// Plane statistics: out[9*(j-1) + q] = the mean over plane j of value q.
__global__ void k_plane_totals(const double *part, int C2, int splits, double cells, double *out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 9 * C2) return;
    const int j = t / 9, q = t - 9 * j;
    const double *p = part + ((size_t)q * C2 + j) * splits;
    double s = 0.0;
    for (int v = 0; v < splits; ++v) s += p[v];
    out[t] = s / cells;
}
// Half the sum of n block sums: one block, strided sums in order, then a fixed tree of shuffles.
__global__ void __launch_bounds__(1024) k_energy_total(const double *part, int n, double *out) {
    __shared__ double red[32];
    double e = 0.0;
    for (int q = threadIdx.x; q < n; q += 1024) e += part[q];
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    e = red[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if (threadIdx.x == 0) *out = 0.5 * e;
}

int grid_for(int64_t n) {
    const int64_t b = (n + 255) / 256;
    return (int)(b < 152 * 16 ? (b < 1 ? 1 : b) : 152 * 16);
}

} // namespace

template <class T> void output_pack(const DevState<T> &S, int ncon, int fcur, const CellPack &a, cudaStream_t st) {
    const int64_t n = (int64_t)(a.k1 - a.k0) * S.g.C1 * S.g.C2;
    if (n > 0) k_pack<T><<<grid_for(n), 256, 0, st>>>(S, ncon, fcur, a);
}

template <class T> void output_average_add(const DevState<T> &S, int ncon, const AvgArrays &A, cudaStream_t st) {
    const int64_t n = (int64_t)S.g.C1 * S.g.C2 * S.g.C3;
    k_average_add<T><<<grid_for(n), 256, 0, st>>>(S, ncon, A);
}

template <class T> void output_energy(const DevState<T> &S, int ncon, double *scratch, double *out, cudaStream_t st) {
    const dim3 grid(S.g.C2, stat_splits(S.g));
    k_moments<T, true><<<grid, 32 * kStatWarps, 0, st>>>(S, ncon, scratch);
    k_energy_total<<<1, 1024, 0, st>>>(scratch, (int)(3 * grid.x * grid.y), out);
}

template <class T> void output_plane_stats(const DevState<T> &S, int ncon, double *scratch, double *out, cudaStream_t st) {
    const dim3 grid(S.g.C2, stat_splits(S.g));
    k_moments<T, false><<<grid, 32 * kStatWarps, 0, st>>>(S, ncon, scratch);
    k_plane_totals<<<(9 * S.g.C2 + 127) / 128, 128, 0, st>>>(scratch, S.g.C2, (int)grid.y, (double)S.g.C1 * S.g.C3, out);
}
template void output_plane_stats<double>(const DevState<double> &, int, double *, double *, cudaStream_t);
template void output_plane_stats<float>(const DevState<float> &, int, double *, double *, cudaStream_t);

template void output_pack<double>(const DevState<double> &, int, int, const CellPack &, cudaStream_t);
template void output_pack<float>(const DevState<float> &, int, int, const CellPack &, cudaStream_t);
template void output_average_add<double>(const DevState<double> &, int, const AvgArrays &, cudaStream_t);
template void output_average_add<float>(const DevState<float> &, int, const AvgArrays &, cudaStream_t);
template void output_energy<double>(const DevState<double> &, int, double *, double *, cudaStream_t);
template void output_energy<float>(const DevState<float> &, int, double *, double *, cudaStream_t);

} // namespace ark
