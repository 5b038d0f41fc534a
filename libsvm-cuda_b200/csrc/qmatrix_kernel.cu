// qmatrix_kernel.cu -- whole kernel matrices of small instances, evaluated by
// the whole GPU ahead of the solve.
//
// When an instance's Q-row cache has a slot for every variable, its rows are
// evaluated here, tile by tile, straight into the cache (variable v's row in
// slot v), and the solver then never evaluates a row.  With room for half of the
// matrix the lower triangle alone is kept.  The values are those of
// the solver's own row passes bit for bit: every dot product accumulates in
// feature order (float64, or float32 in the plain form), and K(a, b) is the
// same number as K(b, a), so only the tiles on and below the diagonal are
// evaluated and the others are their transposes.
//
// Why a kernel of its own: a row pass of the solver runs on the one to ten
// blocks of its group, loads every target row once per source row or two, and
// waits out its staging, its barriers and its last loads each time (about 10k
// cycles for 500 targets of 16 features).  A 64 x 64 tile reads 128 rows for
// 4,096 values, on all SMs.
#include <cuda_runtime.h>

#include "engine.hpp"
#include "kernel_math.cuh"

namespace svmb {

namespace {

constexpr int kQT = 64;             // tile edge
constexpr int kQK = 16;             // features per staged slice
constexpr int kQThreads = 128;      // 8 x 16 threads of 8 x 4 values
constexpr int kQPitch = kQT + 2;    // staged slice [feature][row]: rows 16-byte aligned, loads of a warp in distinct banks
constexpr int kQDots = kQT + 1;     // finished tile [row][column]

__device__ __forceinline__ double q_mac(double a, double b, double acc) { return fma(a, b, acc); }
__device__ __forceinline__ float q_mac(float a, float b, float acc) { return fmaf(a, b, acc); }

// T: the type dots accumulate in (products of float32 features are exact in
// float64, so a fused multiply-add rounds as the separate operations do)
template <typename T>
__global__ void __launch_bounds__(kQThreads) q_dense_kernel(const InstanceDesc *__restrict__ insts,
                                                            const int *__restrict__ first, int count, int total)
{
    __shared__ __align__(16) unsigned char raw[kQT * kQDots * 8];
    __shared__ double xa[kQT], xb[kQT];
    __shared__ int ra[kQT], rb[kQT], ya[kQT], yb[kQT];
    static_assert(2 * kQK * kQPitch * 8 <= kQT * kQDots * 8, "the slices share the finished tile's space");
    T *const sa = reinterpret_cast<T *>(raw), *const sb = sa + kQK * kQPitch;
    double *const dots = reinterpret_cast<double *>(raw);
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        // the instance whose tiles hold t, and the tile (bi, bj <= bi) within it
        int lo = 0, hi = count - 1;
        while (lo < hi) {
            const int m = (lo + hi + 1) >> 1;
            if (first[m] <= t) lo = m;
            else hi = m - 1;
        }
        const InstanceDesc &D = insts[lo];
        const int u = t - first[lo], l = D.l;
        int bi = (int)((sqrt(8.0 * (double)u + 1.0) - 1.0) * 0.5);
        while (bi * (bi + 1) / 2 > u) bi--;
        while ((bi + 1) * (bi + 2) / 2 <= u) bi++;
        const int bj = u - bi * (bi + 1) / 2;
        const int p0 = bi * kQT, q0 = bj * kQT;
        __syncthreads();        // the previous tile has been written
        {
            const int r = tid & (kQT - 1), p = (tid < kQT ? p0 : q0) + r;
            const bool in = p < l;
            const int row = in ? D.pos_row[p] : -1;
            (tid < kQT ? ra : rb)[r] = row;
            (tid < kQT ? ya : yb)[r] = in ? D.y[p] : 0;
            (tid < kQT ? xa : xb)[r] = in && D.x.xsq ? D.x.xsq[row] : 0.0;
        }
        __syncthreads();
        T acc[8][4];
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = T(0);
        // a thread moves two 16-byte pieces of each operand per slice: rows
        // tid / 4 and tid / 4 + 32, features 4 (tid % 4) ..; the next slice's are
        // loaded while this one is used
        const int ld = D.x.ld, c4 = 4 * (tid & 3), r0 = tid >> 2;
        const float *const X = D.x.X;
        float4 va[2], vb[2];
        auto load = [&](int k0) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = r0 + 32 * h;
                const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
                const bool in = k0 + c4 < ld;       // ld is a multiple of 4
                va[h] = in && ra[r] >= 0 ? __ldg(reinterpret_cast<const float4 *>(X + (long long)ra[r] * ld + k0 + c4)) : z;
                vb[h] = in && rb[r] >= 0 ? __ldg(reinterpret_cast<const float4 *>(X + (long long)rb[r] * ld + k0 + c4)) : z;
            }
        };
        load(0);
        for (int k0 = 0; k0 < ld; k0 += kQK) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = r0 + 32 * h;
                sa[(c4 + 0) * kQPitch + r] = (T)va[h].x; sa[(c4 + 1) * kQPitch + r] = (T)va[h].y;
                sa[(c4 + 2) * kQPitch + r] = (T)va[h].z; sa[(c4 + 3) * kQPitch + r] = (T)va[h].w;
                sb[(c4 + 0) * kQPitch + r] = (T)vb[h].x; sb[(c4 + 1) * kQPitch + r] = (T)vb[h].y;
                sb[(c4 + 2) * kQPitch + r] = (T)vb[h].z; sb[(c4 + 3) * kQPitch + r] = (T)vb[h].w;
            }
            __syncthreads();
            if (k0 + kQK < ld) load(k0 + kQK);
#pragma unroll
            for (int kk = 0; kk < kQK; kk++) {
                // thread (tx, ty) owns rows 2 tx + 16 i (+1) and columns 4 ty + j
                T av[8], bv[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    av[2 * i] = sa[kk * kQPitch + 2 * tx + 16 * i];
                    av[2 * i + 1] = sa[kk * kQPitch + 2 * tx + 16 * i + 1];
                }
#pragma unroll
                for (int j = 0; j < 4; j++) bv[j] = sb[kk * kQPitch + 4 * ty + j];
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] = q_mac(av[i], bv[j], acc[i][j]);
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) dots[(2 * tx + 16 * (i >> 1) + (i & 1)) * kQDots + 4 * ty + j] = (double)acc[i][j];
        __syncthreads();
        // kernel values row by row: consecutive threads on consecutive columns
        const KernelParams kp = D.kp;
        float *const Q = D.cache.data;
        const long long stride = D.cache.stride;
#pragma unroll 2
        for (int e = tid; e < kQT * kQT; e += kQThreads) {
            const int r = e >> 6, c = e & (kQT - 1);
            const float q = q_value(kp, ya[r] * yb[c], dots[r * kQDots + c], xa[r], xb[c]);
            if (p0 + r < l && q0 + c < l) {
                if (D.resident == kResidentFull) Q[(p0 + r) * stride + q0 + c] = q;
                else if (p0 + r >= q0 + c) Q[tri_at(p0 + r, q0 + c)] = q;
            }
            dots[r * kQDots + c] = (double)q;
        }
        if (bi == bj || D.resident == kResidentTri) continue;
        __syncthreads();
        // the transposed tile: consecutive threads on consecutive rows
        for (int e = tid; e < kQT * kQT; e += kQThreads) {
            const int c = e >> 6, r = e & (kQT - 1);
            if (p0 + r < l && q0 + c < l) Q[(q0 + c) * stride + p0 + r] = (float)dots[r * kQDots + c];
        }
    }
}

}  // namespace

int q_tiles(int l)
{
    const long long t = (l + kQT - 1) / kQT;
    return (int)(t * (t + 1) / 2);
}

cudaError_t load_q_dense(int form)
{
    cudaFuncAttributes at;
    return form == FORM_FP32 ? cudaFuncGetAttributes(&at, (const void *)q_dense_kernel<float>)
                             : cudaFuncGetAttributes(&at, (const void *)q_dense_kernel<double>);
}

cudaError_t launch_q_dense(int form, const InstanceDesc *d_insts, const int *d_first, int count, int total, cudaStream_t s)
{
    const int most = device_sm_count() * 4, blocks = total < most ? total : most;
    if (form == FORM_FP32) q_dense_kernel<float><<<blocks, kQThreads, 0, s>>>(d_insts, d_first, count, total);
    else q_dense_kernel<double><<<blocks, kQThreads, 0, s>>>(d_insts, d_first, count, total);
    return cudaGetLastError();
}

}  // namespace svmb
