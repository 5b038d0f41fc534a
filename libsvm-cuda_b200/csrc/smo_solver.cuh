// smo_solver.cuh -- device-resident SMO solver for C-SVC and nu-SVC (device code).
//
// One persistent launch runs the whole solve of one or more instances (each a
// binary subproblem).  Every instance is owned by a group of `nblocks` thread
// blocks; block `rank` of the group owns a contiguous chunk of the active
// positions [0, A) and a chunk of the inactive tail [A, l).  The state of its
// active chunk (G, alpha, QD, label, bound status, cache column, row id, cache
// slot) lives in the block's shared memory between shrink events.  Per SMO
// iteration there are exactly two record exchanges:
//
//   phase A  take the working index i of the I_up records (nu-SVC: the two
//            tracks' ip/in), evaluate the Q row(s) on the block's chunk where the
//            cache has none, scan the chunk for the second-order j candidate
//            (WSS3, reference svm.cpp:833-930 / :1076-1186)
//   --- records ---
//   phase B  take j, stopping test, evaluate Q_j if missing, two-variable
//            analytic step with box clipping (svm.cpp:636-721, computed
//            redundantly and identically by every block), gradient update
//            G += dQ (svm.cpp:729-735) and G_bar update (:744-769) on the block's
//            chunk, fused with the I_up scan for the next i
//   --- records ---
//
// What bounds an iteration: not bandwidth but the chain of one block's
// barriers, reductions, the records' trip through L2 and the row reads, so
// the chain is kept short.
//   - A phase ends in two block barriers: warps leave their partial results,
//     warp 0 reduces them (three integer warp reductions per arg-max over an
//     order-preserving key instead of five rounds of double shuffles), sends
//     the block's record, polls the group's records and leaves the winner.
//   - A record is a few 16-byte words that each carry the exchange's sequence
//     number, written and read with single 128-bit accesses: a word that shows
//     the number shows its data, so no fence precedes the store and no second
//     round trip follows the poll.  Blocks share nothing else in the loop (a
//     block reads only the Q columns it filled itself); the collective
//     sections, after which chunks move, use release/acquire exchanges.
//   - Where a variable's row is cached is kept beside its position and travels
//     in the record, so a phase knows a hit or a miss as soon as it knows the
//     variable; every block replays the same slot allocation.
//
// Measured, 45 one-vs-one pairs of 3,600 to 21,600 rows, d = 256: kernel 55.7 ms
// with fence-and-flag records, per-set LRU cache lookups and 64-bit shuffles,
// 44.0 ms with the above; 100,000 x 784 exact form 9.27 and 6.87 s.  Row passes
// (see warp_tile_dots) are then two thirds of an iteration there.
//
// Shrinking (svm.cpp:932-1011), gradient reconstruction (:473-513) and the
// initial gradient (:545-572) run inside the same launch as group-collective
// sections on the global copies of the state.  The position permutation of
// shrinking is the reference's (each shrunk position below the new active
// size is swapped with the highest kept position above it), so the
// position-based tie-breaks are identical.  All double arithmetic keeps the
// reference's operand order; the file is compiled with -fmad=false so that no
// multiply-add is contracted.
//
// Every wait is bounded: a poll that exceeds the instance's wait bound (30 s
// unless the host sets another) sets the group's error flag and every block
// of the group returns.
//
// The kernel template smo_persistent<FORM> is instantiated once per
// arithmetic form, each in its own translation unit (smo_form_*.cu), so the
// forms compile in parallel; the launchers are in smo_kernel.cu.
#pragma once
#include "engine.h"
#include "kernel_math.cuh"
#include "tc_sm100.cuh"

#include <cuda_runtime.h>

#include <type_traits>

namespace svmb {
// internal linkage: every form's translation unit has its own copy
namespace {


#define SVMB_INF __longlong_as_double(0x7ff0000000000000ULL)
constexpr double kTau = 1e-12;                     // reference svm.cpp:42
constexpr long long kWaitTimeoutNs = 30000000000LL;  // default bound of a cross-block wait: 30 s
// positions ahead of the one in hand whose Q values a thread of the chunk scans
// has on their way
constexpr int kScanAhead = 3;

// --------------------------------------------------------------------------
// memory-model helpers
// --------------------------------------------------------------------------
__device__ __forceinline__ int ld_acquire_i32(const int *p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_i32(int *p, int v)
{
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_relaxed_i32(const int *p)
{
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// single-copy atomic 128-bit accesses of a record word at L2
__device__ __forceinline__ RecWord ld_word(const RecWord *p)
{
    RecWord w;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(w.lo), "=l"(w.hi) : "l"(p) : "memory");
    return w;
}
__device__ __forceinline__ void st_word(RecWord *p, double d, unsigned x, unsigned seq)
{
    const unsigned long long lo = (unsigned long long)__double_as_longlong(d);
    const unsigned long long hi = (unsigned long long)x | ((unsigned long long)seq << 32);
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}"
                 ::"l"(p), "l"(lo), "l"(hi) : "memory");
}

// --------------------------------------------------------------------------
// source-row staging and the row-block product
// --------------------------------------------------------------------------
// Sources of a row-block product are staged in dynamic shared memory when the
// instance's stage_cap > 0 (dense rows copied; sparse rows scattered into
// zeroed dense vectors), otherwise read from global memory (dense) or merged
// against the target's CSR row (sparse).  `sp[k]` points at source k.
// The exact form stages its sources as float64 (`dbl`): a float -> double
// conversion per use would otherwise outnumber the float64 multiply-adds
// (conversions issue at a quarter of their rate), and the value is the same.
struct StageSlots {
    const void *sp[kSrcBatch];
    int rows[kSrcBatch];
    int ns;
    int dbl;
    // column-keyed table of wide sparse sources (hash_slots > 0): keys, the
    // values [slot][kSrcBatch], and the sources' nonzeros flattened
    // (source k owns [hoff[k], hoff[k+1])); hash = 0 when this pass's sources
    // did not fit and merge walks are used instead
    int hash;
    int hoff[kSrcBatch + 1];
    int *hkeys;
    void *hvals;
};
// staged nonzeros a thread handles at most (a pass holds up to kHashSlots / 2)
constexpr int kHashPer = (kHashSlots / 2 + kThreads - 1) / kThreads;

__device__ __forceinline__ int hash_home(int col) { return (int)(((unsigned)col * 2654435761u) >> 22) & (kHashSlots - 1); }

// the table slot holding column `col`, or -1
__device__ __forceinline__ int hash_find(const int *keys, int col)
{
    int h = hash_home(col);
    while (true) {
        const int k = keys[h];
        if (k == col) return h;
        if (k < 0) return -1;
        h = (h + 1) & (kHashSlots - 1);
    }
}

// which source owns flattened nonzero t (hoff ascending, ns <= kSrcBatch)
__device__ __forceinline__ int hash_owner(const StageSlots &ss, int t)
{
    int k = 0;
    while (k + 1 < ss.ns && t >= ss.hoff[k + 1]) ++k;
    return k;
}

// bytes of one staged value in the form
__host__ __device__ constexpr int stage_elem(int form) { return form == FORM_EXACT ? 8 : 4; }

__device__ void stage_sources(const InstanceDesc &D, float *stage, StageSlots &ss, const int *rows, int ns)
{
    const DevX &x = D.x;
    const bool dbl = D.form == FORM_EXACT && D.stage_cap > 0;
    double *stage_d = reinterpret_cast<double *>(stage);
    if (threadIdx.x < ns) ss.rows[threadIdx.x] = rows[threadIdx.x];
    if (threadIdx.x == 0) {
        ss.ns = ns;
        ss.dbl = dbl ? 1 : 0;
        ss.hash = 0;
    }
    if (x.X) {
        // all sources in one pass: thread e moves 16 bytes of source e / ld4
        const int ld4 = x.ld >> 2;
        if (D.stage_cap > 0) {
            const int total = ns * ld4;
            for (int e = threadIdx.x; e < total; e += blockDim.x) {
                const int k = e / ld4, t = e - k * ld4;
                const float4 v = __ldg(reinterpret_cast<const float4 *>(x.X + (long long)rows[k] * x.ld) + t);
                if (dbl) {
                    double2 *dst = reinterpret_cast<double2 *>(stage_d + (long long)k * D.stage_lds);
                    dst[2 * t] = make_double2((double)v.x, (double)v.y);
                    dst[2 * t + 1] = make_double2((double)v.z, (double)v.w);
                } else {
                    reinterpret_cast<float4 *>(stage + (long long)k * D.stage_lds)[t] = v;
                }
            }
        }
        if (threadIdx.x < ns) {
            const int k = threadIdx.x;
            if (dbl) ss.sp[k] = stage_d + (long long)k * D.stage_lds;
            else if (D.stage_cap > 0) ss.sp[k] = stage + (long long)k * D.stage_lds;
            else ss.sp[k] = x.X + (long long)rows[k] * x.ld;
        }
    } else if (D.hash_slots > 0) {
        // wide sparse sources: every nonzero (column c of source k) goes to the
        // slot of c in the table; a slot shared by several sources holds each
        // one's value, the others stay zero
        if (threadIdx.x == 0) {
            int tot = 0;
            ss.hoff[0] = 0;
            for (int k = 0; k < ns; k++) {
                tot += (int)(x.rowptr[rows[k] + 1] - x.rowptr[rows[k]]);
                ss.hoff[k + 1] = tot;
            }
            ss.hash = tot <= kHashSlots / 2 ? 1 : 0;
            ss.hkeys = reinterpret_cast<int *>(stage);
            ss.hvals = reinterpret_cast<char *>(stage) + kHashSlots * 4;
            ss.dbl = D.form == FORM_EXACT ? 1 : 0;
        }
        __syncthreads();
        for (int t = threadIdx.x; ss.hash && t < ss.hoff[ns]; t += blockDim.x) {
            const int k = hash_owner(ss, t);
            const long long e = x.rowptr[rows[k]] + (t - ss.hoff[k]);
            const int col = x.col[e];
            const float v = x.val[e];
            int h = hash_home(col);
            while (true) {
                const int prev = atomicCAS(&ss.hkeys[h], -1, col);
                if (prev == -1 || prev == col) break;
                h = (h + 1) & (kHashSlots - 1);
            }
            if (D.form == FORM_EXACT) reinterpret_cast<double *>(ss.hvals)[h * kSrcBatch + k] = (double)v;
            else reinterpret_cast<float *>(ss.hvals)[h * kSrcBatch + k] = v;
        }
    } else if (D.stage_cap > 0) {
        for (int k = 0; k < ns; k++) {
            const long long a = x.rowptr[rows[k]], b = x.rowptr[rows[k] + 1];
            if (dbl) {
                double *dst = stage_d + (long long)k * D.stage_lds;
                for (long long e = a + threadIdx.x; e < b; e += blockDim.x) dst[x.col[e]] = (double)x.val[e];
                if (threadIdx.x == 0) ss.sp[k] = dst;
            } else {
                float *dst = stage + (long long)k * D.stage_lds;
                for (long long e = a + threadIdx.x; e < b; e += blockDim.x) dst[x.col[e]] = x.val[e];
                if (threadIdx.x == 0) ss.sp[k] = dst;
            }
        }
    }
    __syncthreads();
}

// Undo a sparse scatter so that the dense vectors are all-zero again.
__device__ void unstage_sources(const InstanceDesc &D, float *stage, StageSlots &ss)
{
    __syncthreads();
    const DevX &x = D.x;
    if (!x.X && D.hash_slots > 0) {
        // every slot this pass filled goes back to empty with zero values: the
        // slots are found first and cleared after a barrier, so that no
        // lookup meets a chain with a hole
        int h[kHashPer], k[kHashPer];
#pragma unroll
        for (int u = 0; u < kHashPer; u++) {
            const int t = threadIdx.x + u * (int)blockDim.x;
            h[u] = -1;
            k[u] = 0;
            if (ss.hash && t < ss.hoff[ss.ns]) {
                k[u] = hash_owner(ss, t);
                h[u] = hash_find(ss.hkeys, x.col[x.rowptr[ss.rows[k[u]]] + (t - ss.hoff[k[u]])]);
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kHashPer; u++) {
            if (h[u] < 0) continue;
            ss.hkeys[h[u]] = -1;
            if (ss.dbl) reinterpret_cast<double *>(ss.hvals)[h[u] * kSrcBatch + k[u]] = 0.0;
            else reinterpret_cast<float *>(ss.hvals)[h[u] * kSrcBatch + k[u]] = 0.0f;
        }
    } else if (!x.X && D.stage_cap > 0) {
        for (int k = 0; k < ss.ns; k++) {
            const long long a = x.rowptr[ss.rows[k]], b = x.rowptr[ss.rows[k] + 1];
            if (ss.dbl) {
                double *dst = reinterpret_cast<double *>(stage) + (long long)k * D.stage_lds;
                for (long long e = a + threadIdx.x; e < b; e += blockDim.x) dst[x.col[e]] = 0.0;
            } else {
                float *dst = stage + (long long)k * D.stage_lds;
                for (long long e = a + threadIdx.x; e < b; e += blockDim.x) dst[x.col[e]] = 0.0f;
            }
        }
    }
    __syncthreads();
}

// q_value as one function: inlined at every use (up to 8 sources per target,
// each with every kernel type's code) it made the row passes several times
// larger than the instruction caches
__device__ __noinline__ float q_of(int yy, double dot, double xsq_a, double xsq_b);

template <int FORM>
struct Acc {
    typedef typename std::conditional<FORM == FORM_EXACT, double, float>::type type;
};

template <int FORM>
__device__ __forceinline__ typename Acc<FORM>::type mac(float a, float b, typename Acc<FORM>::type acc)
{
    if (FORM == FORM_EXACT) return fma((double)a, (double)b, (double)acc);
    return fmaf(a, b, (float)acc);
}
// a source staged as float64 (exact form): only the target value is converted
template <int FORM>
__device__ __forceinline__ typename Acc<FORM>::type mac(float a, double b, typename Acc<FORM>::type acc)
{
    return fma((double)a, b, (double)acc);
}

// four staged source values starting at feature 4*i: float4 or two double2
__device__ __forceinline__ float4 src4(const float *p, int i) { return reinterpret_cast<const float4 *>(p)[i]; }
struct D4 { double x, y, z, w; };
__device__ __forceinline__ D4 src4(const double *p, int i)
{
    const double2 a = reinterpret_cast<const double2 *>(p)[2 * i], b = reinterpret_cast<const double2 *>(p)[2 * i + 1];
    return D4{a.x, a.y, b.x, b.y};
}

// Dot products of target row `r` with NS staged sources, accumulated in
// feature order (the order of the reference's Kernel::dot, svm.cpp:305-325:
// only matching indices contribute; zero products leave the sum unchanged).
// Dense rows are streamed 8 x 16 bytes at a time per thread.
template <int FORM, int NS, typename S>
__device__ __forceinline__ void row_dots_n(const InstanceDesc &D, const StageSlots &ss, int ns, int r,
                                           double (&out)[kSrcBatch])
{
    const DevX &x = D.x;
    typedef typename Acc<FORM>::type acc_t;
    acc_t acc[NS];
#pragma unroll
    for (int k = 0; k < NS; k++) acc[k] = acc_t(0);
    if (x.X) {
        const float4 *row = reinterpret_cast<const float4 *>(x.X + (long long)r * x.ld);
        const S *src[NS];
#pragma unroll
        for (int k = 0; k < NS; k++) src[k] = reinterpret_cast<const S *>(ss.sp[k < ns ? k : 0]);
        const int ld4 = x.ld >> 2;
        int c = 0;
        for (; c + 8 <= ld4; c += 8) {
            float4 v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = __ldg(row + c + u);
#pragma unroll
            for (int u = 0; u < 8; u++) {
#pragma unroll
                for (int k = 0; k < NS; k++) {
                    if (NS == kSrcBatch && k >= ns) continue;
                    const auto w = src4(src[k], c + u);
                    acc[k] = mac<FORM>(v[u].x, w.x, acc[k]);
                    acc[k] = mac<FORM>(v[u].y, w.y, acc[k]);
                    acc[k] = mac<FORM>(v[u].z, w.z, acc[k]);
                    acc[k] = mac<FORM>(v[u].w, w.w, acc[k]);
                }
            }
        }
        for (; c < ld4; c++) {
            const float4 v = __ldg(row + c);
#pragma unroll
            for (int k = 0; k < NS; k++) {
                if (NS == kSrcBatch && k >= ns) continue;
                const auto w = src4(src[k], c);
                acc[k] = mac<FORM>(v.x, w.x, acc[k]);
                acc[k] = mac<FORM>(v.y, w.y, acc[k]);
                acc[k] = mac<FORM>(v.z, w.z, acc[k]);
                acc[k] = mac<FORM>(v.w, w.w, acc[k]);
            }
        }
    } else if (D.stage_cap > 0) {
        const long long a = x.rowptr[r], b = x.rowptr[r + 1];
        long long e = a;
        for (; e + 4 <= b; e += 4) {
            int cc[4];
            float vv[4];
#pragma unroll
            for (int u = 0; u < 4; u++) { cc[u] = __ldg(x.col + e + u); vv[u] = __ldg(x.val + e + u); }
#pragma unroll
            for (int u = 0; u < 4; u++) {
#pragma unroll
                for (int k = 0; k < NS; k++) {
                    if (NS == kSrcBatch && k >= ns) continue;
                    acc[k] = mac<FORM>(vv[u], reinterpret_cast<const S *>(ss.sp[k])[cc[u]], acc[k]);
                }
            }
        }
        for (; e < b; e++) {
            const int cc = __ldg(x.col + e);
            const float vv = __ldg(x.val + e);
#pragma unroll
            for (int k = 0; k < NS; k++) {
                if (NS == kSrcBatch && k >= ns) continue;
                acc[k] = mac<FORM>(vv, reinterpret_cast<const S *>(ss.sp[k])[cc], acc[k]);
            }
        }
    } else if (ss.hash) {
        // the target's nonzeros in column order, each looked up in the
        // sources' table: only matching columns contribute, in the order of
        // the reference's merge (svm.cpp:305-325)
        const long long a = x.rowptr[r], b = x.rowptr[r + 1];
        const int *keys = ss.hkeys;
        const S *vals = reinterpret_cast<const S *>(ss.hvals);
        long long e = a;
        for (; e + 4 <= b; e += 4) {
            int cc[4];
            float vv[4];
#pragma unroll
            for (int u = 0; u < 4; u++) { cc[u] = __ldg(x.col + e + u); vv[u] = __ldg(x.val + e + u); }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int h = hash_find(keys, cc[u]);
                if (h < 0) continue;
#pragma unroll
                for (int k = 0; k < NS; k++) {
                    if (NS == kSrcBatch && k >= ns) continue;
                    acc[k] = mac<FORM>(vv[u], vals[h * kSrcBatch + k], acc[k]);
                }
            }
        }
        for (; e < b; e++) {
            const int h = hash_find(keys, __ldg(x.col + e));
            if (h < 0) continue;
            const float vv = __ldg(x.val + e);
#pragma unroll
            for (int k = 0; k < NS; k++) {
                if (NS == kSrcBatch && k >= ns) continue;
                acc[k] = mac<FORM>(vv, vals[h * kSrcBatch + k], acc[k]);
            }
        }
    } else {
        // merge walk of two sorted index lists in global memory
        const long long a = x.rowptr[r], b = x.rowptr[r + 1];
#pragma unroll
        for (int k = 0; k < NS; k++) {
            if (k >= ns) continue;
            const long long sa = x.rowptr[ss.rows[k]], sb = x.rowptr[ss.rows[k] + 1];
            long long e = a, f = sa;
            acc_t s = acc_t(0);
            while (e < b && f < sb) {
                const int ce = __ldg(x.col + e), cf = __ldg(x.col + f);
                if (ce == cf) {
                    s = mac<FORM>(__ldg(x.val + e), __ldg(x.val + f), s);
                    ++e;
                    ++f;
                } else if (ce > cf) {
                    ++f;
                } else {
                    ++e;
                }
            }
            acc[k] = s;
        }
    }
#pragma unroll
    for (int k = 0; k < NS; k++) out[k] = (double)acc[k];
}

template <int FORM>
__device__ __forceinline__ void row_dots(const InstanceDesc &D, const StageSlots &ss, int ns, int r,
                                         double (&out)[kSrcBatch])
{
    if (FORM == FORM_EXACT && ss.dbl) {
        if (ns == 1) row_dots_n<FORM, 1, double>(D, ss, ns, r, out);
        else if (ns == 2) row_dots_n<FORM, 2, double>(D, ss, ns, r, out);
        else row_dots_n<FORM, kSrcBatch, double>(D, ss, ns, r, out);
    } else {
        if (ns == 1) row_dots_n<FORM, 1, float>(D, ss, ns, r, out);
        else if (ns == 2) row_dots_n<FORM, 2, float>(D, ss, ns, r, out);
        else row_dots_n<FORM, kSrcBatch, float>(D, ss, ns, r, out);
    }
}

// --------------------------------------------------------------------------
// reductions with the reference's tie rules
// --------------------------------------------------------------------------
// argmax, ties -> larger index ("if (v >= best)" scanning upward, svm.cpp:851,860)
__device__ __forceinline__ void better_max(double &v, int &i, double v2, int i2)
{
    if (v2 > v || (v2 == v && i2 > i)) { v = v2; i = i2; }
}

// Order-preserving key of a number that is not NaN (-0 counts as +0); 0 is
// below every number's key.
typedef unsigned long long u64;
__device__ __forceinline__ u64 key_of(double v)
{
    const long long b = __double_as_longlong(__dadd_rn(v, 0.0));
    return (u64)b ^ ((u64)(b >> 63) | 0x8000000000000000ull);
}
__device__ __forceinline__ double key_value(u64 k)
{
    const u64 b = (k >> 63) ? k ^ 0x8000000000000000ull : ~k;
    return __longlong_as_double((long long)b);
}
// the largest key of the warp
__device__ __forceinline__ u64 warp_max_key(u64 k)
{
    const unsigned hi = (unsigned)(k >> 32), lo = (unsigned)k;
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    return ((u64)mh << 32) | ml;
}
// the largest key of the warp and, among the lanes that hold it, the largest
// index (ties go to the larger index); every lane gets both.  (Stopping after
// the high words when one lane holds the maximum, by a vote, was slower: the
// reductions are short, the branch is not.)
__device__ __forceinline__ void warp_best(u64 &k, int &i)
{
    const u64 m = warp_max_key(k);
    i = __reduce_max_sync(0xffffffffu, k == m ? i : -1);
    k = m;
}

__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ int warp_sum_i(int v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct RedScratch {
    double v[4][kWarps];
    int i[kWarps];
};

// Maxima of N values over the block; the result is in every thread.
template <int N>
__device__ void block_max(RedScratch &s, double (&v)[N])
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < N; k++) v[k] = warp_max(v[k]);
    __syncthreads();
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < N; k++) s.v[k][w] = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; k++) v[k] = warp_max(lane < kWarps ? s.v[k][lane] : -SVMB_INF);
}

__device__ int block_sum_i(RedScratch &s, int v)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    v = warp_sum_i(v);
    __syncthreads();
    if (lane == 0) s.i[w] = v;
    __syncthreads();
    int tot = lane < kWarps ? s.i[lane] : 0;
    tot = warp_sum_i(tot);
    __syncthreads();
    return tot;
}

// exclusive prefix over the block of a 0/1 flag, in thread order; the block
// total goes to *total.
__device__ int block_excl_scan(RedScratch &s, int flag, int *total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned bal = __ballot_sync(0xffffffffu, flag);
    const int in_warp = __popc(bal & ((1u << lane) - 1u));
    __syncthreads();
    if (lane == 0) s.i[w] = __popc(bal);
    __syncthreads();
    int before = 0, tot = 0;
    for (int k = 0; k < kWarps; k++) {
        const int c = s.i[k];
        if (k < w) before += c;
        tot += c;
    }
    __syncthreads();
    *total = tot;
    return before + in_warp;
}

// --------------------------------------------------------------------------
// per-block solver context
// --------------------------------------------------------------------------
// flags of an active position: label, bound status (ST_*), whole row cached,
// row evaluated ahead of need and not yet used
constexpr int kFlagPos = 1, kFlagStatus = 1, kFlagFull = 8, kFlagAhead = 16;   // status at bits 1-2
__device__ __forceinline__ int flag_y(unsigned f) { return (f & kFlagPos) ? +1 : -1; }
__device__ __forceinline__ unsigned char flag_s(unsigned f) { return (unsigned char)((f >> kFlagStatus) & 3u); }
__device__ __forceinline__ unsigned char flags_of(int y, unsigned char s, unsigned slotword)
{
    return (unsigned char)((y > 0 ? kFlagPos : 0) | (s << kFlagStatus) | ((slotword >> 13) & (kFlagFull | kFlagAhead)));
}
// a slot with its flags, as it travels in records and in D.pos_slot
constexpr unsigned kSlotFull = 1u << 16, kSlotAhead = 1u << 17;
__device__ __forceinline__ unsigned slot_word(unsigned slot, unsigned f) { return slot | ((f & (kFlagFull | kFlagAhead)) << 13); }
// a position and its label as they travel in records
constexpr unsigned kNoPos = 0xffffffffu;
__device__ __forceinline__ unsigned pos_code(int p, int y) { return (unsigned)p * 2u + (y > 0 ? 1u : 0u); }
__device__ __forceinline__ int code_pos(unsigned c) { return c == kNoPos ? -1 : (int)(c >> 1); }
__device__ __forceinline__ int code_y(unsigned c) { return (c & 1u) ? +1 : -1; }

// work counters of a solve, kept by thread 0
enum { kCntActive, kCntQ, kCntLook, kCntMiss, kCntFill, kCntAhead, kCntTargets, kCnt };

constexpr int kPollWarps = (kMaxGroupBlocks + 31) / 32;   // each polls the records of 32 blocks
static_assert(kPollWarps < kWarps, "a warp is left for the prefetch candidates");

// The winning records of a phase as one poll warp saw them.
//   phase A, track t: words 4t..: {-y G, pos_code} {alpha, column} {QD, slot} {-, row}
//   phase B:          {decrease, pos_code} {G, column} {alpha, row} {QD, slot} {Gmax2, Q_ij} {Gmax2 of y=-1, -}
// (nu-SVC has two tracks; C-SVC uses track 0 and the first Gmax2)
struct WinA { double d[2 * kWordsI]; unsigned x[2 * kWordsI]; };
struct WinB { double d[kWordsJ]; unsigned x[kWordsJ]; };
// a prefetch candidate: priority, position and label, column, row, slot (kNoSlot: not cached)
struct Cand { double v; unsigned pc, col, row, slot; };

// what every thread of the block knows about its part of the instance; thread 0
// writes it, between barriers
struct Ctx {
    float *stage;           // source staging area (dynamic smem)
    float *tile;            // per-warp 32-row transpose tiles (dense rows)
    int choff;              // my chunk of [0,A): its offset in dynamic shared memory
    int rank, nb;
    int A;                  // active size
    int a0, a1;             // my chunk of [0,A)
    int t0, t1;             // my chunk of [A,l)
    int phase;              // exchange counter: selects the record buffer and sequence number
    uint32_t tcbase;        // FORM_BF16X3: shared address of the operand stages (1024-aligned)
    long long tc_g;         // tensor-core steps issued so far (mbarrier phase parities)
    long long fg;           // steps of the fill pipeline so far (its mbarrier phase parities)
    int fstages;            // operand stages of the fill pipeline (3 or 4, by the stage area)
};

struct Shared {
    InstanceDesc D;
    Ctx c;
    RedScratch red;
    StageSlots ss;
    // warps' partial results of a phase: keys and positions
    u64 wk[3][kWarps];
    int wi[2][kWarps], wp[kWarps];
    float wq[kWarps];               // the Q value of a warp's j candidate
    WinA wa[kPollWarps];
    WinB wb[kPollWarps];
    Cand cand[kPrefetchCand];       // single-block groups: the block's own candidates
    long long cnt[kCnt], prof[8], tstart;
    unsigned prof32[8];             // cycles since the last flush
    unsigned ahead_used;            // rows evaluated ahead of need and used later (every block counts its own)
    int fail;
    // slot allocation, replayed identically by every block: the next slot to
    // look at, whether slots are being reused, and the reference bits
    int hand, reused;
    unsigned ref[kRefSlots / 32];
    int srcpos[kSrcBatch];
    int srcrow[kSrcBatch];
    int nsrc;
    int stop_at;
    // rows of the current fill pass: row id, label, slot, position (with how
    // many of them are evaluated ahead of need)
    int frow[kPrefetchMax], fy[kPrefetchMax], fslot[kPrefetchMax], fpos[kPrefetchMax], fcol[kPrefetchMax];
    int nfill, nneed;
    // per source of the fill pass running now: norm, label, destination row
    double fsx[kPrefetchMax];
    int fsy[kPrefetchMax];
    float *fsd[kPrefetchMax];
    // tensor-core block products (FORM_BF16X3, FORM_FP16X3): sources of the current pass
    // (row id, position, alpha, norm, C, inverse scale, label, status), the
    // pipeline's mbarriers (one per operand stage) and the TMEM base address
    int tsrow[kTcMaxN], tspos[kTcMaxN];
    double tsa[kTcMaxN], tsx[kTcMaxN], tsc[kTcMaxN], tsi[kTcMaxN];
    signed char tsy[kTcMaxN];
    unsigned char tss[kTcMaxN];
    uint64_t tbar[kTcStages];
    uint32_t tmem;
    // the fill pipeline's mbarriers: operand stage loaded / free, accumulator
    // written / read; fabort is set by a role whose wait ran out
    uint64_t ffull[kFillStagesMax], fempty[kFillStagesMax], faccf[kFillAcc], facce[kFillAcc];
    int fabort;
    Partial lrec[2];                // single-block groups keep their two exchange records here
};

// The block's shared state, reachable by its address from every device function
// (a reference passed to a function that is not inlined would make each
// access a generic one).
__device__ __forceinline__ Shared &block_shared()
{
    __shared__ Shared s;
    return s;
}
extern __shared__ __align__(128) unsigned char dyn[];

__device__ __noinline__ float q_of(int yy, double dot, double xsq_a, double xsq_b)
{
    return q_value(block_shared().D.kp, yy, dot, xsq_a, xsq_b);
}

// the block's chunk of the active state, in dynamic shared memory
struct Chunk {
    double *G, *A, *QD;
    int *Col, *Row;
    unsigned short *Slot;
    unsigned char *F;       // kFlag*
};
__device__ __forceinline__ Chunk chunk_at(int off, int cap)
{
    Chunk k;
    k.G = reinterpret_cast<double *>(dyn + off);
    k.A = k.G + cap;
    k.QD = k.A + cap;
    k.Col = reinterpret_cast<int *>(k.QD + cap);
    k.Row = k.Col + cap;
    k.Slot = reinterpret_cast<unsigned short *>(k.Row + cap);
    k.F = reinterpret_cast<unsigned char *>(k.Slot + cap);
    return k;
}


// the active size and my chunks of [0,A) and [A,l); called by every thread
__device__ __forceinline__ void set_active(int A)
{
    Ctx &c = block_shared().c;
    __syncthreads();
    if (threadIdx.x == 0) {
        const long long n = A, m = block_shared().D.l - A;
        c.A = A;
        c.a0 = (int)(n * c.rank / c.nb);
        c.a1 = (int)(n * (c.rank + 1) / c.nb);
        c.t0 = A + (int)(m * c.rank / c.nb);
        c.t1 = A + (int)(m * (c.rank + 1) / c.nb);
    }
    __syncthreads();
}

__device__ __forceinline__ Partial *my_partial()
{
    Ctx &c = block_shared().c;
    if (c.nb == 1) return block_shared().lrec + (c.phase & 1);
    return block_shared().D.partials + (long long)(c.phase & 1) * c.nb + c.rank;
}
__device__ __forceinline__ const Partial *prev_partials()
{
    Ctx &c = block_shared().c;
    if (c.nb == 1) return block_shared().lrec + ((c.phase - 1) & 1);
    return block_shared().D.partials + (long long)((c.phase - 1) & 1) * c.nb;
}

// Publish my record of this phase and wait for everybody's (group barrier).
__device__ __noinline__ bool exchange()
{
    Ctx &c = block_shared().c;
    __syncthreads();
    const int want = c.phase + 1;
    Partial *mine = my_partial();
    int ok = 1;
    if (c.nb > 1) {
        // the release store orders this thread's writes and, through the
        // barrier above, the whole block's before the record is seen
        if (threadIdx.x == 0) st_release_i32(&mine->seq, want);
        const Partial *all = block_shared().D.partials + (long long)(c.phase & 1) * c.nb;
        const long long limit = block_shared().D.wait_ns > 0 ? block_shared().D.wait_ns : kWaitTimeoutNs;
        for (int b = threadIdx.x; b < c.nb; b += blockDim.x) {
            const long long t0 = (long long)tc::global_ns();
            long long spins = 0;
            // spin with relaxed loads; one acquire load of the awaited value
            // then synchronizes with the record's release store
            while (ld_relaxed_i32(&all[b].seq) != want) {
                if ((++spins & 63) == 0) {
                    if (ld_relaxed_i32(&block_shared().D.sync->error) != 0 || (long long)tc::global_ns() - t0 > limit) {
                        atomicExch(&block_shared().D.sync->error, 1);
                        ok = 0;
                        break;
                    }
                }
            }
            if (ok) (void)ld_acquire_i32(&all[b].seq);
        }
    }
    // the pollers' acquire loads, followed by the barrier, order every later
    // read of this block after the other blocks' releases
    ok = __syncthreads_and(ok);
    if (threadIdx.x == 0) c.phase++;
    __syncthreads();
    return ok != 0;
}

__device__ __forceinline__ double get_C(const InstanceDesc &D, int y) { return y > 0 ? D.Cp : D.Cn; }

__device__ __forceinline__ unsigned char status_of(double a, double C)
{
    if (a >= C) return ST_UPPER;            // reference svm.cpp:441-449
    if (a <= 0) return ST_LOWER;
    return ST_FREE;
}

// chunk state: global -> shared / shared -> global (mutable fields only)
__device__ __noinline__ void chunk_load()
{
    Ctx &c = block_shared().c;
    const InstanceDesc &D = block_shared().D;
    const Chunk ck = chunk_at(c.choff, block_shared().D.chunk_cap);
    for (int k = threadIdx.x; k < c.a1 - c.a0; k += blockDim.x) {
        const int p = c.a0 + k;
        const unsigned w = (unsigned)D.pos_slot[p];
        ck.G[k] = D.G[p];
        ck.A[k] = D.alpha[p];
        ck.QD[k] = D.QD[p];
        ck.Col[k] = D.pos_local[p];
        ck.Row[k] = D.pos_row[p];
        ck.Slot[k] = (unsigned short)(w & 0xffffu);
        ck.F[k] = flags_of(D.y[p], D.status[p], w);
    }
    __syncthreads();
}
__device__ __noinline__ void chunk_store()
{
    Ctx &c = block_shared().c;
    const InstanceDesc &D = block_shared().D;
    const Chunk ck = chunk_at(c.choff, block_shared().D.chunk_cap);
    __syncthreads();
    for (int k = threadIdx.x; k < c.a1 - c.a0; k += blockDim.x) {
        const int p = c.a0 + k;
        D.G[p] = ck.G[k];
        D.alpha[p] = ck.A[k];
        D.status[p] = flag_s(ck.F[k]);
        D.pos_slot[p] = (int)slot_word(ck.Slot[k], ck.F[k]);
    }
}

// Sum over the group's blocks of per-block counters of the previous exchange.
__device__ void group_counts(int slot, int *below, int *above, int *total)
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    const Partial *all = prev_partials();
    int b_lo = 0, b_hi = 0, tot = 0;
    for (int b = threadIdx.x; b < c.nb; b += blockDim.x) {
        const int v = c.nb == 1 ? all[b].n[slot] : __ldcg(&all[b].n[slot]);
        tot += v;
        if (b < c.rank) b_lo += v;
        if (b > c.rank) b_hi += v;
    }
    *below = block_sum_i(sh.red, b_lo);
    *above = block_sum_i(sh.red, b_hi);
    *total = block_sum_i(sh.red, tot);
}

// --------------------------------------------------------------------------
// row-block accumulation on the global state: for every target position e in
// [lo,hi), in source order over the positions s < src_end selected by the
// predicate,
//   G[e] += alpha_s * Q[s][e]  and, with `with_bar`, for upper-bound s,
//   G_bar[e] += C_s * Q[s][e].
// This is the initial gradient (svm.cpp:559-570) and the gradient
// reconstruction (svm.cpp:493-512); per target the additions happen in the
// same order as in the reference.
// --------------------------------------------------------------------------
template <int FORM>
__device__ __noinline__ void accumulate_rows(int src_end, int pick_free_only, int with_bar, int lo, int hi)
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    const InstanceDesc &D = block_shared().D;
    const int cap = D.stage_cap > 0 ? D.stage_cap : kSrcBatch;
    int scan = 0;
    while (true) {
        if (threadIdx.x == 0) sh.nsrc = 0;
        __syncthreads();
        while (scan < src_end) {
            const int p = scan + threadIdx.x;
            int sel = 0;
            if (p < src_end) {
                const unsigned char s = D.status[p];
                sel = pick_free_only ? (s == ST_FREE) : (s != ST_LOWER);
            }
            int tot;
            const int pre = block_excl_scan(sh.red, sel, &tot);
            const int have = sh.nsrc;
            const int room = cap - have;
            if (sel && pre < room) sh.srcpos[have + pre] = p;
            const int take = tot < room ? tot : room;
            if (take < tot && sel && pre == take) sh.stop_at = threadIdx.x;
            __syncthreads();
            const int consumed = take == tot ? (int)blockDim.x : sh.stop_at;
            __syncthreads();
            if (threadIdx.x == 0) sh.nsrc = have + take;
            scan += consumed;
            __syncthreads();
            if (sh.nsrc == cap) break;
        }
        const int ns = sh.nsrc;
        if (ns == 0) break;
        if (threadIdx.x < ns) sh.srcrow[threadIdx.x] = D.pos_row[sh.srcpos[threadIdx.x]];
        __syncthreads();
        stage_sources(D, c.stage, sh.ss, sh.srcrow, ns);
        for (int e = lo + threadIdx.x; e < hi; e += blockDim.x) {
            double dots[kSrcBatch];
            const int r = D.pos_row[e];
            row_dots<FORM>(D, sh.ss, ns, r, dots);
            double g = D.G[e];
            double gb = with_bar ? D.G_bar[e] : 0.0;
            const int ye = D.y[e];
            const double xe = D.x.xsq ? D.x.xsq[r] : 0.0;
            for (int k = 0; k < ns; k++) {
                const int sp = sh.srcpos[k];
                const int ys = D.y[sp];
                const double xs = D.x.xsq ? D.x.xsq[sh.srcrow[k]] : 0.0;
                const float q = q_of(ys * ye, dots[k], xs, xe);
                g = __dadd_rn(g, __dmul_rn(D.alpha[sp], (double)q));
                if (with_bar && D.status[sp] == ST_UPPER) gb = __dadd_rn(gb, __dmul_rn(get_C(D, ys), (double)q));
            }
            D.G[e] = g;
            if (with_bar) D.G_bar[e] = gb;
        }
        unstage_sources(D, c.stage, sh.ss);
        if (ns < cap) break;
    }
}

// --------------------------------------------------------------------------
// tensor-core block products (FORM_BF16X3, FORM_FP16X3)
// --------------------------------------------------------------------------
// dot(x_t, x_s) for the targets t in [lo,hi) -- chunk-local indices into the
// shared-memory chunk, or with `global_targets` positions of the global state
// -- against the ns <= tc_n sources whose row ids are in sh.tsrow, with the
// split of the form (x = hi + lo in bf16, or x 2^e = hi + lo in fp16;
// hi.lo + lo.hi + hi.hi, 3 MMAs per K-step of 16).
//
// Each step is one 64-feature chunk of one 128-target tile; its 12 MMAs start
// a fresh float32 accumulator in TMEM (two, alternating), and while the next
// chunk's MMAs run, the threads add the finished chunk into float64 registers:
// the tensor core's float32 accumulation then spans 64 features only, so its
// rounding stays at the level of a float32 dot product of that length.  The
// cross terms are issued before hi.hi so that they are added while the
// accumulator is small.  When a tile's last chunk is absorbed, `epi(tile_lo,
// acc)` runs on every thread: warp w holds TMEM lanes 32(w%4).. (targets) and,
// if 16(w/4) < N, columns 16(w/4)..+15 (sources) of the tile in acc[16].
//
// Operand stages (kTcStages deep) are filled by cp.async with 16-byte pieces
// of gathered rows into 128B-swizzled K-major tiles by all warps but the
// last; lane 0 of the last warp issues the MMAs and commits each step to its
// stage's mbarrier, queueing step g before step g-1 is waited for.  Every
// commit is waited for exactly once, in order, so the phase parities follow
// from the running step counter c.tc_g.  A wait that times out sets the group's error flag and
// the product returns false.
template <class Epi>
__device__ bool tc_product(int ns, int lo, int hi, bool global_targets, Epi &&epi)
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    const InstanceDesc &D = block_shared().D;
    const Chunk ck = chunk_at(c.choff, block_shared().D.chunk_cap);
    const long long tcg = c.tc_g;
    const int NK = D.x.nchunk;
    const int ntiles = hi > lo ? (hi - lo + kTcM - 1) / kTcM : 0;
    const int total = ntiles * NK;
    if (total <= 0 || ns <= 0) return true;
    const int N = (ns + 15) & ~15;                      // MMA N for M = 128: multiple of 16
    const uint32_t idesc = D.form == FORM_TF32 ? tc::idesc_tf32_f32(kTcM, N) : tc::idesc_f16_f32(kTcM, N, D.form == FORM_BF16X3);
    const uint32_t sbytes = (uint32_t)tc_stage_bytes(D.tc_n);
    const uint32_t a_lo = kTcM * 128u;                  // target lo tile
    const uint32_t b_hi = 2u * kTcM * 128u;             // source hi tile
    const uint32_t b_lo = b_hi + (uint32_t)D.tc_n * 128u;
    const long long rs = (long long)NK * 2 * kSplitChunk;
    const uint16_t *Xs = D.x.Xs;
    const int warp = threadIdx.x >> 5;
    const int lg = warp & 3, cg = warp >> 2;
    const bool reader = cg * 16 < N;
    // the last warp issues the MMAs and takes no part in the loads, so that
    // the issue overlaps the other warps' absorb and loads
    const int issuer = (int)(blockDim.x >> 5) - 1;
    const int nload = (int)blockDim.x - 32;
    auto load = [&](int g) {
        if (warp == issuer) return;
        const int tile = g / NK, kc = g - tile * NK;
        const uint32_t sa = c.tcbase + (uint32_t)((tcg + g) % kTcStages) * sbytes;
        const int tb = lo + tile * kTcM;
        for (int i = threadIdx.x; i < kTcM * 16; i += nload) {
            const int r = i >> 4, q = i & 15;
            const int t = tb + r;
            const bool ok = t < hi;
            const int row = ok ? (global_targets ? D.pos_row[t] : ck.Row[t]) : 0;
            tc::cp_async16(sa + (q >= 8 ? a_lo : 0u) + tc::sw128_offset(r, q & 7),
                           Xs + (long long)row * rs + kc * 128 + q * 8, ok ? 16u : 0u);
        }
        for (int i = threadIdx.x; i < N * 16; i += nload) {
            const int r = i >> 4, q = i & 15;
            const bool ok = r < ns;
            const int row = ok ? sh.tsrow[r] : 0;
            tc::cp_async16(sa + (q >= 8 ? b_lo : b_hi) + tc::sw128_offset(r, q & 7),
                           Xs + (long long)row * rs + kc * 128 + q * 8, ok ? 16u : 0u);
        }
    };
    double acc[16];
#pragma unroll
    for (int k = 0; k < 16; k++) acc[k] = 0.0;
    // add the finished chunk of global step Gs (its MMAs have completed) into acc
    auto absorb = [&](long long Gs) {
        tc::tc_fence_after();
        if (reader) {
            float v[16];
            tc::tmem_ld16(sh.tmem + ((uint32_t)(lg * 32) << 16) + (uint32_t)((Gs & 1) * kTcMaxN + cg * 16), v);
#pragma unroll
            for (int k = 0; k < 16; k++) acc[k] = __dadd_rn(acc[k], (double)v[k]);
        }
    };
    auto finish_tile = [&](int tile) {
        epi(lo + tile * kTcM, acc);
#pragma unroll
        for (int k = 0; k < 16; k++) acc[k] = 0.0;
    };
    for (int g = 0; g < kTcStages - 1; g++) {
        if (g < total) load(g);
        tc::cp_async_commit();
    }
    bool ok = true;
    for (int g = 0; g < total; g++) {
        const long long G = tcg + g;
        const int tile = g / NK, kc = g - tile * NK;
        // step g has landed: the groups of steps g+1 .. g+kTcStages-2 may still be pending
        tc::cp_async_wait<kTcStages - 2>();
        tc::fence_async_smem();
        __syncthreads();
        // step g's MMAs go in before step g-1's are waited for, so the tensor
        // core always has the next step queued.  Its accumulator (G & 1) was
        // last read by the absorb of step G-2, which ended before the barrier
        // that closed the previous iteration.
        if (threadIdx.x == (unsigned)(issuer * 32)) {
            tc::tc_fence_after();
            const uint32_t sa = c.tcbase + (uint32_t)(G % kTcStages) * sbytes;
            const uint32_t dst = sh.tmem + (uint32_t)((G & 1) * kTcMaxN);
            if (D.form == FORM_TF32) {
                // the two 128-byte halves hold features 0..31 and 32..63 of the chunk
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int kk = 0; kk < 4; kk++)
                        tc::mma_tf32(dst, tc::sw128_desc(sa + (h ? a_lo : 0u) + kk * 32),
                                     tc::sw128_desc(sa + (h ? b_lo : b_hi) + kk * 32), idesc, h > 0 || kk > 0);
            } else {
#pragma unroll
                // the small cross terms of the whole chunk first, then hi.hi (the
                // tensor core's fp32 accumulation rounds toward zero; see the
                // kernel-block kernel): dots measured 2x less biased this way
                for (int kk = 0; kk < 4; kk++) {
                    const uint64_t ah = tc::sw128_desc(sa + kk * 32), al = tc::sw128_desc(sa + a_lo + kk * 32);
                    const uint64_t bh = tc::sw128_desc(sa + b_hi + kk * 32), bl = tc::sw128_desc(sa + b_lo + kk * 32);
                    tc::mma_bf16(dst, ah, bl, idesc, kk > 0);
                    tc::mma_bf16(dst, al, bh, idesc, true);
                }
#pragma unroll
                for (int kk = 0; kk < 4; kk++)
                    tc::mma_bf16(dst, tc::sw128_desc(sa + kk * 32), tc::sw128_desc(sa + b_hi + kk * 32), idesc, true);
            }
            tc::mma_commit(&sh.tbar[G % kTcStages]);
        }
        bool w = true;
        if (g >= 1) {
            // step g-1's MMAs have read their stage and written their accumulator
            w = tc::mbar_wait(&sh.tbar[(G - 1) % kTcStages], (unsigned)(((G - 1) / kTcStages) & 1));
            if (w) {
                absorb(G - 1);
                if (kc == 0) finish_tile(tile - 1);
            }
        }
        // the stage of step g-1 is free: step g + kTcStages - 1 goes there
        if (w && g + kTcStages - 1 < total) load(g + kTcStages - 1);
        tc::cp_async_commit();
        tc::tc_fence_before();
        ok = __syncthreads_and(w) != 0;
        if (!ok) break;
    }
    if (ok) {
        const long long G = tcg + total - 1;
        ok = __syncthreads_and(tc::mbar_wait(&sh.tbar[G % kTcStages], (unsigned)((G / kTcStages) & 1))) != 0;
        if (ok) {
            absorb(G);
            finish_tile(ntiles - 1);
            tc::tc_fence_before();
        }
    }
    tc::cp_async_wait<0>();
    if (threadIdx.x == 0) c.tc_g += total;
    if (!ok && threadIdx.x == 0) atomicExch(&D.sync->error, 1);
    __syncthreads();
    return ok;
}

// tensor-core form of fill_rows: Q rows of ns (<= kPrefetchMax) sources into
// cache slots, on my chunk of [0,A) (tail = 0) or of [A,l) (tail = 1).
//
// A warp-specialised pipeline over the steps (one 64-feature chunk of one
// 128-target tile) with no block barrier per step:
//   warps kFillLoad0..  load a step's target tile and source rows into a free
//                       operand stage (cp.async), wait for their own copies,
//                       fence them into the async proxy and arrive on ffull;
//   warp 4, one lane    waits for ffull and for a free accumulator, issues the
//                       step's MMAs and commits them to fempty (stage free) and
//                       faccf (accumulator written);
//   warps 0-3           (TMEM lanes = the tile's 128 targets) wait for faccf,
//                       add the fp32 chunk into fp64 registers, arrive on facce,
//                       and write the tile's Q values after its last chunk.
// The MMAs, their order and the fp64 flush are those of tc_product, so the Q
// values are the same bit for bit.  Every wait is bounded; a role whose wait
// runs out sets fabort, which ends the other roles' waits.
__device__ __noinline__ bool fill_rows_tc(int ns, int tail)
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    const InstanceDesc &D = block_shared().D;
    const Chunk ck = chunk_at(c.choff, block_shared().D.chunk_cap);
    const long long fg = c.fg;
    if (ns == 0) return true;
    if (threadIdx.x < ns) {
        // the sources' row, norm, inverse scale, label and destination row
        const int k = threadIdx.x;
        sh.tsrow[k] = sh.frow[k];
        sh.fsx[k] = D.x.xsq[sh.frow[k]];
        sh.tsi[k] = D.x.xinv ? D.x.xinv[sh.frow[k]] : 1.0;
        sh.fsy[k] = sh.fy[k];
        sh.fsd[k] = D.cache.data + (long long)sh.fslot[k] * D.cache.stride;
    }
    __syncthreads();
    const int lo = tail ? c.t0 : 0, hi = tail ? c.t1 : c.a1 - c.a0;
    const int NK = D.x.nchunk;
    const int ntiles = hi > lo ? (hi - lo + kTcM - 1) / kTcM : 0;
    const int total = ntiles * NK;
    if (total <= 0) return true;
    const int S = c.fstages;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int *abort = &sh.fabort;
    constexpr uint32_t kStage = (uint32_t)fill_stage_bytes();
    constexpr uint32_t a_lo = kTcM * 128u;                       // target lo tile
    constexpr uint32_t b_hi = 2u * kTcM * 128u;                  // source hi tile
    constexpr uint32_t b_lo = b_hi + (uint32_t)kFillN * 128u;    // source lo tile
    const long long rs = (long long)NK * 2 * kSplitChunk;
    if (warp < 4) {
        // ---- readers and epilogue: target t = tile base + warp * 32 + lane.
        // The target's row norm, scale, label and cache column are loaded when
        // its tile starts, so the epilogue waits on no global load.
        double acc[kPrefetchMax];
#pragma unroll
        for (int k = 0; k < kPrefetchMax; k++) acc[k] = 0.0;
        int a = (int)(fg % kFillAcc);
        unsigned ph = (unsigned)((fg / kFillAcc) & 1);
        int kc = 0, tile = 0;
        int yp = 0, col = 0;
        bool tok = false;
        double xe = 0.0, ie = 1.0;
        for (int g = 0; g < total; g++) {
            if (kc == 0) {
                const int t = lo + tile * kTcM + warp * 32 + lane;
                tok = t < hi;
                if (tok) {
                    int r;
                    if (tail) {
                        r = D.pos_row[t];
                        yp = D.y[t];
                        col = D.pos_local[t];
                    } else {
                        r = ck.Row[t];
                        yp = flag_y(ck.F[t]);
                        col = ck.Col[t];
                    }
                    xe = D.x.xsq[r];
                    ie = D.x.xinv ? D.x.xinv[r] : 1.0;
                }
            }
            if (!tc::mbar_wait_or(&sh.faccf[a], ph, abort)) {
                *abort = 1;
                break;
            }
            tc::tc_fence_after();
            float v[kPrefetchMax];
            tc::tmem_ld8(sh.tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(a * kFillN), v);
#pragma unroll
            for (int k = 0; k < kPrefetchMax; k++) acc[k] = __dadd_rn(acc[k], (double)v[k]);
            tc::tc_fence_before();
            tc::mbar_arrive(&sh.facce[a]);
            if (++a == kFillAcc) {
                a = 0;
                ph ^= 1u;
            }
            if (++kc == NK) {
                if (tok) {
#pragma unroll
                    for (int k = 0; k < kPrefetchMax; k++)
                        if (k < ns)
                            __stcg(sh.fsd[k] + col, q_of(sh.fsy[k] * yp,
                                                            __dmul_rn(__dmul_rn(acc[k], ie), sh.tsi[k]), sh.fsx[k], xe));
                }
#pragma unroll
                for (int k = 0; k < kPrefetchMax; k++) acc[k] = 0.0;
                kc = 0;
                tile++;
            }
        }
    } else if (warp == 4) {
        // ---- MMA issue
        if (lane == 0) {
            const uint32_t idesc = D.form == FORM_TF32 ? tc::idesc_tf32_f32(kTcM, kFillN)
                                                       : tc::idesc_f16_f32(kTcM, kFillN, D.form == FORM_BF16X3);
            int s = (int)(fg % S), a = (int)(fg % kFillAcc);
            unsigned phs = (unsigned)((fg / S) & 1), pha = (unsigned)((fg / kFillAcc) & 1);
            int issued = 0;
            for (int g = 0; g < total; g++) {
                if (!tc::mbar_wait_or(&sh.ffull[s], phs, abort) || !tc::mbar_wait_or(&sh.facce[a], pha ^ 1u, abort)) {
                    *abort = 1;
                    break;
                }
                tc::tc_fence_after();
                const uint32_t sa = c.tcbase + (uint32_t)s * kStage;
                const uint32_t dst = sh.tmem + (uint32_t)(a * kFillN);
                if (D.form == FORM_TF32) {
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int kk = 0; kk < 4; kk++)
                            tc::mma_tf32(dst, tc::sw128_desc(sa + (h ? a_lo : 0u) + kk * 32),
                                         tc::sw128_desc(sa + (h ? b_lo : b_hi) + kk * 32), idesc, h > 0 || kk > 0);
                } else {
                    // cross terms of the chunk first, then hi.hi (as in tc_product)
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {
                        tc::mma_bf16(dst, tc::sw128_desc(sa + kk * 32), tc::sw128_desc(sa + b_lo + kk * 32), idesc,
                                     kk > 0);
                        tc::mma_bf16(dst, tc::sw128_desc(sa + a_lo + kk * 32), tc::sw128_desc(sa + b_hi + kk * 32),
                                     idesc, true);
                    }
#pragma unroll
                    for (int kk = 0; kk < 4; kk++)
                        tc::mma_bf16(dst, tc::sw128_desc(sa + kk * 32), tc::sw128_desc(sa + b_hi + kk * 32), idesc, true);
                }
                tc::mma_commit(&sh.fempty[s]);
                tc::mma_commit(&sh.faccf[a]);
                issued++;
                if (++s == S) {
                    s = 0;
                    phs ^= 1u;
                }
                if (++a == kFillAcc) {
                    a = 0;
                    pha ^= 1u;
                }
            }
            if (issued < total && issued > 0) {
                // stopped early: let the MMAs already issued finish before the
                // stages and the accumulators are given up
                const long long G = fg + issued - 1;
                tc::mbar_wait(&sh.fempty[G % S], (unsigned)((G / S) & 1));
            }
        }
        __syncwarp();
    } else {
        // ---- operand loads: piece i of a step is a 16-byte piece of a target
        // row (i < 16 * kTcM) or of a source row; the pieces of a thread keep
        // their rows for a whole tile, only the chunk moves
        constexpr int kLoaders = kThreads - kFillLoad0 * 32;
        constexpr int kPieces = (16 * kTcM + 16 * kPrefetchMax + kLoaders - 1) / kLoaders;
        const int lt = threadIdx.x - kFillLoad0 * 32;
        const uint16_t *Xs = D.x.Xs;
        const uint16_t *src[kPieces];
        uint32_t off[kPieces];
        int s = (int)(fg % S), sd = s;
        unsigned phs = (unsigned)((fg / S) & 1);
        int kc = 0, tile = 0;
        bool run = true;
        // up to S - 1 steps in flight; a landed step is handed to the MMA
        // before this thread waits for a free stage, so that the MMAs of
        // consecutive steps queue back to back
        for (int g = 0; g < total + S - 1; g++) {
            if (g >= S - 1 && run) {
                // step g - (S - 1) has landed (S - 2 younger groups may be pending)
                tc::cp_async_wait_n(S - 2);
                tc::fence_async_smem();
                tc::mbar_arrive(&sh.ffull[sd]);
                if (++sd == S) sd = 0;
            }
            if (g < total && run) {
                if (kc == 0) {
                    const int tb = lo + tile * kTcM;
#pragma unroll
                    for (int j = 0; j < kPieces; j++) {
                        const int i = lt + j * kLoaders;
                        src[j] = nullptr;
                        off[j] = 0;
                        if (i < 16 * kTcM) {
                            const int r = i >> 4, q = i & 15, t = tb + r;
                            if (t < hi) {
                                const int row = tail ? D.pos_row[t] : ck.Row[t];
                                src[j] = Xs + (long long)row * rs + q * 8;
                                off[j] = (q >= 8 ? a_lo : 0u) + tc::sw128_offset(r, q & 7);
                            }
                        } else if (i < 16 * kTcM + 16 * ns) {
                            const int r = (i - 16 * kTcM) >> 4, q = i & 15;
                            src[j] = Xs + (long long)sh.tsrow[r] * rs + q * 8;
                            off[j] = (q >= 8 ? b_lo : b_hi) + tc::sw128_offset(r, q & 7);
                        }
                    }
                }
                if (!tc::mbar_wait_or(&sh.fempty[s], phs ^ 1u, abort)) {
                    *abort = 1;
                    run = false;
                } else {
                    const uint32_t sa = c.tcbase + (uint32_t)s * kStage;
#pragma unroll
                    for (int j = 0; j < kPieces; j++)
                        if (src[j]) tc::cp_async16(sa + off[j], src[j] + kc * 128, 16u);
                }
                if (++s == S) {
                    s = 0;
                    phs ^= 1u;
                }
                if (++kc == NK) {
                    kc = 0;
                    tile++;
                }
            }
            tc::cp_async_commit();
        }
        tc::cp_async_wait<0>();
    }
    tc::tc_fence_before();
    __syncthreads();
    const bool ok = *abort == 0;
    if (threadIdx.x == 0) {
        c.fg += total;
        if (!ok) atomicExch(&D.sync->error, 1);
    }
    __syncthreads();
    tc::tc_fence_after();
    return ok;
}

// tensor-core form of accumulate_rows: sources are taken kTcMaxN (tc_n) at a
// time; per target the contributions of one pass are summed in source order
// in four column groups, which are then added in a fixed order
__device__ __noinline__ bool accumulate_rows_tc(int src_end, int pick_free_only, int with_bar, int lo, int hi)
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    const InstanceDesc &D = block_shared().D;
    const int cap = D.tc_n;
    int scan = 0;
    double *red = reinterpret_cast<double *>(c.tile);   // [2][4][kTcM] partial sums (aux area)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lg = warp & 3, cg = warp >> 2;
    while (true) {
        if (threadIdx.x == 0) sh.nsrc = 0;
        __syncthreads();
        while (scan < src_end) {
            const int p = scan + threadIdx.x;
            int sel = 0;
            if (p < src_end) {
                const unsigned char s = D.status[p];
                sel = pick_free_only ? (s == ST_FREE) : (s != ST_LOWER);
            }
            int tot;
            const int pre = block_excl_scan(sh.red, sel, &tot);
            const int have = sh.nsrc;
            const int room = cap - have;
            if (sel && pre < room) sh.tspos[have + pre] = p;
            const int take = tot < room ? tot : room;
            if (take < tot && sel && pre == take) sh.stop_at = threadIdx.x;
            __syncthreads();
            const int consumed = take == tot ? (int)blockDim.x : sh.stop_at;
            __syncthreads();
            if (threadIdx.x == 0) sh.nsrc = have + take;
            scan += consumed;
            __syncthreads();
            if (sh.nsrc == cap) break;
        }
        const int ns = sh.nsrc;
        if (ns == 0) break;
        if (threadIdx.x < ns) {
            const int sp = sh.tspos[threadIdx.x];
            const int r = D.pos_row[sp];
            const int y = D.y[sp];
            sh.tsrow[threadIdx.x] = r;
            sh.tsa[threadIdx.x] = D.alpha[sp];
            sh.tsx[threadIdx.x] = D.x.xsq[r];
            sh.tsi[threadIdx.x] = D.x.xinv ? D.x.xinv[r] : 1.0;
            sh.tsc[threadIdx.x] = get_C(D, y);
            sh.tsy[threadIdx.x] = (signed char)y;
            sh.tss[threadIdx.x] = D.status[sp];
        }
        __syncthreads();
        const bool ok = tc_product(ns, lo, hi, true, [&](int tlo, const double *acc) {
            const int t = tlo + lg * 32 + lane;
            double part = 0.0, partb = 0.0;
            if (cg * 16 < ns && t < hi) {
                const int r = D.pos_row[t];
                const int ye = D.y[t];
                const double xe = D.x.xsq[r];
                const double ie = D.x.xinv ? D.x.xinv[r] : 1.0;
#pragma unroll
                for (int k = 0; k < 16; k++) {
                    const int s = cg * 16 + k;
                    if (s < ns) {
                        const double dot = __dmul_rn(__dmul_rn(acc[k], ie), sh.tsi[s]);
                        const float q = q_of(sh.tsy[s] * ye, dot, sh.tsx[s], xe);
                        part = __dadd_rn(part, __dmul_rn(sh.tsa[s], (double)q));
                        if (with_bar && sh.tss[s] == ST_UPPER) partb = __dadd_rn(partb, __dmul_rn(sh.tsc[s], (double)q));
                    }
                }
            }
            red[cg * kTcM + lg * 32 + lane] = part;
            red[4 * kTcM + cg * kTcM + lg * 32 + lane] = partb;
            __syncthreads();
            if (cg == 0 && t < hi) {
                double g = D.G[t];
                for (int k = 0; k < 4; k++) g = __dadd_rn(g, red[k * kTcM + lg * 32 + lane]);
                D.G[t] = g;
                if (with_bar) {
                    double gb = D.G_bar[t];
                    for (int k = 0; k < 4; k++) gb = __dadd_rn(gb, red[4 * kTcM + k * kTcM + lg * 32 + lane]);
                    D.G_bar[t] = gb;
                }
            }
            __syncthreads();
        });
        if (!ok) return false;
        if (ns < cap) break;
    }
    return true;
}

// The same sums for a resident instance: the Q values are read from the cache,
// consecutive threads on neighbouring columns, instead of evaluated again.
// Sources go through shared memory a batch at a time: `batch` is a whole block
// of positions for the CUDA-core forms, whose sums run source by source, and
// one tensor-core pass for the others, whose sums run in four groups of 16.
template <int FORM>
__device__ __noinline__ void accumulate_resident(int src_end, int pick_free_only, int with_bar, int lo, int hi)
{
    Shared &sh = block_shared();
    const InstanceDesc &D = sh.D;
    constexpr bool tensor = is_tc_form(FORM);
    const int cap = tensor ? D.tc_n : kThreads;
    // the staging area holds the batch: alpha, C of the sources at the bound (0: not), column
    double *const ba = reinterpret_cast<double *>(dyn), *const bc = ba + kThreads;
    int *const bcol = reinterpret_cast<int *>(bc + kThreads);
    const float *const Q = D.cache.data;
    const long long stride = D.cache.stride;
    const bool tri = D.resident == kResidentTri;
    int scan = 0;
    while (true) {
        if (threadIdx.x == 0) sh.nsrc = 0;
        __syncthreads();
        while (scan < src_end) {
            const int p = scan + threadIdx.x;
            int sel = 0;
            unsigned char st = ST_LOWER;
            if (p < src_end) {
                st = D.status[p];
                sel = pick_free_only ? (st == ST_FREE) : (st != ST_LOWER);
            }
            int tot;
            const int pre = block_excl_scan(sh.red, sel, &tot);
            const int have = sh.nsrc, room = cap - have;
            if (sel && pre < room) {
                ba[have + pre] = D.alpha[p];
                bc[have + pre] = st == ST_UPPER ? get_C(D, D.y[p]) : 0.0;
                bcol[have + pre] = D.pos_local[p];
            }
            const int take = tot < room ? tot : room;
            if (take < tot && sel && pre == take) sh.stop_at = threadIdx.x;
            __syncthreads();
            const int consumed = take == tot ? (int)blockDim.x : sh.stop_at;
            __syncthreads();
            if (threadIdx.x == 0) sh.nsrc = have + take;
            scan += consumed;
            __syncthreads();
            if (sh.nsrc == cap) break;
        }
        const int ns = sh.nsrc;
        if (ns == 0) break;
        for (int e = lo + threadIdx.x; e < hi; e += blockDim.x) {
            const int ecol = D.pos_local[e];
            const float *const Qe = Q + ecol;
            double g = D.G[e], gb = with_bar ? D.G_bar[e] : 0.0;
            constexpr int kGroup = tensor ? 16 : 8;     // loads in flight; a tensor form's partial sum
            for (int k0 = 0; k0 < ns; k0 += kGroup) {
                float q[kGroup];
#pragma unroll
                for (int u = 0; u < kGroup; u++) q[u] = k0 + u >= ns ? 0.0f : tri ? Q[tri_at(bcol[k0 + u], ecol)] : Qe[bcol[k0 + u] * stride];
                double part = tensor ? 0.0 : g, partb = tensor ? 0.0 : gb;
#pragma unroll
                for (int u = 0; u < kGroup; u++) {
                    if (k0 + u >= ns) break;
                    part = __dadd_rn(part, __dmul_rn(ba[k0 + u], (double)q[u]));
                    const double C = bc[k0 + u];
                    if (with_bar && C != 0.0) partb = __dadd_rn(partb, __dmul_rn(C, (double)q[u]));
                }
                g = tensor ? __dadd_rn(g, part) : part;
                gb = tensor ? __dadd_rn(gb, partb) : partb;
            }
            D.G[e] = g;
            if (with_bar) D.G_bar[e] = gb;
        }
        __syncthreads();
        if (ns < cap) break;
    }
}

// the row-block product of the form: CUDA cores or tensor cores
template <int FORM>
__device__ bool accumulate(int src_end, int pick_free_only, int with_bar, int lo, int hi)
{
    if (block_shared().D.resident) {
        accumulate_resident<FORM>(src_end, pick_free_only, with_bar, lo, hi);
        return true;
    }
    if constexpr (is_tc_form(FORM)) {
        return accumulate_rows_tc(src_end, pick_free_only, with_bar, lo, hi);
    } else {
        accumulate_rows<FORM>(src_end, pick_free_only, with_bar, lo, hi);
        return true;
    }
}

// gradient reconstruction (reference svm.cpp:473-513); group collective on the
// global state (the caller has stored its chunk)
template <int FORM>
__device__ bool reconstruct()
{
    Ctx &c = block_shared().c;
    const InstanceDesc &D = block_shared().D;
    if (c.A == D.l) return true;
    if (D.lazy_gbar) {
        // G = p + sum over every alpha > 0 (active or not) of alpha * Q, on the inactive positions
        for (int e = c.t0 + threadIdx.x; e < c.t1; e += blockDim.x) D.G[e] = D.p[e];
        __syncthreads();
        if (!accumulate<FORM>(D.l, 0, 0, c.t0, c.t1)) return false;
        return exchange();
    }
    for (int e = c.t0 + threadIdx.x; e < c.t1; e += blockDim.x) D.G[e] = __dadd_rn(D.G_bar[e], D.p[e]);
    __syncthreads();
    if (!accumulate<FORM>(c.A, 1, 0, c.t0, c.t1)) return false;
    return exchange();
}

// --------------------------------------------------------------------------
// shrinking (reference svm.cpp:932-1011 / Solver_NU :1188-1258)
// --------------------------------------------------------------------------
__device__ __forceinline__ bool be_shrunk(int nu, unsigned char s, int y, double G, const double *g)
{
    if (!nu) {
        if (s == ST_UPPER) return y == +1 ? (-G > g[0]) : (-G > g[1]);
        if (s == ST_LOWER) return y == +1 ? (G > g[1]) : (G > g[0]);
        return false;
    }
    if (s == ST_UPPER) return y == +1 ? (-G > g[0]) : (-G > g[3]);
    if (s == ST_LOWER) return y == +1 ? (G > g[1]) : (G > g[2]);
    return false;
}

__device__ __forceinline__ void swap_pos(const InstanceDesc &D, int a, int b)
{
    double t;
    t = D.G[a]; D.G[a] = D.G[b]; D.G[b] = t;
    t = D.G_bar[a]; D.G_bar[a] = D.G_bar[b]; D.G_bar[b] = t;
    t = D.alpha[a]; D.alpha[a] = D.alpha[b]; D.alpha[b] = t;
    t = D.p[a]; D.p[a] = D.p[b]; D.p[b] = t;
    t = D.QD[a]; D.QD[a] = D.QD[b]; D.QD[b] = t;
    signed char ty = D.y[a]; D.y[a] = D.y[b]; D.y[b] = ty;
    unsigned char ts = D.status[a]; D.status[a] = D.status[b]; D.status[b] = ts;
    int ti = D.pos_local[a]; D.pos_local[a] = D.pos_local[b]; D.pos_local[b] = ti;
    ti = D.pos_row[a]; D.pos_row[a] = D.pos_row[b]; D.pos_row[b] = ti;
    ti = D.pos_slot[a]; D.pos_slot[a] = D.pos_slot[b]; D.pos_slot[b] = ti;
}

// widen the active set to l after a reconstruction (chunk reloaded).  Only
// complete rows stay cached, and of an inactive variable's only those whose
// slot no other row has taken since.
__device__ void widen()
{
    Ctx &c = block_shared().c;
    const InstanceDesc &D = block_shared().D;
    set_active(D.l);
    for (int p = c.a0 + threadIdx.x; p < c.a1 && !D.resident; p += blockDim.x) {
        const unsigned w = (unsigned)D.pos_slot[p], slot = w & 0xffffu;
        if (slot == kNoSlot) continue;
        if (!(w & kSlotFull) || __ldcg(&D.cache.tag[slot]) != D.pos_local[p]) D.pos_slot[p] = kNoSlot;
    }
    chunk_load();
}

// the whole gradient reconstructed and the active set widened (svm.cpp:598-611)
template <int FORM>
__device__ __noinline__ bool reopen()
{
    chunk_store();
    if (!exchange()) return false;
    if (!reconstruct<FORM>()) return false;
    widen();
    return true;
}

template <int FORM>
__device__ __noinline__ bool do_shrinking(int &unshrink)
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    const InstanceDesc &D = block_shared().D;
    const Chunk ck = chunk_at(c.choff, block_shared().D.chunk_cap);
    const int nu = D.nu;
    const int n = c.a1 - c.a0;
    // 1. maximal violations over the active set (C-SVC: Gmax1, Gmax2; nu: Gmax1..4)
    {
        double v[4] = {-SVMB_INF, -SVMB_INF, -SVMB_INF, -SVMB_INF};
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            const unsigned char s = flag_s(ck.F[k]);
            const double G = ck.G[k];
            const int y = flag_y(ck.F[k]);
            if (!nu) {
                if (y == +1) {
                    if (s != ST_UPPER) v[0] = fmax(v[0], -G);
                    if (s != ST_LOWER) v[1] = fmax(v[1], G);
                } else {
                    if (s != ST_UPPER) v[1] = fmax(v[1], -G);
                    if (s != ST_LOWER) v[0] = fmax(v[0], G);
                }
            } else {
                if (s != ST_UPPER) { if (y == +1) v[0] = fmax(v[0], -G); else v[3] = fmax(v[3], -G); }
                if (s != ST_LOWER) { if (y == +1) v[1] = fmax(v[1], G); else v[2] = fmax(v[2], G); }
            }
        }
        block_max<4>(sh.red, v);
        if (threadIdx.x == 0) {
            Partial *pp = my_partial();
            for (int k = 0; k < 4; k++) pp->v[k] = v[k];
        }
    }
    chunk_store();     // the swaps and a reconstruction work on the global state
    if (!exchange()) return false;
    double g[4];
    {
        const Partial *all = prev_partials();
        double v[4] = {-SVMB_INF, -SVMB_INF, -SVMB_INF, -SVMB_INF};
        for (int b = threadIdx.x; b < c.nb; b += blockDim.x)
            for (int k = 0; k < 4; k++) v[k] = fmax(v[k], c.nb == 1 ? all[b].v[k] : __ldcg(&all[b].v[k]));
        block_max<4>(sh.red, v);
        for (int k = 0; k < 4; k++) g[k] = v[k];
    }
    const double gap = nu ? fmax(__dadd_rn(g[0], g[1]), __dadd_rn(g[2], g[3])) : __dadd_rn(g[0], g[1]);
    if (!unshrink && gap <= __dmul_rn(D.eps, 10.0)) {
        unshrink = 1;
        if (!reconstruct<FORM>()) return false;
        widen();
    }
    // 2. shrunk positions per block -> new active size K
    {
        int cnt = 0;
        for (int k = threadIdx.x; k < c.a1 - c.a0; k += blockDim.x)
            cnt += be_shrunk(nu, flag_s(ck.F[k]), flag_y(ck.F[k]), ck.G[k], g) ? 1 : 0;
        cnt = block_sum_i(sh.red, cnt);
        if (threadIdx.x == 0) my_partial()->n[0] = cnt;
    }
    if (!exchange()) return false;
    int K;
    {
        int below, above, tot;
        group_counts(0, &below, &above, &tot);
        K = c.A - tot;
    }
    // 3. holes = shrunk positions in [0,K) ascending, movers = kept positions in [K,A) descending
    {
        int h = 0, m = 0;
        for (int k = threadIdx.x; k < c.a1 - c.a0; k += blockDim.x) {
            const int p = c.a0 + k;
            const bool s = be_shrunk(nu, flag_s(ck.F[k]), flag_y(ck.F[k]), ck.G[k], g);
            if (p < K && s) h++;
            if (p >= K && !s) m++;
        }
        h = block_sum_i(sh.red, h);
        m = block_sum_i(sh.red, m);
        if (threadIdx.x == 0) { Partial *pp = my_partial(); pp->n[0] = h; pp->n[1] = m; }
    }
    if (!exchange()) return false;
    int hole_base, movers_below, movers_above, total_movers, dummy0, dummy1;
    group_counts(0, &hole_base, &dummy0, &dummy1);
    group_counts(1, &movers_below, &movers_above, &total_movers);
    int *holes = D.scratch;
    int *movers = D.scratch + D.l;
    {
        int h_run = 0, m_run = 0;
        for (int base = 0; base < c.a1 - c.a0; base += blockDim.x) {
            const int k = base + threadIdx.x;
            const int p = c.a0 + k;
            bool s = false;
            if (p < c.a1) s = be_shrunk(nu, flag_s(ck.F[k]), flag_y(ck.F[k]), ck.G[k], g);
            const int isH = (p < c.a1 && p < K && s) ? 1 : 0;
            const int isM = (p < c.a1 && p >= K && !s) ? 1 : 0;
            int totH, totM;
            const int preH = block_excl_scan(sh.red, isH, &totH);
            const int preM = block_excl_scan(sh.red, isM, &totM);
            if (isH) holes[hole_base + h_run + preH] = p;
            if (isM) {
                const int asc = movers_below + m_run + preM;        // ascending rank among movers
                movers[total_movers - 1 - asc] = p;                 // descending pairing order
            }
            h_run += totH;
            m_run += totM;
        }
    }
    if (!exchange()) return false;
    // 4. swap pair r: holes[r] <-> movers[r] (the reference's swap_index loop)
    for (long long r = (long long)c.rank * blockDim.x + threadIdx.x; r < total_movers; r += (long long)c.nb * blockDim.x)
        swap_pos(D, __ldcg(&holes[r]), __ldcg(&movers[r]));
    if (!exchange()) return false;
    set_active(K);
    chunk_load();
    return true;
}

// --------------------------------------------------------------------------
// I_up scan of my chunk (first half of WSS3): per track the max of -y_t G_t
// with its payload.  C-SVC uses track 0 only; nu-SVC: track 0 = y=+1, 1 = y=-1.
// --------------------------------------------------------------------------
// Prefetch priority of a position: how strongly it violates optimality on
// either side, max(-y G over I_up, y G over I_low) -- the quantities whose
// extremes WSS picks from, so high-priority rows are likely to be needed soon.
__device__ __forceinline__ double prefetch_priority(int y, unsigned char s, double G)
{
    double up = -SVMB_INF, low = -SVMB_INF;
    if (y == +1) {
        if (s != ST_UPPER) up = -G;
        if (s != ST_LOWER) low = G;
    } else {
        if (s != ST_LOWER) up = G;
        if (s != ST_UPPER) low = -G;
    }
    return fmax(up, low);
}

// Wait until the W words at p carry sequence number `want`; false when the
// group's error flag is set or the wait's bound runs out.
template <int W>
__device__ __forceinline__ bool poll_words(const InstanceDesc &D, const RecWord *p, unsigned want, RecWord (&w)[W])
{
    long long t0 = 0;
    for (unsigned spins = 1;; spins++) {
        bool all = true;
#pragma unroll
        for (int k = 0; k < W; k++) w[k] = ld_word(p + k);
#pragma unroll
        for (int k = 0; k < W; k++) all = all && (unsigned)(w[k].hi >> 32) == want;
        if (all) return true;
        if ((spins & 255u) == 0) {
            const long long now = (long long)tc::global_ns();
            if (t0 == 0) t0 = now;
            const long long limit = D.wait_ns > 0 ? D.wait_ns : kWaitTimeoutNs;
            if (ld_relaxed_i32(&D.sync->error) != 0 || now - t0 > limit) {
                atomicExch(&D.sync->error, 1);
                return false;
            }
        }
    }
}

// One poll warp's part of a phase-A exchange: the records of blocks 32 warp ..
// + 31, the best of each of the T tracks left in sh.wa[warp].
template <int T>
__device__ __forceinline__ void poll_iup(unsigned seq, int warp, int lane)
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    const int b = warp * 32 + lane;
    RecWord w[kWordsI * T];
    bool ok = true;
    if (b < c.nb) ok = poll_words<kWordsI * T>(sh.D, sh.D.words + (long long)b * kRecWords + kWordA, seq, w);
    if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) sh.fail = 1;
        return;
    }
#pragma unroll
    for (int t = 0; t < T; t++) {
        const int p = b < c.nb ? code_pos((unsigned)w[kWordsI * t].hi) : -1;
        u64 key = p >= 0 ? key_of(__longlong_as_double((long long)w[kWordsI * t].lo)) : 0;
        int best = p;
        warp_best(key, best);
        if (best >= 0 ? p == best : lane == 0) {
#pragma unroll
            for (int e = 0; e < kWordsI; e++) {
                sh.wa[warp].d[kWordsI * t + e] = __longlong_as_double((long long)w[kWordsI * t + e].lo);
                sh.wa[warp].x[kWordsI * t + e] = (unsigned)w[kWordsI * t + e].hi;
            }
        }
    }
}

// Exchange of the block's I_up maxima (per track, with payload) and, with
// `ahead`, publication of its most violating positions (prefetch candidates:
// the best of each warp, top kPrefetchCand).  The group's winners are in sh.wa.
template <int nu>
__device__ __forceinline__ bool iup_publish(unsigned seq, bool ahead, const double (&v)[2],
                                            const int (&ix)[2], double pv, int pix)
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    const Chunk ck = chunk_at(c.choff, block_shared().D.chunk_cap);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u64 k0 = ix[0] >= 0 ? key_of(v[0]) : 0, k1 = 0;
    int p0 = ix[0], p1 = -1;
    warp_best(k0, p0);
    if (nu) {
        k1 = ix[1] >= 0 ? key_of(v[1]) : 0;
        p1 = ix[1];
        warp_best(k1, p1);
    }
    if (ahead) {
        u64 kp = pix >= 0 && pv > -SVMB_INF ? key_of(pv) : 0;
        int pp = kp ? pix : -1;
        warp_best(kp, pp);
        if (lane == 0) {
            sh.wk[2][warp] = kp;
            sh.wp[warp] = pp;
        }
    }
    if (lane == 0) {
        sh.wk[0][warp] = k0;
        sh.wi[0][warp] = p0;
        sh.wk[1][warp] = k1;
        sh.wi[1][warp] = p1;
    }
    __syncthreads();
    RecWord *mine = sh.D.words + (long long)c.rank * kRecWords;
    if (warp < kPollWarps) {
        if (warp == 0) {
            k0 = lane < kWarps ? sh.wk[0][lane] : 0;
            p0 = lane < kWarps ? sh.wi[0][lane] : -1;
            warp_best(k0, p0);
            if (nu) {
                k1 = lane < kWarps ? sh.wk[1][lane] : 0;
                p1 = lane < kWarps ? sh.wi[1][lane] : -1;
                warp_best(k1, p1);
            }
            if (lane < (nu ? 2 : 1) * kWordsI) {
                // lane 4t + e builds word e of track t, without branches: words 0 to
                // 2 carry the 1st to 3rd of G, alpha and QD
                const int p = lane < kWordsI ? p0 : p1, e = lane & (kWordsI - 1), q = p >= 0 ? p - c.a0 : 0;
                double d = ck.G[min(e, 2) * sh.D.chunk_cap + q];
                const unsigned f = ck.F[q];
                if (e == 0 && flag_y(f) > 0) d = -d;
                const unsigned col = (unsigned)ck.Col[q], row = (unsigned)ck.Row[q], slot = slot_word(ck.Slot[q], f);
                unsigned x = e == 0 ? pos_code(p, flag_y(f)) : e == 1 ? col : e == 2 ? slot : row;
                if (p < 0) {
                    d = -SVMB_INF;
                    x = kNoPos;
                }
                if (c.nb == 1) {
                    sh.wa[0].d[lane] = d;
                    sh.wa[0].x[lane] = x;
                } else {
                    st_word(mine + kWordA + lane, d, x, seq);
                }
            }
            __syncwarp();
        }
        if (c.nb > 1 && warp * 32 < c.nb) {
            if (nu) poll_iup<2>(seq, warp, lane);
            else poll_iup<1>(seq, warp, lane);
        }
    } else if (warp == kPollWarps && ahead) {
        // the warps' best by rank: lane w counts the warps ahead of warp w
        const u64 k = lane < kWarps ? sh.wk[2][lane] : 0;
        const int p = lane < kWarps ? sh.wp[lane] : -1;
        int rank = 0;
#pragma unroll
        for (int j = 0; j < kWarps; j++) {
            const u64 kj = __shfl_sync(0xffffffffu, k, j);
            const int pj = __shfl_sync(0xffffffffu, p, j);
            rank += kj > k || (kj == k && pj > p) ? 1 : 0;
        }
        const int found = __popc(__ballot_sync(0xffffffffu, p >= 0));
        Cand cd{-SVMB_INF, kNoPos, 0u, 0u, (unsigned)kNoSlot};
        int at = -1;
        if (p >= 0) {
            const int q = p - c.a0;
            cd.v = key_value(k);
            cd.pc = pos_code(p, flag_y(ck.F[q]));
            cd.col = (unsigned)ck.Col[q];
            cd.row = (unsigned)ck.Row[q];
            cd.slot = ck.Slot[q];
            if (rank < kPrefetchCand) at = rank;
        }
        // the places no warp takes are marked empty by lanes kWarps ..
        if (lane >= kWarps && lane < kWarps + kPrefetchCand - found) at = found + lane - kWarps;
        if (at >= 0) {
            if (c.nb == 1) {
                sh.cand[at] = cd;
            } else {
                st_word(mine + kWordCand + 2 * at, cd.v, cd.pc, seq);
                st_word(mine + kWordCand + 2 * at + 1, __longlong_as_double((long long)cd.col | ((long long)cd.row << 32)),
                        cd.slot, seq);
            }
        }
    }
    __syncthreads();
    return sh.fail == 0;
}

template <int nu>
__device__ __noinline__ bool scan_iup(unsigned seq)
{
    Ctx &c = block_shared().c;
    const Chunk ck = chunk_at(c.choff, block_shared().D.chunk_cap);
    double v[2] = {-SVMB_INF, -SVMB_INF};
    int ix[2] = {-1, -1};
    double pv = -SVMB_INF;
    int pix = -1;
    for (int k = threadIdx.x; k < c.a1 - c.a0; k += blockDim.x) {
        const unsigned char s = flag_s(ck.F[k]);
        const double G = ck.G[k];
        const int y = flag_y(ck.F[k]);
        if (y == +1) {
            if (s != ST_UPPER) better_max(v[0], ix[0], -G, c.a0 + k);
        } else {
            if (s != ST_LOWER) better_max(v[nu], ix[nu], G, c.a0 + k);
        }
        better_max(pv, pix, prefetch_priority(y, s, G), c.a0 + k);
    }
    return iup_publish<nu>(seq, block_shared().D.prefetch > 1, v, ix, pv, pix);
}

// One poll warp's part of a phase-B exchange (W words a record).
template <int W>
__device__ __forceinline__ void poll_j(unsigned seq, int warp, int lane)
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    const int b = warp * 32 + lane;
    RecWord w[W];
    bool ok = true;
    if (b < c.nb) ok = poll_words<W>(sh.D, sh.D.words + (long long)b * kRecWords + kWordB, seq, w);
    if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) sh.fail = 1;
        return;
    }
    const int p = b < c.nb ? code_pos((unsigned)w[0].hi) : -1;
    u64 key = p >= 0 ? key_of(__longlong_as_double((long long)w[0].lo)) : 0;
    int best = p;
    warp_best(key, best);
    const u64 g2 = warp_max_key(b < c.nb ? key_of(__longlong_as_double((long long)w[4].lo)) : 0);
    u64 g2n = 0;
    if (W > 5) g2n = warp_max_key(b < c.nb ? key_of(__longlong_as_double((long long)w[W - 1].lo)) : 0);
    if (best >= 0 ? p == best : lane == 0) {
#pragma unroll
        for (int e = 0; e < W; e++) {
            if (e < 4) sh.wb[warp].d[e] = __longlong_as_double((long long)w[e].lo);
            sh.wb[warp].x[e] = (unsigned)w[e].hi;
        }
    }
    if (lane == 0) {
        sh.wb[warp].d[4] = key_value(g2);
        if (W > 5) sh.wb[warp].d[5] = key_value(g2n);
    }
}

// Exchange of the block's second-order j candidate (largest decrease, with
// payload) and its Gmax2 maxima; the group's are in sh.wb.
template <int nu>
__device__ __forceinline__ bool j_publish(unsigned seq, double dec, int jx, float jq, double g2,
                                          double g2n)
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    const Chunk ck = chunk_at(c.choff, block_shared().D.chunk_cap);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u64 k = jx >= 0 ? key_of(dec) : 0;
    int p = jx;
    warp_best(k, p);
    u64 kg = warp_max_key(key_of(g2)), kn = 0;
    if (nu) kn = warp_max_key(key_of(g2n));
    if (jx == p && p >= 0) sh.wq[warp] = jq;
    if (lane == 0) {
        sh.wk[0][warp] = k;
        sh.wi[0][warp] = p;
        sh.wk[1][warp] = kg;
        sh.wk[2][warp] = kn;
    }
    __syncthreads();
    if (warp < kPollWarps) {
        if (warp == 0) {
            const int m = lane & (kWarps - 1), mi = sh.wi[0][m];
            const float mq = sh.wq[m];
            k = sh.wk[0][m];
            p = mi;
            warp_best(k, p);
            kg = warp_max_key(sh.wk[1][m]);
            if (nu) kn = warp_max_key(sh.wk[2][m]);
            const float jqv = __shfl_sync(0xffffffffu, mq, __ffs(__ballot_sync(0xffffffffu, mi == p)) - 1);
            if (lane < kWordsJ) {
                // without branches: words 1 to 3 carry the 1st to 3rd of G, alpha and QD
                const int q = p >= 0 ? p - c.a0 : 0;
                const double g = ck.G[min(max(lane - 1, 0), 2) * sh.D.chunk_cap + q];
                const unsigned f = ck.F[q], col = (unsigned)ck.Col[q], row = (unsigned)ck.Row[q], slot = slot_word(ck.Slot[q], f);
                const u64 kd = lane == 0 ? k : lane == 4 ? kg : kn;
                const double d = lane >= 1 && lane <= 3 ? g : nu || lane < 5 ? key_value(kd) : 0.0;
                const unsigned x = p < 0 ? kNoPos : lane == 0 ? pos_code(p, flag_y(f)) : lane == 1 ? col : lane == 2 ? row :
                                   lane == 3 ? slot : __float_as_uint(jqv);
                if (c.nb == 1) {
                    sh.wb[0].d[lane] = d;
                    sh.wb[0].x[lane] = x;
                } else {
                    st_word(sh.D.words + (long long)c.rank * kRecWords + kWordB + lane, d, x, seq);
                }
            }
            __syncwarp();
        }
        if (c.nb > 1 && warp * 32 < c.nb) {
            if (nu) poll_j<kWordsJ>(seq, warp, lane);
            else poll_j<kWordsJ - 1>(seq, warp, lane);
        }
    }
    __syncthreads();
    return sh.fail == 0;
}

// which poll warp's record of track t wins (larger value, ties to the larger position)
__device__ __noinline__ int win_iup(int np, int t)
{
    Shared &sh = block_shared();
    int e = 0;
    for (int k = 1; k < np; k++) {
        const double a = sh.wa[e].d[kWordsI * t], b = sh.wa[k].d[kWordsI * t];
        const int pa = code_pos(sh.wa[e].x[kWordsI * t]), pb = code_pos(sh.wa[k].x[kWordsI * t]);
        if (pb >= 0 && (pa < 0 || b > a || (b == a && pb > pa))) e = k;
    }
    return e;
}
__device__ __noinline__ int win_j(int np)
{
    Shared &sh = block_shared();
    int e = 0;
    for (int k = 1; k < np; k++) {
        const double a = sh.wb[e].d[0], b = sh.wb[k].d[0];
        const int pa = code_pos(sh.wb[e].x[0]), pb = code_pos(sh.wb[k].x[0]);
        if (pb >= 0 && (pa < 0 || b > a || (b == a && pb > pa))) e = k;
    }
    return e;
}

// Dot products of the 32 rows of a warp (lane L owns row r) with up to 8
// staged dense sources.  The 32 rows are read in 16-column slices with
// coalesced 64-byte pieces per row (cp.async, 16 bytes per lane) into 32 x 16
// shared tiles (pieces swizzled).  The warp's tiles form a ring of
// D.tile_bufs slices: all but the one in use are in flight, so a warp moves
// tile_bufs slices per memory round trip.  Every lane accumulates ITS row in
// feature order from the tile -- the reference's summation order.
// shared-memory loads by 32-bit shared-window address (volatile: they stay
// after the cp.async wait and __syncwarp that publish the tile)
__device__ __forceinline__ float4 lds_f4(uint32_t a)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ double2 lds_d2(uint32_t a)
{
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
    return v;
}
// four staged source values at byte address a: float4, or two double2
__device__ __forceinline__ float4 src4_at(uint32_t a, float) { return lds_f4(a); }
__device__ __forceinline__ D4 src4_at(uint32_t a, double)
{
    const double2 p = lds_d2(a), q = lds_d2(a + 16);
    return D4{p.x, p.y, q.x, q.y};
}

// what a fill pass's warps need of the descriptor, in registers
struct TileJob {
    const float *X;
    int ld;             // multiple of 4
    int bufs;           // tiles in the warp's ring
    uint32_t sstride;   // the staged sources lie this many bytes apart
    uint32_t src0, tile;
};

template <int FORM, int NS, typename S>
__device__ __forceinline__ void warp_tile_dots(const TileJob &J, int ns, int r, double (&out)[kPrefetchMax])
{
    typedef typename Acc<FORM>::type acc_t;
    const int lane = threadIdx.x & 31;
    const int ld = J.ld;
    const float *X = J.X;
    acc_t acc[NS];
#pragma unroll
    for (int k = 0; k < NS; k++) acc[k] = acc_t(0);
    const uint32_t src0 = J.src0, sstride = J.sstride, tile_s = J.tile;
    // a slice is 32 rows x 4 pieces of 16 bytes; lane L moves pieces L + 32i
    // (i < 4): row (L + 32i) / 4, piece L % 4.  Row t of a tile = the row of lane t.
    const float *prow[4];
#pragma unroll
    for (int i = 0; i < 4; i++) prow[i] = X + (long long)__shfl_sync(0xffffffffu, r, (lane + 32 * i) >> 2) * ld + 4 * (lane & 3);
    auto issue = [&](int c0, int buf) {
        if (c0 < ld) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int t = (lane + 32 * i) >> 2;
                const bool ok = c0 + 4 * (lane & 3) < ld;     // ld is a multiple of 4
                // piece c of tile row t sits at piece position c ^ ((t >> 1) & 3): the
                // 16-byte reads of 8 consecutive lanes then hit distinct banks
                tc::cp_async16(tile_s + (uint32_t)((buf * 32 * kTileStride + t * kTileStride + 4 * ((lane & 3) ^ ((t >> 1) & 3))) * 4),
                               prow[i] + (ok ? c0 : 0), ok ? 16u : 0u);
            }
        }
        tc::cp_async_commit();
    };
    const int nb = J.bufs;
    // prologue: slices 0 .. nb-2 in flight
    for (int p = 0; p + 1 < nb; p++) issue(16 * p, p);
    for (int c0 = 0, s = 0; c0 < ld; c0 += 16) {
        // slice s + nb - 1 goes to the buffer used by slice s - 1 (consumed
        // before the __syncwarp that ended the previous step)
        issue(c0 + 16 * (nb - 1), s == 0 ? nb - 1 : s - 1);
        tc::cp_async_wait_n(nb - 1);                     // slice s has landed (for this lane)
        __syncwarp();
        const uint32_t cur = tile_s + (uint32_t)(s * 32 * kTileStride * 4 + lane * kTileStride * 4);
        auto step = [&](int q) {    // columns c0 + q .. c0 + q + 3
            const float4 xv = lds_f4(cur + (uint32_t)(16 * ((q >> 2) ^ ((lane >> 1) & 3))));
            const uint32_t soff = (uint32_t)((c0 + q) * (int)sizeof(S));
#pragma unroll
            for (int k = 0; k < NS; k++) {
                const auto w = src4_at(src0 + (uint32_t)(k < ns ? k : 0) * sstride + soff, S());
                acc[k] = mac<FORM>(xv.x, w.x, acc[k]);
                acc[k] = mac<FORM>(xv.y, w.y, acc[k]);
                acc[k] = mac<FORM>(xv.z, w.z, acc[k]);
                acc[k] = mac<FORM>(xv.w, w.w, acc[k]);
            }
        };
        if (FORM == FORM_EXACT && ld - c0 >= 16) {
            // a whole slice, its four steps unrolled (the fp32 form keeps the
            // loop: eight float4 sources per step would not fit registers)
#pragma unroll
            for (int q = 0; q < 16; q += 4) step(q);
        } else {
            const int lim = ld - c0 < 16 ? ld - c0 : 16;    // multiple of 4
            for (int q = 0; q < lim; q += 4) step(q);
        }
        __syncwarp();
        s = s + 1 == nb ? 0 : s + 1;
    }
#pragma unroll
    for (int k = 0; k < NS; k++) out[k] = (double)acc[k];
}

// Evaluate the Q rows of `ns` (<= kPrefetchMax, <= stage_cap when staged)
// sources into cache slots on my chunk of [0,A) (tail = 0, from shared
// memory) or of [A,l) (tail = 1, global state).
template <int FORM, typename S>
__device__ __forceinline__ void tile_dots_ns(const TileJob &J, int ns, int r, double (&dots)[kPrefetchMax])
{
    switch (ns) {
    case 1: warp_tile_dots<FORM, 1, S>(J, ns, r, dots); break;
    case 2: warp_tile_dots<FORM, 2, S>(J, ns, r, dots); break;
    case 3: warp_tile_dots<FORM, 3, S>(J, ns, r, dots); break;
    case 4: warp_tile_dots<FORM, 4, S>(J, ns, r, dots); break;
    case 5: warp_tile_dots<FORM, 5, S>(J, ns, r, dots); break;
    case 6: warp_tile_dots<FORM, 6, S>(J, ns, r, dots); break;
    default: warp_tile_dots<FORM, 8, S>(J, ns, r, dots); break;
    }
}

template <int FORM>
__device__ __noinline__ void fill_rows(int ns, int tail)
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    const InstanceDesc &D = block_shared().D;
    const Chunk ck = chunk_at(c.choff, block_shared().D.chunk_cap);
    if (ns == 0) return;
    // per-source constants of this pass, read from shared memory where used
    if (threadIdx.x < ns) {
        const int k = threadIdx.x;
        sh.fsx[k] = D.x.xsq ? D.x.xsq[sh.frow[k]] : 0.0;
        sh.fsy[k] = sh.fy[k];
        sh.fsd[k] = D.cache.data + (long long)sh.fslot[k] * D.cache.stride;
    }
    stage_sources(D, c.stage, sh.ss, sh.frow, ns);   // ends with a barrier
    const int lo = tail ? c.t0 : 0, hi = tail ? c.t1 : c.a1 - c.a0;
    const double *const xsq = D.x.xsq;
    if (D.x.X && D.stage_cap > 0) {
        // dense rows, staged sources: warp-tiled, whole warps per 32 positions
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        float *const tile = c.tile + warp * (D.tile_bufs * 32 * kTileStride);
        const TileJob job{D.x.X, D.x.ld, D.tile_bufs, (uint32_t)(D.stage_lds * stage_elem(FORM)), tc::smem_addr(sh.ss.sp[0]), tc::smem_addr(tile)};
        for (int base = lo + warp * 32; base < hi; base += blockDim.x) {
            const int k = base + lane;
            const bool valid = k < hi;
            const int kk = valid ? k : base;     // idle lanes repeat a valid row
            int r, yp, col;
            if (tail) {
                r = D.pos_row[kk];
                yp = D.y[kk];
                col = D.pos_local[kk];
            } else {
                r = ck.Row[kk];
                yp = flag_y(ck.F[kk]);
                col = ck.Col[kk];
            }
            // the target's norm is loaded before the dots so that its latency hides behind them
            const double xe = xsq ? xsq[r] : 0.0;
            double dots[kPrefetchMax];
            // staged sources are float64 in the exact form
            if (FORM == FORM_EXACT) tile_dots_ns<FORM, double>(job, ns, r, dots);
            else tile_dots_ns<FORM, float>(job, ns, r, dots);
            if (valid) {
#pragma unroll
                for (int s2 = 0; s2 < kPrefetchMax; s2++)
                    if (s2 < ns) sh.fsd[s2][col] = q_of(sh.fsy[s2] * yp, dots[s2], sh.fsx[s2], xe);
            }
        }
    } else {
        for (int k = lo + threadIdx.x; k < hi; k += blockDim.x) {
            int r, yp, col;
            if (tail) {
                r = D.pos_row[k];
                yp = D.y[k];
                col = D.pos_local[k];
            } else {
                r = ck.Row[k];
                yp = flag_y(ck.F[k]);
                col = ck.Col[k];
            }
            double dots[kSrcBatch];
            row_dots<FORM>(D, sh.ss, ns, r, dots);
            const double xe = xsq ? xsq[r] : 0.0;
#pragma unroll
            for (int s2 = 0; s2 < kPrefetchMax; s2++)
                if (s2 < ns) sh.fsd[s2][col] = q_of(sh.fsy[s2] * yp, dots[s2], sh.fsx[s2], xe);
        }
    }
    unstage_sources(D, c.stage, sh.ss);
}

// the fill pass of the form (the rows listed in sh.f*): CUDA cores or tensor cores
template <int FORM>
__device__ __forceinline__ bool fill(int ns, int tail)
{
    if constexpr (is_tc_form(FORM)) {
        return fill_rows_tc(ns, tail);
    } else {
        fill_rows<FORM>(ns, tail);
        return true;
    }
}

// --------------------------------------------------------------------------
// Q-row cache slots
// --------------------------------------------------------------------------
// A slot is taken by a hand that goes round the slots and passes over those
// used since its last visit (it clears their reference bits) and over the two
// the phase still reads.  Rows evaluated ahead of need get no reference bit
// until they are used.  With more slots than bits the hand just goes round.
// Every block takes the same slots in the same order.  The `taken` slots the
// pass already has in sh.fslot stay its own (a pass takes at most nslots - 2).
__device__ int take_slot(int keep0, int keep1, int taken, bool used)
{
    Shared &sh = block_shared();
    const int n = sh.D.cache.nslots;
    int s = sh.hand;
    while (true) {
        if (s >= n) {
            s = 0;
            sh.reused = 1;
        }
        bool free = s != keep0 && s != keep1;
        for (int t = 0; t < taken; t++) free = free && s != sh.fslot[t];
        if (free) {
            if (n > kRefSlots) break;
            const unsigned m = 1u << (s & 31), w = sh.ref[s >> 5];
            if (!(w & m)) {
                if (used) sh.ref[s >> 5] = w | m;
                break;
            }
            sh.ref[s >> 5] = w & ~m;
        }
        s++;
    }
    sh.hand = s + 1;
    return s;
}
__device__ __forceinline__ void touch_slot(int s)
{
    Shared &sh = block_shared();
    if (sh.D.cache.nslots <= kRefSlots) sh.ref[s >> 5] |= 1u << (s & 31);
}

// The block's positions learn the fill pass's slots: whoever held one loses
// it, the variables of the pass get theirs.  Position k belongs to thread
// k % kThreads here as everywhere; the fill begins with a barrier.
__device__ __forceinline__ void claim_slots()
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    const Chunk ck = chunk_at(c.choff, block_shared().D.chunk_cap);
    const int n = c.a1 - c.a0, nf = sh.nfill;
    if (sh.reused) {
        for (int k = threadIdx.x; k < n; k += kThreads) {
            const int s = ck.Slot[k];
            for (int t = 0; t < nf; t++)
                if (s == sh.fslot[t]) {
                    ck.Slot[k] = kNoSlot;
                    ck.F[k] = (unsigned char)(ck.F[k] & ~(kFlagFull | kFlagAhead));
                }
        }
    }
    for (int t = 0; t < nf; t++) {
        const int k = sh.fpos[t] - c.a0;
        if (k >= 0 && k < n && (k & (kThreads - 1)) == (int)threadIdx.x) {
            ck.Slot[k] = (unsigned short)sh.fslot[t];
            ck.F[k] = (unsigned char)((ck.F[k] & ~(kFlagFull | kFlagAhead)) | (c.A == sh.D.l ? kFlagFull : 0) |
                                      (t >= sh.nneed ? kFlagAhead : 0));
        }
    }
    if (c.rank == 0 && threadIdx.x < nf) sh.D.cache.tag[sh.fslot[threadIdx.x]] = sh.fcol[threadIdx.x];
}
static_assert((kThreads & (kThreads - 1)) == 0, "a position's thread is found by masking");

// Phase A without the row of track 0 and / or 1 (their records in wa[e0], wa[e1]):
// the missing rows are evaluated together with the rows of the group's most
// violating positions (this only fills the cache; it never changes which
// pair is chosen).
template <int FORM>
__device__ __noinline__ bool miss_iup(unsigned seq, int e0, int e1, int need0, int need1)
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    const InstanceDesc &D = sh.D;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        const int nneed = need0 + need1;
        const int i0 = code_pos(sh.wa[e0].x[0]), i1 = D.nu ? code_pos(sh.wa[e1].x[kWordsI]) : -1;
        const int held0 = i0 >= 0 && !need0 ? (int)(sh.wa[e0].x[2] & 0xffffu) : -1;
        const int held1 = i1 >= 0 && !need1 ? (int)(sh.wa[e1].x[kWordsI + 2] & 0xffffu) : -1;
        if (lane == 0) {
            int nf = 0;
            for (int t = 0; t < 2; t++) {
                if (!(t ? need1 : need0)) continue;
                const unsigned *x = sh.wa[t ? e1 : e0].x + kWordsI * t;
                sh.fslot[nf] = take_slot(held0, held1, nf, true);
                sh.fpos[nf] = code_pos(x[0]);
                sh.fy[nf] = code_y(x[0]);
                sh.fcol[nf] = (int)x[1];
                sh.frow[nf] = (int)x[3];
                nf++;
            }
            sh.nneed = nf;
        }
        __syncwarp();
        int nf = nneed;
        const int want = D.prefetch - nneed;
        const int most = min(D.prefetch, D.cache.nslots - 2);
        if (want > 0 && most > nneed) {
            // the group's candidates, each lane keeping its best two; then `want`
            // rounds of the warp's best (the lowest lane on equal priorities)
            u64 k1 = 0, k2 = 0;
            Cand c1{}, c2{};
            bool ok = true;
            for (int e = lane; e < c.nb * kPrefetchCand; e += 32) {
                Cand cd;
                if (c.nb == 1) {
                    cd = sh.cand[e];
                } else {
                    RecWord w[2];
                    ok = ok && poll_words<2>(D, D.words + (long long)(e / kPrefetchCand) * kRecWords + kWordCand +
                                                    2 * (e % kPrefetchCand), seq, w);
                    if (!ok) break;
                    cd.v = __longlong_as_double((long long)w[0].lo);
                    cd.pc = (unsigned)w[0].hi;
                    cd.col = (unsigned)w[1].lo;
                    cd.row = (unsigned)(w[1].lo >> 32);
                    cd.slot = (unsigned)w[1].hi;
                }
                const int p = code_pos(cd.pc);
                if (p < 0 || p == i0 || p == i1) continue;
                const u64 k = key_of(cd.v);
                if (k > k1) {
                    k2 = k1;
                    c2 = c1;
                    k1 = k;
                    c1 = cd;
                } else if (k > k2) {
                    k2 = k;
                    c2 = cd;
                }
            }
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) sh.fail = 1;
            } else {
                for (int r = 0; r < want && nf < most; r++) {
                    const u64 m = warp_max_key(k1);
                    if (m == 0) break;
                    const int who = __ffs(__ballot_sync(0xffffffffu, k1 == m)) - 1;
                    int took = 0;
                    if (lane == who) {
                        if (c1.slot == kNoSlot) {
                            took = 1;
                            sh.fslot[nf] = take_slot(held0, held1, nf, false);
                            sh.fpos[nf] = code_pos(c1.pc);
                            sh.fy[nf] = code_y(c1.pc);
                            sh.fcol[nf] = (int)c1.col;
                            sh.frow[nf] = (int)c1.row;
                        }
                        k1 = k2;
                        c1 = c2;
                        k2 = 0;
                    }
                    nf += __shfl_sync(0xffffffffu, took, who);
                    __syncwarp();
                }
            }
        }
        if (lane == 0) sh.nfill = nf;
    }
    __syncthreads();
    if (sh.fail) return false;
    const int ns = sh.nfill;
    if (threadIdx.x == 0) {
        sh.cnt[kCntAhead] += ns - sh.nneed;
        sh.cnt[kCntMiss] += sh.nneed;
        sh.cnt[kCntQ] += (long long)ns * c.A;
        sh.cnt[kCntTargets] += c.A;
        sh.cnt[kCntFill]++;
    }
    claim_slots();
    return fill<FORM>(ns, 0);
}

// Phase B without the row of j (its record in wb[e]).
template <int FORM>
__device__ __noinline__ bool miss_j(int e, int slot0, int slot1)
{
    Ctx &c = block_shared().c;
    Shared &sh = block_shared();
    if (threadIdx.x == 0) {
        const unsigned *x = sh.wb[e].x;
        sh.fslot[0] = take_slot(slot0, slot1, 0, true);
        sh.fpos[0] = code_pos(x[0]);
        sh.fy[0] = code_y(x[0]);
        sh.fcol[0] = (int)x[1];
        sh.frow[0] = (int)x[2];
        sh.nfill = sh.nneed = 1;
        sh.cnt[kCntMiss]++;
        sh.cnt[kCntQ] += c.A;
        sh.cnt[kCntTargets] += c.A;
        sh.cnt[kCntFill]++;
    }
    __syncthreads();
    claim_slots();
    return fill<FORM>(1, 0);
}

// two-variable analytic step with box clipping (svm.cpp:636-721): alpha_i and
// alpha_j in ai and aj become their new values
__device__ __forceinline__ void pair_step(int yi, int yj, double QDi, double QDj, float Qij, double Gi, double Gj, double C_i,
                                          double C_j, double &ai, double &aj)
{
    if (yi != yj) {
        double quad_coef = __dadd_rn(__dadd_rn(QDi, QDj), (double)__fmul_rn(2.0f, Qij));
        if (quad_coef <= 0) quad_coef = kTau;
        const double delta = __ddiv_rn(__dsub_rn(-Gi, Gj), quad_coef);
        const double diff = __dsub_rn(ai, aj);
        ai = __dadd_rn(ai, delta);
        aj = __dadd_rn(aj, delta);
        if (diff > 0) {
            if (aj < 0) { aj = 0; ai = diff; }
        } else {
            if (ai < 0) { ai = 0; aj = -diff; }
        }
        if (diff > __dsub_rn(C_i, C_j)) {
            if (ai > C_i) { ai = C_i; aj = __dsub_rn(C_i, diff); }
        } else {
            if (aj > C_j) { aj = C_j; ai = __dadd_rn(C_j, diff); }
        }
    } else {
        double quad_coef = __dsub_rn(__dadd_rn(QDi, QDj), (double)__fmul_rn(2.0f, Qij));
        if (quad_coef <= 0) quad_coef = kTau;
        const double delta = __ddiv_rn(__dsub_rn(Gi, Gj), quad_coef);
        const double sum = __dadd_rn(ai, aj);
        ai = __dsub_rn(ai, delta);
        aj = __dadd_rn(aj, delta);
        if (sum > C_i) {
            if (ai > C_i) { ai = C_i; aj = __dsub_rn(sum, C_i); }
        } else {
            if (aj < 0) { aj = 0; ai = sum; }
        }
        if (sum > C_j) {
            if (aj > C_j) { aj = C_j; ai = __dsub_rn(sum, C_j); }
        } else {
            if (ai < 0) { ai = 0; aj = sum; }
        }
    }
}

// Row i and / or j completed over the inactive positions.
template <int FORM>
__device__ __noinline__ bool fill_tail(bool ti, bool tj, int i, int yi, int row_i, int slot_i, int j, int yj, int row_j,
                                       int slot_j)
{
    Shared &sh = block_shared();
    Ctx &c = sh.c;
    const Chunk ck = chunk_at(c.choff, sh.D.chunk_cap);
    const int ns = (ti ? 1 : 0) + (tj ? 1 : 0);
    __syncthreads();    // the last fill's list is no longer read
    if (threadIdx.x == 0) {
        if (ti) {
            sh.frow[0] = row_i;
            sh.fy[0] = yi;
            sh.fslot[0] = slot_i;
        }
        if (tj) {
            sh.frow[ns - 1] = row_j;
            sh.fy[ns - 1] = yj;
            sh.fslot[ns - 1] = slot_j;
        }
        sh.cnt[kCntQ] += (long long)ns * (sh.D.l - c.A);
        sh.cnt[kCntTargets] += sh.D.l - c.A;
    }
    __syncthreads();
    if (!fill<FORM>(ns, 1)) return false;
    const int ki = i - c.a0, kj = j - c.a0;
    if (ti && i >= c.a0 && i < c.a1 && (ki & (kThreads - 1)) == (int)threadIdx.x) ck.F[ki] |= kFlagFull;
    if (tj && j >= c.a0 && j < c.a1 && (kj & (kThreads - 1)) == (int)threadIdx.x) ck.F[kj] |= kFlagFull;
    return true;
}

// G_bar of all my positions after i and / or j reached or left their bound
// (svm.cpp:744-769): G_bar -+ C Q for each of the two that did.
// Row: const float * or TriRow.
template <class Row>
__device__ __noinline__ void update_gbar(Row Qi, bool bar_i, bool sub_i, double C_i, Row Qj, bool bar_j, bool sub_j, double C_j)
{
    Shared &sh = block_shared();
    const InstanceDesc &D = sh.D;
    Ctx &c = sh.c;
    const Chunk ck = chunk_at(c.choff, D.chunk_cap);
    auto bar = [&](double g, int col) {
        if (bar_i) { const double q = (double)Qi[col]; g = sub_i ? __dsub_rn(g, __dmul_rn(C_i, q)) : __dadd_rn(g, __dmul_rn(C_i, q)); }
        if (bar_j) { const double q = (double)Qj[col]; g = sub_j ? __dsub_rn(g, __dmul_rn(C_j, q)) : __dadd_rn(g, __dmul_rn(C_j, q)); }
        return g;
    };
    const int n = c.a1 - c.a0;
    for (int k = threadIdx.x; k < n; k += kThreads) D.G_bar[c.a0 + k] = bar(D.G_bar[c.a0 + k], ck.Col[k]);
    for (int p = c.t0 + threadIdx.x; p < c.t1; p += kThreads) D.G_bar[p] = bar(D.G_bar[p], D.pos_local[p]);
}

// num / quad roughly, as an integer that orders like it: the high word (20 bits
// of mantissa) + 1 of num times an approximate reciprocal with one Newton step,
// which together are off by less than 2^-30.  A quotient that is not safe to estimate
// (quad or the result at the ends of the exponent range, NaN) is given the
// value of an infinite one.
__device__ __forceinline__ unsigned rough_quotient(double num, double quad)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(quad));
    r = fma(r, fma(-quad, r, 1.0), r);
    const unsigned hq = (unsigned)__double2hiint(quad);
    const unsigned h = (unsigned)__double2hiint(__dmul_rn(num, r)) & 0x7fffffffu;
    return hq - 0x01000000u > 0x7d000000u ? 0x7ff00000u : h + 1u;
}
// what a rough quotient must reach to be divided exactly when the best one is
// `top`: two below it (one is what truncation can cost), or everything when the
// best is not a safe estimate.  Without the Newton step the line had to lie
// 64 below, which let in most of a one-vs-one pair's untouched positions (equal
// gradients, kernel values near 0) and sent every warp through its positions again.
__device__ __forceinline__ unsigned rough_least(unsigned top)
{
    return top >= 0x7fe00000u || top <= 0x00200000u ? 1u : top - 2u;
}

// an empty staging area: sparse sources are scattered into zeroed dense
// vectors, or into a table without keys
template <int FORM>
__device__ void stage_clear(float *stage)
{
    const InstanceDesc &D = block_shared().D;
    if (!D.x.X && D.stage_cap > 0)
        for (long long k = threadIdx.x; k < (long long)D.stage_lds * D.stage_cap * (stage_elem(FORM) / 4); k += blockDim.x)
            stage[k] = 0.0f;
    if (!D.x.X && D.hash_slots > 0) {
        int *keys = reinterpret_cast<int *>(stage);
        for (int k = threadIdx.x; k < kHashSlots; k += blockDim.x) keys[k] = -1;
        float *vals = reinterpret_cast<float *>(reinterpret_cast<char *>(stage) + kHashSlots * 4);
        for (int k = threadIdx.x; k < kHashSlots * kSrcBatch * (stage_elem(FORM) / 4); k += blockDim.x) vals[k] = 0.0f;
    }
    __syncthreads();
}

// --------------------------------------------------------------------------
// the persistent solver
// --------------------------------------------------------------------------
__device__ __forceinline__ void put_counters(SolveOut &o)
{
    Shared &sh = block_shared();
    o.sum_active = sh.cnt[kCntActive];
    o.q_evals = sh.cnt[kCntQ];
    o.lookups = sh.cnt[kCntLook];
    o.hits = sh.cnt[kCntLook] - sh.cnt[kCntMiss];
    o.fills = sh.cnt[kCntFill];
    o.prefetched = sh.cnt[kCntAhead];
    o.prefetch_used = (long long)sh.ahead_used;
    o.fill_targets = sh.cnt[kCntTargets];
    for (int k = 0; k < 8; k++) o.prof[k] = sh.prof[k];
}

// A block's context, its work counters and the initial state (svm.cpp:525-572,
// QD svm.cpp:1321-1327) on the global copies; the block's chunk is loaded.
template <int FORM>
__device__ __noinline__ bool start_solve(int rank)
{
    Shared &sh = block_shared();
    const InstanceDesc &D = sh.D;
    Ctx &c = sh.c;
    if (threadIdx.x == 0) {
        c.rank = rank;
        c.nb = D.nblocks;
        c.phase = 0;
        c.tcbase = 0;
        c.tc_g = 0;
        c.fg = 0;
        c.fstages = fill_stages(D.tc_n);
        // dynamic shared memory: [tensor-core stages][stage][tiles][G][alpha][QD][col][row][slot][flags]
        size_t off = 0;
        if constexpr (is_tc_form(FORM)) {
            const uint32_t raw = tc::smem_addr(dyn);
            c.tcbase = (raw + 1023u) & ~1023u;
            off = (size_t)tc_area_bytes(D.tc_n);
        }
        c.stage = reinterpret_cast<float *>(dyn + off);
        off += (size_t)D.stage_cap * D.stage_lds * stage_elem(FORM);
        if (D.hash_slots > 0) off += (size_t)hash_bytes(FORM);
        off = (off + 127) & ~(size_t)127;   // 64-byte tile rows: two to a 128-byte line
        c.tile = reinterpret_cast<float *>(dyn + off);
        c.choff = (int)(off + aux_bytes(FORM, D.tile_bufs));
    }
    set_active(D.l);
    if (threadIdx.x == 0) {
        for (int k = 0; k < kCnt; k++) sh.cnt[k] = 0;
        if (D.resident) sh.cnt[kCntQ] = (long long)D.l * D.l;
        for (int k = 0; k < 8; k++) {
            sh.prof[k] = 0;
            sh.prof32[k] = 0;
        }
        sh.tstart = clock64();
        sh.ahead_used = 0;
        sh.fail = 0;
        sh.hand = 0;
        sh.reused = 0;
    }
    for (int k = threadIdx.x; k < kRefSlots / 32; k += blockDim.x) sh.ref[k] = 0;
    stage_clear<FORM>(c.stage);
    const int l = D.l;
    for (int p = c.a0 + threadIdx.x; p < c.a1; p += blockDim.x) {
        D.pos_local[p] = p;      // positions start as local indices
        D.pos_slot[p] = D.resident ? (int)((unsigned)p | kSlotFull) : kNoSlot;
        D.status[p] = status_of(D.alpha[p], get_C(D, D.y[p]));
        const int r = D.pos_row[p];
        const double xs = D.x.xsq ? D.x.xsq[r] : 0.0;
        // dot(x,x) in feature order is exactly what xsq holds
        D.QD[p] = kernel_from_dot(D.kp, xs, xs, xs);
        D.G[p] = D.p[p];
        D.G_bar[p] = 0.0;
    }
    if (!exchange()) return false;
    // a resident matrix whose evaluation gave up leaves the group's error flag
    if (__syncthreads_or(D.resident && ld_relaxed_i32(&D.sync->error))) return false;
    int any = 0;
    for (int p = threadIdx.x; p < l; p += blockDim.x) any |= D.alpha[p] > 0 ? 1 : 0;
    any = __syncthreads_or(any);
    if (any) {
        if (!accumulate<FORM>(l, 0, D.lazy_gbar ? 0 : 1, c.a0, c.a1)) return false;
        if (!exchange()) return false;
    }
    chunk_load();
    return true;
}

// rho (svm.cpp:1013-1049 / 1260-1308), objective (:795-802), alpha out (:805-808)
__device__ __noinline__ void finish_solve(int nu, long long iter, int status, int unshrink)
{
    Shared &sh = block_shared();
    const InstanceDesc &D = sh.D;
    Ctx &c = sh.c;
    const int l = D.l, rank = c.rank;
    // The sums run sequentially in position order (bit-exact with the reference), on block 0.
    if (rank == 0) {
        // the staging area is no longer needed
        double *chv = reinterpret_cast<double *>(dyn), *chg = chv + kThreads;
        unsigned char *chs = reinterpret_cast<unsigned char *>(chg + kThreads);
        signed char *chy = reinterpret_cast<signed char *>(chs + kThreads);
        __syncthreads();
        double ub = SVMB_INF, lb = -SVMB_INF, sum_free = 0;
        int nr_free = 0;
        double ub1 = SVMB_INF, ub2 = SVMB_INF, lb1 = -SVMB_INF, lb2 = -SVMB_INF, sf1 = 0, sf2 = 0;
        int nf1 = 0, nf2 = 0;
        double objv = 0;
        const int A = c.A;
        for (int base = 0; base < l; base += blockDim.x) {
            const int p = base + threadIdx.x;
            if (p < l) {
                chs[threadIdx.x] = D.status[p];
                chy[threadIdx.x] = D.y[p];
                chg[threadIdx.x] = D.G[p];
                chv[threadIdx.x] = __dmul_rn(D.alpha[p], __dadd_rn(D.G[p], D.p[p]));
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                const int lim = l - base < (int)blockDim.x ? l - base : (int)blockDim.x;
                for (int k = 0; k < lim; k++) {
                    objv = __dadd_rn(objv, chv[k]);
                    if (base + k >= A) continue;
                    const unsigned char s = chs[k];
                    const int y = chy[k];
                    const double G = chg[k];
                    if (!nu) {
                        const double yG = __dmul_rn((double)y, G);
                        if (s == ST_UPPER) { if (y == -1) ub = fmin(ub, yG); else lb = fmax(lb, yG); }
                        else if (s == ST_LOWER) { if (y == +1) ub = fmin(ub, yG); else lb = fmax(lb, yG); }
                        else { ++nr_free; sum_free = __dadd_rn(sum_free, yG); }
                    } else {
                        if (y == +1) {
                            if (s == ST_UPPER) lb1 = fmax(lb1, G);
                            else if (s == ST_LOWER) ub1 = fmin(ub1, G);
                            else { ++nf1; sf1 = __dadd_rn(sf1, G); }
                        } else {
                            if (s == ST_UPPER) lb2 = fmax(lb2, G);
                            else if (s == ST_LOWER) ub2 = fmin(ub2, G);
                            else { ++nf2; sf2 = __dadd_rn(sf2, G); }
                        }
                    }
                }
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            SolveOut o;
            o.iters = iter;
            o.status = status;
            o.active_size = c.A;
            o.unshrink = unshrink;
            o.obj = __ddiv_rn(objv, 2.0);
            o.gap = 0;
            put_counters(o);
            o.prof[kProfTotal] = clock64() - sh.tstart;
            if (!nu) {
                o.rho = nr_free > 0 ? __ddiv_rn(sum_free, (double)nr_free) : __ddiv_rn(__dadd_rn(ub, lb), 2.0);
                o.r = 0;
                o.nr_free = nr_free;
            } else {
                const double r1 = nf1 > 0 ? __ddiv_rn(sf1, (double)nf1) : __ddiv_rn(__dadd_rn(ub1, lb1), 2.0);
                const double r2 = nf2 > 0 ? __ddiv_rn(sf2, (double)nf2) : __ddiv_rn(__dadd_rn(ub2, lb2), 2.0);
                o.r = __ddiv_rn(__dadd_rn(r1, r2), 2.0);
                o.rho = __ddiv_rn(__dsub_rn(r1, r2), 2.0);
                o.nr_free = nf1 + nf2;
            }
            *D.out = o;
        }
    }
    {
        const int lo = (int)((long long)l * rank / c.nb), hi = (int)((long long)l * (rank + 1) / c.nb);
        for (int p = lo + threadIdx.x; p < hi; p += blockDim.x) D.alpha_local[D.pos_local[p]] = D.alpha[p];
    }
}

// a wait ran out: the group's error
__device__ __noinline__ void fail_solve(long long iter, int unshrink)
{
    Shared &sh = block_shared();
    const InstanceDesc &D = sh.D;
    Ctx &c = sh.c;
    const int rank = c.rank;
    if (threadIdx.x == 0 && rank == 0) {
        SolveOut o;
        o.iters = iter; o.rho = 0; o.obj = 0; o.r = 0; o.status = -1; o.active_size = c.A;
        o.unshrink = unshrink; o.nr_free = 0; o.gap = 0;
        put_counters(o);
        *D.out = o;
    }
}

// NU: Solver_NU (two tracks) or Solver
template <int FORM, bool NU>
__device__ __noinline__ void solve_instance(int rank)
{
    Shared &sh = block_shared();
    const InstanceDesc &D = sh.D;
    Ctx &c = sh.c;
    if (!start_solve<FORM>(rank)) {
        fail_solve(0, 0);
        return;
    }
    const int l = D.l;
    constexpr int nu = NU ? 1 : 0;
    const Chunk ck = chunk_at(c.choff, D.chunk_cap);
    unsigned seq = 0;       // sequence number of the last record exchange
    long long iter = 0;
    int unshrink = 0;
    int status = 0;
    // section timers of thread 0: the loop adds 32-bit cycle counts (an add that
    // waits for nothing) and folds them every 1000 iterations
    unsigned tmark = (unsigned)clock();
#define SVMB_PROF(k)                                   \
    do {                                               \
        if (threadIdx.x == 0) {                        \
            const unsigned now_ = (unsigned)clock();   \
            atomicAdd(&sh.prof32[k], now_ - tmark);    \
            tmark = now_;                              \
        }                                              \
    } while (0)
    auto fold = [&]() {
        if (threadIdx.x == 0)
            for (int k = 0; k < 8; k++) {
                sh.prof[k] += sh.prof32[k];
                sh.prof32[k] = 0;
            }
    };
    {
        const long long max_iter = D.max_iter;
        int counter = (l < 1000 ? l : 1000) + 1;
        if (!scan_iup<nu>(++seq)) goto fail;
        const int np = (c.nb + 31) >> 5;
        // slots are never taken back when every variable has one
        const bool evicts = D.cache.nslots < l;
        const bool ahead = D.prefetch > 1;
        long long passes = 0, sum_from = 0;     // phase-A passes; iterations already in the active-size sum
        auto count_active = [&]() {
            if (threadIdx.x == 0) sh.cnt[kCntActive] += (iter - sum_from) * c.A;
            sum_from = iter;
        };

        while (iter < max_iter) {
            if (--counter == 0) {
                counter = l < 1000 ? l : 1000;
                fold();
                count_active();
                if (D.shrinking) {
                    SVMB_PROF(kProfBUpdate);
                    if (!do_shrinking<FORM>(unshrink)) goto fail;
                    if (!scan_iup<nu>(++seq)) goto fail;
                    SVMB_PROF(kProfShrink);
                }
            }
            int widened = 0;
        select_again:
            // ======================= phase A =======================
            const int n = c.a1 - c.a0;
            const int e0 = np > 1 ? win_iup(np, 0) : 0, e1 = nu && np > 1 ? win_iup(np, 1) : 0;
            const WinA &w0 = sh.wa[e0], &w1 = sh.wa[e1];
            const int i0 = code_pos(w0.x[0]), i1 = nu ? code_pos(w1.x[kWordsI]) : -1;
            const double Gmax0 = w0.d[0], Gmax1 = nu ? w1.d[kWordsI] : -SVMB_INF;
            int slot0 = i0 >= 0 ? (int)(w0.x[2] & 0xffffu) : -1, slot1 = i1 >= 0 ? (int)(w1.x[kWordsI + 2] & 0xffffu) : -1;
            {
                const int need0 = slot0 == kNoSlot ? 1 : 0, need1 = slot1 == kNoSlot ? 1 : 0;
                passes++;
                if (evicts && threadIdx.x == 0) {
                    if (i0 >= 0 && !need0) touch_slot(slot0);
                    if (i1 >= 0 && !need1) touch_slot(slot1);
                }
                SVMB_PROF(kProfAReduce);
                if (need0 | need1) {
                    if (!miss_iup<FORM>(seq, e0, e1, need0, need1)) goto fail;
                    if (need0) slot0 = sh.fslot[0];
                    if (need1) slot1 = sh.fslot[need0];
                }
                SVMB_PROF(kProfAFill);
            }
            const float *const Qi0 = i0 >= 0 ? D.cache.data + (long long)slot0 * D.cache.stride : nullptr;
            const float *const Qi1 = i1 >= 0 ? D.cache.data + (long long)slot1 * D.cache.stride : nullptr;
            {
                // second-order j scan on my chunk (svm.cpp:869-924 / :1120-1174): the
                // largest decrease (Gmax + y G)^2 / quad, ties to the larger position.
                // Exact divisions are long, so rough quotients come first and only
                // those that may be the warp's best are divided: about one per warp.
                // A thread keeps its best rough quotient with its
                // terms, and its second best; it goes over its positions once more
                // in the rare case that both are in reach.
                double dec = -SVMB_INF, g2 = -SVMB_INF, g2n = -SVMB_INF;
                int jx = -1;
                const double QDi0 = w0.d[2], QDi1 = w1.d[kWordsI + 2];
                const double two_yi0 = __dmul_rn(2.0, (double)code_y(w0.x[0]));
                // numerator and denominator of position k; false: not a candidate
                auto quotient = [&](int k, float q, double &num, double &quad) -> bool {
                    const unsigned f = ck.F[k];
                    const unsigned char s = flag_s(f);
                    const bool pos = (f & kFlagPos) != 0;
                    if (s == (pos ? ST_LOWER : ST_UPPER)) return false;
                    const double G = ck.G[k], Gm = pos || !nu ? Gmax0 : Gmax1;
                    const double yG = pos ? G : -G;
                    const double grad_diff = __dadd_rn(Gm, yG);
                    if (pos || !nu) g2 = fmax(g2, yG);
                    else g2n = fmax(g2n, yG);
                    if (!(grad_diff > 0)) return false;
                    const double cross = nu ? (double)__fmul_rn(2.0f, q) : __dmul_rn(pos ? two_yi0 : -two_yi0, (double)q);
                    quad = __dsub_rn(__dadd_rn(pos || !nu ? QDi0 : QDi1, ck.QD[k]), cross);
                    num = __dmul_rn(grad_diff, grad_diff);
                    if (!(quad > 0)) quad = kTau;
                    return true;
                };
                unsigned r1 = 0, r2 = 0;
                int k1 = -1;
                double num1 = 0.0, quad1 = 1.0;
                float q1 = 0.0f, jq = 0.0f;
                auto row_at = [&](int k) -> float {
                    const float *Qr = (nu && !(ck.F[k] & kFlagPos)) ? Qi1 : Qi0;
                    return Qr ? Qr[ck.Col[k]] : 0.0f;
                };
                // a rolled loop, its Q_i values kScanAhead positions ahead
                float qn[kScanAhead];
#pragma unroll
                for (int u = 0; u < kScanAhead; u++) {
                    const int k = threadIdx.x + u * kThreads;
                    qn[u] = k < n ? row_at(k) : 0.0f;
                }
#pragma unroll 1
                for (int k = threadIdx.x; k < n; k += kThreads) {
                    const float q = qn[0];
#pragma unroll
                    for (int u = 0; u + 1 < kScanAhead; u++) qn[u] = qn[u + 1];
                    if (k + kScanAhead * kThreads < n) qn[kScanAhead - 1] = row_at(k + kScanAhead * kThreads);
                    double num, quad;
                    if (!quotient(k, q, num, quad)) continue;
                    const unsigned r = rough_quotient(num, quad);
                    if (r > r1) {
                        r2 = r1;
                        r1 = r;
                        k1 = k;
                        num1 = num;
                        quad1 = quad;
                        q1 = q;
                    } else if (r > r2) {
                        r2 = r;
                    }
                }
                __syncwarp();
                const unsigned least = rough_least(__reduce_max_sync(0xffffffffu, r1));
                if (r2 >= least) {
#pragma unroll 1
                    for (int k = threadIdx.x; k < n; k += kThreads) {
                        const float q = row_at(k);
                        double num, quad;
                        if (!quotient(k, q, num, quad) || rough_quotient(num, quad) < least) continue;
                        better_max(dec, jx, __ddiv_rn(num, quad), c.a0 + k);
                        if (jx == c.a0 + k) jq = q;
                    }
                } else if (r1 >= least) {
                    better_max(dec, jx, __ddiv_rn(num1, quad1), c.a0 + k1);
                    jq = q1;
                }
                __syncwarp();
                if (!j_publish<nu>(++seq, dec, jx, jq, g2, g2n)) goto fail;
            }
            SVMB_PROF(kProfAScan);

            // ======================= phase B =======================
            const int eb = np > 1 ? win_j(np) : 0;
            const WinB &wj = sh.wb[eb];
            const int j = code_pos(wj.x[0]);
            {
                double gm = sh.wb[0].d[4], gmn = nu ? sh.wb[0].d[5] : -SVMB_INF;
                for (int k = 1; k < np; k++) {
                    gm = fmax(gm, sh.wb[k].d[4]);
                    if (nu) gmn = fmax(gmn, sh.wb[k].d[5]);
                }
                bool stop;
                if (!nu) stop = __dadd_rn(Gmax0, gm) < D.eps;
                else stop = fmax(__dadd_rn(Gmax0, gm), __dadd_rn(Gmax1, gmn)) < D.eps;
                if (stop || j < 0) {
                    if (widened) break;
                    // reconstruct the whole gradient, widen, select again (svm.cpp:598-611)
                    count_active();
                    if (c.A < l && !reopen<FORM>()) goto fail;
                    widened = 1;
                    if (!scan_iup<nu>(++seq)) goto fail;
                    goto select_again;
                }
                if (widened) counter = 1;
            }
            ++iter;
            // the working pair; nu-SVC takes i from the track of y_j (svm.cpp:1179-1182)
            const int yj = code_y(wj.x[0]);
            const int tr = (nu && yj != +1) ? 1 : 0;
            const WinA &wi = tr ? w1 : w0;
            const int i = tr ? i1 : i0;
            const int yi = tr ? -1 : code_y(w0.x[0]);
            const double Gi = tr ? Gmax1 : (yi == +1 ? -Gmax0 : Gmax0);
            const double alpha_i = wi.d[kWordsI * tr + 1], QDi = wi.d[kWordsI * tr + 2];
            const int slot_i = tr ? slot1 : slot0;
            const float Qij = __uint_as_float(wj.x[4]);     // (of the track of y_j)
            const double Gj = wj.d[1], alpha_j = wj.d[2], QDj = wj.d[3];
            // Q_j row
            int slot_j = (int)(wj.x[3] & 0xffffu);
            {
                const bool need = slot_j == kNoSlot;
                if (evicts && !need && threadIdx.x == 0) touch_slot(slot_j);
                SVMB_PROF(kProfBReduce);
                if (need) {
                    if (!miss_j<FORM>(eb, slot0, slot1)) goto fail;
                    slot_j = sh.fslot[0];
                }
            }
            // identical in every block
            const double C_i = get_C(D, yi), C_j = get_C(D, yj);
            double ai = alpha_i, aj = alpha_j;
            pair_step(yi, yj, QDi, QDj, Qij, Gi, Gj, C_i, C_j, ai, aj);
            const double dai = __dsub_rn(ai, alpha_i);
            const double daj = __dsub_rn(aj, alpha_j);
            const unsigned char old_si = status_of(alpha_i, C_i), old_sj = status_of(alpha_j, C_j);
            const unsigned char new_si = status_of(ai, C_i), new_sj = status_of(aj, C_j);
            const bool bar_i = !D.lazy_gbar && (old_si == ST_UPPER) != (new_si == ST_UPPER);
            const bool bar_j = !D.lazy_gbar && (old_sj == ST_UPPER) != (new_sj == ST_UPPER);
            // complete rows for the G_bar update: fill the tail [A,l) where missing
            if ((bar_i || bar_j) && c.A < l) {
                const bool ti = bar_i && !(wi.x[kWordsI * tr + 2] & kSlotFull), tj = bar_j && !(wj.x[3] & kSlotFull);
                if (!fill_tail<FORM>(ti, tj, i, yi, (int)wi.x[kWordsI * tr + 3], slot_i, j, yj, (int)wj.x[2], slot_j)) goto fail;
            }
            SVMB_PROF(kProfBFill);
            // the owners of i and j take their new alpha and status (a position is
            // read and written by its own thread only until the next barrier)
            {
                auto take = [&](int p, double a, unsigned char st) {
                    const int k = p - c.a0;
                    if (k < 0 || k >= n || (k & (kThreads - 1)) != (int)threadIdx.x) return;
                    const unsigned f = ck.F[k];
                    if (f & kFlagAhead) atomicAdd(&sh.ahead_used, 1u);
                    ck.A[k] = a;
                    ck.F[k] = (unsigned char)((f & ~((3u << kFlagStatus) | kFlagAhead)) | ((unsigned)st << kFlagStatus));
                };
                take(i, ai, new_si);
                take(j, aj, new_sj);
            }
            // G update on my chunk (svm.cpp:732-735) + G_bar (svm.cpp:744-769) + next I_up scan
            {
                const float *Qi = D.cache.data + (long long)slot_i * D.cache.stride;
                const float *Qj = D.cache.data + (long long)slot_j * D.cache.stride;
                double v[2] = {-SVMB_INF, -SVMB_INF};
                int ix[2] = {-1, -1};
                double pv = -SVMB_INF;
                int pix = -1;
                // rolled like the j scan, Q_i and Q_j kScanAhead positions ahead
                float qi[kScanAhead], qj[kScanAhead];
#pragma unroll
                for (int u = 0; u < kScanAhead; u++) {
                    const int k = threadIdx.x + u * kThreads;
                    const int col = k < n ? ck.Col[k] : 0;
                    qi[u] = k < n ? Qi[col] : 0.0f;
                    qj[u] = k < n ? Qj[col] : 0.0f;
                }
#pragma unroll 1
                for (int k = threadIdx.x; k < n; k += kThreads) {
                    const double qid = (double)qi[0], qjd = (double)qj[0];
#pragma unroll
                    for (int u = 0; u + 1 < kScanAhead; u++) {
                        qi[u] = qi[u + 1];
                        qj[u] = qj[u + 1];
                    }
                    if (k + kScanAhead * kThreads < n) {
                        const int col = ck.Col[k + kScanAhead * kThreads];
                        qi[kScanAhead - 1] = Qi[col];
                        qj[kScanAhead - 1] = Qj[col];
                    }
                    const double G = __dadd_rn(ck.G[k], __dadd_rn(__dmul_rn(qid, dai), __dmul_rn(qjd, daj)));
                    ck.G[k] = G;
                    const unsigned f = ck.F[k];
                    const unsigned char s = flag_s(f);
                    const bool pos = (f & kFlagPos) != 0;
                    const bool up = s != (pos ? ST_UPPER : ST_LOWER);
                    const double yG = pos ? -G : G;
                    if (up) {
                        if (pos || !nu) better_max(v[0], ix[0], yG, c.a0 + k);
                        else better_max(v[1], ix[1], yG, c.a0 + k);
                    }
                    if (ahead) better_max(pv, pix, s == ST_FREE ? fabs(G) : (up ? yG : -yG), c.a0 + k);
                }
                __syncwarp();
                if (bar_i || bar_j) update_gbar(Qi, bar_i, old_si == ST_UPPER, C_i, Qj, bar_j, old_sj == ST_UPPER, C_j);
                if (!iup_publish<nu>(++seq, ahead, v, ix, pv, pix)) goto fail;
            }
            SVMB_PROF(kProfBUpdate);
        }

        count_active();
        fold();
        if (threadIdx.x == 0) sh.cnt[kCntLook] = passes * (nu ? 2 : 1) + iter;
        chunk_store();
        if (!exchange()) goto fail;
        if (iter >= max_iter) {
            status = 1;
            if (c.A < l) {
                if (!reconstruct<FORM>()) goto fail;
                set_active(l);
            }
        }
    }
    finish_solve(nu, iter, status, unshrink);
    return;
fail:
    fail_solve(iter, unshrink);
#undef SVMB_PROF
}

// Tell the host, through a word of mapped host memory, that every block of the
// instance has written its results (a request loop collects the instance and
// reuses its SMs while the rest of the launch runs on).
__device__ void signal_done(const InstanceDesc &D)
{
    if (!D.done_flag) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence_system();
        if (atomicAdd(&D.sync->finished, 1u) == (unsigned)D.nblocks - 1u) {
            __threadfence_system();
            *(volatile int *)D.done_flag = 1;
        }
    }
}

template <int FORM>
__global__ void __launch_bounds__(kThreads, 1)
smo_persistent(const InstanceDesc *__restrict__ insts, const int *__restrict__ block_inst)
{
    Shared &sh = block_shared();
    const int inst = block_inst[blockIdx.x];
    // the descriptor is read all through the solve: a copy in shared memory
    for (int k = threadIdx.x; k < (int)(sizeof(InstanceDesc) / 4); k += blockDim.x)
        reinterpret_cast<int *>(&sh.D)[k] = reinterpret_cast<const int *>(&insts[inst])[k];
    __syncthreads();
    const InstanceDesc &D = sh.D;
    const int rank = blockIdx.x - D.block0;
    if constexpr (is_tc_form(FORM)) {
        // mbarriers of the tensor-core pipeline and the TMEM accumulator (one block per SM)
        if (threadIdx.x == 0) {
            for (int k = 0; k < kTcStages; k++) tc::mbar_init(&sh.tbar[k], 1);
            for (int k = 0; k < kFillStagesMax; k++) {
                tc::mbar_init(&sh.ffull[k], kThreads - kFillLoad0 * 32);
                tc::mbar_init(&sh.fempty[k], 1);
            }
            for (int k = 0; k < kFillAcc; k++) {
                tc::mbar_init(&sh.faccf[k], 1);
                tc::mbar_init(&sh.facce[k], kTcM);
            }
            sh.fabort = 0;
            tc::mbar_init_fence();
        }
        if (threadIdx.x < 32) {
            tc::tmem_alloc(&sh.tmem, 2 * kTcMaxN);
            tc::tmem_relinquish();
        }
        tc::tc_fence_before();
        __syncthreads();
        tc::tc_fence_after();
    }
    if (D.nu) solve_instance<FORM, true>(rank);
    else solve_instance<FORM, false>(rank);
    signal_done(D);
    if constexpr (is_tc_form(FORM)) {
        tc::tc_fence_before();
        __syncthreads();
        if (threadIdx.x < 32) tc::tmem_dealloc(sh.tmem, 2 * kTcMaxN);
    }
}

// Whole kernel matrices of sparse instances (their caches hold every row):
// block t takes a group of source variables, stages them as a row pass does
// and walks the targets from its first source on; the values left of the
// diagonal are copied from the right.  Bound by the target walks: 8 bytes and
// one or two table probes per stored value for up to 8 sources.
template <int FORM>
__global__ void __launch_bounds__(kThreads, 1)
smo_rows(const InstanceDesc *__restrict__ insts, const int *__restrict__ first, int count, int total)
{
    Shared &sh = block_shared();
    const InstanceDesc &D = sh.D;
    int cur = -1;
    float *const stage = reinterpret_cast<float *>(dyn);
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        int lo = 0, hi = count - 1;
        while (lo < hi) {
            const int m = (lo + hi + 1) >> 1;
            if (first[m] <= t) lo = m;
            else hi = m - 1;
        }
        if (lo != cur) {
            // another instance: its descriptor, and an empty staging area
            cur = lo;
            __syncthreads();
            for (int k = threadIdx.x; k < (int)(sizeof(InstanceDesc) / 4); k += blockDim.x)
                reinterpret_cast<int *>(&sh.D)[k] = reinterpret_cast<const int *>(&insts[lo])[k];
            __syncthreads();
            stage_clear<FORM>(stage);
        }
        const int l = D.l, cap = D.stage_cap > 0 ? D.stage_cap : kSrcBatch;
        const int p0 = (t - first[lo]) * cap, ns = min(cap, l - p0);
        if (threadIdx.x < ns) {
            const int row = D.pos_row[p0 + threadIdx.x];
            sh.frow[threadIdx.x] = row;
            sh.fy[threadIdx.x] = D.y[p0 + threadIdx.x];
            sh.fsx[threadIdx.x] = D.x.xsq ? D.x.xsq[row] : 0.0;
        }
        __syncthreads();
        stage_sources(D, stage, sh.ss, sh.frow, ns);
        float *const Q = D.cache.data;
        const long long stride = D.cache.stride;
        for (int p = p0 + threadIdx.x; p < l; p += blockDim.x) {
            const int r = D.pos_row[p], yp = D.y[p];
            double dots[kSrcBatch];
            row_dots<FORM>(D, sh.ss, ns, r, dots);
            const double xe = D.x.xsq ? D.x.xsq[r] : 0.0;
#pragma unroll
            for (int k = 0; k < kSrcBatch; k++) {
                if (k >= ns) break;
                const float q = q_of(sh.fy[k] * yp, dots[k], sh.fsx[k], xe);
                if (D.resident == kResidentTri) {
                    if (p >= p0 + k) Q[tri_at(p, p0 + k)] = q;
                    continue;
                }
                Q[(long long)(p0 + k) * stride + p] = q;
                if (p >= p0 + ns) Q[(long long)p * stride + p0 + k] = q;
            }
        }
        unstage_sources(D, stage, sh.ss);
    }
}

}  // namespace
}  // namespace svmb
