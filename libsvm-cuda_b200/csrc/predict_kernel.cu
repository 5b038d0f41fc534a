// predict_kernel.cu -- decision values of the reference's svm_predict_values
// (reference libsvm/svm.cpp:2569-2643) for a batch of rows on the device.
//
// kvalue[t][s] = K(x_t, SV_s) with the prediction-time kernel of the reference
// (Kernel::k_function, svm.cpp:327-384: RBF walks the squared difference over
// the union of nonzero features in index order, no norm trick).  Each pair's
// sum runs sequentially over the two classes' SVs in model order, exactly as
// the reference, so decision values match it bit for bit (rows and SVs are
// kept as the doubles the caller's svm_node lists hold).
// The file is compiled with -fmad=false.
//
// Kernel values are kept SV-major, kv[s][t] for the t-th test row of a chunk,
// so that the pair sums (each in model order over the two classes' SVs)
// read consecutive words across a warp.  Dense rows take
// a tiled kernel: a block computes 64 test rows x 64 SVs, 16 features at a
// time staged in shared memory, 4 x 4 values per thread.  With a
// tensor-core predict form the values come from the split-product kernel
// block of the SVs' split copy (kept with the model) and the chunk's.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include "engine.hpp"
#include "predict.hpp"

namespace svmb {

namespace {

struct Rows {
    // dense [n][ld] or CSR, values in float64: a model's SVs (read from a
    // model file, say) and the caller's rows are doubles, and the exact form
    // evaluates the reference's kernel on exactly those values.  Each array
    // grows on demand and is reused by later uploads (capacities in bytes)
    double *X = nullptr;
    long long *rowptr = nullptr;
    int *col = nullptr;
    double *val = nullptr;
    size_t capX = 0, capRp = 0, capCol = 0, capVal = 0;
    int n = 0, ld = 0;
    bool dense = true;
    void release()
    {
        cudaFree(X); cudaFree(rowptr); cudaFree(col); cudaFree(val);
        X = nullptr; rowptr = nullptr; col = nullptr; val = nullptr;
        capX = capRp = capCol = capVal = 0;
    }
    size_t held() const { return capX + capRp + capCol + capVal; }
};

// device buffer of at least `bytes`, reallocated only when it must grow
template <typename T>
cudaError_t grow(T *&p, size_t &cap, size_t bytes)
{
    if (bytes <= cap && p) return cudaSuccess;
    cudaFree(p);
    p = nullptr;
    cap = 0;
    const size_t want = std::max<size_t>(bytes, 256);
    cudaError_t e = cudaMalloc(&p, want);
    if (e == cudaSuccess) cap = want;
    return e;
}

__device__ __forceinline__ double powi_p(double base, int times)
{
    double tmp = base, ret = 1.0;
    for (int t = times; t > 0; t /= 2) {
        if (t % 2 == 1) ret = __dmul_rn(ret, tmp);
        tmp = __dmul_rn(tmp, tmp);
    }
    return ret;
}

struct KP {
    int type, degree;
    double gamma, coef0;
};

// kvalue for rows given as CSR in global memory (merge walks, svm.cpp:305-384)
__device__ double kval_csr(const KP &kp, const long long *rpa, const int *ca, const double *va, int a,
                           const long long *rpb, const int *cb, const double *vb, int b)
{
    long long e = rpa[a], ee = rpa[a + 1], f = rpb[b], ff = rpb[b + 1];
    double sum = 0.0;
    if (kp.type == 2) {
        while (e < ee && f < ff) {
            const int x = ca[e], y = cb[f];
            if (x == y) {
                const double d = __dsub_rn(va[e], vb[f]);
                sum = __dadd_rn(sum, __dmul_rn(d, d));
                ++e; ++f;
            } else if (x > y) {
                sum = __dadd_rn(sum, __dmul_rn(vb[f], vb[f]));
                ++f;
            } else {
                sum = __dadd_rn(sum, __dmul_rn(va[e], va[e]));
                ++e;
            }
        }
        for (; e < ee; ++e) sum = __dadd_rn(sum, __dmul_rn(va[e], va[e]));
        for (; f < ff; ++f) sum = __dadd_rn(sum, __dmul_rn(vb[f], vb[f]));
        return exp(__dmul_rn(-kp.gamma, sum));
    }
    while (e < ee && f < ff) {
        const int x = ca[e], y = cb[f];
        if (x == y) { sum = __dadd_rn(sum, __dmul_rn(va[e], vb[f])); ++e; ++f; }
        else if (x > y) ++f;
        else ++e;
    }
    if (kp.type == 0) return sum;
    if (kp.type == 1) return powi_p(__dadd_rn(__dmul_rn(kp.gamma, sum), kp.coef0), kp.degree);
    return tanh(__dadd_rn(__dmul_rn(kp.gamma, sum), kp.coef0));
}

constexpr int kPT = 64;   // test rows per tile (dense path)
constexpr int kPS = 64;   // SVs per tile
constexpr int kPK = 16;   // features per staged slice

__device__ __forceinline__ double kfinish(const KP &kp, double acc)
{
    if (kp.type == 2) return exp(__dmul_rn(-kp.gamma, acc));
    if (kp.type == 0) return acc;
    if (kp.type == 1) return powi_p(__dadd_rn(__dmul_rn(kp.gamma, acc), kp.coef0), kp.degree);
    return tanh(__dadd_rn(__dmul_rn(kp.gamma, acc), kp.coef0));
}

// dense path: a 64 x 64 tile of K(test, SV), out[s][t] (ldo = nt).  Thread
// (ty, tx) of 16 x 16 owns test rows t0 + tx + 16i and SVs s0 + 4ty + j; every
// value accumulates over the features in order, as the reference's walk does
// (RBF: the squared difference; a feature zero in both adds nothing).
__global__ void __launch_bounds__(256) kvalue_tile(KP kp, const double *__restrict__ T, int nt,
                                                  const double *__restrict__ S, int ns, int ld,
                                                  double *__restrict__ out)
{
    __shared__ double ta[kPK][kPT + 1];
    __shared__ double sb[kPK][kPS + 1];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int t0 = blockIdx.y * kPT, s0 = blockIdx.x * kPS;
    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0;
    // loader: 64 rows x 16 features = 256 pieces of 4 doubles per operand, one per thread
    const int lr = tid >> 2, lc = (tid & 3) * 4;
    for (int k0 = 0; k0 < ld; k0 += kPK) {
        const int c = k0 + lc;
        double2 a0 = make_double2(0.0, 0.0), a1 = a0, b0 = a0, b1 = a0;
        if (t0 + lr < nt && c < ld) {
            const double2 *p = reinterpret_cast<const double2 *>(T + (long long)(t0 + lr) * ld + c);
            a0 = __ldg(p);
            a1 = __ldg(p + 1);
        }
        if (s0 + lr < ns && c < ld) {
            const double2 *p = reinterpret_cast<const double2 *>(S + (long long)(s0 + lr) * ld + c);
            b0 = __ldg(p);
            b1 = __ldg(p + 1);
        }
        __syncthreads();
        ta[lc][lr] = a0.x; ta[lc + 1][lr] = a0.y; ta[lc + 2][lr] = a1.x; ta[lc + 3][lr] = a1.y;
        sb[lc][lr] = b0.x; sb[lc + 1][lr] = b0.y; sb[lc + 2][lr] = b1.x; sb[lc + 3][lr] = b1.y;
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kPK; kk++) {
            double av[4], bv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) av[i] = ta[kk][tx + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; j++) bv[j] = sb[kk][4 * ty + j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (kp.type == 2) {
                        const double d = __dsub_rn(av[i], bv[j]);
                        acc[i][j] = __dadd_rn(acc[i][j], __dmul_rn(d, d));
                    } else {
                        acc[i][j] = __dadd_rn(acc[i][j], __dmul_rn(av[i], bv[j]));
                    }
                }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int sv = s0 + 4 * ty + j;
        if (sv >= ns) continue;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int t = t0 + tx + 16 * i;
            if (t < nt) out[(long long)sv * nt + t] = kfinish(kp, acc[i][j]);
        }
    }
}

// sparse path: out[s][t] = K(test t, SV s) by merge walks, consecutive threads on consecutive test rows
__global__ void kvalue_csr(KP kp, Rows T, Rows S, double *__restrict__ out)
{
    const long long total = (long long)T.n * S.n;
    for (long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x; id < total; id += (long long)gridDim.x * blockDim.x) {
        const int s = (int)(id / T.n), t = (int)(id % T.n);
        out[id] = kval_csr(kp, T.rowptr, T.col, T.val, t, S.rowptr, S.col, S.val, s);
    }
}

// Pair sums, each sequential over the two classes' SVs in model order
// (svm.cpp:2606-2631).  A sum is one chain of dependent additions, so a thread
// that also fetches and multiplies each term waits out a memory round trip per
// few terms (a single row against 1,500 SVs: 125 us); and with a thread per
// row and pair every kernel value is read once per pair its class is in (9 times
// with 10 classes: 3.6 ms for 6,000 rows x 20,000 SVs).  Two kernels:
//   few sums   a block per (row, pair): all threads form the products of the
//              next piece in shared memory while one adds up the previous one;
//   many rows  a thread per row walks all SVs once and keeps every pair's sum:
//              classes come in order, so a pair's first class is added before its
//              second, as the reference does.
constexpr int kPiece = 1024;     // products per piece of a sum

__device__ __forceinline__ void pair_classes(int p, int nr_class, int &i, int &j)
{
    i = 0;
    int rem = p;
    while (rem >= nr_class - 1 - i) { rem -= nr_class - 1 - i; ++i; }
    j = i + 1 + rem;
}

__global__ void __launch_bounds__(256) pair_sums_few(const double *__restrict__ kv, int nt, int ns, int nr_class,
                                                     const int *__restrict__ start, const int *__restrict__ nsv,
                                                     const double *__restrict__ coef, const double *__restrict__ rho,
                                                     double *__restrict__ dec)
{
    __shared__ __align__(16) double prod[2][kPiece];
    const int npair = nr_class * (nr_class - 1) / 2;
    const long long total = (long long)nt * npair;
    for (long long id = blockIdx.x; id < total; id += gridDim.x) {
        const int p = (int)(id / nt), t = (int)(id % nt);
        int i, j;
        pair_classes(p, nr_class, i, j);
        const double *coef1 = coef + (long long)(j - 1) * ns, *coef2 = coef + (long long)i * ns;
        const int ni = nsv[i], n = ni + nsv[j], s1 = start[i], s2 = start[j] - ni;
        const int pieces = (n + kPiece - 1) / kPiece;
        double sum = 0;
        // threads 32.. form piece q + 1 while thread 0 adds piece q
        auto form = [&](int q, int from, int step) {
            const int hi = min(n, (q + 1) * kPiece);
            for (int e = q * kPiece + from; e < hi; e += step) {
                const bool one = e < ni;
                const int s = e + (one ? s1 : s2);
                prod[q & 1][e - q * kPiece] = __dmul_rn(one ? coef1[s] : coef2[s], kv[(long long)s * nt + t]);
            }
        };
        form(0, threadIdx.x, blockDim.x);
        __syncthreads();
        for (int q = 0; q < pieces; q++) {
            if (threadIdx.x >= 32) {
                if (q + 1 < pieces) form(q + 1, threadIdx.x - 32, blockDim.x - 32);
            } else if (threadIdx.x == 0) {
                const double *v = prod[q & 1];
                const int m = min(kPiece, n - q * kPiece);
                int e = 0;
                for (; e + 16 <= m; e += 16) {
                    double2 w[8];
#pragma unroll
                    for (int u = 0; u < 8; u++) w[u] = reinterpret_cast<const double2 *>(v + e)[u];
#pragma unroll
                    for (int u = 0; u < 8; u++) sum = __dadd_rn(__dadd_rn(sum, w[u].x), w[u].y);
                }
                for (; e < m; e++) sum = __dadd_rn(sum, v[e]);
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) dec[(long long)t * npair + p] = __dsub_rn(sum, rho[p]);
        __syncthreads();
    }
}

constexpr int kSumRows = 64;     // test rows per block
constexpr int kSumGroups = 4;    // threads per row, each with a share of a class's partners
constexpr int kSumSv = 32;       // SVs per staged tile
constexpr int kSumStages = 5;
constexpr int kSumMost = 3;      // partners per thread and walk, at most
constexpr int kSumStage = kSumSv * (kSumRows + kSumGroups * kSumMost);       // doubles per stage
constexpr int kSumSmem = kSumStages * kSumStage * 8;

__device__ __forceinline__ void cp_async8(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// N: partners per thread (a class of k has k - 1; its SVs are walked again when
// they are more than kSumGroups * kSumMost).  Bound by HBM: the
// kernel values come from there once, four staged tiles ahead (8-byte copies: an odd
// number of rows leaves no wider alignment).  With plain loads, eight ahead
// per thread, 6,000 rows x 20,000 SVs x 10 classes took 4.5 ms.
template <int N>
__global__ void __launch_bounds__(kSumRows *kSumGroups) pair_sums_many(const double *__restrict__ kv, int nt, int ns,
                                                                        int nr_class, const int *__restrict__ start,
                                                                        const int *__restrict__ nsv,
                                                                        const double *__restrict__ coef,
                                                                        const double *__restrict__ rho,
                                                                        double *__restrict__ dec)
{
    extern __shared__ __align__(16) double stages[];
    const int npair = nr_class * (nr_class - 1) / 2;
    const int tid = threadIdx.x, row = tid % kSumRows, grp = tid / kSumRows;
    const int t0 = blockIdx.x * kSumRows, t = t0 + row;
    const bool in = t < nt;
    double *const mine = dec + (long long)(in ? t : 0) * npair;     // the row's running sums, one per pair
    // the tile the next copies take: class lc, partners from lr, SVs from ls
    int lc = 0, lr = 0, ls = 0;
    auto next_class = [&]() {
        while (lc < nr_class && nsv[lc] == 0) lc++;
        lr = 0;
        if (lc < nr_class) ls = start[lc];
    };
    next_class();
    int to = 0, from = 0;       // stages to copy into / to use
    auto copy = [&]() {
        if (lc < nr_class) {
            double *const kt = stages + to * kSumStage, *const ct = kt + kSumSv * kSumRows;
            const int end = start[lc] + nsv[lc];
            for (int e = tid; e < kSumSv * kSumRows; e += kSumRows * kSumGroups) {
                const int s = ls + e / kSumRows, tt = t0 + e % kSumRows;
                if (s < end && tt < nt) cp_async8(kt + e, kv + (long long)s * nt + tt);
            }
            for (int e = tid; e < kSumSv * kSumGroups * N; e += kSumRows * kSumGroups) {
                const int r = lr + e / kSumSv, s = ls + e % kSumSv;
                if (s < end && r < nr_class - 1) cp_async8(ct + e, coef + (long long)r * ns + s);
            }
            ls += kSumSv;
            if (ls >= end) {
                lr += kSumGroups * N;
                ls = start[lc];
                if (lr >= nr_class - 1) {
                    lc++;
                    next_class();
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        to = to + 1 == kSumStages ? 0 : to + 1;
    };
    for (int q = 0; q < kSumStages - 1; q++) copy();
    for (int c = 0; c < nr_class; c++) {
        const int end = start[c] + nsv[c];
        for (int r0 = 0; r0 < nr_class - 1; r0 += kSumGroups * N) {
            // partner r of class c is class r (r < c) or r + 1, its coefficients row r of coef
            double sum[N];
            int pair[N];
            bool second[N];
#pragma unroll
            for (int u = 0; u < N; u++) {
                const int r = r0 + grp * N + u, o = r < c ? r : r + 1, i = min(c, o), j = max(c, o);
                pair[u] = r < nr_class - 1 && in ? i * (nr_class - 1) - i * (i - 1) / 2 + j - i - 1 : -1;
                second[u] = o < c;
                sum[u] = pair[u] >= 0 && second[u] ? mine[pair[u]] : 0.0;
            }
            for (int sb = start[c]; sb < end; sb += kSumSv) {
                asm volatile("cp.async.wait_group %0;" ::"n"(kSumStages - 2) : "memory");
                __syncthreads();        // the tile has landed, and everyone is done with the one before
                copy();
                const double *const kt = stages + from * kSumStage + row;
                const double *const ct = stages + from * kSumStage + kSumSv * kSumRows + grp * N * kSumSv;
                const int m = min(kSumSv, end - sb);
#pragma unroll 4
                for (int e = 0; e < m; e++) {
                    const double k = kt[e * kSumRows];
#pragma unroll
                    for (int u = 0; u < N; u++) sum[u] = __dadd_rn(sum[u], __dmul_rn(ct[u * kSumSv + e], k));
                }
                from = from + 1 == kSumStages ? 0 : from + 1;
            }
#pragma unroll
            for (int u = 0; u < N; u++)     // a pair is complete after its second class
                if (pair[u] >= 0) mine[pair[u]] = second[u] ? __dsub_rn(sum[u], rho[pair[u]]) : sum[u];
        }
        __syncthreads();        // another thread of the row may hold the pair next
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The kernel for nt rows: the estimated time of both, in additions of one
// chain (about 10 cycles).  Few: the sums go round the GPU's block places (8
// per SM), each the length of its pair.  Many: a block of 64 rows takes about 30
// cycles per SV.  One row, 1,500 SVs, 2 classes: few.  6,000 rows, 20,000
// SVs, 10 classes: many.
cudaError_t launch_pair_sums(const double *kv, int nt, int ns, int nr_class, const int *start, const int *nsv,
                             const double *coef, const double *rho, double *dec)
{
    const double npair = 0.5 * nr_class * (nr_class - 1);
    const double pair_len = 2.0 * ns / nr_class;
    const int blocks = (nt + kSumRows - 1) / kSumRows;
    const double sms = device_sm_count();
    const double few = std::ceil(nt * npair / (sms * 8)) * (pair_len + 200.0);
    const double many = std::ceil(blocks / (sms * 2)) * (ns + 500.0 * nr_class) * 3.0;
    if (few <= many) {
        pair_sums_few<<<(int)std::min<double>(nt * npair, sms * 8), 256>>>(kv, nt, ns, nr_class, start, nsv, coef, rho, dec);
        return cudaGetLastError();
    }
    const int r = nr_class - 1;
    auto *const fn = r <= kSumGroups ? pair_sums_many<1> : r <= 2 * kSumGroups ? pair_sums_many<2> : pair_sums_many<3>;
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSumSmem);
    if (e != cudaSuccess) return e;
    fn<<<blocks, kSumRows * kSumGroups, kSumSmem>>>(kv, nt, ns, nr_class, start, nsv, coef, rho, dec);
    return cudaGetLastError();
}

// Tensor forms: kv[t][s] row-major; one warp per (test row, pair), the lanes
// summing every 32nd SV of each class in model order and the lane sums
// combined by a fixed shuffle tree (the order is the same on every run; the
// exact form keeps the reference's sequential sums in pair_sums)
__global__ void pair_sums_rows(const double *__restrict__ kv, int nt, int ns, int nr_class, const int *__restrict__ start,
                               const int *__restrict__ nsv, const double *__restrict__ coef, const double *__restrict__ rho,
                               double *__restrict__ dec)
{
    const int npair = nr_class * (nr_class - 1) / 2;
    const long long total = (long long)nt * npair;
    const int lane = threadIdx.x & 31;
    const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long id = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; id < total; id += warps) {
        const int t = (int)(id / npair), p = (int)(id % npair);
        int i = 0, rem = p;
        while (rem >= nr_class - 1 - i) { rem -= nr_class - 1 - i; ++i; }
        const int j = i + 1 + rem;
        const double *k = kv + (long long)t * ns;
        const double *coef1 = coef + (long long)(j - 1) * ns;
        const double *coef2 = coef + (long long)i * ns;
        double sum = 0;
        for (int q = lane; q < nsv[i]; q += 32) sum = __dadd_rn(sum, __dmul_rn(coef1[start[i] + q], k[start[i] + q]));
        for (int q = lane; q < nsv[j]; q += 32) sum = __dadd_rn(sum, __dmul_rn(coef2[start[j] + q], k[start[j] + q]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum = __dadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, o));
        if (lane == 0) dec[(long long)t * npair + p] = __dsub_rn(sum, rho[p]);
    }
}

struct Session {
    // fingerprint
    const svm_node *const *SV = nullptr;
    const double *coef0 = nullptr;
    int l = 0, nr_class = 0;
    double rho0 = 0;
    // device copy
    Rows sv;
    Rows sv_csr;                // CSR copy of dense SVs for the merge path (made on first need)
    std::unique_ptr<DeviceRows> sv_tc;   // the SVs in a tensor predict form (split copy), made on first need
    int d = 0, base = 1;
    double *coef = nullptr, *rho = nullptr;
    int *start = nullptr, *nsv = nullptr;
    void release()
    {
        sv.release();
        sv_csr.release();
        sv_tc.reset();
        cudaFree(coef); cudaFree(rho); cudaFree(start); cudaFree(nsv);
        coef = rho = nullptr;
        start = nsv = nullptr;
    }
};

std::mutex g_mu;
std::map<const svm_model *, std::unique_ptr<Session>> g_sessions;
int g_predict_form = FORM_EXACT;

// Per-process prediction buffers, grown on demand and kept (a loop of
// single-row svm_predict calls allocates nothing after its first call).
struct Workspace {
    double *kv = nullptr, *dec = nullptr;
    int *err = nullptr;
    size_t cap_kv = 0, cap_dec = 0, cap_err = 0;
    Rows T;                     // test rows of the current chunk
    // test rows of a tensor form: CSR with float32 values, norms, split copy
    char *t_block = nullptr;
    uint16_t *t_Xs = nullptr;
    double *t_xinv = nullptr;
    size_t cap_t = 0, cap_Xs = 0, cap_xinv = 0;
    char *pin = nullptr;        // page-locked staging of test rows and decision values (at most kPinMost)
    size_t cap_pin = 0, asked_pin[2] = {0, 0};      // what there is; the most that each use asked for without getting it
    size_t held() const { return cap_kv + cap_dec + cap_t + cap_Xs + cap_xinv + cap_pin + T.held(); }
    void release()
    {
        cudaFree(kv); cudaFree(dec); cudaFree(err); cudaFree(t_block); cudaFree(t_Xs); cudaFree(t_xinv);
        T.release();
        if (pin) cudaFreeHost(pin);
        *this = Workspace();
    }
} g_ws;
constexpr size_t kPinMost = 512u << 20, kPinLeast = 1u << 20;
// With no model left, buffers above this are given back.  Smaller ones stay:
// a cross-validation makes and frees a model per fold, and allocating (the
// page-locked staging above all) anew for each took 15 to 40 ms of a call
// whose solves take 1.3 ms, on hosts where such calls are slow.
constexpr size_t kKeepMost = 64u << 20;

// Host staging of at least `bytes`: page-locked and kept, or ordinary memory of
// the call.  Page-locking costs 1 to 5 ms per MB, more than it saves in one call: it
// waits for the second use that needs more than there is, of test rows and of
// models' support vectors each (a model's are staged once).  8,192 rows x 64 after a
// small call: 7 to 28 ms locked at once, 2.8 ms in ordinary memory; later calls
// 0.55 and 1.3 ms.
enum StagingUse { kStageRows, kStageModel };
char *staging(size_t bytes, std::unique_ptr<char[]> &fallback, StagingUse use)
{
    size_t &asked = g_ws.asked_pin[use];
    if (bytes <= g_ws.cap_pin) return g_ws.pin;
    if (bytes <= asked) {
        if (g_ws.pin) cudaFreeHost(g_ws.pin);
        g_ws.pin = nullptr;
        g_ws.cap_pin = 0;
        const size_t want = std::min(kPinMost, std::max(bytes + bytes / 4, kPinLeast));
        if (cudaHostAlloc((void **)&g_ws.pin, want, cudaHostAllocDefault) == cudaSuccess) {
            g_ws.cap_pin = want;
            return g_ws.pin;
        }
        cudaGetLastError();
        g_ws.pin = nullptr;
    }
    if (bytes <= kPinMost) asked = std::max(asked, std::max(bytes, kPinLeast));
    fallback.reset(new char[bytes]);
    return fallback.get();
}
// host loops over fewer rows than this stay on the calling thread (waking the
// others takes longer)
[[maybe_unused]] constexpr int kParallelRows = 128;

#define PK(call)                                                                  \
    do {                                                                          \
        cudaError_t e_ = (call);                                                  \
        if (e_ != cudaSuccess) {                                                  \
            set_error(std::string(#call) + ": " + cudaGetErrorString(e_));        \
            return -1;                                                            \
        }                                                                         \
    } while (0)

// the nodes of every row counted: rp[r + 1] - rp[r]
void count_nodes(const svm_node *const *x, int n, long long *rp)
{
    rp[0] = 0;
#pragma omp parallel for schedule(static) if (n > kParallelRows)
    for (int r = 0; r < n; r++) {
        long long c = 0;
        for (const svm_node *p = x[r]; p->index != -1; ++p) c++;
        rp[(size_t)r + 1] = c;
    }
    for (int r = 0; r < n; r++) rp[(size_t)r + 1] += rp[r];
}

// The copies are queued on the default stream; the caller waits for it before
// the next use of the staging.
int upload_nodes(const svm_node *const *x, int n, int d, int base, bool dense, Rows &out, StagingUse use)
{
    out.n = n;
    out.dense = dense;
    out.ld = (d + 3) & ~3;
    if (out.ld == 0) out.ld = 4;
    std::unique_ptr<char[]> fallback;
    if (dense) {
        const size_t bytes = (size_t)std::max(n, 1) * out.ld * sizeof(double);
        double *h = (double *)staging(bytes, fallback, use);
        if (n == 0) memset(h, 0, bytes);
#pragma omp parallel for schedule(static) if (n > kParallelRows)
        for (int r = 0; r < n; r++) {
            double *row = h + (size_t)r * out.ld;
            memset(row, 0, sizeof(double) * out.ld);
            for (const svm_node *p = x[r]; p->index != -1; ++p) {
                const int c = p->index - base;
                if (c >= 0 && c < out.ld) row[c] = p->value;
            }
        }
        PK(grow(out.X, out.capX, bytes));
        PK(xfer_async(out.X, h, bytes, cudaMemcpyHostToDevice, 0));
        if (fallback) PK(cudaStreamSynchronize(0));
    } else {
        std::vector<long long> rp((size_t)n + 1, 0);
        count_nodes(x, n, rp.data());
        const size_t nnz = (size_t)std::max<long long>(rp[n], 1);
        const size_t b_val = ((size_t)n + 1) * sizeof(long long), b_col = b_val + nnz * sizeof(double);
        char *h = staging(b_col + nnz * sizeof(int), fallback, use);
        memcpy(h, rp.data(), b_val);
        double *val = (double *)(h + b_val);
        int *col = (int *)(h + b_col);
        if (rp[n] == 0) {
            val[0] = 0.0;
            col[0] = 0;
        }
#pragma omp parallel for schedule(static) if (n > kParallelRows)
        for (int r = 0; r < n; r++) {
            long long k = rp[r];
            for (const svm_node *p = x[r]; p->index != -1; ++p, ++k) {
                col[k] = p->index - base;
                val[k] = p->value;
            }
        }
        PK(grow(out.rowptr, out.capRp, b_val));
        PK(grow(out.col, out.capCol, nnz * sizeof(int)));
        PK(grow(out.val, out.capVal, nnz * sizeof(double)));
        PK(xfer_async(out.rowptr, h, b_val, cudaMemcpyHostToDevice, 0));
        PK(xfer_async(out.col, col, nnz * sizeof(int), cudaMemcpyHostToDevice, 0));
        PK(xfer_async(out.val, val, nnz * sizeof(double), cudaMemcpyHostToDevice, 0));
        if (fallback) PK(cudaStreamSynchronize(0));
    }
    return 0;
}

Session *get_session(const svm_model *m)
{
    auto it = g_sessions.find(m);
    if (it != g_sessions.end()) {
        Session *s = it->second.get();
        if (s->SV == m->SV && s->l == m->l && s->nr_class == m->nr_class &&
            s->coef0 == (m->nr_class > 1 ? m->sv_coef[0] : nullptr) && s->rho0 == (m->nr_class > 1 ? m->rho[0] : 0.0))
            return s;
        s->release();
        g_sessions.erase(it);
    }
    std::unique_ptr<Session> s(new Session());
    s->SV = m->SV;
    s->l = m->l;
    s->nr_class = m->nr_class;
    s->coef0 = m->nr_class > 1 ? m->sv_coef[0] : nullptr;
    s->rho0 = m->nr_class > 1 ? m->rho[0] : 0.0;
    int maxi = 0;
    long long nnz = 0;
    for (int i = 0; i < m->l; i++)
        for (const svm_node *p = m->SV[i]; p->index != -1; ++p) { maxi = std::max(maxi, p->index); nnz++; }
    s->base = 0;
    s->d = maxi + 1;
    const bool dense = m->l == 0 || (double)nnz >= 0.25 * (double)m->l * s->d || (double)m->l * s->d * 4 < 32e6;
    if (upload_nodes(m->SV, m->l, s->d, s->base, dense, s->sv, kStageModel) != 0) return nullptr;
    if (cudaStreamSynchronize(0) != cudaSuccess) {      // the staging is used again
        set_error("upload of the support vectors failed");
        return nullptr;
    }
    const int k = m->nr_class, npair = k * (k - 1) / 2;
    std::vector<double> coef((size_t)std::max(k - 1, 1) * std::max(m->l, 1), 0.0);
    for (int j = 0; j < k - 1; j++)
        for (int i = 0; i < m->l; i++) coef[(size_t)j * m->l + i] = m->sv_coef[j][i];
    std::vector<int> start(std::max(k, 1), 0), nsv(std::max(k, 1), 0);
    // one-class and SVR models have no classes: all SVs form one group and
    // the value is the single "pair" sum over it (svm.cpp:2571-2587)
    for (int i = 0; i < k; i++) nsv[i] = m->nSV ? m->nSV[i] : (i == 0 ? m->l : 0);
    for (int i = 1; i < k; i++) start[i] = start[i - 1] + nsv[i - 1];
    std::vector<double> rho(std::max(npair, 1), 0.0);
    for (int p = 0; p < npair; p++) rho[p] = m->rho[p];
    if (cudaMalloc(&s->coef, coef.size() * 8) != cudaSuccess || cudaMalloc(&s->rho, rho.size() * 8) != cudaSuccess ||
        cudaMalloc(&s->start, start.size() * 4) != cudaSuccess || cudaMalloc(&s->nsv, nsv.size() * 4) != cudaSuccess) {
        set_error("device allocation for prediction failed");
        s->release();
        return nullptr;
    }
    xfer(s->coef, coef.data(), coef.size() * 8, cudaMemcpyHostToDevice);
    xfer(s->rho, rho.data(), rho.size() * 8, cudaMemcpyHostToDevice);
    xfer(s->start, start.data(), start.size() * 4, cudaMemcpyHostToDevice);
    xfer(s->nsv, nsv.data(), nsv.size() * 4, cudaMemcpyHostToDevice);
    Session *raw = s.get();
    g_sessions[m] = std::move(s);
    return raw;
}

// rows as host CSR (0-based columns) of width d
int rows_to_device(const svm_node *const *x, int n, int d, int form, DeviceRows &out)
{
    // CSR of the rows (columns = libsvm indices), counted and filled in
    // parallel over rows
    std::vector<long long> rp((size_t)n + 1, 0);
#pragma omp parallel for schedule(static)
    for (int r = 0; r < n; r++) {
        long long c = 0;
        for (const svm_node *p = x[r]; p->index != -1; ++p) c++;
        rp[(size_t)r + 1] = c;
    }
    for (int r = 0; r < n; r++) rp[(size_t)r + 1] += rp[r];
    std::vector<int> col((size_t)std::max<long long>(rp[n], 1), 0);
    std::vector<float> val(col.size(), 0.0f);
#pragma omp parallel for schedule(static)
    for (int r = 0; r < n; r++) {
        long long k = rp[r];
        for (const svm_node *p = x[r]; p->index != -1; ++p, ++k) {
            col[k] = p->index;
            val[k] = (float)p->value;
        }
    }
    if (upload_csr(rp.data(), col.data(), val.data(), n, d, out, -1, 0) != 0) return -1;
    return out.prepare_form(form, 0);
}

// The test rows of a call in a tensor form: CSR in the kept workspace, its
// norms and split copy.  `out` borrows the buffers (see BorrowedRows).
int tensor_rows(const svm_node *const *x, int n, int d, int form, DeviceRows &out)
{
    std::vector<long long> rp((size_t)n + 1, 0);
    count_nodes(x, n, rp.data());
    const size_t nnz = (size_t)std::max<long long>(rp[n], 1);
    auto al = [](size_t v) { return (v + 255) & ~size_t(255); };
    const size_t b_col = al(((size_t)n + 1) * 8), b_val = al(b_col + nnz * 4), up = b_val + nnz * 4;
    const size_t b_sq = al(up), total = b_sq + (size_t)n * 8;
    std::unique_ptr<char[]> fallback;
    char *h = staging(up, fallback, kStageRows);
    memcpy(h, rp.data(), ((size_t)n + 1) * 8);
    int *col = (int *)(h + b_col);
    float *val = (float *)(h + b_val);
#pragma omp parallel for schedule(static) if (n > kParallelRows)
    for (int r = 0; r < n; r++) {
        long long k = rp[r];
        for (const svm_node *p = x[r]; p->index != -1; ++p, ++k) {
            col[k] = p->index;
            val[k] = (float)p->value;
        }
    }
    out.n = n;
    out.d = d > 0 ? d : 1;
    out.ld = (out.d + 3) & ~3;
    out.nnz = rp[n];
    out.nchunk = std::max(1, (out.d + kSplitChunk - 1) / kSplitChunk);
    const size_t b_Xs = (size_t)n * out.nchunk * 2 * kSplitChunk * sizeof(uint16_t);
    PK(grow(g_ws.t_block, g_ws.cap_t, total));
    PK(grow(g_ws.t_Xs, g_ws.cap_Xs, b_Xs));
    if (form == FORM_FP16X3) PK(grow(g_ws.t_xinv, g_ws.cap_xinv, (size_t)n * 8));
    out.rowptr = (long long *)g_ws.t_block;
    out.col = (int *)(g_ws.t_block + b_col);
    out.val = (float *)(g_ws.t_block + b_val);
    out.xsq[FORM_EXACT] = (double *)(g_ws.t_block + b_sq);
    PK(xfer_async(g_ws.t_block, h, up, cudaMemcpyHostToDevice, 0));
    if (fallback) PK(cudaStreamSynchronize(0));
    PK(launch_xsq(out.view(FORM_EXACT), n, out.xsq[FORM_EXACT], FORM_EXACT, 0));
    count_launch();
    PK(cudaMemsetAsync(g_ws.t_Xs, 0, b_Xs, 0));
    PK(launch_split(out, form, out.nchunk, g_ws.t_Xs, form == FORM_FP16X3 ? g_ws.t_xinv : nullptr, 0));
    out.Xs = g_ws.t_Xs;
    out.xinv = form == FORM_FP16X3 ? g_ws.t_xinv : nullptr;
    out.split_form = form;
    return 0;
}
// a DeviceRows frees its split copy: one that borrows it lets go first
struct BorrowedRows : DeviceRows {
    ~BorrowedRows()
    {
        Xs = nullptr;
        xinv = nullptr;
    }
};

// The SVs' split (or tf32) copy for tensor-core kernel values, made once per
// model, form and width: both row sets of the block product need the same
// split width, and test rows wider than the SVs widen it (their extra
// features still count in the RBF norms).
int prepare_tensor_svs(const svm_model *m, Session *s, int width, int form)
{
    width = std::max(width, s->d);
    if (s->sv_tc && s->sv_tc->split_form == form && s->sv_tc->d >= width) return 0;
    s->sv_tc.reset(new DeviceRows());
    if (rows_to_device(m->SV, m->l, width, form, *s->sv_tc) != 0) {
        s->sv_tc.reset();
        return -1;
    }
    return 0;
}

}  // namespace

int predict_set_form(int form)
{
    if (form != FORM_EXACT && !is_tc_form(form)) return -1;
    std::lock_guard<std::mutex> g(g_mu);
    g_predict_form = form;
    return 0;
}

void predict_forget(const svm_model *model)
{
    std::lock_guard<std::mutex> g(g_mu);
    auto it = g_sessions.find(model);
    if (it != g_sessions.end()) {
        it->second->release();
        g_sessions.erase(it);
        if (g_sessions.empty() && g_ws.held() > kKeepMost) g_ws.release();
    }
}

int predict_batch(const svm_model *m, const svm_node *const *rows, int n, double *labels, double *dec_out)
{
    const int type = m->param.svm_type;
    if (type < C_SVC || type > NU_SVR) {
        set_error("unknown svm_type in the model");
        return -1;
    }
    if (m->param.kernel_type == PRECOMPUTED) {
        set_error("precomputed kernels are not supported on the GPU");
        return -1;
    }
    const bool classify = type == C_SVC || type == NU_SVC;
    std::lock_guard<std::mutex> g(g_mu);
    Session *s = get_session(m);
    if (!s) return -1;
    const int k = m->nr_class, npair = k * (k - 1) / 2;
    if (n == 0) return 0;
    KP kp{m->param.kernel_type, m->param.degree, m->param.gamma, m->param.coef0};
    std::vector<double> dec((size_t)n * std::max(npair, 1), 0.0);
    if (npair > 0 && m->l > 0) {
        // the test rows go to the device once; kernel values are made in
        // chunks of rows whose value block stays below a quarter of the free
        // device memory (at most 4 GB)
        const bool trace = getenv("SVMB_TRACE") && *getenv("SVMB_TRACE") == '1';
        const auto c0 = std::chrono::steady_clock::now();
        // (asking for the free memory takes longer than a small call's kernels:
        // not when the block in hand, or the least one allowed, will do)
        const long long per_row = (long long)m->l * 8;
        long long budget = std::max<long long>((long long)g_ws.cap_kv, 64LL << 20);
        if (n * per_row > budget) {
            size_t free_b = 0, total_b = 0;
            if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) free_b = 1ull << 32;
            budget = std::max(budget, std::min<long long>(4LL << 30, (long long)(free_b / 4)));
        }
        const int chunk = (int)std::max<long long>(1, std::min<long long>(n, budget / per_row));
        PK(grow(g_ws.kv, g_ws.cap_kv, (size_t)chunk * per_row));
        PK(grow(g_ws.dec, g_ws.cap_dec, (size_t)chunk * npair * 8));
        double *kv = g_ws.kv, *d_dec = g_ws.dec;
        // test rows: features beyond the SVs' width cannot meet an SV feature in a
        // dot product but still count in the RBF distance, so widen to cover them
        int maxi = s->d - 1;
#pragma omp parallel for schedule(static) reduction(max : maxi) if (n > kParallelRows)
        for (int r = 0; r < n; r++)
            for (const svm_node *p = rows[r]; p->index != -1; ++p) maxi = std::max(maxi, p->index);
        const bool wider = maxi + 1 > s->d;
        const bool tensor = is_tc_form(g_predict_form);
        const bool dense = !tensor && s->sv.dense && !wider;
        Rows &T = g_ws.T;
        BorrowedRows Ttc;
        if (tensor) {
            if (prepare_tensor_svs(m, s, maxi + 1, g_predict_form) != 0) return -1;
            if (tensor_rows(rows, n, s->sv_tc->d, g_predict_form, Ttc) != 0) return -1;
        } else if (dense) {
            if (upload_nodes(rows, n, s->d, s->base, true, T, kStageRows) != 0) return -1;
        } else {
            if (s->sv.dense && !s->sv_csr.rowptr) {
                if (upload_nodes(m->SV, m->l, s->d, s->base, false, s->sv_csr, kStageModel) != 0) return -1;
                PK(cudaStreamSynchronize(0));       // the staging is used again
            }
            if (upload_nodes(rows, n, maxi + 1, s->base, false, T, kStageRows) != 0) return -1;
        }
        int *d_err = nullptr;
        if (tensor) {
            PK(grow(g_ws.err, g_ws.cap_err, sizeof(int)));
            d_err = g_ws.err;
            PK(cudaMemsetAsync(d_err, 0, sizeof(int), 0));
        }
        const auto c1 = std::chrono::steady_clock::now();
        KernelParams kpk{m->param.kernel_type, m->param.degree, m->param.gamma, m->param.coef0};
        for (int t0 = 0; t0 < n; t0 += chunk) {
            const int tn = std::min(chunk, n - t0);
            if (tensor) {
                PK(launch_kernel_block2(Ttc, *s->sv_tc, kpk, g_predict_form, t0, tn, m->l, kv, m->l, 0, d_err, 0));
            } else if (dense) {
                dim3 grid((m->l + kPS - 1) / kPS, (tn + kPT - 1) / kPT);
                kvalue_tile<<<grid, 256>>>(kp, T.X + (long long)t0 * T.ld, tn, s->sv.X, m->l, s->sv.ld, kv);
                count_launch();
            } else {
                const Rows &Sc = s->sv.dense ? s->sv_csr : s->sv;
                Rows Tc = T;               // a view of rows t0 .. t0+tn (row pointers stay absolute)
                Tc.rowptr = T.rowptr + t0;
                Tc.n = tn;
                kvalue_csr<<<(int)std::min<long long>(((long long)tn * m->l + 255) / 256, 148 * 16), 256>>>(kp, Tc, Sc, kv);
                count_launch();
            }
            if (tensor)
                pair_sums_rows<<<(int)std::min<long long>(((long long)tn * npair * 32 + 255) / 256, 148 * 16), 256>>>(
                    kv, tn, m->l, k, s->start, s->nsv, s->coef, s->rho, d_dec);
            else
                PK(launch_pair_sums(kv, tn, m->l, k, s->start, s->nsv, s->coef, s->rho, d_dec));
            count_launch();
            // (the test rows have left the staging once these kernels have run)
            const size_t bytes = (size_t)tn * npair * 8;
            char *const to = (char *)(dec.data() + (size_t)t0 * npair), *const h = bytes <= g_ws.cap_pin ? g_ws.pin : to;
            cudaError_t e = cudaSuccess;
            if (t0 == 0) e = cudaStreamSynchronize(0);
            if (e == cudaSuccess) e = xfer_async(h, d_dec, bytes, cudaMemcpyDeviceToHost, 0);
            if (e == cudaSuccess) e = cudaStreamSynchronize(0);
            if (e != cudaSuccess) {
                set_error(std::string("prediction kernels failed: ") + cudaGetErrorString(e));
                return -1;
            }
            if (h != to) memcpy(to, h, bytes);
        }
        if (tensor) {
            int herr = 0;
            PK(xfer(&herr, d_err, sizeof(int), cudaMemcpyDeviceToHost));
            if (herr) {
                set_error("tensor-core kernel values: a wait timed out");
                return -1;
            }
        }
        if (trace) {
            const auto c2 = std::chrono::steady_clock::now();
            auto ms = [](std::chrono::steady_clock::time_point a, std::chrono::steady_clock::time_point b) {
                return std::chrono::duration<double, std::milli>(b - a).count();
            };
            fprintf(stderr, "[svmb] predict rows=%d svs=%d chunks=%d rows_to_device=%.2fms values+sums=%.2fms\n", n,
                    m->l, (n + chunk - 1) / chunk, ms(c0, c1), ms(c1, c2));
        }
    } else if (npair > 0) {
        for (int t = 0; t < n; t++)
            for (int p = 0; p < npair; p++) dec[(size_t)t * npair + p] = -m->rho[p];
    }
#pragma omp parallel for schedule(static) if (n > kParallelRows)
    for (int t = 0; t < n; t++) {
        if (!classify) {
            // one-class: the side of the boundary; SVR: the value (svm.cpp:2585-2587)
            const double v = dec[t];
            labels[t] = type == ONE_CLASS ? (v > 0 ? 1 : -1) : v;
            if (dec_out) dec_out[t] = v;
            continue;
        }
        // votes, ties to the lowest class index (svm.cpp:2627-2637)
        std::vector<int> vote(std::max(k, 1), 0);
        int p = 0;
        for (int i = 0; i < k; i++)
            for (int j = i + 1; j < k; j++) {
                if (dec[(size_t)t * npair + p] > 0) ++vote[i];
                else ++vote[j];
                p++;
            }
        int best = 0;
        for (int i = 1; i < k; i++)
            if (vote[i] > vote[best]) best = i;
        labels[t] = m->label ? m->label[best] : 0;
        if (dec_out)
            for (int q = 0; q < npair; q++) dec_out[(size_t)t * npair + q] = dec[(size_t)t * npair + q];
    }
    return 0;
}

}  // namespace svmb
