// smo_resident.cuh -- the solver loop of resident instances (device code).
//
// An instance whose kernel matrix is in its cache before the solve needs no
// row pass, no cache decisions and no prefetching, so its iteration is the bare
// chain
//
//   i known -> row Q_i -> j scan -> block's best -> group's best -> step,
//   row Q_j -> update and I_up scan -> block's best -> group's best -> next i
//
// What bounds it: latency (L2 row reads, block barriers, the trip between
// blocks) and, just as much, instruction fetch: the general loop executes
// more code per iteration than the instruction cache holds, and the mere
// presence of its cold paths cost 20%.  Hence a loop of its own with nothing
// else in it, and:
//   - the group is one thread-block cluster of up to kClusterMax blocks, and a
//     record goes straight into every block's shared memory (st.async, which
//     also counts its bytes on the receiver's mbarrier).  Through L2 an exchange
//     took about 2.2k cycles; this one about half.
//   - every warp waits on that mbarrier itself and takes the winner from the
//     records, so a phase has one block barrier instead of two.
// The records are double-buffered by exchange parity: a block overwrites a
// buffer two exchanges of the same kind later, when every block's warps have
// gone through a barrier after their last read of it.
//
// Measured (whole svm_train calls; the general loop as it was before this one,
// with its fence-and-flag records and row passes, then this loop): 500 x 16 8.0
// and 1.5 ms, 4000 x 64 66.5 and 11.1 ms (8 blocks), epsilon-SVR 2500 x 8 450
// and 90 ms, 6000 sparse rows of 20000 columns (a triangle, 16 blocks) 484 and
// 52 ms.  An iteration takes 3.3 to 4.4 us; instruction-cache misses fell
// from 225 to 13 per iteration.
//
// Choices, arithmetic and tie rules are the general loop's; the collective
// sections (shrinking, reconstruction, start and end) are the same functions.
#pragma once
#include "smo_solver.cuh"

namespace svmb {
namespace {

// a record word as st.async writes it
struct alignas(16) ResWord {
    double d;
    unsigned x, pad;
};
constexpr int kResWords = 9;        // 8 words per block and buffer, and one that keeps blocks in distinct banks
static_assert(2 * kWordsI < kResWords && kWordsJ < kResWords, "record buffers are too small");
struct ResRecords {
    ResWord a[2][kClusterMax][kResWords], b[2][kClusterMax][kResWords];
    uint64_t bar_a, bar_b;
};
__device__ __forceinline__ ResRecords &res_records()
{
    __shared__ ResRecords r;
    return r;
}

__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, int rank)
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
    return a;
}
__device__ __forceinline__ void st_async_word(uint32_t addr, double d, unsigned x, uint32_t bar)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(addr), "r"((unsigned)b), "r"((unsigned)(b >> 32)), "r"(x), "r"(0u), "r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_cluster(uint64_t *bar, unsigned parity)
{
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(tc::smem_addr(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// the slow part of a wait: until the group's error flag is set or the bound runs out
__device__ __noinline__ bool mbar_wait_long(uint64_t *bar, unsigned parity)
{
    const InstanceDesc &D = block_shared().D;
    const long long t0 = (long long)tc::global_ns(), limit = D.wait_ns > 0 ? D.wait_ns : kWaitTimeoutNs;
    for (unsigned k = 1;; k++) {
        if (mbar_try_cluster(bar, parity)) return true;
        if ((k & 63u) == 0 && (ld_relaxed_i32(&D.sync->error) != 0 || (long long)tc::global_ns() - t0 > limit)) {
            atomicExch(&D.sync->error, 1);
            return false;
        }
    }
}
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t *bar, unsigned parity)
{
#pragma unroll 1
    for (int k = 0; k < 64; k++)
        if (mbar_try_cluster(bar, parity)) return true;
    return mbar_wait_long(bar, parity);
}

// Row i of a resident matrix: a row of its own, or a row and a column of the triangle.
struct TriRow {
    const float *Q;
    unsigned i;
    __device__ __forceinline__ float operator[](int c) const { return Q[tri_at(i, (unsigned)c)]; }
};
template <bool TRI>
struct RowOf {
    typedef const float *type;
    static __device__ __forceinline__ type at(const float *Q, long long stride, int i) { return Q + (long long)i * stride; }
};
template <>
struct RowOf<true> {
    typedef TriRow type;
    static __device__ __forceinline__ type at(const float *Q, long long, int i) { return TriRow{Q, (unsigned)i}; }
};

// The block's I_up maxima (per track) to every block of the cluster, then the
// group's.  ok: this warp's last wait did not run out.  Returns 1 when the
// records are in buffer (count - 1) & 1, 0 when this warp's wait ran out (its
// next barrier must be a __syncthreads_or), -1 when another warp's last one did.
template <int nu>
__device__ __forceinline__ int res_exchange_iup(unsigned &count, bool ok, const double (&v)[2], const int (&ix)[2])
{
    Shared &sh = block_shared();
    ResRecords &R = res_records();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned par = count & 1u;
    const Ctx &c = sh.c;
    const Chunk ck = chunk_at(c.choff, sh.D.chunk_cap);
    u64 k0 = ix[0] >= 0 ? key_of(v[0]) : 0, k1 = 0;
    int p0 = ix[0], p1 = -1;
    warp_best(k0, p0);
    if (nu) {
        k1 = ix[1] >= 0 ? key_of(v[1]) : 0;
        p1 = ix[1];
        warp_best(k1, p1);
    }
    if (lane == 0) {
        sh.wk[0][warp] = k0;
        sh.wi[0][warp] = p0;
        if (nu) {
            sh.wk[1][warp] = k1;
            sh.wi[1][warp] = p1;
        }
    }
    if (__syncthreads_or(!ok)) return -1;
    if (warp == 0) {
        constexpr int W = (nu ? 2 : 1) * kWordsI;
        const int m = lane & (kWarps - 1);      // (both halves of the warp see every warp's result)
        k0 = sh.wk[0][m];
        p0 = sh.wi[0][m];
        warp_best(k0, p0);
        if (nu) {
            k1 = sh.wk[1][m];
            p1 = sh.wi[1][m];
            warp_best(k1, p1);
        }
        // a lane builds word e of the record and sends it to blocks lane / W, + 32 / W ..
        // (without branches: word w of a track is the w-th of G, alpha and QD)
        const int e = lane & (W - 1), w = e & (kWordsI - 1), p = nu && e >= kWordsI ? p1 : p0;
        const int q = p >= 0 ? p - c.a0 : 0;
        double d = ck.G[min(w, 2) * sh.D.chunk_cap + q];
        const unsigned f = ck.F[q], col = (unsigned)ck.Col[q];
        if (w == 0 && flag_y(f) > 0) d = -d;
        unsigned x = w == 0 ? pos_code(p, flag_y(f)) : col;
        if (p < 0) {
            d = -SVMB_INF;
            x = kNoPos;
        }
        if (lane == 0) mbar_expect(&R.bar_a, (unsigned)(c.nb * W * 16));
        const uint32_t dst = tc::smem_addr(&R.a[par][c.rank][e]), bar = tc::smem_addr(&R.bar_a);
        for (int b = lane / W; b < c.nb; b += 32 / W) st_async_word(cluster_addr(dst, b), d, x, cluster_addr(bar, b));
        __syncwarp();
    }
    count++;
    return mbar_wait_cluster(&R.bar_a, par) ? 1 : 0;
}

// The same for the block's second-order j candidate and its Gmax2 maxima.
template <int nu>
__device__ __forceinline__ int res_exchange_j(unsigned &count, bool ok, double dec, int jx, float jq, double g2, double g2n)
{
    Shared &sh = block_shared();
    ResRecords &R = res_records();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned par = count & 1u;
    const Ctx &c = sh.c;
    const Chunk ck = chunk_at(c.choff, sh.D.chunk_cap);
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
        if (nu) sh.wk[2][warp] = kn;
    }
    if (__syncthreads_or(!ok)) return -1;
    if (warp == 0) {
        constexpr int W = nu ? kWordsJ : kWordsJ - 1;
        const int m = lane & (kWarps - 1), mi = sh.wi[0][m];
        const float mq = sh.wq[m];
        k = sh.wk[0][m];
        p = mi;
        warp_best(k, p);
        kg = warp_max_key(sh.wk[1][m]);
        if (nu) kn = warp_max_key(sh.wk[2][m]);
        // (without branches: words 1 to 3 are the 1st to 3rd of G, alpha and QD)
        const int e = lane & 7, q = p >= 0 ? p - c.a0 : 0;
        const double g = ck.G[min(max(e - 1, 0), 2) * sh.D.chunk_cap + q];
        const unsigned f = ck.F[q], col = (unsigned)ck.Col[q];
        const u64 kd = e == 0 ? k : e == 4 ? kg : kn;
        const double d = e >= 1 && e <= 3 ? g : key_value(kd);
        const float jqv = __shfl_sync(0xffffffffu, mq, __ffs(__ballot_sync(0xffffffffu, mi == p)) - 1);
        const unsigned x = p < 0 ? kNoPos : e == 0 ? pos_code(p, flag_y(f)) : e == 1 ? col : __float_as_uint(jqv);
        if (lane == 0) mbar_expect(&R.bar_b, (unsigned)(c.nb * W * 16));
        const uint32_t dst = tc::smem_addr(&R.b[par][c.rank][e]), bar = tc::smem_addr(&R.bar_b);
        if (e < W)
            for (int b = lane >> 3; b < c.nb; b += 4) st_async_word(cluster_addr(dst, b), d, x, cluster_addr(bar, b));
        __syncwarp();
    }
    count++;
    return mbar_wait_cluster(&R.bar_b, par) ? 1 : 0;
}

// the block whose record word 0 wins (largest value, ties to the larger position)
__device__ __forceinline__ int res_win(const ResWord (&r)[kClusterMax][kResWords], int word, int nb)
{
    if (nb == 1) return 0;
    const int lane = threadIdx.x & 31;
    const int p = lane < nb ? code_pos(r[lane][word].x) : -1;
    u64 key = p >= 0 ? key_of(r[lane][word].d) : 0;
    int best = p;
    warp_best(key, best);
    return best < 0 ? 0 : __ffs(__ballot_sync(0xffffffffu, p == best)) - 1;
}
// the largest d of a word over the blocks
__device__ __forceinline__ double res_max(const ResWord (&r)[kClusterMax][kResWords], int word, int nb)
{
    if (nb == 1) return r[0][word].d;
    const int lane = threadIdx.x & 31;
    return key_value(warp_max_key(lane < nb ? key_of(r[lane][word].d) : 0));
}

template <int nu>
__device__ __noinline__ int res_scan_iup(unsigned &count)
{
    Ctx &c = block_shared().c;
    const Chunk ck = chunk_at(c.choff, block_shared().D.chunk_cap);
    double v[2] = {-SVMB_INF, -SVMB_INF};
    int ix[2] = {-1, -1};
    for (int k = threadIdx.x; k < c.a1 - c.a0; k += kThreads) {
        const unsigned f = ck.F[k];
        const bool pos = (f & kFlagPos) != 0;
        const double yG = pos ? -ck.G[k] : ck.G[k];
        if (flag_s(f) == (pos ? ST_UPPER : ST_LOWER)) continue;
        if (pos || !nu) better_max(v[0], ix[0], yG, c.a0 + k);
        else better_max(v[1], ix[1], yG, c.a0 + k);
    }
    return res_exchange_iup<nu>(count, true, v, ix);
}

template <int FORM, bool NU, bool TRI>
__device__ __noinline__ void solve_resident(int rank)
{
    constexpr int nu = NU ? 1 : 0;
    Shared &sh = block_shared();
    ResRecords &R = res_records();
    const InstanceDesc &D = sh.D;
    const Ctx &c = sh.c;
    if (!start_solve<FORM>(rank)) {
        fail_solve(0, 0);
        return;
    }
    if (D.mute == 1 && rank == D.nblocks - 1) return;
    const Chunk ck = chunk_at(c.choff, D.chunk_cap);
    const int l = D.l, nb = D.nblocks;
    typedef typename RowOf<TRI>::type Row;
    const float *const Q = D.cache.data;
    const long long stride = D.cache.stride;
    unsigned ka = 0, kb = 0;        // exchanges so far
    long long iter = 0, sum_from = 0;
    int unshrink = 0, status = 0, ok = 0;
    unsigned tmark = (unsigned)clock();
    auto mark = [&](int k) {
        if (threadIdx.x == 0) {
            const unsigned now = (unsigned)clock();
            atomicAdd(&sh.prof32[k], now - tmark);
            tmark = now;
        }
    };
    // counters of thread 0: active positions, phase-A passes, and the timers in 64 bits
    auto fold = [&]() {
        if (threadIdx.x == 0) {
            sh.cnt[kCntActive] += (iter - sum_from) * c.A;
            for (int k = 0; k < 8; k++) {
                sh.prof[k] += sh.prof32[k];
                sh.prof32[k] = 0;
            }
        }
        sum_from = iter;
    };
    int counter = (l < 1000 ? l : 1000) + 1;
    if ((ok = res_scan_iup<nu>(ka)) < 0) goto fail;
    while (iter < D.max_iter) {
        if (--counter == 0) {
            if (__syncthreads_or(!ok)) goto fail;
            counter = l < 1000 ? l : 1000;
            fold();
            if (D.shrinking) {
                mark(kProfBUpdate);
                if (!do_shrinking<FORM>(unshrink)) goto fail;
                if ((ok = res_scan_iup<nu>(ka)) < 0) goto fail;
                mark(kProfShrink);
            }
        }
        int widened = 0;
    select_again:
        // ======================= phase A: the j scan =======================
        const unsigned pa = (ka - 1) & 1u;
        const int n = c.a1 - c.a0, a0 = c.a0;
        const int e0 = ok ? res_win(R.a[pa], 0, nb) : 0, e1 = nu && ok ? res_win(R.a[pa], kWordsI, nb) : 0;
        const ResWord *const w0 = R.a[pa][e0], *const w1 = R.a[pa][e1] + kWordsI;
        int i0 = -1, i1 = -1;
        Row Qi0 = RowOf<TRI>::at(Q, stride, 0), Qi1 = Qi0;
        double dec = -SVMB_INF, g2 = -SVMB_INF, g2n = -SVMB_INF;
        int jx = -1;
        float jq = 0.0f;
        if (ok) {
            i0 = code_pos(w0[0].x);
            if (i0 >= 0) Qi0 = RowOf<TRI>::at(Q, stride, (int)w0[1].x);
            if (nu) {
                i1 = code_pos(w1[0].x);
                if (i1 >= 0) Qi1 = RowOf<TRI>::at(Q, stride, (int)w1[1].x);
            }
        }
        if (i0 >= 0 || (nu && i1 >= 0)) {
            const double Gmax0 = w0[0].d, Gmax1 = nu ? w1[0].d : 0.0;
            const double QDi0 = w0[2].d, QDi1 = nu ? w1[2].d : 0.0;
            const double two_yi0 = __dmul_rn(2.0, (double)code_y(w0[0].x));
            // the general loop's scan: rough quotients first, see there
            auto row_at = [&](int k) -> float {
                if (!nu) return Qi0[ck.Col[k]];
                if (ck.F[k] & kFlagPos) return i0 >= 0 ? Qi0[ck.Col[k]] : 0.0f;
                return i1 >= 0 ? Qi1[ck.Col[k]] : 0.0f;
            };
            auto quotient = [&](int k, float q, double &num, double &quad) -> bool {
                const unsigned f = ck.F[k];
                const bool pos = (f & kFlagPos) != 0;
                if (flag_s(f) == (pos ? ST_LOWER : ST_UPPER)) return false;
                const double G = ck.G[k], yG = pos ? G : -G;
                const double grad_diff = __dadd_rn(pos || !nu ? Gmax0 : Gmax1, yG);
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
            float q1 = 0.0f;
            float qn = threadIdx.x < n ? row_at(threadIdx.x) : 0.0f;
#pragma unroll 1
            for (int k = threadIdx.x; k < n; k += kThreads) {
                const float q = qn;
                if (k + kThreads < n) qn = row_at(k + kThreads);    // one position ahead
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
                    double num, quad;
                    const float q = row_at(k);
                    if (!quotient(k, q, num, quad) || rough_quotient(num, quad) < least) continue;
                    better_max(dec, jx, __ddiv_rn(num, quad), a0 + k);
                    if (jx == a0 + k) jq = q;
                }
            } else if (r1 >= least) {
                better_max(dec, jx, __ddiv_rn(num1, quad1), a0 + k1);
                jq = q1;
            }
        } else if (ok) {
            // no candidate i at all: only the Gmax2 maxima matter
            for (int k = threadIdx.x; k < n; k += kThreads) {
                const unsigned f = ck.F[k];
                const bool pos = (f & kFlagPos) != 0;
                if (flag_s(f) == (pos ? ST_LOWER : ST_UPPER)) continue;
                if (pos || !nu) g2 = fmax(g2, pos ? ck.G[k] : -ck.G[k]);
                else g2n = fmax(g2n, -ck.G[k]);
            }
        }
        __syncwarp();
        if ((ok = res_exchange_j<nu>(kb, ok != 0, dec, jx, jq, g2, g2n)) < 0) goto fail;
        mark(kProfAScan);

        // ======================= phase B: step and update =======================
        const unsigned pb = (kb - 1) & 1u;
        const int eb = ok ? res_win(R.b[pb], 0, nb) : 0;
        const ResWord *const wj = R.b[pb][eb];
        double v[2] = {-SVMB_INF, -SVMB_INF};
        int ix[2] = {-1, -1};
        if (ok) {
            const int j = code_pos(wj[0].x);
            // the working pair; nu-SVC takes i from the track of y_j (svm.cpp:1179-1182)
            const int yj = code_y(wj[0].x);
            const int tr = nu && j >= 0 && yj != +1 ? 1 : 0;
            const ResWord *const wi = tr ? w1 : w0;
            const int i = tr ? i1 : i0, yi = tr ? -1 : code_y(w0[0].x);
            const Row Qi = tr ? Qi1 : Qi0, Qj = RowOf<TRI>::at(Q, stride, j >= 0 ? (int)wj[1].x : 0);
            int k = threadIdx.x;
            float qin = 0.0f, qjn = 0.0f;
            if (j >= 0 && k < n) {      // on their way during the stopping test and the step
                qin = Qi[ck.Col[k]];
                qjn = Qj[ck.Col[k]];
            }
            const double Gmax0 = w0[0].d, Gmax1 = nu ? w1[0].d : 0.0;
            const double gm = res_max(R.b[pb], 4, nb), gmn = nu ? res_max(R.b[pb], 5, nb) : 0.0;
            const bool stop = (!nu ? __dadd_rn(Gmax0, gm) : fmax(__dadd_rn(Gmax0, gm), __dadd_rn(Gmax1, gmn))) < D.eps;
            if (stop || j < 0) {
                if (__syncthreads_or(0)) goto fail;
                if (widened) break;
                fold();
                if (c.A < l && !reopen<FORM>()) goto fail;
                widened = 1;
                if ((ok = res_scan_iup<nu>(ka)) < 0) goto fail;
                goto select_again;
            }
            if (widened) counter = 1;
            ++iter;
            const double alpha_i = wi[1].d, alpha_j = wj[2].d;
            const double C_i = get_C(D, yi), C_j = get_C(D, yj);
            double ai = alpha_i, aj = alpha_j;
            pair_step(yi, yj, wi[2].d, wj[3].d, __uint_as_float(wj[4].x),
                      tr ? Gmax1 : (yi == +1 ? -Gmax0 : Gmax0), wj[1].d, C_i, C_j, ai, aj);
            const double dai = __dsub_rn(ai, alpha_i), daj = __dsub_rn(aj, alpha_j);
            const unsigned char new_si = status_of(ai, C_i), new_sj = status_of(aj, C_j);
            // the owners of i and j take their new alpha and status (a position is
            // read and written by its own thread only until the next barrier)
            auto take = [&](int p, double a, unsigned char st) {
                const int q = p - a0;
                if (q < 0 || q >= n || (q & (kThreads - 1)) != (int)threadIdx.x) return;
                ck.A[q] = a;
                ck.F[q] = (unsigned char)((ck.F[q] & ~(3u << kFlagStatus)) | ((unsigned)st << kFlagStatus));
            };
            take(i, ai, new_si);
            take(j, aj, new_sj);
            // G update (svm.cpp:732-735) + next I_up scan
#pragma unroll 1
            for (; k < n; k += kThreads) {
                const double qi = (double)qin, qj = (double)qjn;
                if (k + kThreads < n) {
                    qin = Qi[ck.Col[k + kThreads]];
                    qjn = Qj[ck.Col[k + kThreads]];
                }
                const double G = __dadd_rn(ck.G[k], __dadd_rn(__dmul_rn(qi, dai), __dmul_rn(qj, daj)));
                ck.G[k] = G;
                const unsigned f = ck.F[k];
                const bool pos = (f & kFlagPos) != 0;
                if (flag_s(f) != (pos ? ST_UPPER : ST_LOWER)) {
                    if (pos || !nu) better_max(v[0], ix[0], pos ? -G : G, a0 + k);
                    else better_max(v[1], ix[1], G, a0 + k);
                }
            }
            if (!D.lazy_gbar) {
                const unsigned char old_si = status_of(alpha_i, C_i), old_sj = status_of(alpha_j, C_j);
                const bool bar_i = (old_si == ST_UPPER) != (new_si == ST_UPPER), bar_j = (old_sj == ST_UPPER) != (new_sj == ST_UPPER);
                if (bar_i || bar_j) update_gbar(Qi, bar_i, old_si == ST_UPPER, C_i, Qj, bar_j, old_sj == ST_UPPER, C_j);
            }
        }
        __syncwarp();
        if ((ok = res_exchange_iup<nu>(ka, ok != 0, v, ix)) < 0) goto fail;
        mark(kProfBUpdate);
    }
    if (__syncthreads_or(!ok)) goto fail;
    fold();
    if (threadIdx.x == 0) sh.cnt[kCntLook] = (long long)kb * (nu ? 2 : 1) + iter;
    chunk_store();
    if (!exchange()) goto fail;
    if (iter >= D.max_iter) {
        status = 1;
        if (c.A < l) {
            if (!reconstruct<FORM>()) goto fail;
            set_active(l);
        }
    }
    finish_solve(nu, iter, status, unshrink);
    return;
fail:
    // Nobody waits for the records this block sent last: they land (well within
    // this pause) before it lets the others leave.
    __nanosleep(100000);
    fail_solve(iter, unshrink);
}

__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Every instance owns one cluster (nblocks blocks); clusters never wait for one
// another, so a launch may hold more of them than the GPU runs at a time.
template <int FORM>
__global__ void __launch_bounds__(kThreads, 1)
smo_cluster(const InstanceDesc *__restrict__ insts, const int *__restrict__ block_inst)
{
    Shared &sh = block_shared();
    ResRecords &R = res_records();
    const int inst = block_inst[blockIdx.x];
    for (int k = threadIdx.x; k < (int)(sizeof(InstanceDesc) / 4); k += blockDim.x)
        reinterpret_cast<int *>(&sh.D)[k] = reinterpret_cast<const int *>(&insts[inst])[k];
    if (threadIdx.x == 0) {
        tc::mbar_init(&R.bar_a, 1);
        tc::mbar_init(&R.bar_b, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int rank = blockIdx.x - sh.D.block0;
    if (threadIdx.x == 0 && sh.D.mute > 1 && rank == sh.D.nblocks - 1) sh.D.max_iter = sh.D.mute - 2;
    cluster_sync();     // no block sends before every block's mbarriers exist
    // (the tensor forms' values differ in the last bits with the operands swapped:
    // their matrices are whole)
    if constexpr (!is_tc_form(FORM)) {
        if (sh.D.resident == kResidentTri) {
            if (sh.D.nu) solve_resident<FORM, true, true>(rank);
            else solve_resident<FORM, false, true>(rank);
        }
    }
    if (sh.D.resident == kResidentFull) {
        if (sh.D.nu) solve_resident<FORM, true, false>(rank);
        else solve_resident<FORM, false, false>(rank);
    }
    signal_done(sh.D);
    __syncthreads();
    cluster_sync();     // no block leaves while another may still send to it
}

}  // namespace
}  // namespace svmb
