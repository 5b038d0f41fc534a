// A stand-in for the CUDA runtime and the kernel launchers, so that the host
// side of the engine (plans, the request loop, its bookkeeping) runs without a
// GPU.  Device memory is host memory, a stream is a thread that works off its
// queue, and a "solve" lasts 1 us per row (fake_us_per_row) and returns the
// iteration count l and alpha = 1 for every variable.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

#include "engine.hpp"
#include "predict.hpp"

namespace {

struct Stream {
    std::mutex mu;
    std::condition_variable cv, idle;
    std::deque<std::function<void()>> queue;
    bool busy = false, stop = false;
    std::atomic<int> solving{0};        // launches of the solver queued or at work
    std::thread worker;
    Stream()
    {
        worker = std::thread([this] {
            std::unique_lock<std::mutex> lk(mu);
            while (true) {
                cv.wait(lk, [&] { return stop || !queue.empty(); });
                if (queue.empty()) return;
                auto f = std::move(queue.front());
                queue.pop_front();
                busy = true;
                lk.unlock();
                f();
                lk.lock();
                busy = false;
                if (queue.empty()) idle.notify_all();
            }
        });
    }
    void push(std::function<void()> f)
    {
        std::lock_guard<std::mutex> g(mu);
        queue.push_back(std::move(f));
        cv.notify_one();
    }
    void sync()
    {
        std::unique_lock<std::mutex> lk(mu);
        idle.wait(lk, [&] { return queue.empty() && !busy; });
    }
    ~Stream()
    {
        {
            std::lock_guard<std::mutex> g(mu);
            stop = true;
            cv.notify_one();
        }
        worker.join();
    }
};
struct Event {
    std::mutex mu;
    std::condition_variable cv;
    int pending = 0;
};
Stream &stream(cudaStream_t s)
{
    static Stream *def = new Stream();
    return s ? *(Stream *)s : *def;
}
cudaError_t got(void **p, size_t n)
{
    *p = malloc(n);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}

std::atomic<int> blocks_now{0}, blocks_peak{0}, cluster_launches{0}, general_launches{0};
std::atomic<long long> us_per_row{1}, h2d_bytes{0};
std::atomic<int> waits{0};           // calls that wait for the device
std::atomic<int> frees_behind{0};    // memory given back behind a launch at work: who gets it waits for that launch


void solve(const svmb::InstanceDesc *insts, const int *map, int blocks)
{
    const int now = blocks_now += blocks;
    int peak = blocks_peak;
    while (now > peak && !blocks_peak.compare_exchange_weak(peak, now)) {}
    // the instances run side by side: in the order of their lengths
    std::vector<int> order;
    for (int b = 0; b < blocks; b++)
        if (order.empty() || order.back() != map[b]) order.push_back(map[b]);
    std::sort(order.begin(), order.end(), [&](int a, int b) { return insts[a].l < insts[b].l; });
    long long at = 0;
    for (int k : order) {
        const svmb::InstanceDesc D = insts[k];
        const long long end = D.l * us_per_row;
        std::this_thread::sleep_for(std::chrono::microseconds(end - at));
        at = end;
        svmb::SolveOut o{};
        o.iters = D.l;
        *D.out = o;
        for (int p = 0; p < D.l; p++) D.alpha_local[p] = 1.0;
        blocks_now -= D.nblocks;
        if (D.done_flag) __atomic_store_n(D.done_flag, 1, __ATOMIC_RELEASE);
    }
}
cudaError_t launch(const svmb::InstanceDesc *insts, const int *map, int blocks, cudaStream_t s)
{
    Stream *const st = &stream(s);
    st->solving++;
    st->push([=] {
        solve(insts, map, blocks);
        st->solving--;
    });
    return cudaSuccess;
}
cudaError_t nothing() { return cudaSuccess; }

}  // namespace

extern "C" {
int fake_peak_blocks() { return blocks_peak.exchange(0); }
int fake_cluster_launches() { return cluster_launches.exchange(0); }
int fake_general_launches() { return general_launches.exchange(0); }
long long fake_h2d_bytes() { return h2d_bytes.exchange(0); }
int fake_frees_behind_a_launch() { return frees_behind.exchange(0); }
int fake_waits() { return waits.exchange(0); }
void fake_us_per_row(long long us) { us_per_row = us; }

int omp_get_max_threads() { return 1; }

cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : a == cudaDevAttrMaxSharedMemoryPerMultiprocessor ? 233472 : 148;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return waits++, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int)
{
    memset(p, 0, sizeof *p);
    p->multiProcessorCount = 148;
    p->major = 10;
    return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = (cudaEvent_t) new Event, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventSynchronize(cudaEvent_t ev)
{
    Event *e = (Event *)ev;
    std::unique_lock<std::mutex> lk(e->mu);
    e->cv.wait(lk, [&] { return e->pending == 0; });
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    cudaEventSynchronize(e);
    delete (Event *)e;
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1, cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t ev)
{
    Event *e = (Event *)ev;
    std::lock_guard<std::mutex> g(e->mu);
    return e->pending ? cudaErrorNotReady : cudaSuccess;
}
cudaError_t cudaEventRecordWithFlags(cudaEvent_t ev, cudaStream_t s, unsigned)
{
    Event *e = (Event *)ev;
    {
        std::lock_guard<std::mutex> g(e->mu);
        e->pending++;
    }
    stream(s).push([e] {
        std::lock_guard<std::mutex> g(e->mu);
        e->pending--;
        e->cv.notify_all();
    });
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { return waits++, got(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return got(p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return got(p, n); }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { return *d = h, cudaSuccess; }
cudaError_t cudaFree(void *p)
{
    if (p) waits++;
    return free(p), cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { return waits++, free(p), cudaSuccess; }
cudaError_t cudaFreeAsync(void *p, cudaStream_t s)
{
    if (!p) return cudaErrorInvalidValue;
    if (stream(s).solving) frees_behind++;
    return stream(s).push([p] { free(p); }), cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { return *f = *t = size_t(64) << 30, cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { return waits++, memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind kind, cudaStream_t st)
{
    if (kind == cudaMemcpyHostToDevice) h2d_bytes += (long long)n;
    return stream(st).push([=] { memcpy(d, s, n); }), cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t s) { return stream(s).push([=] { memset(d, v, n); }), cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return *s = (cudaStream_t) new Stream, cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return waits++, stream(s).sync(), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s)
{
    ((Stream *)s)->sync();
    delete (Stream *)s;
    return cudaSuccess;
}
// no graphs: the engine then issues the stream work directly
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}

namespace svmb {
int smo_static_smem() { return 8192; }
size_t smo_cluster_smem(int) { return 214000; }
cudaError_t smo_max_clusters(int, int c, size_t, int *n) { return *n = 148 / c, cudaSuccess; }
cudaError_t smo_max_blocks(int, size_t, int *n) { return *n = 1, cudaSuccess; }
cudaError_t load_solver_kernels(int) { return nothing(); }
int q_tiles(int l) { return (l + 63) / 64 * ((l + 63) / 64 + 1) / 2; }
cudaError_t launch_q_dense(int, const InstanceDesc *, const int *, int, int, cudaStream_t) { return nothing(); }
cudaError_t launch_q_sparse(int, const InstanceDesc *, const int *, int, int, size_t, cudaStream_t) { return nothing(); }
cudaError_t launch_q_tensor(int, const InstanceDesc *, int, cudaStream_t) { return nothing(); }
cudaError_t launch_xsq(const DevX &, int, double *, int, cudaStream_t) { return nothing(); }
cudaError_t launch_split(const DeviceRows &, int, int, uint16_t *, double *, cudaStream_t) { return nothing(); }
cudaError_t launch_scatter_dense(const long long *, const int *, const float *, int, int, float *, cudaStream_t) { return nothing(); }
cudaError_t launch_kernel_block(const DeviceRows &, const KernelParams &, int, const int *, int, const int *, int, double *,
                                long long, int *, cudaStream_t) { return nothing(); }
cudaError_t launch_smo(int, const InstanceDesc *d, const int *map, int n, size_t, bool, cudaStream_t s)
{
    general_launches++;
    return launch(d, map, n, s);
}
cudaError_t launch_smo_cluster(int, const InstanceDesc *d, const int *map, int n, int, size_t, cudaStream_t s)
{
    cluster_launches++;
    return launch(d, map, n, s);
}
int predict_batch(const svm_model *, const svm_node *const *, int, double *, double *) { return -1; }
void predict_forget(const svm_model *) {}
int predict_set_form(int) { return 0; }
}  // namespace svmb
