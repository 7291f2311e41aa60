// Context, device memory and state transfer helpers.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <system_error>
#include <thread>

#include "context.h"
#include "device_common.cuh"

namespace qb {

Context &ctx()
{
    static Context c;
    return c;
}

double wall_seconds()
{
    using namespace std::chrono;
    return duration<double>(system_clock::now().time_since_epoch()).count();
}

void *dev_alloc(size_t bytes)
{
    void *p = nullptr;
    if (bytes == 0) return nullptr;
    QB_CUDA(cudaMallocAsync(&p, bytes, ctx().stream));
    return p;
}

void *dev_try_alloc(size_t bytes)
{
    void *p = nullptr;
    const cudaError_t e = cudaMallocAsync(&p, bytes, ctx().stream);
    if (e == cudaErrorMemoryAllocation) {
        (void)cudaGetLastError();  // not sticky
        return nullptr;
    }
    QB_CUDA(e);
    return p;
}

void dev_free(void *p)
{
    if (p) cudaFreeAsync(p, ctx().stream);
}

namespace {

// One pinned slot.  The first slot's transfer and the last slot's host copy
// overlap nothing, so small slots shorten both ends; with 1 MB the copies' own
// cost shows.  ms for 191 MB device -> host / 32 MB device -> host / 1.5 GB
// host -> device, with 8 workers and 8 MB slots 6.2 / 1.9 / 41, 8 and 2 MB
// 5.4 / 1.2 / 36, 12 and 2 MB 4.9 / 1.2 / 35, 16 and 1 MB 4.8 / 1.3 / 43 (16
// host cores).  Four processes on that host at once copy 2 x 15 MiB up in
// 2.7-3.3 ms with 12 workers each, 1.2-2.5 with 8.
constexpr size_t kStageBytes = 2u << 20;
constexpr unsigned kStageWorkers = 12;
// The smallest copies that go through the slots: starting and joining the
// workers takes 0.15 ms.  ms of two copies in one call / through the slots.
// Up, from arrays that are not in the host's caches: 3 MiB 0.68 / 0.59-0.76,
// 4.5 MiB 0.95 / 0.65, 7.5 MiB 1.50 / 0.90, 12 MiB 2.37 / 1.22 (the same array
// again: 0.41 / 0.54, 0.55 / 0.62, 0.85 / 0.82, 1.32 / 1.07).  Down: 4.5 MiB
// 0.65 / 0.68, 7.5 MiB 0.88-1.03 / 0.90-0.98, 9 MiB 1.12-1.21 / 0.97-1.03, 12 MiB
// 1.57 / 1.15.  The first staged copy after QPHIX_init also makes the slots
// and streams, 45-100 ms.
constexpr size_t kStageMinUp = 4u << 20, kStageMinDown = 8u << 20;

void make_staging(Context &c)
{
    HostStaging &h = c.staging;
    if (h.workers) return;
    const unsigned hw = std::thread::hardware_concurrency();
    const int w = (int)std::max(1u, std::min(kStageWorkers, hw * 3 / 4));
    for (int i = 0; i < w; ++i) {
        cudaStream_t s;
        QB_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        h.streams.push_back(s);
        for (int k = 0; k < 2; ++k) {
            void *p = nullptr;
            QB_CUDA(cudaHostAlloc(&p, kStageBytes, cudaHostAllocDefault));
            h.slots.push_back(static_cast<char *>(p));
            cudaEvent_t e;
            QB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
            h.done.push_back(e);
        }
        h.workers = i + 1;
    }
}

// f(0) .. f(n - 1), each in a thread of its own; where the system refuses a
// thread, the caller does what is left.
template <typename F>
void run_workers(int n, F f)
{
    std::vector<std::thread> th;
    th.reserve(n);
    try {
        for (int w = 0; w < n; ++w) th.emplace_back(f, w);
    } catch (const std::system_error &) {
    }
    for (int w = (int)th.size(); w < n; ++w) f(w);
    for (auto &t : th) t.join();
}

}  // namespace

void free_staging()
{
    HostStaging &h = ctx().staging;
    for (auto s : h.streams) cudaStreamDestroy(s);
    for (auto p : h.slots) cudaFreeHost(p);
    for (auto e : h.done) cudaEventDestroy(e);
    h = HostStaging{};
}

void h2d_copy(void *dst, const void *src, size_t bytes)
{
    Context &c = ctx();
    if (bytes == 0) return;
    // only plain pageable host memory is staged; pinned, managed or device
    // memory goes by one copy (direction from the unified address space)
    cudaPointerAttributes at{};
    const bool pageable = cudaPointerGetAttributes(&at, src) != cudaSuccess || at.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();  // an unregistered pointer is not an error here
    if (!pageable || bytes < kStageMinUp) {
        QB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, c.stream));
        QB_CUDA(cudaStreamSynchronize(c.stream));
        return;
    }
    make_staging(c);
    // work already queued on the library stream (e.g. a memset of dst)
    // finishes before the worker streams write dst
    QB_CUDA(cudaStreamSynchronize(c.stream));
    HostStaging &h = c.staging;
    const int W = h.workers;
    std::atomic<int> failed{0};
    run_workers(W, [&](int w) {
        if (cudaSetDevice(c.device) != cudaSuccess) { failed = 1; return; }
        // contiguous part of the source, 4 KiB aligned
        const size_t lo = (bytes * w / W) & ~(size_t)4095, hi = w + 1 == W ? bytes : (bytes * (w + 1) / W) & ~(size_t)4095;
        int k = 0;
        for (size_t off = lo; off < hi; off += kStageBytes, ++k) {
            const size_t n = std::min(kStageBytes, hi - off);
            const int sl = 2 * w + (k & 1);
            if (k >= 2 && cudaEventSynchronize(h.done[sl]) != cudaSuccess) { failed = 1; break; }
            std::memcpy(h.slots[sl], static_cast<const char *>(src) + off, n);
            if (cudaMemcpyAsync(static_cast<char *>(dst) + off, h.slots[sl], n, cudaMemcpyHostToDevice,
                                h.streams[w]) != cudaSuccess ||
                cudaEventRecord(h.done[sl], h.streams[w]) != cudaSuccess) {
                failed = 1;
                break;
            }
        }
        if (cudaStreamSynchronize(h.streams[w]) != cudaSuccess) failed = 1;
    });
    if (failed) throw Error("host to device copy through pinned staging failed");
}

void d2h_copy(void *dst, const void *src, size_t bytes)
{
    Context &c = ctx();
    if (bytes == 0) return;
    cudaPointerAttributes at{};
    const bool pageable = cudaPointerGetAttributes(&at, dst) != cudaSuccess || at.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();  // an unregistered pointer is not an error here
    if (!pageable || bytes < kStageMinDown) {
        QB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, c.stream));
        QB_CUDA(cudaStreamSynchronize(c.stream));
        return;
    }
    make_staging(c);
    // the kernels that produce src finish before the worker streams read it
    QB_CUDA(cudaStreamSynchronize(c.stream));
    HostStaging &h = c.staging;
    const int W = h.workers;
    std::atomic<int> failed{0};
    run_workers(W, [&](int w) {
        if (cudaSetDevice(c.device) != cudaSuccess) { failed = 1; return; }
        const size_t lo = (bytes * w / W) & ~(size_t)4095, hi = w + 1 == W ? bytes : (bytes * (w + 1) / W) & ~(size_t)4095;
        // chunk k goes device -> slot k&1 while the host copies chunk k-1 out of the other slot
        size_t prev_off = 0, prev_n = 0;
        int k = 0;
        auto drain = [&](int slot) {
            if (cudaEventSynchronize(h.done[slot]) != cudaSuccess) { failed = 1; return false; }
            std::memcpy(static_cast<char *>(dst) + prev_off, h.slots[slot], prev_n);
            return true;
        };
        for (size_t off = lo; off < hi; off += kStageBytes, ++k) {
            const size_t n = std::min(kStageBytes, hi - off);
            const int sl = 2 * w + (k & 1);
            if (cudaMemcpyAsync(h.slots[sl], static_cast<const char *>(src) + off, n, cudaMemcpyDeviceToHost,
                                h.streams[w]) != cudaSuccess ||
                cudaEventRecord(h.done[sl], h.streams[w]) != cudaSuccess) {
                failed = 1;
                break;
            }
            if (k > 0 && !drain(2 * w + ((k - 1) & 1))) break;
            prev_off = off;
            prev_n = n;
        }
        if (!failed && k > 0) drain(2 * w + ((k - 1) & 1));
        if (cudaStreamSynchronize(h.streams[w]) != cudaSuccess) failed = 1;
    });
    if (failed) throw Error("device to host copy through pinned staging failed");
}

void check_lattice(const int L[4], const char *who)
{
    const std::string w(who);
    for (int i = 0; i < 4; ++i)
        if (L[i] <= 0) throw Error(w + ": non-positive lattice extent");
    if (L[0] % 2) throw Error(w + ": Nx must be even");
    if ((L[0] / 2) % 2 != 0) throw Error(w + ": Nx/2 must be even");
    if (L[1] % 4 || L[2] % 4 || L[3] % 4) throw Error(w + ": Ny, Nz and Nt must be multiples of 4");
    const long long V = (long long)L[0] * L[1] * L[2] * L[3];
    if (V / 2 > (1LL << 30)) throw Error(w + ": lattice too large for 32-bit site indices");
    if (2LL * ((V / 2 + kBlock - 1) / kBlock) > 4LL * kMaxPartials)
        throw Error(w + ": lattice too large for one GPU's reduction scratch");
}

static size_t cx_bytes(Prec p) { return p == Prec::Double ? 16 : (p == Prec::Single ? 8 : 4); }

VecBlock alloc_vec(Prec p)
{
    Context &c = ctx();
    VecBlock b;
    b.data = dev_alloc(vec_bytes(p, c.g.vh));
    QB_CUDA(cudaMemsetAsync(b.data, 0, vec_bytes(p, c.g.vh), c.stream));
    return b;
}

void free_vec(VecBlock &b)
{
    dev_free(b.data);
    b.data = nullptr;
}

LinkSet alloc_links(Prec p) { return alloc_links(p, ctx().g.vh); }

LinkSet alloc_links(Prec p, int vh)
{
    Context &c = ctx();
    LinkSet ls;
    const size_t bytes = (size_t)kMats * 9 * vh * cx_bytes(p);
    for (int cb = 0; cb < 2; ++cb) {
        ls.blk[cb] = dev_alloc(bytes);
        QB_CUDA(cudaMemsetAsync(ls.blk[cb], 0, bytes, c.stream));
    }
    ls.prec = p;
    ls.valid = true;
    return ls;
}

void free_links(LinkSet &ls)
{
    for (int cb = 0; cb < 2; ++cb) {
        dev_free(ls.blk[cb]);
        dev_free(ls.sign[cb]);
        dev_free(ls.lam[cb]);
        ls.blk[cb] = nullptr;
        ls.sign[cb] = nullptr;
        ls.lam[cb] = nullptr;
    }
    ls.valid = false;
    ls.mirrored = -1;
    ls.recon = 0;
}

void upload_state()
{
    Context &c = ctx();
    QB_CUDA(cudaMemcpyAsync(c.d_state, c.h_state, sizeof(SolverState), cudaMemcpyHostToDevice, c.stream));
    // the pinned mirror is edited again right after; let the copy land first
    QB_CUDA(cudaStreamSynchronize(c.stream));
}

void download_state()
{
    Context &c = ctx();
    QB_CUDA(cudaMemcpyAsync(c.h_state, c.d_state, sizeof(SolverState), cudaMemcpyDeviceToHost, c.stream));
    sync_check();
}

void sync_check()
{
    Context &c = ctx();
    QB_CUDA(cudaStreamSynchronize(c.stream));
    // only kernels with bounded waits write the failure word
    if (!c.d_err || !c.err_armed) return;
    c.err_armed = false;
    int e = 0;
    QB_CUDA(cudaMemcpy(&e, c.d_err, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) {
        QB_CUDA(cudaMemsetAsync(c.d_err, 0, sizeof(int), c.stream));
        throw Error(std::string(e == kErrLoopWait ? "a grid barrier of the solver loop" : "a Dslash pipeline wait") +
                    " timed out on the GPU; the call's results are invalid");
    }
}

}  // namespace qb
