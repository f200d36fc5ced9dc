// transfer.cu -- copies between the device and a caller's pageable memory.
//
// A plain copy from or to pageable memory is staged by the driver on one
// host thread; taking a result into fresh memory also faults its pages in
// one by one.  Large copies therefore go through pinned chunks with several
// host threads: each thread takes the next chunk, moves
// it over the bus and copies it between its pinned buffer and its own part
// of the caller's memory.  Measured on a host with 16 cores: five 33 MB
// snapshots into fresh memory 76 ms plainly (with one more host copy each),
// a 85 MB field 17 ms.  Small copies and pinned memory take the plain path, and
// so does a copy that gets no chunk: none can be pinned, or all are in use.
#include <atomic>
#include <mutex>
#include <system_error>
#include <thread>

#include "runtime_internal.h"

namespace prt {

namespace {

// The largest part of a copy one thread has in hand, and the size from which
// a copy is worth the threads (they cost about 0.2 ms together).
constexpr size_t kChunk = size_t(1) << 20;
constexpr size_t kStagedFrom = size_t(4) << 20;
// Copies of a device that run on chunks at a time: 32 MiB of pinned memory, and
// 32 host threads.
constexpr int kSets = 4;

// The sets of chunks of a device; a copy has one to itself while it runs.  A
// set given back may still be the source of a copy in flight on its last
// user's stream; its chunks' events say when (work).
struct DeviceSets {
    Transfer set[kSets];
    bool lent[kSets] = {};
    int contexts = 0;
};
std::mutex sets_mu;
constexpr int kDevices = 64;  // a device beyond has none
DeviceSets sets_of[kDevices];

Transfer* take_set(int device) {
    if (device >= kDevices) return nullptr;
    std::lock_guard<std::mutex> lk(sets_mu);
    DeviceSets& d = sets_of[device];
    for (int i = 0; i < kSets; ++i)
        if (!d.lent[i]) {
            d.lent[i] = true;
            return &d.set[i];
        }
    return nullptr;
}

void give_set(int device, Transfer* t) {
    std::lock_guard<std::mutex> lk(sets_mu);
    DeviceSets& d = sets_of[device];
    d.lent[t - d.set] = false;
}

bool pageable(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// One thread's share: chunks in turn until none is left or one has failed.
void work(const prt_ctx* ctx, Transfer* t, int w, char* host, char* dev, size_t bytes, bool out,
          std::atomic<size_t>* next, std::atomic<int>* error) noexcept {
    cudaStream_t s = ctx->stream;
    cudaError_t e = cudaSetDevice(ctx->device);
    while (e == cudaSuccess && error->load() == 0) {
        const size_t at = next->fetch_add(kChunk);
        if (at >= bytes) return;
        const size_t len = std::min(kChunk, bytes - at);
        // the buffer's last copy, of this call or an earlier one, is done
        e = cudaEventSynchronize(t->ev[w]);
        if (e != cudaSuccess) break;
        if (out) {
            e = cudaMemcpyAsync(t->pin[w], dev + at, len, cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaEventRecord(t->ev[w], s);
            if (e == cudaSuccess) e = cudaEventSynchronize(t->ev[w]);
            if (e == cudaSuccess) memcpy(host + at, t->pin[w], len);
        } else {
            memcpy(t->pin[w], host + at, len);
            e = cudaMemcpyAsync(dev + at, t->pin[w], len, cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess) e = cudaEventRecord(t->ev[w], s);
        }
    }
    if (e != cudaSuccess) error->store((int)e);
}

// Whether the copy ran on pinned chunks, with its error in *e.
bool staged(prt_ctx* ctx, char* host, char* dev, size_t bytes, bool out, cudaError_t* e) {
    if (bytes < kStagedFrom || !pageable(host)) return false;
    Transfer* t = take_set(ctx->device);
    if (!t) return false;
    const unsigned cores = std::thread::hardware_concurrency();
    const int want = t->ensure(
        (int)std::min<size_t>({(size_t)Transfer::kWorkers, (size_t)std::max(1u, cores / 2),
                               (bytes + kChunk - 1) / kChunk}),
        kChunk);
    std::atomic<size_t> next{0};
    std::atomic<int> error{0};
    std::thread th[Transfer::kWorkers];
    for (int w = 1; w < want; ++w) {
        try {
            th[w] = std::thread(work, ctx, t, w, host, dev, bytes, out, &next, &error);
        } catch (const std::system_error&) {
            break;  // no thread to be had: the others take its chunks
        }
    }
    if (want) work(ctx, t, 0, host, dev, bytes, out, &next, &error);
    for (int w = 1; w < want; ++w)
        if (th[w].joinable()) th[w].join();
    give_set(ctx->device, t);
    *e = (cudaError_t)error.load();
    return want > 0;
}

}  // namespace

int Transfer::ensure(int workers, size_t chunk) {
    for (; n < workers; ++n) {
        if (cudaHostAlloc(&pin[n], chunk, cudaHostAllocDefault) != cudaSuccess) break;
        if (cudaEventCreateWithFlags(&ev[n], cudaEventDisableTiming) != cudaSuccess) {
            cudaFreeHost(pin[n]);
            break;
        }
    }
    if (n < workers) cudaGetLastError();  // the copy goes another way
    return std::min(n, workers);
}

void Transfer::release() {
    for (; n > 0; --n) {
        cudaEventDestroy(ev[n - 1]);
        cudaFreeHost(pin[n - 1]);
    }
}

void transfer_open(int device) {
    if (device >= kDevices) return;
    std::lock_guard<std::mutex> lk(sets_mu);
    sets_of[device].contexts += 1;
}

void transfer_close(int device) {
    if (device >= kDevices) return;
    std::lock_guard<std::mutex> lk(sets_mu);
    DeviceSets& d = sets_of[device];
    if (--d.contexts > 0) return;
    for (Transfer& t : d.set) t.release();
}

cudaError_t copy_out(prt_ctx* ctx, void* host, const void* dev, size_t bytes) {
    cudaError_t e = cudaSuccess;
    if (staged(ctx, static_cast<char*>(host), const_cast<char*>(static_cast<const char*>(dev)), bytes,
               true, &e))
        return e;
    e = cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, ctx->stream);
    return e == cudaSuccess ? cudaStreamSynchronize(ctx->stream) : e;
}

cudaError_t copy_in(prt_ctx* ctx, void* dev, const void* host, size_t bytes) {
    cudaError_t e = cudaSuccess;
    if (staged(ctx, const_cast<char*>(static_cast<const char*>(host)), static_cast<char*>(dev), bytes,
               false, &e))
        return e;
    return cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, ctx->stream);
}

}  // namespace prt
