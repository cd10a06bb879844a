// Copies between pageable host arrays and the device for the host-pointer entry points.
//
// The driver moves a pageable array through a staging buffer of its own with one host thread: 8 - 12 GB/s, less where the
// destination's pages are touched for the first time, while PCIe carries 50. Here a few threads of the context move 64 KiB
// pieces between the caller's array and a ring of pinned slots, and the copy engine works on one slot while they fill (or
// empty) the next. Between jobs the threads spin for about 100 us -- the pieces are microseconds long -- and then sleep. A
// context owns its threads and its ring (8 MiB, made by the first large copy, given back with the context or asca_ctx_trim).
#include "common.cuh"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>

namespace {
constexpr size_t SLOT = (size_t)1 << 20, PIECE = (size_t)64 << 10;
constexpr int SLOTS = 8, MAX_WORKERS = 7;
static_assert(SLOT / PIECE < 65536, "pieces of a job are counted in 16 bits");
}  // namespace

struct asca_hostcopy {
    char* ring = nullptr;
    cudaEvent_t done[SLOTS] = {};
    bool used[SLOTS] = {};
    unsigned next = 0;
    // one job at a time: pieces are claimed by counter, the caller takes part and waits for the last
    std::vector<std::thread> workers;
    std::mutex mu;
    std::condition_variable cv;
    std::atomic<int> asleep{0};
    std::atomic<bool> quit{false};
    std::atomic<uint64_t> job{0};       // (job number << 32) | (pieces << 16) | pieces claimed
    std::atomic<uint32_t> finished{0};
    char* dst = nullptr;
    const char* src = nullptr;
    size_t bytes = 0;

    void piece(uint32_t i) {
        const size_t at = (size_t)i * PIECE, n = bytes - at < PIECE ? bytes - at : PIECE;
        memcpy(dst + at, src + at, n);
        finished.fetch_add(1, std::memory_order_acq_rel);
    }
    // claims pieces of the current job until none are left; the job number keeps a late thread off the next job's pieces
    void help(uint64_t number) {
        for (;;) {
            uint64_t j = job.load(std::memory_order_acquire);
            const uint32_t total = (uint32_t)j >> 16, at = (uint32_t)j & 0xffff;
            if ((j >> 32) != number || at >= total) return;
            if (job.compare_exchange_weak(j, j + 1, std::memory_order_acq_rel)) piece(at);
        }
    }
    void work() {
        uint64_t seen = 0;
        while (!quit.load(std::memory_order_acquire)) {
            const auto idle = std::chrono::steady_clock::now() + std::chrono::microseconds(100);
            uint64_t number;
            while ((number = job.load(std::memory_order_acquire) >> 32) == seen && std::chrono::steady_clock::now() < idle) {
#if defined(__x86_64__)
                __builtin_ia32_pause();
#endif
            }
            if (number == seen) {
                std::unique_lock<std::mutex> lk(mu);
                asleep.fetch_add(1);
                cv.wait(lk, [&] { return (job.load() >> 32) != seen || quit.load(); });
                asleep.fetch_sub(1);
                continue;
            }
            help(number);
            seen = number;
        }
    }
    void copy(void* d, const void* s, size_t n) {
        if (n <= PIECE || workers.empty()) {
            memcpy(d, s, n);
            return;
        }
        // (the previous job is complete, so no thread reads these fields; the job number publishes them)
        dst = (char*)d; src = (const char*)s; bytes = n;
        finished.store(0, std::memory_order_relaxed);
        const uint32_t total = (uint32_t)((n + PIECE - 1) / PIECE);
        const uint64_t number = (job.load(std::memory_order_relaxed) >> 32) + 1;
        job.store(number << 32 | (uint64_t)total << 16);
        if (asleep.load() > 0) {
            std::lock_guard<std::mutex> lk(mu);   // (a thread between its check and its wait holds it)
            cv.notify_all();
        }
        help(number);
        while (finished.load(std::memory_order_acquire) < total) {
#if defined(__x86_64__)
            __builtin_ia32_pause();
#endif
        }
    }
};

// What a caller's array is. The copies below touch a pageable array from the host, so anything else is told apart first: pinned
// memory goes to the copy engine as it is (at full speed), managed memory too, and a device address is refused.
enum class Mem { pageable, pinned, managed };
static int host_array(asca_ctx* ctx, const void* p, Mem* kind) {
    cudaPointerAttributes at;
    *kind = Mem::pageable;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return ASCA_OK;
    }
    ASCA_REQUIRE(ctx, at.type != cudaMemoryTypeDevice, "a host array is expected here, got a device address");
    if (at.type == cudaMemoryTypeHost) *kind = Mem::pinned;
    else if (at.type == cudaMemoryTypeManaged) *kind = Mem::managed;
    return ASCA_OK;
}

static asca_hostcopy* hostcopy(asca_ctx* ctx) {
    if (ctx->hostcopy) return ctx->hostcopy;
    asca_hostcopy* h = new asca_hostcopy();
    bool ok = cudaHostAlloc((void**)&h->ring, SLOT * SLOTS, cudaHostAllocDefault) == cudaSuccess;
    for (int i = 0; ok && i < SLOTS; ++i) ok = cudaEventCreateWithFlags(&h->done[i], cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        for (auto e : h->done)
            if (e) cudaEventDestroy(e);
        if (h->ring) cudaFreeHost(h->ring);
        delete h;
        return nullptr;
    }
    const unsigned cores = std::thread::hardware_concurrency();
    const int n = cores > 2 ? std::min<int>(MAX_WORKERS, (int)cores / 2 - 1) : 0;   // half the cores, the caller among them
    for (int i = 0; i < n; ++i) {
        try {
            h->workers.emplace_back([h] { h->work(); });
        } catch (...) {
            break;   // fewer threads, same copies
        }
    }
    ctx->hostcopy = h;
    return h;
}

void asca_hostcopy_free(asca_ctx* ctx) {
    asca_hostcopy* h = ctx->hostcopy;
    if (!h) return;
    {
        std::lock_guard<std::mutex> lk(h->mu);
        h->quit = true;
    }
    h->cv.notify_all();
    for (auto& t : h->workers) t.join();
    for (auto e : h->done) cudaEventDestroy(e);
    cudaFreeHost(h->ring);
    delete h;
    ctx->hostcopy = nullptr;
}

int asca_copy_in(asca_ctx* ctx, void* dst, const void* src, size_t bytes) {
    Mem kind;
    ASCA_TRY(host_array(ctx, src, &kind));
    if (bytes <= PIECE && kind != Mem::managed) return asca_stage_in(ctx, dst, src, bytes);
    asca_hostcopy* h = kind != Mem::pageable ? nullptr : hostcopy(ctx);
    if (!h) {
        ASCA_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream));
        return ASCA_OK;
    }
    for (size_t at = 0; at < bytes; at += SLOT) {
        const size_t n = std::min(SLOT, bytes - at);
        const unsigned s = h->next++ % SLOTS;
        if (h->used[s]) ASCA_CUDA(ctx, cudaEventSynchronize(h->done[s]));
        h->copy(h->ring + s * SLOT, (const char*)src + at, n);
        ASCA_CUDA(ctx, cudaMemcpyAsync((char*)dst + at, h->ring + s * SLOT, n, cudaMemcpyHostToDevice, ctx->stream));
        ASCA_CUDA(ctx, cudaEventRecord(h->done[s], ctx->stream));
        h->used[s] = true;
    }
    return ASCA_OK;
}

// Small arrays arrive with the asca_ctx_sync that ends the call, large ones before this returns.
int asca_copy_out(asca_ctx* ctx, void* dst, const void* src, size_t bytes) {
    Mem kind;
    ASCA_TRY(host_array(ctx, dst, &kind));
    if (bytes <= PIECE && kind != Mem::managed) return asca_stage_out(ctx, dst, src, bytes);
    asca_hostcopy* h = kind != Mem::pageable ? nullptr : hostcopy(ctx);
    if (!h) {
        ASCA_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
        return ASCA_OK;
    }
    const size_t slots = (bytes + SLOT - 1) / SLOT;
    const unsigned first = h->next;
    h->next += (unsigned)slots;
    auto request = [&](size_t i) -> int {
        const unsigned s = (first + (unsigned)i) % SLOTS;
        const size_t at = i * SLOT;
        ASCA_CUDA(ctx, cudaMemcpyAsync(h->ring + s * SLOT, (const char*)src + at, std::min(SLOT, bytes - at), cudaMemcpyDeviceToHost, ctx->stream));
        ASCA_CUDA(ctx, cudaEventRecord(h->done[s], ctx->stream));
        h->used[s] = true;
        return ASCA_OK;
    };
    // (earlier uploads read their slots in stream order before these copies write them)
    for (size_t i = 0; i < slots && i < SLOTS; ++i) ASCA_TRY(request(i));
    for (size_t i = 0; i < slots; ++i) {
        const unsigned s = (first + (unsigned)i) % SLOTS;
        const size_t at = i * SLOT;
        ASCA_CUDA(ctx, cudaEventSynchronize(h->done[s]));
        h->copy((char*)dst + at, h->ring + s * SLOT, std::min(SLOT, bytes - at));
        if (i + SLOTS < slots) ASCA_TRY(request(i + SLOTS));
    }
    return ASCA_OK;
}
