// The driver copies pageable memory through one thread, at 11 GB/s each way on a
// B200 host, and a fresh array's first touch falls to the same thread (382 MB
// down into a new array: 82 ms), where the link moves 55 GB/s.  Here each of up
// to eight threads moves every eighth 1 MB piece through two pinned buffers of
// its own, so that pieces are copied (and touched) in parallel and beside the
// transfers of others.  Small copies (split_bytes), copies of memory that is
// already pinned, and copies while another thread has the buffers go the plain way.
// Upload / download / download into a new array on a 16-core host: 382 MB 34.6 /
// 19.8 / 82 ms plain, 8.8 / 10.1 / 19.4 so; 24 MB 1.25 / 1.26 / 1.23 and 0.85 / 0.76 / 0.78.
#include "hostcopy.cuh"

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>

#include <sched.h>
#include <sys/mman.h>
#include <unistd.h>

namespace glac {

namespace {

constexpr size_t kPiece = (size_t)1 << 20;
constexpr int kThreads = 8, kSlots = 2;
constexpr size_t kLeastSplit = (size_t)10 << 20;  // see split_bytes
constexpr size_t kPinnedBytes = kThreads * kSlots * kPiece, kHugePage = (size_t)2 << 20;
// The buffers cost 1.8 ms, 3.6 the first time, to make and give back (16 MB of huge
// pages; 10 ms by cudaHostAlloc).  A copy of 64 MB saves that by itself (up
// 4.0 -> 1.7 ms, down 3.0 -> 1.8); smaller ones get the buffers once 256 MB, 13 ms
// of plain copies, have gone without.  A context made for one
// configuration of 24 MB, loaded, read and closed does without: 6 ms, 26 where
// buffers are made for its copies; one of 75 MB takes 11 ms, 14 by plain copies.
constexpr size_t kPinBytes = (size_t)64 << 20, kPinAfter = (size_t)256 << 20;

std::mutex g_hold_mu;   // g_holders and the buffers' lifetime
int g_holders = 0;
std::mutex g_use_mu;    // one transfer at a time
void *g_mapped = nullptr;  // the buffers' mapping
pid_t g_owner = 0;         // the process that made it
char *g_pinned = nullptr;  // the buffers: kThreads x kSlots pieces
size_t g_plain = 0;     // bytes that went the plain way for want of the buffers

// Cores this process may run on.
int usable_cores() {
    cpu_set_t set;
    if (sched_getaffinity(0, sizeof(set), &set) == 0) return CPU_COUNT(&set);
    return (int)std::thread::hardware_concurrency();
}
// The size from which a copy is split: 10 MB on four cores or more, below which
// starting the threads costs what they save; 16 MB on three; on two, where they only
// share the copying that one thread does, 128 MB; on one never.  Microseconds plain /
// split, up and then down, on a B200 host: 16 cores 8 MB 415 / 419, 406 / 394, 10 MB
// 517 / 475, 510 / 448, 16 MB 829 / 670, 830 / 648; 4 cores 8 MB 425 / 523, 425 / 419,
// 12 MB 620 / 579, 625 / 518; 3 cores 10 MB 510 / 554, 507 / 540, 16 MB 809 / 753, 781 /
// 793; 2 cores 24 MB 1204 / 1343, 1159 / 1303, 96 MB 8304 / 5648, 4548 / 5224, 192 MB
// 16627 / 11339, 9132 / 9577; 1 core 192 MB 17053 / 16090, 9774 / 16528.
size_t split_bytes() {
    const int cores = usable_cores();
    return cores >= 4 ? kLeastSplit : cores == 3 ? (size_t)16 << 20 : cores == 2 ? (size_t)128 << 20 : SIZE_MAX;
}

bool pageable(const void *host) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// Piece `c` of the copy by thread k's slot; `to_device` picks the direction.
cudaError_t worker(int k, int threads, char *dev, char *host, size_t bytes, int device, cudaStream_t st,
                   bool to_device, std::atomic<int> *failed) {
    cudaError_t e = cudaSetDevice(device);
    cudaEvent_t ev[kSlots] = {nullptr, nullptr};
    for (int i = 0; i < kSlots && e == cudaSuccess; i++) e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
    const size_t pieces = (bytes + kPiece - 1) / kPiece;
    auto size = [&](size_t c) { return std::min(kPiece, bytes - c * kPiece); };
    auto slot = [&](int i) { return g_pinned + ((size_t)k * kSlots + i) * kPiece; };
    // pending[i]: the piece whose transfer uses slot i
    size_t pending[kSlots];
    bool busy[kSlots] = {false, false};
    auto finish = [&](int i) {
        if (!busy[i]) return;
        const cudaError_t w = cudaEventSynchronize(ev[i]);
        if (e == cudaSuccess) e = w;
        if (!to_device && e == cudaSuccess) memcpy(host + pending[i] * kPiece, slot(i), size(pending[i]));
        busy[i] = false;
    };
    int i = 0;
    for (size_t c = k; c < pieces && e == cudaSuccess && !failed->load(); c += threads, i ^= 1) {
        finish(i);
        if (e != cudaSuccess) break;
        if (to_device) memcpy(slot(i), host + c * kPiece, size(c));
        e = to_device ? cudaMemcpyAsync(dev + c * kPiece, slot(i), size(c), cudaMemcpyHostToDevice, st)
                      : cudaMemcpyAsync(slot(i), dev + c * kPiece, size(c), cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess) break;
        pending[i] = c;
        busy[i] = true;
        const cudaError_t r = cudaEventRecord(ev[i], st);
        if (r != cudaSuccess) {
            cudaStreamSynchronize(st);  // the slot is not left while a transfer may use it
            e = r;
        }
    }
    finish(i);
    finish(i ^ 1);
    for (cudaEvent_t v : ev)
        if (v) cudaEventDestroy(v);
    if (e != cudaSuccess) failed->store(1);
    return e;
}

cudaError_t split_copy(char *dev, char *host, size_t bytes, int device, cudaStream_t st, bool to_device) {
    const int threads = (int)std::min<size_t>(kThreads, (bytes + kPiece - 1) / kPiece);
    std::atomic<int> failed{0};
    cudaError_t err[kThreads];
    std::thread pool[kThreads];
    int made = 1;
    // threads that cannot be started, for want of a thread or of memory, leave their
    // pieces to fewer: the count is fixed only once they all run
    std::atomic<int> count{0};
    auto run = [&](int k) {
        int n;
        while ((n = count.load()) == 0) std::this_thread::yield();
        err[k] = k < n ? worker(k, n, dev, host, bytes, device, st, to_device, &failed) : cudaSuccess;
    };
    try {
        for (; made < threads; made++) pool[made] = std::thread(run, made);
    } catch (...) {
    }
    count.store(made);
    run(0);
    cudaError_t e = err[0];
    for (int k = 1; k < made; k++) {
        pool[k].join();
        if (e == cudaSuccess) e = err[k];
    }
    return e;
}

// The buffers: whole huge pages where the system gives them, which are quick to
// pin.  A forked child gets none of them (their pages must not become copies of
// what the driver has pinned) and leaves what may lie at their place alone.
void unpin_buffers() {
    if (g_owner == getpid()) {
        if (g_pinned) cudaHostUnregister(g_pinned);
        if (g_mapped) munmap(g_mapped, kPinnedBytes + kHugePage);
    }
    g_pinned = nullptr;
    g_mapped = nullptr;
}
void pin_buffers() {
    void *m = mmap(nullptr, kPinnedBytes + kHugePage, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (m == MAP_FAILED) return;
    g_mapped = m;
    g_owner = getpid();
    char *p = reinterpret_cast<char *>(((uintptr_t)m + kHugePage - 1) / kHugePage * kHugePage);
    madvise(m, kPinnedBytes + kHugePage, MADV_DONTFORK);
    madvise(p, kPinnedBytes, MADV_HUGEPAGE);
    for (size_t i = 0; i < kPinnedBytes; i += kHugePage) reinterpret_cast<volatile char *>(p)[i] = 0;
    if (cudaHostRegister(p, kPinnedBytes, cudaHostRegisterPortable) == cudaSuccess) {
        g_pinned = p;
        return;
    }
    cudaGetLastError();
    unpin_buffers();
}

// Whether a copy goes through the buffers, which are made for it if it pays alone
// or if enough has gone the plain way without them.
bool take_buffers(size_t bytes) {
    if (!g_pinned) {
        g_plain += bytes;
        if (bytes < kPinBytes && g_plain < kPinAfter) return false;
        g_plain = 0;
        pin_buffers();
    }
    return g_pinned != nullptr;
}

cudaError_t copy(char *dev, char *host, size_t bytes, int device, cudaStream_t st, bool to_device) {
    if (bytes >= kLeastSplit && bytes >= split_bytes() && pageable(host)) {
        std::unique_lock<std::mutex> use(g_use_mu, std::try_to_lock);
        if (use.owns_lock() && take_buffers(bytes)) return split_copy(dev, host, bytes, device, st, to_device);
    }
    if (to_device) return cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
    const cudaError_t e = cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st);
    return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
}

}  // namespace

cudaError_t copy_to_device(void *dev, const void *host, size_t bytes, int device, cudaStream_t st) {
    return copy(static_cast<char *>(dev), static_cast<char *>(const_cast<void *>(host)), bytes, device, st, true);
}
cudaError_t copy_to_host(void *host, const void *dev, size_t bytes, int device, cudaStream_t st) {
    return copy(static_cast<char *>(const_cast<void *>(dev)), static_cast<char *>(host), bytes, device, st, false);
}

void hostcopy_hold() {
    std::lock_guard<std::mutex> lock(g_hold_mu);
    g_holders++;
}
void hostcopy_drop() {
    std::lock_guard<std::mutex> lock(g_hold_mu);
    if (--g_holders > 0) return;
    std::lock_guard<std::mutex> use(g_use_mu);
    unpin_buffers();
    g_plain = 0;
}

}  // namespace glac
