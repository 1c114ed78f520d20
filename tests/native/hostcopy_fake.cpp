// The host side of the field copies (hostcopy.cu) on a fake CUDA runtime whose
// copies are memcpy.  argv: hardware threads, then one step after another:
//   up N | down N    a copy of N bytes, checked; prints the number of transfers it took
//   fail             from here on a thread's state finds no memory
//   hold | drop      a holder comes or goes; drop prints the bytes pinned after it
//   pinned           prints the bytes pinned now and how often memory was pinned
#include "hostcopy.cu"

#include <cstdio>
#include <cstdlib>
#include <map>
#include <new>
#include <string>
#include <vector>

static std::atomic<int> g_copies{0};
static std::mutex g_mu;
static std::map<void *, size_t> g_regions;
static int g_pins = 0;
static unsigned g_hw = 1;
static std::atomic<bool> g_fail{false};
static std::thread::id g_main;

unsigned int std::thread::hardware_concurrency() noexcept { return g_hw; }

void *operator new(size_t n) {
    if (g_fail.load() && std::this_thread::get_id() == g_main) throw std::bad_alloc();
    if (void *p = malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

static size_t pinned() {
    std::lock_guard<std::mutex> l(g_mu);
    size_t n = 0;
    for (auto &r : g_regions) n += r.second;
    return n;
}
static cudaError_t pin(void *p, size_t n) {
    std::lock_guard<std::mutex> l(g_mu);
    g_regions[p] = n;
    g_pins++;
    return cudaSuccess;
}
static cudaError_t unpin(void *p) {
    std::lock_guard<std::mutex> l(g_mu);
    return g_regions.erase(p) ? cudaSuccess : cudaErrorInvalidValue;
}

extern "C" {
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(1);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    g_copies++;
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    *p = malloc(n);
    return pin(*p, n);
}
cudaError_t cudaFreeHost(void *p) {
    const cudaError_t e = unpin(p);
    free(p);
    return e;
}
cudaError_t cudaHostRegister(void *p, size_t n, unsigned) { return pin(p, n); }
cudaError_t cudaHostUnregister(void *p) { return unpin(p); }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *) { return cudaSuccess; }
}

int main(int argc, char **argv) {
    g_main = std::this_thread::get_id();
    g_hw = (unsigned)atoi(argv[1]);
    std::vector<char> dev, host;
    for (int i = 2; i < argc; i++) {
        const std::string s = argv[i];
        if (s == "fail") g_fail = true;
        else if (s == "hold") glac::hostcopy_hold();
        else if (s == "drop") {
            glac::hostcopy_drop();
            printf("%zu\n", pinned());
        } else if (s == "pinned") printf("%zu %d\n", pinned(), g_pins);
        else {
            const size_t n = (size_t)atoll(argv[++i]);
            const bool up = s == "up", fail = g_fail.exchange(false);
            dev.assign(n, 0);
            host.assign(n, 0);
            std::vector<char> &src = up ? host : dev;
            for (size_t k = 0; k < n; k++) src[k] = (char)(k * 31 + (k >> 11));
            g_copies = 0;
            g_fail = fail;
            const cudaError_t e = up ? glac::copy_to_device(dev.data(), host.data(), n, 0, nullptr)
                                     : glac::copy_to_host(host.data(), dev.data(), n, 0, nullptr);
            g_fail = false;
            if (e != cudaSuccess || dev != host) {
                printf("wrong\n");
                return 1;
            }
            g_fail = fail;
            printf("%d\n", g_copies.load());
        }
    }
    return 0;
}
