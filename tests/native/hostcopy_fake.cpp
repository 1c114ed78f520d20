// The host side of the field copies (hostcopy.cu) on a fake CUDA runtime whose
// copies are memcpy.  argv: the cores that the process may use (-n: n in the machine,
// and no affinity mask to be had), then one step after another:
//   up N | down N    a copy of N bytes, checked; prints the number of transfers it took
//   fail             the third and every later thread of the copies that follow finds no memory
//   hold | drop      a holder comes or goes; drop prints the bytes pinned after it
//   pinned           prints the bytes pinned now and how often memory was pinned
//   forked           a child puts memory of its own where the buffers were, drops its
//                    holder and uses that memory; prints its exit status
#include "hostcopy.cu"

#include <cstdio>
#include <cstdlib>
#include <new>
#include <sched.h>
#include <string>
#include <sys/wait.h>
#include <vector>

static std::atomic<int> g_copies{0};
static std::mutex g_mu;
struct Region {
    void *p;
    size_t n;
};
static Region g_regions[16];  // no allocation of the fake's own
static int g_pins = 0;
static int g_cores = 1;
static bool g_fail = false;         // of the main thread, which makes the threads
static thread_local int g_left = -1;  // allocations until the first that fails; below 0: none does

unsigned int std::thread::hardware_concurrency() noexcept { return (unsigned)abs(g_cores); }
extern "C" int sched_getaffinity(pid_t, size_t n, cpu_set_t *set) noexcept {
    if (g_cores < 0) return -1;
    memset(set, 0, n);
    for (int k = 0; k < g_cores; k++) CPU_SET_S(k, n, set);
    return 0;
}

void *operator new(size_t n) {
    if (g_left == 0) throw std::bad_alloc();
    if (g_left > 0) g_left--;
    if (void *p = malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

static size_t pinned() {
    std::lock_guard<std::mutex> l(g_mu);
    size_t n = 0;
    for (const Region &r : g_regions) n += r.n;
    return n;
}
static cudaError_t move(void *from, void *to, size_t n) {
    std::lock_guard<std::mutex> l(g_mu);
    for (Region &r : g_regions)
        if (r.p == from) {
            r = Region{to, n};
            return cudaSuccess;
        }
    return cudaErrorInvalidValue;
}
static cudaError_t pin(void *p, size_t n) {
    g_pins++;
    return move(nullptr, p, n);
}
static cudaError_t unpin(void *p) { return move(p, nullptr, 0); }

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
}

int main(int argc, char **argv) {
    g_cores = atoi(argv[1]);
    std::vector<char> dev, host;
    for (int i = 2; i < argc; i++) {
        const std::string s = argv[i];
        if (s == "fail") g_fail = true;
        else if (s == "hold") glac::hostcopy_hold();
        else if (s == "drop") {
            glac::hostcopy_drop();
            printf("%zu\n", pinned());
        } else if (s == "pinned") printf("%zu %d\n", pinned(), g_pins);
        else if (s == "forked") {
            fflush(stdout);
            const pid_t child = fork();
            if (child == 0) {
                void *p = mmap(glac::g_mapped, 4096, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_FIXED, -1, 0);
                glac::hostcopy_drop();
                *static_cast<volatile char *>(p) = 1;
                _exit(pinned() > 0 ? 0 : 2);  // nor does the child unpin what is not its own
            }
            int status = -1;
            waitpid(child, &status, 0);
            printf("%d\n", status);
        }
        else {
            const size_t n = (size_t)atoll(argv[++i]);
            const bool up = s == "up";
            dev.assign(n, 0);
            host.assign(n, 0);
            std::vector<char> &src = up ? host : dev;
            for (size_t k = 0; k < n; k++) src[k] = (char)(k * 31 + (k >> 11));
            g_copies = 0;
            g_left = g_fail ? 2 : -1;
            const cudaError_t e = up ? glac::copy_to_device(dev.data(), host.data(), n, 0, nullptr)
                                     : glac::copy_to_host(host.data(), dev.data(), n, 0, nullptr);
            g_left = -1;
            if (e != cudaSuccess || dev != host) {
                printf("wrong\n");
                return 1;
            }
            printf("%d\n", g_copies.load());
        }
    }
    return 0;
}
