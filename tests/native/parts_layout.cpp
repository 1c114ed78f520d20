// The stand-alone measurement's parts inside a link field and a force
// (PlaneParts, lattice.cuh), compiled for the host.  argv[1]: sites.  Prints
// "<fp32|fp64> <0|1: every check held> <admitted by field_offsets_fit>".
#include "lattice.cuh"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

using namespace glac;

// Every slot's first and last element: 32-bit offsets equal to the 64-bit ones,
// inside the buffer and below the plaquettes.
template <typename T> bool offsets_hold(int Vh) {
    const bool fp64 = sizeof(T) == 8;
    const size_t chunk = 16, chunks = 8 * sizeof(T) / chunk, vh32 = (size_t)round32(Vh);
    char *field = reinterpret_cast<char *>((uintptr_t)1 << 40), *force = reinterpret_cast<char *>((uintptr_t)1 << 41);
    const PlaneParts<T> v = plane_parts_view<T>(field, force, Vh);
    char *plaq = reinterpret_cast<char *>(v.plaq);
    bool ok = plaq >= field && plaq + 12 * (size_t)Vh * sizeof(T) <= field + field_bytes(Vh, fp64);
    for (int k = 0; k < 12; k++)
        for (int par = 0; par < 2; par++)
            for (int s : {0, 31, Vh / 2, Vh - 1}) {
                const bool low = k < PlaneParts<T>::kLow;
                const int dir = low ? k : k - PlaneParts<T>::kLow;
                const uint32_t got = (low ? v.lo : v.hi).base(dir, par, s);
                const uint64_t want = (uint64_t)(2 * dir + par) * chunks * vh32 + (uint64_t)(s >> 5) * 32 * chunks +
                                      (uint64_t)(s & 31);
                const uint64_t end = (want + 32 * (chunks - 1) + 1) * chunk;
                ok = ok && got == want && (low ? field + end <= plaq : end <= force_bytes(Vh, fp64));
            }
    return ok;
}

// All parts and plaquettes written, then read back; the bytes behind both buffers stay.
template <typename T> bool round_trip(int Vh) {
    const bool fp64 = sizeof(T) == 8;
    const size_t fb = field_bytes(Vh, fp64), zb = force_bytes(Vh, fp64), guard = 4096;
    char *field = static_cast<char *>(aligned_alloc(256, (fb + guard + 255) / 256 * 256));
    char *force = static_cast<char *>(aligned_alloc(256, (zb + guard + 255) / 256 * 256));
    memset(field + fb, 0x5a, guard);
    memset(force + zb, 0x5a, guard);
    const PlaneParts<T> v = plane_parts_view<T>(field, force, Vh);
    auto value = [&](int k, int par, int s) { return T((k * 2 + par) * 1024 + s); };
    for (int k = 0; k < 12; k++)
        for (int par = 0; par < 2; par++)
            for (int s = 0; s < Vh; s++) {
                const T x = value(k, par, s);
                AH8<T> Z;
                Z.a = x; Z.d = -x; Z.b = cx(x, T(1)); Z.c = cx(T(2), x); Z.e = cx(x, T(3));
                v.store(k, par, s, Z);
                v.plaq[(k / 2 * 2 + par) * Vh + s] = x;
            }
    bool ok = true;
    for (int k = 0; k < 12; k++)
        for (int par = 0; par < 2; par++)
            for (int s = 0; s < Vh; s++) {
                const T x = value(k, par, s);
                const AH8<T> Z = v.load(k, par, s);
                ok = ok && Z.a == x && Z.d == -x && Z.b.re == x && Z.b.im == T(1) && Z.c.re == T(2) && Z.c.im == x &&
                     Z.e.re == x && Z.e.im == T(3) && (k % 2 == 0 || v.plaq[(k / 2 * 2 + par) * Vh + s] == x);
            }
    for (size_t i = 0; i < guard; i++) ok = ok && field[fb + i] == 0x5a && force[zb + i] == 0x5a;
    free(field);
    free(force);
    return ok;
}

template <typename T> void check(const char *name, long long V) {
    const bool fits = field_offsets_fit(V, sizeof(T) == 8);
    bool ok = fits ? offsets_hold<T>((int)(V / 2)) : true;
    if (V <= 2048) ok = ok && round_trip<T>((int)(V / 2));
    printf("%s %d %d\n", name, ok, fits);
}

int main(int argc, char **argv) {
    const long long V = argc > 1 ? atoll(argv[1]) : 0;
    check<float>("fp32", V);
    check<double>("fp64", V);
    return 0;
}
