// Launch variants of the kernel families (host code): what a variant's number launches.
//
// A number means the same form from build to build, so that a tuning kept from an
// earlier run stays what it was; variant 0 is each family's default, which follows
// the lattice.
#pragma once

namespace glac {

enum Family { FAM_FLOW = 0, FAM_METRO = 1, FAM_OBS = 2 };
constexpr int kMaxVariants = 4;

// regs: the register cap (0: the compiler's own allocation under 128-thread launch
// bounds).  shape: the flow's site-block shape (0: a link per thread).
struct VariantForm {
    int regs, shape;
};
inline bool operator==(const VariantForm &a, const VariantForm &b) { return a.regs == b.regs && a.shape == b.shape; }
// several warps to a link (split.cu, metro_split.cu)
constexpr VariantForm kSplitForm{-1, 0};

// The flow stage waits on its neighbour links (L2 hits), so resident warps count
// for more than registers: its caps give 16 (FP64) and 24 (FP32) warps per SM.
// Stage 2 on B200, capped / uncapped: FP64 24^3 x 48 440 / 531 us, 16^3 x 32 96 /
// 116; FP32 32^3 x 64 664 / 699, 16^3 x 32 52 / 54.  Variant 0 is variant 1's form
// but on small lattices, where it is the form of several warps to a link (split.cu).
// Metropolis: variant 0 as metro_default_regs says.  Measurement: the caps are an
// ensemble's; a single lattice's kernel takes its variant as blocks per SM
// (observables.cu).
inline int num_variants(Family f, bool fp32) { return f == FAM_FLOW ? 4 : fp32 ? (f == FAM_METRO ? 4 : 3) : 2; }
inline VariantForm variant_form(Family f, bool fp32, int v) {
    constexpr VariantForm flow[2][4] = {{{128, 0}, {128, 0}, {0, 1}, {128, 2}}, {{80, 0}, {80, 0}, {0, 3}, {96, 0}}};
    constexpr VariantForm metro[2][4] = {{{0, 0}, {128, 0}}, {{96, 0}, {96, 0}, {80, 0}, {128, 0}}};
    constexpr VariantForm obs[2][4] = {{{0, 0}, {128, 0}}, {{0, 0}, {128, 0}, {168, 0}}};
    if (v < 0 || v >= num_variants(f, fp32)) return VariantForm{0, 0};
    return (f == FAM_FLOW ? flow : f == FAM_METRO ? metro : obs)[fp32 ? 1 : 0][v];
}

// Register cap of a single lattice's sub-sweep as variant 0.  FP32 takes 96 (five
// blocks per SM), but 128 (four) where a fifth block finds no work, up to one wave of
// blocks, and for the learned spread, whose kernel spills at 96.  Microseconds per
// sweep on B200 at 128 / 96: 12^3 x 24 112 / 115, 24^3 x 48 784 / 776, 32^3 x 64 2275 /
// 2247, all at 1965 MHz; learned 24^3 x 48 898 / 934 (uncapped 930).  FP64 goes
// uncapped (three blocks per SM), but with 128 and a small spill from ten blocks per SM
// on: 16^3 x 32 346 / 329 us, 24^3 x 48 1463 / 1498, 32^3 x 64 4310 / 4432.
inline int metro_default_regs(bool fp32, bool learned, int blocks) {
    if (fp32) return learned || blocks <= 5 * 148 ? 128 : 96;
    return blocks > 10 * 148 ? 128 : 0;
}

// What a variant launches on a single lattice; split: whether its default is kSplitForm.
// The other exponentials have one form, whose stage 1 with the measurement may still be
// the site-per-thread one.
inline VariantForm lattice_flow_form(bool fp32, int v, bool split, bool morningstar) {
    if (v == 0 && split) return kSplitForm;
    const VariantForm f = variant_form(FAM_FLOW, fp32, v);
    return morningstar ? f : VariantForm{0, f.shape == 3 ? 3 : 0};
}
inline VariantForm lattice_metro_form(bool fp32, int v, bool split, bool learned, int blocks) {
    if (v == 0 && split) return kSplitForm;
    return v == 0 ? VariantForm{metro_default_regs(fp32, learned, blocks), 0} : variant_form(FAM_METRO, fp32, v);
}

// same[v]: the first variant with v's form.
template <typename Form> void first_alike(int n, Form form, int *same) {
    for (int v = 0; v < n; v++) {
        same[v] = v;
        for (int w = 0; w < v && same[v] == v; w++)
            if (form(w) == form(v)) same[v] = w;
    }
}

}  // namespace glac
