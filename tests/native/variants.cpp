// The forms of the launch variants (variants.cuh).  Without arguments a line
// "family fp32 variant regs shape" each; with "split morningstar learned blocks" a line
// "family fp32 same[0] ..." for the flow and Metropolis variants of such a lattice.
#include "variants.cuh"

#include <cstdio>
#include <cstdlib>

using namespace glac;

int main(int argc, char **argv) {
    if (argc > 4) {
        const bool split = atoi(argv[1]), morningstar = atoi(argv[2]), learned = atoi(argv[3]);
        const int blocks = atoi(argv[4]);
        for (int f = 0; f < 2; f++)
            for (int p = 0; p < 2; p++) {
                int same[kMaxVariants];
                const int n = num_variants((Family)f, p);
                first_alike(n, [&](int v) {
                    return f == FAM_FLOW ? lattice_flow_form(p, v, split, morningstar)
                                         : lattice_metro_form(p, v, split, learned, blocks);
                }, same);
                printf("%d %d", f, p);
                for (int v = 0; v < n; v++) printf(" %d", same[v]);
                printf("\n");
            }
        return 0;
    }
    for (int f = 0; f < 3; f++)
        for (int p = 0; p < 2; p++)
            for (int v = 0; v < num_variants((Family)f, p); v++) {
                const VariantForm form = variant_form((Family)f, p, v);
                printf("%d %d %d %d %d\n", f, p, v, form.regs, form.shape);
            }
    return 0;
}
