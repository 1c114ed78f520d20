// The forms of the launch variants (variants.cuh): a line "family fp32 variant regs
// shape" each, then "metro fp32 learned blocks regs" of variant 0 at the blocks in argv.
#include "variants.cuh"

#include <cstdio>
#include <cstdlib>

using namespace glac;

int main(int argc, char **argv) {
    for (int f = 0; f < 3; f++)
        for (int p = 0; p < 2; p++)
            for (int v = 0; v < num_variants((Family)f, p); v++) {
                const VariantForm form = variant_form((Family)f, p, v);
                printf("%d %d %d %d %d\n", f, p, v, form.regs, form.shape);
            }
    for (int i = 1; i < argc; i++)
        for (int p = 0; p < 2; p++)
            for (int l = 0; l < 2; l++) printf("%d %d %s %d\n", p, l, argv[i], metro_default_regs(p, l, atoi(argv[i])));
    return 0;
}
