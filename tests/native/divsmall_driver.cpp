// CPU driver for modal::div_small (csrc/divsmall.cuh): reads (double n, double c) pairs from
// stdin, writes (div_small, n / c) per pair.
#include <cstdio>
#include "../../modal-cmb_gb300/csrc/divsmall.cuh"

int main()
{
    double in[2];
    while (fread(in, 8, 2, stdin) == 2) {
        const double o[2] = {modal::div_small(in[0], in[1], 1.0 / in[1]), in[0] / in[1]};
        fwrite(o, 8, 2, stdout);
    }
    return 0;
}
