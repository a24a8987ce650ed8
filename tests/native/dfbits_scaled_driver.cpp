// CPU driver for dfb::scaled (csrc/dfbits.cuh): reads (uint32 float bits, int32 e)
// pairs from stdin, writes (int64 ok, double value) per pair.
#include <cstdio>
#include "../../modal-cmb_gb300/csrc/dfbits.cuh"

int main()
{
    struct { uint32_t u; int32_t e; } in;
    while (fread(&in, 8, 1, stdin) == 1) {
        struct { int64_t ok; double x; } o = {0, 0.0};
        o.ok = dfb::scaled(in.u, in.e, &o.x) ? 1 : 0;
        fwrite(&o, 16, 1, stdout);
    }
    return 0;
}
