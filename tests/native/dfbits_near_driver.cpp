// CPU driver for dfb::near_int (csrc/dfbits.cuh): reads (double x, int64 sh) pairs from
// stdin, writes (int64 ok, int64 F) per pair.
#include <cstdio>
#include "../../modal-cmb_gb300/csrc/dfbits.cuh"

int main()
{
    struct { double x; int64_t sh; } in;
    while (fread(&in, 16, 1, stdin) == 1) {
        long long F = 0;
        const bool ok = dfb::near_int(in.x, (int)in.sh, &F);
        int64_t o[2] = {ok ? 1 : 0, (int64_t)F};
        fwrite(o, 16, 1, stdout);
    }
    return 0;
}
