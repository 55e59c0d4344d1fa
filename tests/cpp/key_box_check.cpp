// The tracer's box test on the high words of positions (allscale_ipic3d_gb300/
// csrc/fp64_int.cuh: key_box, in_key_box) on the host. Reads triples of
// doubles (low, high, x) from argv[1] and writes one byte each: bit 0 the box
// test, bit 1 low <= x <= high. Built so that a signed overflow ends it.
#include <cstdint>
#include <cstdio>

namespace ipg { namespace soft { float soft_host_rcp(float x) { return x; } float soft_host_rsqrt(float x) { return x; } } }
#include "../../allscale_ipic3d_gb300/csrc/fp64_int.cuh"

int main(int argc, char** argv) {
    if (argc < 2) return 2;
    FILE* f = fopen(argv[1], "rb");
    if (!f) return 2;
    double v[3];
    while (fread(v, sizeof v, 1, f) == 1)
        putchar((int)ipg::soft::in_key_box(v[2], ipg::soft::key_box(v[0], v[1])) | (v[0] <= v[2] && v[2] <= v[1]) << 1);
    fclose(f);
    return 0;
}
