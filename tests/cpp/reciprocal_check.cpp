// refine_reciprocal (allscale_ipic3d_gb300/csrc/fp64_int.cuh) on the host: reads
// pairs (d, e) from argv[1] and writes the refinement of 1 / d (1 + e).
#include <cstdint>
#include <cstdio>

namespace ipg { namespace soft { float soft_host_rcp(float x) { return x; } float soft_host_rsqrt(float x) { return x; } } }
#include "../../allscale_ipic3d_gb300/csrc/fp64_int.cuh"

int main(int argc, char** argv) {
    if (argc < 2) return 2;
    FILE* f = fopen(argv[1], "rb");
    if (!f) return 2;
    double v[2];
    while (fread(v, sizeof v, 1, f) == 1) {
        const double r = ipg::soft::refine_reciprocal(v[0], 1.0 / v[0] * (1.0 + v[1]));
        fwrite(&r, sizeof r, 1, stdout);
    }
    fclose(f);
    return 0;
}
