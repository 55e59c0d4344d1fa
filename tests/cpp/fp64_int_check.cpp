// Runs the integer-pipe FP64 arithmetic (allscale_ipic3d_gb300/csrc/
// fp64_int.cuh) on the host against the host's own FP64 operations. The FP32
// estimates the device takes from its approximate instructions are replaced
// by the exact value times 1 + e, e over the instructions' error bounds.
// Reads quadruples of doubles (a, b, c, err in [-1, 1]) from argv[1] and
// writes per quadruple: the number of operations that differ from FP64
// (product, square, triple, sum of magnitudes, quotients), pow25(|a|) and
// whether it is sure.
#include <cmath>
#include <cstdint>
#include <cstdio>

namespace ipg { namespace soft { float soft_host_rcp(float); float soft_host_rsqrt(float); } }
#include "../../allscale_ipic3d_gb300/csrc/fp64_int.cuh"

static double g_err = 0.0;
namespace ipg { namespace soft {
float soft_host_rcp(float x) { return (float)((1.0 / (double)x) * (1.0 + g_err * 0x1p-23)); }
float soft_host_rsqrt(float x) { return (float)((1.0 / std::sqrt((double)x)) * (1.0 + g_err * 0x1.8p-24)); }
}}

int main(int argc, char** argv) {
    using namespace ipg::soft;
    if (argc < 2) return 2;
    FILE* f = fopen(argv[1], "rb");
    if (!f) return 2;
    double v[4];
    while (fread(v, sizeof v, 1, f) == 1) {
        const double a = v[0], b = v[1], c = v[2];
        g_err = v[3];
        const Num A = unpack(a), B = unpack(b), C = unpack(c);
        double bad = 0;
        bad += pack(A) != a;
        bad += pack(mul(A, B)) != a * b;
        bad += pack(mul(mul(A, B), C)) != (a * b) * c;
        bad += pack(sqr(mul(A, B))) != (a * b) * (a * b);
        bad += pack(triple(A)) != 3.0 * a;
        bad += pack(mul(triple(A), B)) != (3.0 * a) * b;
        bad += pack(add_positive(A, B)) != std::fabs(a) + std::fabs(b);
        bad += pack(add_positive(add_positive(sqr(A), sqr(B)), sqr(C))) != (a * a + b * b) + c * c;
        bad += pack(div(A, divisor(B))) != a / b;
        bad += pack(div(mul(A, C), divisor(add_positive(B, C)))) != (a * c) / (std::fabs(b) + std::fabs(c));
        bad += std::signbit(pack(div(A, divisor(B)))) != std::signbit(a / b);
        const double w = std::fabs(b) * std::ldexp(1.0, 1023 - exponent_of(b) + (exponent_of(c) % 90));
        bad += quotient(a, w, 1.0 / w, power_of_two(w)) != a / w;
        bad += quotient(a, 0.125, 8.0, power_of_two(0.125)) != a / 0.125;
        bad += std::signbit(quotient(-0.0, w, 1.0 / w, 0)) != std::signbit(-0.0 / w);
        bad += bits_of(plus_zero(-0.0)) != bits_of(0.0 + -0.0) || plus_zero(a) != a;
        bool sure = false;
        const double p = pack(pow25(unpack(std::fabs(a)), sure));
        const double out[3] = {bad, p, sure ? 1.0 : 0.0};
        fwrite(out, sizeof(double), 3, stdout);
    }
    fclose(f);
    return 0;
}
