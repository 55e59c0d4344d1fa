// FP64 particle kernels: absolute positions. Built with -fmad=false: the
// dipole mover, the export test and the element kernel round as the
// reference's x86 build does; the field mover and the deposit (push64.cuh)
// fuse their products explicitly (__fma_rn).
#include <algorithm>

#include "particles_impl.cuh"
#include "push64.cuh"

namespace ipg {

namespace {
// How a launch over `slots` slots in `tiles` tiles is cut: particles per work
// item, tiles per span, blocks per span and warps per block.
//   * Items are as long as leaves about six warps per sub-partition (152 SMs
//     x 4): an item costs a quarter of a round or more, shorter ones leave
//     a shorter tail and end more evenly. Gather + dipole + deposit, 256
//     particles a cell, ms per push with items of 256 / 64 / 32 / 16: 32^3
//     cells 1.25 / 1.45 / 1.55 / 1.67, 20^3 0.45 / 0.38 / 0.39 / 0.42, 14^3
//     0.40 / 0.162 / 0.145 / 0.150, 10^3 0.39 / 0.127 / 0.074 / 0.063; 24^3 of
//     32 a cell and species 0.283 / 0.199 / 0.227 / 0.215. Items of 128 cut
//     every other cell of 128 in two, and such items leave half a warp idle
//     (32^3 1.50, 20^3 0.43): not used. Without the deposit an item costs
//     next to nothing: 32 (32^3, dipole mover: 64 1.56, 32 1.31).
//   * Spans of 4 tiles leave fewer part-filled warps than single tiles
//     (32^3 1.25 against 1.47, 14^3 0.145 against 0.148, 306k particles 0.081
//     against 0.083); small universes keep a tile per span, whose table is
//     sooner scanned (E x B 8^3: 0.021 against 0.029).
//   * One warp a block: its registers are free as soon as it ends (blocks of 4
//     warps: 32^3 1.39). Items of 8 and 16 with the deposit take four, which
//     join the sums of a cell (Joint64).
//   * A block takes one round of items, where there is no deposit and the
//     launch is large four (32^3, dipole mover: 1.31 -> 1.22).
//   * Items of 32 at most where the dipole can ask for many sub-cycles
//     (many_sub_cycles): a round of 8 particles close to it takes up to 0.25 ms,
//     and an item's rounds follow one another (planet of one cell, bz 30, dipole
//     mover with deposit, push of 26^3 cells of 256: 3.98 ms -> 1.61, of 24^3
//     cells of 64: 0.97 -> 0.63).
struct Shape64 {
    int item, span, parts, warps;
};
Shape64 shape64(int64_t slots, int64_t tiles, bool deposit, bool sub_cycles) {
    constexpr int64_t kSms = 152, kGroups = 6 * kSms * 4 * kWarpItems64;
    Shape64 s{32, 1, 1, 1};
    if (deposit && !sub_cycles) s.item = slots >= kMaxItem64 * kGroups ? kMaxItem64 : 64;
    while (s.item > kGroup64 && slots < s.item * kGroups) s.item /= 2;
    if (tiles >= 2 * kSms) s.span = kMaxSpan64;
    s.parts = s.span * kSlotsPerCta / (s.item * kWarpItems64);
    if (!deposit && tiles >= 6 * kMaxSpan64 * kSms) s.parts /= 4;
    if (deposit && s.item <= 2 * kGroup64) {
        s.warps = Joint64::kWarps;
        s.parts /= s.warps;
    }
    return s;
}

Push64Set push64_set(const Geom& g, const PopSet<double>& S) {
    Push64Set pcs{};
    for (int i = 0; i < S.n; ++i) pcs.c[i] = push64_const(g, S.p[i]);
    return pcs;
}
}  // namespace

bool many_sub_cycles(const Geom& g, double qom) {
    if (g.mft == 0.0 || (g.mover == 1 && !(g.flags & 4u))) return false;
    double r2 = 0.0;  // of the closest point of the domain to the dipole
    for (int a = 0; a < 3; ++a) {
        const double out = std::max(g.origin[a], -(g.origin[a] + g.L[a]));
        if (out > 0.0) r2 += out * out;
    }
    // the planet drops what comes closer
    if (g.object_center[0] == 0.0 && g.object_center[1] == 0.0 && g.object_center[2] == 0.0)
        r2 = std::max(r2, g.planet_r2);
    // too few particles to matter (32^3 cells of 256, |B| above the line within
    // 0.3 cells, field mover: 1.64 ms without the short items, 1.86 with them;
    // within 0.63 cells 2.11 and 1.90)
    const double half = 0.5 * std::min(g.w[0], std::min(g.w[1], g.w[2]));
    r2 = std::max(r2, half * half);
    const double b2 = 4.0 * g.mft * g.mft / (r2 * r2 * r2);  // at the pole
    return g.dt * (4.0 * std::fabs(qom)) * b2 * g.inv_pic >= 8.0;
}

Push64Const push64_const(const Geom& g, const Pop<double>& P) {
    Push64Const c;
    c.d = dipole_species(g.mft, P.qom, g.dt, g.inv_pic);
    c.k1 = P.qom * 0.5 * g.dt;
    // rotations too large for the fast form take the sub-cycle branch
    c.d.e_max = std::min(c.d.e_max, kLargeRotation + 1023 - soft::exponent_of(c.k1));
    c.no_field = g.mft == 0.0 && soft::regular(g.dt, 100) && std::isfinite(c.k1) && std::isfinite(P.qom) &&
                 std::isfinite(4.0 * P.qom * g.dt) && std::isfinite(g.inv_pic);
    c.field_scale = (g.flags & 2u /*IPIC3D_F_GATHER_DIV_VOL*/) ? 1.0 / g.vol : 1.0;
    return c;
}

template <>
int launch_push<double>(const Geom& g, const PopSet<double>& S, int mode, const PushShape&, cudaStream_t st) {
    int64_t tiles = 0, most = 0, slots = 0;
    for (int i = 0; i < S.n; ++i) {
        const int64_t t = (S.p[i].capacity + kSlotsPerCta - 1) / kSlotsPerCta;
        tiles += t;
        most = std::max(most, t);
        slots += S.p[i].capacity;
    }
    if (most <= 0 || (mode != 0 && !g.deposit)) return 0;
    bool sub_cycles = false;
    for (int i = 0; i < S.n; ++i) sub_cycles = sub_cycles || many_sub_cycles(g, S.p[i].qom);
    const Shape64 sh = shape64(slots, tiles, g.deposit != 0, sub_cycles);
    const dim3 grid((unsigned)((most + sh.span - 1) / sh.span), sh.parts, S.n);
    const Push64Set pcs = push64_set(g, S);
    constexpr int kJ = Joint64::kWarps;
    auto run = [&](auto k) {
        k<<<grid, 32 * sh.warps, sh.warps * push64_smem_bytes(sh.span), st>>>(g, S, pcs, sh.span, sh.item);
    };
    const bool joined = sh.warps > 1;
    if (mode != 0) joined ? run(k_push64<false, false, true, kJ>) : run(k_push64<false, false, true, 1>);
    else if (g.mover == 1 && g.deposit)
        joined ? run(k_push64<true, true, true, kJ>) : run(k_push64<true, true, true, 1>);
    else if (g.mover == 1) run(k_push64<true, true, false, 1>);
    else if (g.deposit) joined ? run(k_push64<true, false, true, kJ>) : run(k_push64<true, false, true, 1>);
    else run(k_push64<true, false, false, 1>);
    return 1;
}
template <>
int launch_push_pending<double>(const Geom& g, const PopSet<double>& S, cudaStream_t st) {
    if (S.n <= 0) return 0;
    k_push_pending64<<<dim3(152, S.n), 128, 0, st>>>(g, S, push64_set(g, S));
    return 1;
}
template int launch_inject<double>(const Geom&, const Pop<double>&, double, const double*, const double*, uint64_t,
                                   const uint64_t*, cudaStream_t);
template int launch_place<double>(const Geom&, const PopSet<double>&, cudaStream_t);
template int launch_pending_rotate<double>(const PopSet<double>&, uint64_t*, cudaStream_t);
template int launch_relayout<double>(const Pop<double>&, const Pop<double>&, int, int32_t*, cudaStream_t);
template int launch_pending_count<double>(const Pop<double>&, int32_t*, cudaStream_t);

template <>
int launch_push_batch<double>(const PopJob<double>* jobs, const int2* cta_job, int64_t nctas, int mode,
                              const Geom& g, const BatchTraits& traits, const PushShape&, cudaStream_t st) {
    if (nctas <= 0 || (mode != 0 && !g.deposit)) return 0;
    const Shape64 sh = shape64(nctas * kSlotsPerCta, nctas, g.deposit != 0, traits.sub_cycles);
    const unsigned grid = (unsigned)(nctas * sh.parts);
    constexpr int kJ = Joint64::kWarps;
    auto run = [&](auto k) {
        k<<<grid, 32 * sh.warps, sh.warps * push64_smem_bytes(sh.span), st>>>(jobs, cta_job, sh.span, sh.item,
                                                                              sh.parts);
    };
    const bool joined = sh.warps > 1;
    if (mode != 0) joined ? run(k_push64_batch<false, false, true, kJ>) : run(k_push64_batch<false, false, true, 1>);
    else if (g.mover == 1 && g.deposit)
        joined ? run(k_push64_batch<true, true, true, kJ>) : run(k_push64_batch<true, true, true, 1>);
    else if (g.mover == 1) run(k_push64_batch<true, true, false, 1>);
    else if (g.deposit) joined ? run(k_push64_batch<true, false, true, kJ>) : run(k_push64_batch<true, false, true, 1>);
    else run(k_push64_batch<true, false, false, 1>);
    return 1;
}
template <>
int launch_push_pending_batch<double>(const PopJob<double>* jobs, int njobs, cudaStream_t st) {
    k_push_pending64_batch<<<dim3(2, njobs), 128, 0, st>>>(jobs);
    return 1;
}
template int launch_place_batch<double>(const PopJob<double>*, const int2*, int64_t, cudaStream_t);
template int launch_pending_rotate_batch<double>(const PopJob<double>*, int, cudaStream_t);
template int launch_batch_begin<double>(const PopJob<double>*, int, const InstJob*, int, int64_t, int, uint32_t*,
                                        cudaStream_t);
template int launch_batch_end<double>(const PopJob<double>*, const InstJob*, int, uint32_t*, cudaStream_t);
template int launch_batch_status<double>(const PopJob<double>*, int, JobStatus*, cudaStream_t);
}  // namespace ipg

#include "../../include/ipic3d_types.h"

namespace ipg {

// Particle::updateVelocity + updatePosition (particle.h:24-49), nsteps times,
// uniform E and B: the element kernel behind the Boris known-answer tests.
__global__ void k_boris(ipic3d_particle* p, uint64_t n, double ex, double ey, double ez, double bx, double by,
                        double bz, double dt, uint64_t nsteps, int push_position) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    ipic3d_particle q = p[i];
    for (uint64_t t = 0; t < nsteps; ++t) {
        boris<double>(q.velocity[0], q.velocity[1], q.velocity[2], ex, ey, ez, bx, by, bz, q.qom, dt);
        if (push_position) {
            q.position[0] = q.position[0] + q.velocity[0] * dt;
            q.position[1] = q.position[1] + q.velocity[1] * dt;
            q.position[2] = q.position[2] + q.velocity[2] * dt;
        }
    }
    p[i] = q;
}

int launch_boris(const void* parts, uint64_t n, const double E[3], const double B[3], double dt, uint64_t nsteps,
                 int push_position, void* out, cudaStream_t st) {
    (void)parts;
    k_boris<<<(unsigned)((n + 127) / 128), 128, 0, st>>>((ipic3d_particle*)out, n, E[0], E[1], E[2], B[0], B[1], B[2],
                                                          dt, nsteps, push_position);
    return 1;
}

}  // namespace ipg
