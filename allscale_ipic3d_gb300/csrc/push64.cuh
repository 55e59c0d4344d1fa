// The FP64 push: mover (cell.h:896-964) + export (cell.h:975-1159) in place,
// fused with the cloud-in-cell deposit (cell.h:787-824, scatter form).
//
// GB300's FP64 pipe bounds it (one warp instruction per 64 to 76 cycles and
// SM sub-partition), so what counts is the number of FP64 instructions a
// warp issues -- idle lanes cost as much as busy ones -- and how many warps
// share the work of a small universe. Per 32 particles of a step with field
// gather, dipole and deposit:
//   * the field is the cell's trilinear polynomial about its centre, built
//     once per work item from the 8 corners: 42 fused multiply-adds (the sum
//     over corners: about 130 multiplications and additions);
//   * the dipole's |r|^-5, the rotation's 2 / (1 + |t|^2) and the deposit's
//     weights are fused forms without divisions (the export test keeps the
//     reference's own differences from the cell centre);
//   * comparisons run on the doubles' bit patterns in the integer pipe;
//   * the deposit sums the centred monomial moments as the FP32 push does
//     (push32_pipe.cuh): 35 operations, and 40 per work item for the
//     reduction over its lanes and the corner sums.
// 183 FP64 instructions (items' shares and idle lanes included) in place of
// 541 before. The dipole mover without the gather rounds exactly as the
// reference does (dipole64.cuh). Measured push per step, before and after:
// 8.4M particles, gather + dipole + deposit 9.18 -> 2.89 ms (FP64 pipe 86 %
// busy); 306k particles, two species, gather + deposit 0.593 -> 0.151 ms;
// 33k particles 0.140 -> 0.028 ms (a warp's serial chain); 1.05M particles,
// dipole mover, a sixth of them leaving their cells 0.489 -> 0.160 ms (FP64
// pipe 58 %, integer 42 %). Loading a round's particles a round ahead
// changed nothing.
//
// Work. A work item is up to `item` particles of one cell, pushed by a group
// of 8 lanes, 8 particles at a time (slots are 8-aligned: full 64-byte
// segments); four items share a warp. Groups of 8 rather than whole warps
// keep the lanes busy where cells hold few particles or end unevenly, at the
// price of a reduction per 8 lanes; a cell of more than `item` particles is
// cut evenly, so that the items of a warp end together. A block of 1 to 4
// warps takes the items of `span` consecutive 1024-slot tiles, or of a part
// of them (gridDim.y parts): cells of up to a tile belong to the span they
// start in, larger ones are cut at its boundaries.
#pragma once

#include "dipole64.cuh"

namespace ipg {

constexpr int kGroup64 = 8;
constexpr int kMaxWarps64 = 4;
constexpr int kWarpItems64 = 32 / kGroup64;  // work items of a warp at a time
constexpr int kCoefStride64 = 50;  // 48 + 2: the four groups of a warp read different banks

// ---- field --------------------------------------------------------------------

// Approximations of the FP64 unit's seed instructions (relative error at
// most 2^-20), refined below.
__device__ __forceinline__ double seed_rsqrt(double x) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}
__device__ __forceinline__ double seed_rcp(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}

// 1 / d: y (1 + e + e^2), e = 1 - d y
__device__ __forceinline__ double reciprocal(double d) {
    const double y = seed_rcp(d);
    const double e = __fma_rn(-d, y, 1.0);
    return __fma_rn(y, __fma_rn(e, e, e), y);
}

// r2^(-5/2) out of the integer path's range: y = r2^(-1/2) by y (1 + e / 2 + 3 e^2 / 8), e = 1 - r2 y^2, and
// one correction of y^5 from the residual of y^2
__device__ __forceinline__ double inverse_pow25(double r2) {
    double y = seed_rsqrt(r2);
    const double e = __fma_rn(-__dmul_rn(r2, y), y, 1.0);
    y = __fma_rn(y, __dmul_rn(e, __fma_rn(0.375, e, 0.5)), y);
    const double y2 = __dmul_rn(y, y);
    const double f = __dmul_rn(__dmul_rn(y2, y2), y);
    const double d = __fma_rn(-r2, y2, 1.0);
    return __fma_rn(f, __dmul_rn(2.5, d), f);
}

// The field of a cell in 64-bit fixed point. A component's 8 corner values
// share the largest one's exponent e_max: fixed = value 2^(1081 - e_max), below
// 2^59, so that one unit is 2^-59 of the largest corner (FP64's own rounding
// is 2^-53 of it). The trilinear polynomial's coefficients are differences of
// these integers, exact, and the position in the cell is a 64-bit fraction:
// a product is the high half of 64 x 64 bits. Seven of them and seven sums per
// component take about 150 integer-pipe cycles per warp; the seven FP64
// multiply-adds they replace took 448 of the FP64 pipe, which bounds the
// push.

// coefficients of 1, x, y, xy, z, xz, yz, xyz (index = bits x | y << 1 | z << 2)
__device__ __forceinline__ int64_t scaled(int64_t c, uint64_t r) {  // floor(c r / 2^64)
    return (int64_t)(__umul64hi((uint64_t)c, r) - (c < 0 ? r : 0));
}
__device__ __forceinline__ int64_t poly_fixed(const int64_t* c, uint64_t x, uint64_t y, uint64_t z) {
    const int64_t xz = c[5] + scaled(c[7], y);
    const int64_t gx = c[1] + scaled(c[3], y) + scaled(xz, z);
    const int64_t gy = c[2] + scaled(c[6], z);
    return c[0] + scaled(c[4], z) + scaled(gy, y) + scaled(gx, x);
}
// v with exponent e as fixed point for e_max >= e
__device__ __forceinline__ int64_t to_fixed(double v, int e_max) {
    const soft::Num n = soft::unpack(v);
    const int d = e_max - n.e;
    const int64_t t = n.e == 0 || d > 59 ? 0 : (int64_t)((n.m << 6) >> d);
    return n.sign ? -t : t;
}
__device__ __forceinline__ double from_fixed(int64_t v, int e_max) {
    if (v == 0) return 0.0;
    const uint64_t a = v < 0 ? (uint64_t)-v : (uint64_t)v;
    const int n = __clzll((long long)a);
    const uint64_t m = a << n;
    soft::Num r;
    r.m = (m >> 11) + ((m >> 10) & 1);
    r.e = e_max - n + 5;
    r.sign = v < 0 ? 0x80000000u : 0u;
    return soft::pack(r);
}
// e_max a component may have (0: all corners are zero); others take FP64
__device__ __forceinline__ bool fixed_range(int e_max) { return e_max == 0 || (uint32_t)(e_max - 200) <= 1600u; }

// A coordinate s about the cell's centre, in cell widths, as the fraction
// (1/2 + s) 2^64; only for |s| <= 1/2.
__device__ __forceinline__ bool in_cell(double s) {
    return (soft::bits_of(s) & 0x7fffffffffffffffull) <= 0x3fe0000000000000ull;
}
__device__ __forceinline__ uint64_t fraction(double s) {
    const soft::Num n = soft::unpack(s);
    const int sh = 1022 - n.e;
    const uint64_t t = n.e == 0 || sh > 63 ? 0 : (n.m << 11) >> sh;
    constexpr uint64_t kHalf = 1ull << 63;
    if (n.sign) return kHalf - t;
    return t == kHalf ? ~0ull : kHalf + t;  // 1/2 + 1/2: one unit below 1
}

// The corner node k = x | y << 1 | z << 2 of a cell: its E, B.
__device__ __forceinline__ const double* corner_field(const Geom& g, int cx, int cy, int cz, int k) {
    return g.field + 9 * field_index(g, cx + 1 + (k & 1), cy + 1 + ((k >> 1) & 1), cz + 1 + (k >> 2));
}

// A node value with the gather's normalisation (none: no FP64 instruction).
__device__ __forceinline__ double field_value(const Push64Const& pc, double v) {
    return soft::bits_of(pc.field_scale) == 0x3ff0000000000000ull ? v : v * pc.field_scale;
}

// E, B at (x, y, z) about the centre of a cell, by one thread in FP64: the
// positions outside the cell (a particle that crossed more than a cell) and
// the values out of the fixed-point range.
__device__ __noinline__ void gather_fp64(const Geom& g, int cx, int cy, int cz, double scale, double x, double y,
                                         double z, double* F) {
    for (int q = 0; q < 6; ++q) {
        double f = 0.0;
        for (int k = 0; k < 8; ++k) {
            const double w = ((k & 1) ? 0.5 + x : 0.5 - x) * ((k & 2) ? 0.5 + y : 0.5 - y) *
                             ((k & 4) ? 0.5 + z : 0.5 - z);
            f = __fma_rn(corner_field(g, cx, cy, cz, k)[q], w, f);
        }
        F[q] = f * scale;
    }
}

// ---- mover ----------------------------------------------------------------------

// Boris rotations and positions (particle.h:24-49), fused: ns sub-cycles of
// dts, k = q/m dts / 2.
__device__ __forceinline__ void boris64(const double (&F)[6], double k, double dts, int ns, PState<double>& p) {
    const double tx = __dmul_rn(k, F[3]), ty = __dmul_rn(k, F[4]), tz = __dmul_rn(k, F[5]);
    const double den = __fma_rn(tx, tx, __fma_rn(ty, ty, __fma_rn(tz, tz, 1.0)));
    const double y = reciprocal(den), f = __dadd_rn(y, y);
    const double sx = __dmul_rn(tx, f), sy = __dmul_rn(ty, f), sz = __dmul_rn(tz, f);
    for (int s = 0; s < ns; ++s) {
        const double mx = __fma_rn(k, F[0], p.u), my = __fma_rn(k, F[1], p.v), mz = __fma_rn(k, F[2], p.w);
        const double px = __fma_rn(my, tz, __fma_rn(-mz, ty, mx));
        const double py = __fma_rn(mz, tx, __fma_rn(-mx, tz, my));
        const double pz = __fma_rn(mx, ty, __fma_rn(-my, tx, mz));
        p.u = __fma_rn(k, F[0], __fma_rn(py, sz, __fma_rn(-pz, sy, mx)));
        p.v = __fma_rn(k, F[1], __fma_rn(pz, sx, __fma_rn(-px, sz, my)));
        p.w = __fma_rn(k, F[2], __fma_rn(px, sy, __fma_rn(-py, sx, mz)));
        p.x = __fma_rn(p.u, dts, p.x);
        p.y = __fma_rn(p.v, dts, p.y);
        p.z = __fma_rn(p.w, dts, p.z);
    }
}

// The field mover's step from the gathered E, B in F.
__device__ __forceinline__ void move_field64(const Geom& g, const Push64Const& pc, double qom, double (&F)[6],
                                             PState<double>& p) {
    if (g.flags & 4u /*IPIC3D_F_DIPOLE_IN_GATHER*/) {
        const double r2 = __fma_rn(p.x, p.x, __fma_rn(p.y, p.y, __dmul_rn(p.z, p.z)));
        // mft / r2^2.5 on the integer pipe
        double f;
        if (pc.d.usable && soft::regular(r2, 200)) {
            bool sure;  // either neighbour will do where it is not
            f = soft::pack(soft::div(pc.d.mft, soft::divisor(soft::pow25(soft::unpack(r2), sure))));
        } else {
            f = __dmul_rn(g.mft, inverse_pow25(r2));
        }
        const double z3 = __dmul_rn(3.0, p.z), zf = __dmul_rn(z3, f);
        F[3] = __fma_rn(p.x, zf, F[3]);
        F[4] = __fma_rn(p.y, zf, F[4]);
        F[5] = __fma_rn(__fma_rn(z3, p.z, -r2), f, F[5]);
    }
    // one sub-cycle is sure below an exponent; else the reference's rule
    const int e = max(max(soft::exponent_of(F[3]), soft::exponent_of(F[4])), soft::exponent_of(F[5]));
    if (e <= pc.d.e_max) {
        boris64(F, pc.k1, g.dt, 1, p);
    } else {
        double dts;
        const double bmag = (F[3] * F[3] + F[4] * F[4]) + F[5] * F[5];
        const int ns = sub_cycles_dt(g.dt, g.c, g.inv_pic, qom, bmag, dts);
        boris64(F, qom * 0.5 * dts, dts, ns, p);
    }
}

// The dipole mover's step (cell.h:939-960), rounded as the reference's.
__device__ __forceinline__ void move_dipole64(const Geom& g, const Push64Const& pc, double qom, PState<double>& p) {
    if (pc.d.usable && coordinates_regular(p.x, p.y, p.z) &&
        dipole_rotate(pc.d, p.x, p.y, p.z, squared_position(p.x, p.y, p.z), p.u, p.v, p.w)) {
        advance_position(p.x, p.y, p.z, p.u, p.v, p.w, g.dt);
        return;
    }
    double r2 = p.x * p.x;
    r2 += p.y * p.y;
    r2 += p.z * p.z;
    const double fac1 = g.mft / pow25_rn(r2);
    const double bx = 3.0 * p.x * p.z * fac1;
    const double by = 3.0 * p.y * p.z * fac1;
    const double bz = (2.0 * (p.z * p.z) - (p.x * p.x) - (p.y * p.y)) * fac1;
    double bmag = bx * bx;
    bmag += by * by;
    bmag += bz * bz;
    double dts;
    const int ns = sub_cycles_dt(g.dt, g.c, g.inv_pic, qom, bmag, dts);
    for (int s = 0; s < ns; ++s) {
        boris_e0(p.u, p.v, p.w, bx, by, bz, qom, dts);
        p.x = p.x + p.u * dts;  // updatePosition (particle.h:24-26)
        p.y = p.y + p.v * dts;
        p.z = p.z + p.w * dts;
    }
}

// ---- export ---------------------------------------------------------------------

// A particle's cell: its coordinates, centre (getCenterOfCell,
// universe_properties.h:139-142), and what the export can leave out.
struct Cell64 {
    int x, y, z;
    double cen[3];
    bool near_planet;  // the planet can reach a particle that stays in the cell
    bool far_planet;   // it cannot reach one that is at most a cell away
    bool edge;         // a face of the cell lies on the domain boundary
};

__device__ __forceinline__ double cell_centre(const Geom& g, int a, int pos) {
    return (g.origin[a] + (double)pos * g.w[a]) + g.half_w[a];
}
// Distance along axis a from the planet's centre to the cell's box, in FP32;
// the comparison with planet_reach adds the margin.
__device__ __forceinline__ float planet_gap(const Geom& g, int a, double cen) {
    return fabsf((float)(cen - g.object_center[a])) - (float)g.half_w[a];
}
// A particle further than this from the planet's centre is outside the planet
// whatever the rounding (a 64th of a cell and 10^-5 of the radius of margin).
__device__ __forceinline__ float planet_reach(const Geom& g) {
    const float w = fmaxf(fmaxf((float)g.w[0], (float)g.w[1]), (float)g.w[2]);
    return sqrtf((float)g.planet_r2) * 1.00001f + w * (1.f / 64.f);
}
// The flags from the three gaps (NaN and overflow: near, not far).
__device__ __forceinline__ void planet_flags(const Geom& g, const float (&gap)[3], float reach, Cell64& c) {
    float in2 = 0.f, out2 = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float in = fmaxf(gap[a], 0.f), out = fmaxf(gap[a] - (float)g.w[a], 0.f);
        in2 += in * in;
        out2 += out * out;
    }
    c.near_planet = !(in2 > reach * reach);
    c.far_planet = out2 > reach * reach;
    c.edge = c.x == 0 || c.y == 0 || c.z == 0 || c.x == g.sx - 1 || c.y == g.sy - 1 || c.z == g.sz - 1;
}

__device__ __forceinline__ uint64_t magnitude_bits(double x) { return soft::bits_of(x) & 0x7fffffffffffffffull; }
// |x| > lim (lim >= 0); false for NaN, as the FP64 comparison
__device__ __forceinline__ bool beyond(double x, double lim) {
    const uint64_t b = magnitude_bits(x);
    return b > soft::bits_of(lim) && b <= 0x7ff0000000000000ull;
}
__device__ __forceinline__ bool is_negative(double x) { return (int64_t)soft::bits_of(x) < 0; }

// The rare parts of the export sit behind calls, so that the FP64
// instructions of all of them are not issued for every leaver.
struct Walled {
    double p;
    int inverts, drops;
};
// The wall rule of one axis (cell.h:1102-1121): reflecting faces shift by half
// a cell and invert the velocity, open ones drop.
__device__ __noinline__ Walled wall64(double p, double rel, double half, int pos, int size, int lo, int hi) {
    Walled r = {p, 0, 0};
    if (!beyond(rel, half)) return r;
    const bool low = is_negative(rel);
    const int bc = low ? (pos == 0 ? lo : 1) : (pos == size - 1 ? hi : 1);
    r.drops = bc == 2;
    r.inverts = bc == 0;
    if (bc == 0) r.p = low ? p + half : p - half;
    return r;
}
__device__ __noinline__ bool inside_planet64(double dx, double dy, double dz, double limit) {
    double r2 = dx * dx;
    r2 += dy * dy;
    r2 += dz * dz;
    return r2 <= limit;  // cell.h:1123-1128
}
__device__ __noinline__ double wrap64(double p, double length, int periodic) { return periodic ? p + length : p; }

// exportParticles (cell.h:1093-1146) for a moved particle: walls, planet,
// move to a neighbour. rel: the position relative to the cell's centre.
__device__ __forceinline__ int export64(const Geom& g, const Cell64& c, PState<double>& p, double (&rel)[3],
                                        int& dest) {
    rel[0] = p.x - c.cen[0];
    rel[1] = p.y - c.cen[1];
    rel[2] = p.z - c.cen[2];
    if (!c.near_planet && magnitude_bits(rel[0]) <= soft::bits_of(g.half_w[0]) &&
        magnitude_bits(rel[1]) <= soft::bits_of(g.half_w[1]) && magnitude_bits(rel[2]) <= soft::bits_of(g.half_w[2]))
        return kStay;
    const int pos[3] = {c.x, c.y, c.z}, size[3] = {g.sx, g.sy, g.sz};
    double P[3] = {p.x, p.y, p.z};
    if (c.edge) {
        int inverts = 0, drops = 0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const Walled r = wall64(P[a], rel[a], g.half_w[a], pos[a], size[a], g.bc_lo[a], g.bc_hi[a]);
            P[a] = r.p;
            inverts |= r.inverts;
            drops |= r.drops;
        }
        if (inverts) {
            p.u = soft::from_bits(soft::bits_of(p.u) ^ 0x8000000000000000ull);
            p.v = soft::from_bits(soft::bits_of(p.v) ^ 0x8000000000000000ull);
            p.w = soft::from_bits(soft::bits_of(p.w) ^ 0x8000000000000000ull);
        }
        if (drops) return kDrop;
        rel[0] = P[0] - c.cen[0];
        rel[1] = P[1] - c.cen[1];
        rel[2] = P[2] - c.cen[2];
    }
    // the planet: settled by the cell for a particle within a cell width of
    // its centre
    if (!(c.far_planet && magnitude_bits(rel[0]) <= soft::bits_of(g.w[0]) &&
          magnitude_bits(rel[1]) <= soft::bits_of(g.w[1]) && magnitude_bits(rel[2]) <= soft::bits_of(g.w[2])) &&
        inside_planet64(P[0] - g.object_center[0], P[1] - g.object_center[1], P[2] - g.object_center[2],
                        g.planet_r2))
        return kDrop;
    int n[3];
    bool out = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        int t = pos[a];
        if (beyond(rel[a], g.half_w[a])) {
            out = true;
            t += is_negative(rel[a]) ? -1 : 1;
            if (t < 0) {
                t += size[a];
                P[a] = wrap64(P[a], g.L[a], g.bc_lo[a] == 1);
            } else if (t >= size[a]) {
                t -= size[a];
                P[a] = wrap64(P[a], -g.L[a], g.bc_hi[a] == 1);
            }
        }
        n[a] = t;
    }
    p.x = P[0];
    p.y = P[1];
    p.z = P[2];
    if (!out) return kStay;
    dest = cell_id(g, n[0], n[1], n[2]);
    return kMove;
}

// ---- one particle of any cell (those that waited for a slot) ---------------------
// The same operations as the bulk push, so that a particle's arithmetic does
// not depend on the path it takes.
__device__ __forceinline__ int step_one64(const Geom& g, const Push64Const& pc, int cell, double qom,
                                          PState<double>& p, int& dest) {
    Cell64 c;
    cell_coords(g, cell, c.x, c.y, c.z);
    const int pos[3] = {c.x, c.y, c.z};
    float gap[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        c.cen[a] = cell_centre(g, a, pos[a]);
        gap[a] = planet_gap(g, a, c.cen[a]);
    }
    planet_flags(g, gap, planet_reach(g), c);
    if (g.mover == 1) {
        const double x = (p.x - c.cen[0]) * g.inv_w[0], y = (p.y - c.cen[1]) * g.inv_w[1],
                     z = (p.z - c.cen[2]) * g.inv_w[2];
        double F[6];
        bool fixed = in_cell(x) && in_cell(y) && in_cell(z);
        int e_max[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            int e = 0;
            bool zero = true;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const double v = field_value(pc, __ldg(corner_field(g, c.x, c.y, c.z, k) + q));
                e = max(e, soft::exponent_of(v));
                zero = zero && (soft::bits_of(v) << 1) == 0;
            }
            e_max[q] = e;
            fixed = fixed && fixed_range(e) && (e != 0 || zero);
        }
        if (fixed) {
            const uint64_t rx = fraction(x), ry = fraction(y), rz = fraction(z);
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                int64_t v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    v[k] = to_fixed(field_value(pc, __ldg(corner_field(g, c.x, c.y, c.z, k) + q)), e_max[q]);
#pragma unroll
                for (int bit = 1; bit < 8; bit <<= 1)
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (k & bit) v[k] -= v[k ^ bit];
                F[q] = from_fixed(poly_fixed(v, rx, ry, rz), e_max[q]);
            }
        } else {
            gather_fp64(g, c.x, c.y, c.z, pc.field_scale, x, y, z, F);
        }
        move_field64(g, pc, qom, F, p);
    } else {
        move_dipole64(g, pc, qom, p);
    }
    double rel[3];
    return export64(g, c, p, rel, dest);
}

// ---- the bulk push ---------------------------------------------------------------
constexpr int kMaxSpan64 = 4;

// A block's dynamic shared memory: the cells of its span, their coefficients
// per group.
struct Push64Smem {
    int64_t* start;  // [cells + 1]
    int64_t* coef;   // [groups][kCoefStride64]
    int* count;      // [cells]
    int* first;      // [cells + 1] items before the cell's
};
__host__ __device__ constexpr size_t push64_smem_bytes(int span, int warps) {
    const int cells = span * kMaxCellsPerCta;
    return (size_t)(cells + 2) / 2 * 2 * sizeof(int64_t) + (size_t)warps * kWarpItems64 * kCoefStride64 * sizeof(double) +
           (size_t)(2 * cells + 1) * sizeof(int);
}
__device__ __forceinline__ Push64Smem push64_smem(int span, int warps) {
    extern __shared__ __align__(16) unsigned char push64_raw[];
    const int cells = span * kMaxCellsPerCta;
    Push64Smem sm;
    sm.start = reinterpret_cast<int64_t*>(push64_raw);
    sm.coef = sm.start + (cells + 2) / 2 * 2;  // 16-byte aligned
    sm.count = reinterpret_cast<int*>(sm.coef + warps * kWarpItems64 * kCoefStride64);
    sm.first = sm.count + cells;
    return sm;
}

// Slots [lo, hi) of cell i that belong to the block's span [base, top).
__device__ __forceinline__ void span_range64(const Push64Smem& sm, int i, int64_t base, int64_t top, int64_t& lo,
                                             int64_t& hi) {
    const int64_t s = sm.start[i];
    lo = s;
    hi = s + sm.count[i];
    if (sm.start[i + 1] - s > kSlotsPerCta) {
        lo = max(lo, base);
        hi = min(hi, top);
    } else if (s < base) {
        hi = lo;
    }
    if (hi < lo) hi = lo;
}

// Bookkeeping of the warp's leavers and drops of one round: outbox, arrival
// lists, holes (a group's slots are of one cell: one atomic per group). The
// round trips -- hole slots, arrival slots, outbox slots -- are issued
// together before any result is used: in the .inp run every round has
// leavers.
__device__ __forceinline__ void leave64(const Geom& g, const Pop<double>& P, int outcome, int cell, int64_t cstart,
                                        int64_t slot, int dest, const PState<double>& p, bool deposit,
                                        uint32_t& nmig, uint32_t& nrem) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, gl = lane & (kGroup64 - 1);
    const unsigned below = (1u << lane) - 1u, group = 0xffu << (lane & ~(kGroup64 - 1));
    const bool leave = outcome == kMove, hole = leave || outcome == kDrop;
    const unsigned lb = __ballot_sync(kAll, leave), hb = __ballot_sync(kAll, hole) & group;
    int hk = 0, ak = 0;
    if (hb && gl == 0) hk = atomicAdd(P.hole_cnt + cell, __popc(hb));
    uint32_t o = 0, id = 0u;
    int64_t ds = 0, de = 0;
    if (leave) {
        ak = atomicAdd(P.arr_cnt + dest, 1);
        ds = P.start[dest];
        de = P.start[dest + 1];
        if (P.id) id = P.id[slot];
    }
    if (lb && lane == 0) o = atomicAdd(&P.ctr->outbox, (uint32_t)__popc(lb));
    o = __shfl_sync(kAll, o, 0) + __popc(lb & below);
    if (leave) {
        Mover<double> m;
        m.cell = dest;
        m.id = id;
        m.x = p.x; m.y = p.y; m.z = p.z;
        m.u = p.u; m.v = p.v; m.w = p.w;
        const bool in_box = o < P.outbox_cap;  // sized for one entry per slot: never full
        if (in_box) P.outbox[o] = m;
        else atomicAdd(&P.ctr->lost, 1u);
        if (ak < (int)(de - ds)) {
            P.arr_list[ds + ak] = in_box ? (int32_t)o : 0;
        } else {  // the destination's slots are short: wait a step
            const uint32_t pi = atomicAdd(&P.ctr->pending_out, 1u);
            if (pi < P.pending_cap) P.pending_out[pi] = m;
            else atomicAdd(&P.ctr->lost, 1u);
        }
        ++nmig;
    }
    hk = __shfl_sync(kAll, hk, 0, kGroup64) + __popc(hb & below);
    if (hole) P.hole_list[cstart + hk] = (int32_t)slot;
    if (outcome == kDrop) ++nrem;
    if (deposit && lb) warp_deposit_leavers<double>(g, leave, dest, p, P.q);
}

// kStep: mover + export (else the deposit of the particles as they are);
// kField: field-gather mover (else the dipole mover); kDep: deposit.
template <bool kStep, bool kField, bool kDep>
__device__ __forceinline__ void push64_body(const Geom& g, const Pop<double>& P, const Push64Const& pc, int64_t tile,
                                            int span, int part, int parts, int item) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int gl = lane & (kGroup64 - 1), sub = lane / kGroup64;
    const Push64Smem sm = push64_smem(span, warps);
    // the cells of the span: consecutive tiles' cells follow one another
    const int64_t base = tile * kSlotsPerCta, top = min(base + (int64_t)span * kSlotsPerCta, P.capacity);
    const int2 cc = __ldg(P.cta_cells + tile), ce = __ldg(P.cta_cells + (top - 1) / kSlotsPerCta);
    const int c0 = cc.x, nc = ce.x + ce.y - cc.x;
    for (int i = threadIdx.x; i <= nc; i += blockDim.x) sm.start[i] = P.start[c0 + i];
    for (int i = threadIdx.x; i < nc; i += blockDim.x) sm.count[i] = P.count[c0 + i];
    __syncthreads();
    if (warp == 0) {  // items before each cell
        int before = 0;
        for (int b = 0; b < nc; b += 32) {
            const int i = b + lane;
            int n = 0;
            if (i < nc) {
                int64_t lo, hi;
                span_range64(sm, i, base, top, lo, hi);
                n = ((int)(hi - lo) + item - 1) / item;
            }
            int incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(kAll, incl, o);
                if (lane >= o) incl += t;
            }
            if (i < nc) sm.first[i] = before + incl - n;
            before += __shfl_sync(kAll, incl, 31);
        }
        if (lane == 0) sm.first[nc] = before;
    }
    __syncthreads();
    const int total = sm.first[nc];
    int64_t* const coef = sm.coef + (warp * kWarpItems64 + sub) * kCoefStride64;
    const float reach = planet_reach(g);
    uint32_t nmig = 0, nrem = 0;

    for (int j0 = (part * warps + warp) * kWarpItems64; j0 < total; j0 += parts * warps * kWarpItems64) {
        const int j = min(j0 + sub, total - 1);
        int i = 0;
        {
            int hi = nc - 1;
            while (i < hi) {
                const int mid = (i + hi + 1) >> 1;
                if (sm.first[mid] <= j) i = mid; else hi = mid - 1;
            }
        }
        int64_t lo, end;
        span_range64(sm, i, base, top, lo, end);
        const int pieces = sm.first[i + 1] - sm.first[i];
        const int piece = ((int)(end - lo) + pieces * kGroup64 - 1) / (pieces * kGroup64) * kGroup64;
        const int64_t a = lo + (int64_t)(j - sm.first[i]) * piece;
        int len = max(0, (int)min((int64_t)piece, end - a));
        if (j0 + sub >= total) len = 0;
        const int cell = c0 + i;
        const int64_t cstart = sm.start[i];
        Cell64 c;
        cell_coords(g, cell, c.x, c.y, c.z);
        {   // lane 0, 1, 2 of the group: the axis' centre
            const double cen = gl < 3 ? cell_centre(g, gl, gl == 0 ? c.x : gl == 1 ? c.y : c.z) : 0.0;
            const float mine = gl < 3 ? planet_gap(g, gl, cen) : 0.f;
            float gap[3];
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                c.cen[b] = __shfl_sync(kAll, cen, b, kGroup64);
                gap[b] = __shfl_sync(kAll, mine, b, kGroup64);
            }
            planet_flags(g, gap, reach, c);
        }
        // lane k: corner k, then coefficient k; the components' exponents in
        // pairs (every lane of the group has them)
        uint32_t exps[3] = {0u, 0u, 0u};
        bool fixed = true;
        if (kStep && kField) {
            const double* f = corner_field(g, c.x, c.y, c.z, gl);
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                const double v = field_value(pc, __ldg(f + q));
                int e = soft::exponent_of(v);
                bool zero = (soft::bits_of(v) << 1) == 0;
#pragma unroll
                for (int bit = 1; bit < 8; bit <<= 1) e = max(e, __shfl_xor_sync(kAll, e, bit));
                fixed = fixed && fixed_range(e) && (e != 0 || zero);
                int64_t n = to_fixed(v, e);
#pragma unroll
                for (int bit = 1; bit < 8; bit <<= 1) {
                    const int64_t o = __shfl_xor_sync(kAll, n, bit);
                    if (gl & bit) n -= o;
                }
                coef[q * 8 + gl] = n;
                exps[q >> 1] |= (uint32_t)e << (16 * (q & 1));
            }
            fixed = (__ballot_sync(kAll, fixed) >> (sub * kGroup64) & 0xffu) == 0xffu;
            __syncwarp();
        }
        double acc[kDep ? 32 : 1];
        if (kDep) {
#pragma unroll
            for (int l = 0; l < 32; ++l) acc[l] = 0.0;
        }
        int stay = 0;
        const int rounds = __reduce_max_sync(kAll, (len + kGroup64 - 1) / kGroup64);
        for (int r = 0; r < rounds; ++r) {
            const int k = r * kGroup64 + gl;
            const bool has = k < len;
            const int64_t slot = a + k;
            // lanes without a particle: the cell's centre at rest, which adds
            // nothing to the moments but the count, taken apart
            PState<double> p = {c.cen[0], c.cen[1], c.cen[2], 0.0, 0.0, 0.0};
            if (has) p = {P.x[slot], P.y[slot], P.z[slot], P.u[slot], P.v[slot], P.w[slot]};
            double rel[3];
            if (kStep) {
                if (kField) {
                    const double x = (p.x - c.cen[0]) * g.inv_w[0], y = (p.y - c.cen[1]) * g.inv_w[1],
                                 z = (p.z - c.cen[2]) * g.inv_w[2];
                    double F[6];
                    if (fixed && in_cell(x) && in_cell(y) && in_cell(z)) {
                        const uint64_t rx = fraction(x), ry = fraction(y), rz = fraction(z);
#pragma unroll
                        for (int q = 0; q < 6; ++q)
                            F[q] = from_fixed(poly_fixed(coef + 8 * q, rx, ry, rz),
                                              (int)(exps[q >> 1] >> (16 * (q & 1)) & 0xffffu));
                    } else {
                        double T[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
                        if (has) gather_fp64(g, c.x, c.y, c.z, pc.field_scale, x, y, z, T);
#pragma unroll
                        for (int q = 0; q < 6; ++q) F[q] = T[q];
                    }
                    move_field64(g, pc, P.qom, F, p);
                } else if (has) {
                    move_dipole64(g, pc, P.qom, p);
                }
                int dest = cell;
                int outcome = has ? export64(g, c, p, rel, dest) : -1;
                if (outcome == kStay) {
                    P.x[slot] = p.x; P.y[slot] = p.y; P.z[slot] = p.z;
                    P.u[slot] = p.u; P.v[slot] = p.v; P.w[slot] = p.w;
                }
                if (__any_sync(kAll, outcome > kStay))
                    leave64(g, P, outcome, cell, cstart, slot, dest, p, kDep, nmig, nrem);
                if (kDep) {
                    stay += outcome == kStay;
                    if (outcome != kStay) {
                        rel[0] = rel[1] = rel[2] = 0.0;
                        p.u = p.v = p.w = 0.0;
                    }
                }
            } else {
                rel[0] = p.x - c.cen[0];
                rel[1] = p.y - c.cen[1];
                rel[2] = p.z - c.cen[2];
                stay += has;
            }
            if (kDep) {
                const double x = rel[0] * g.inv_w[0], y = rel[1] * g.inv_w[1], z = rel[2] * g.inv_w[2];
                const double xy = x * y, xz = x * z, yz = y * z;
                const double M[8] = {1.0, x, y, xy, z, xz, yz, xy * z};
                const double Q[3] = {p.u, p.v, p.w};
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    acc[8 * q] = acc[8 * q] + Q[q];
#pragma unroll
                    for (int m = 1; m < 8; ++m) acc[8 * q + m] = __fma_rn(Q[q], M[m], acc[8 * q + m]);
                }
#pragma unroll
                for (int m = 1; m < 8; ++m) acc[24 + m] = acc[24 + m] + M[m];
            }
        }
        if (kDep) {
            // over the group's lanes: lane m is left with moment m of each Q
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int off = 4; off >= 1; off >>= 1) {
                    const bool up = (gl & off) != 0;
#pragma unroll
                    for (int m = 0; m < off; ++m) {
                        const double send = up ? acc[8 * q + m] : acc[8 * q + m + off];
                        const double keep = up ? acc[8 * q + m + off] : acc[8 * q + m];
                        acc[8 * q + m] = keep + __shfl_xor_sync(kAll, send, off);
                    }
                }
            stay = __reduce_add_sync(0xffu << (sub * kGroup64), stay);
            if (gl == 0) acc[24] = (double)stay;
            // moments -> corner sums (weights 1/2 -+ s), one axis at a time
#pragma unroll
            for (int bit = 1; bit < 8; bit <<= 1)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const double o = __shfl_xor_sync(kAll, acc[8 * q], bit);
                    acc[8 * q] = (gl & bit) ? __fma_rn(0.5, o, acc[8 * q]) : __fma_rn(0.5, acc[8 * q], -o);
                }
            if (stay > 0) {
                const int64_t n =
                    node_index(g, c.x + (gl & 1), c.y + ((gl >> 1) & 1), c.z + (gl >> 2));
#pragma unroll
                for (int q = 0; q < 3; ++q) atomicAdd(g.J + 3 * n + q, P.q * acc[8 * q]);
                atomicAdd(g.rho + n, P.q * acc[24]);
            }
        }
    }
    if (kStep) {
        nmig = __reduce_add_sync(kAll, nmig);
        nrem = __reduce_add_sync(kAll, nrem);
        if (lane == 0) {
            if (nmig) atomicAdd(&P.ctr->migrated, nmig);
            if (nrem) atomicAdd(&P.ctr->removed, nrem);
        }
    }
}

// Block (span, part) of population blockIdx.z of the set.
template <bool kStep, bool kField, bool kDep>
__global__ void __launch_bounds__(32 * kMaxWarps64, kDep ? 3 : 5)
    k_push64(Geom g, const __grid_constant__ PopSet<double> S, const __grid_constant__ Push64Set pcs, int span,
             int item) {
    const Pop<double>& P = S.p[blockIdx.z];
    const int64_t tile = (int64_t)blockIdx.x * span;
    if (tile * kSlotsPerCta >= P.capacity) return;
    push64_body<kStep, kField, kDep>(g, P, pcs.c[blockIdx.z], tile, span, blockIdx.y, gridDim.y, item);
}

// Batched: cta_job[blockIdx.x] = (job, tile of the job); the span starts at
// every span-th tile of a job.
template <bool kStep, bool kField, bool kDep>
__global__ void __launch_bounds__(32 * kMaxWarps64, kDep ? 3 : 5)
    k_push64_batch(const PopJob<double>* __restrict__ jobs, const int2* __restrict__ cta_job, int span, int item) {
    __shared__ PopJob<double> job;
    const int2 cj = __ldg(cta_job + blockIdx.x);
    if (cj.y % span != 0) return;
    load_job(job, jobs + cj.x);
    push64_body<kStep, kField, kDep>(job.g, job.P, job.pc, cj.y, span, blockIdx.y, gridDim.y, item);
}

// ---- particles that waited for a slot ---------------------------------------------
// Entries t0, t0 + stride, ... of the pending list.
__device__ __forceinline__ void push_pending64_body(const Geom& g, const Pop<double>& P, const Push64Const& pc,
                                                    uint32_t t0, uint32_t stride) {
    const uint32_t n = *P.pending_in_count;
    const double q = P.q;
    for (uint32_t i = t0; i < n; i += stride) {
        const Mover<double> m = P.pending_in[i];
        PState<double> p = {m.x, m.y, m.z, m.u, m.v, m.w};
        int dest = m.cell;
        const int outcome = step_one64(g, pc, m.cell, P.qom, p, dest);
        if (outcome == kDrop) {
            atomicAdd(&P.ctr->removed, 1u);
            continue;
        }
        if (outcome == kMove) atomicAdd(&P.ctr->migrated, 1u);
        const Mover<double> o = {dest, m.id, p.x, p.y, p.z, p.u, p.v, p.w};
        const uint32_t k = atomicAdd(&P.ctr->outbox, 1u);
        if (k < P.outbox_cap) {
            P.outbox[k] = o;
            register_arrival(P, k, o);
        } else {
            atomicAdd(&P.ctr->lost, 1u);
        }
        if (g.deposit) deposit_one<double>(g, dest, p, q);
    }
}

__global__ void k_push_pending64(Geom g, const __grid_constant__ PopSet<double> S,
                                 const __grid_constant__ Push64Set pcs) {
    push_pending64_body(g, S.p[blockIdx.y], pcs.c[blockIdx.y], blockIdx.x * blockDim.x + threadIdx.x,
                        gridDim.x * blockDim.x);
}

__global__ void k_push_pending64_batch(const PopJob<double>* __restrict__ jobs) {
    const PopJob<double>& J = jobs[blockIdx.y];
    push_pending64_body(J.g, J.P, J.pc, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

}  // namespace ipg
