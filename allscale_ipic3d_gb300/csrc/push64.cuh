// The FP64 push: mover (cell.h:896-964) + export (cell.h:975-1159) in place,
// fused with the cloud-in-cell deposit (cell.h:787-824, scatter form).
//
// GB300's FP64 pipe bounds it (one warp instruction per 64 to 76 cycles and
// SM sub-partition), so what counts is the number of FP64 instructions a
// warp issues -- idle lanes cost as much as busy ones -- then how many warps
// there are to fill the gaps, and the size of the loop (four or five warps a
// sub-partition, each elsewhere in it, share the instruction cache). Per 32
// particles of a step with field gather, dipole and deposit:
//   * the field is the cell's trilinear polynomial, built once per work item
//     from the 8 corners, and the deposit the moments of the work item's
//     particles: both in 64-bit fixed point on the integer pipe (poly_fixed,
//     Moments64);
//   * the dipole's |r|^-5 on the integer pipe (fp64_int.cuh), the rotation's
//     2 / (1 + |t|^2) without a division (the export test keeps the
//     reference's own differences from the cell centre);
//   * comparisons run on the doubles' bit patterns in the integer pipe;
//   * rare parts (walls, planet, sub-cycles, positions outside the cell) are
//     calls: predicated off they would still take the FP64 pipe.
// 62 FP64 instructions (items' shares and idle lanes included) and 2,700
// others in place of 541 FP64 ones before. The dipole mover without the
// gather rounds exactly as the reference does (dipole64.cuh). Measured push
// per step, before and after: 8.4M particles, gather + dipole + deposit
// 9.18 -> 1.30 ms (FP64 pipe 66 % busy, issue slots 46 %); 306k particles,
// two species, gather + deposit 0.593 -> 0.085 ms; 33k particles 0.140 ->
// 0.022 ms (a warp's serial chain); 1.05M particles, dipole mover, a sixth of
// them leaving their cells 0.489 -> 0.150 ms (FP64 pipe 58 %, integer 42 %).
// Loading a round's particles a round ahead changed nothing.
//
// Work. A work item is up to `item` particles of one cell, pushed by a group
// of 8 lanes, 8 particles at a time (slots are 8-aligned: full 64-byte
// segments); four items share a warp. Groups of 8 rather than whole warps
// keep the lanes busy where cells hold few particles or end unevenly, at the
// price of a reduction per 8 lanes; a cell of more than `item` particles is
// cut evenly, so that the items of a warp end together. The push and the
// moments are two passes over an item: their registers are not live together,
// and the second knows the components' exponents (one pass: 168 registers,
// 12 warps per SM; two: 128 and 16, 2.02 -> 1.87 ms, the particles' second
// read from L1 and L2). A block is one warp, which takes the items of `span`
// consecutive 1024-slot tiles, or every gridDim.y-th four of them: cells of
// up to a tile belong to the span they start in, larger ones are cut at its
// boundaries. Short items with the deposit: blocks of four warps (Joint64).
#pragma once

#include "dipole64.cuh"

namespace ipg {

constexpr int kGroup64 = 8;
constexpr int kWarpItems64 = 32 / kGroup64;  // work items of a warp at a time
constexpr int kCoefStride64 = 50;  // 48 + 2: the four groups of a warp read different banks

// ---- field --------------------------------------------------------------------

// 1 / d from the FP64 unit's approximation (relative error below 2^-20).
__device__ __forceinline__ double reciprocal(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    return soft::refine_reciprocal(d, y);
}

// mft / r2^2.5 out of the integer path's range.
__device__ __noinline__ double dipole_factor(double mft, double r2) { return mft / pow25_rn(r2); }

// The field of a cell in 64-bit fixed point. A component's 8 corner values
// share the largest one's exponent e_max: fixed = value 2^(1081 - e_max), below
// 2^59, so that one unit is 2^-59 of the largest corner (FP64's own rounding
// is 2^-53 of it; a corner below 2^-6 of the largest keeps fewer than 53 bits,
// which shows only at positions that the others hardly reach). The trilinear
// polynomial's coefficients are differences of these integers, exact, and the
// position in the cell is a 64-bit fraction: a product is the high half of 64
// x 64 bits. Seven of them and seven sums per component take about 150
// integer-pipe cycles per warp; the seven FP64 multiply-adds they replace took
// 448 of the FP64 pipe, which bounds the push.

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
// q times the same, rounded once
__device__ __forceinline__ double times_fixed(double q, int64_t v, int e_max) {
    const soft::Num c = soft::unpack(q);
    const uint64_t a = v < 0 ? (uint64_t)-v : (uint64_t)v;
    int n = __clzll((long long)a);
    uint64_t p = __umul64hi(a << (n & 63), c.m << 11);
    if ((int64_t)p >= 0) {
        p <<= 1;
        ++n;
    }
    soft::Num r;
    r.m = (p >> 11) + ((p >> 10) & 1);
    r.e = e_max + c.e - 1017 - n;
    r.sign = (v < 0 ? 0x80000000u : 0u) ^ c.sign;
    if (v == 0 || c.e == 0 || c.e == 2047 || r.e < 1 || r.e > 2045) return q * from_fixed(v, e_max);
    return soft::pack(r);
}
// e_max a component may have (0: all corners are zero); others take FP64
__device__ __forceinline__ bool fixed_range(int e_max) { return e_max == 0 || (uint32_t)(e_max - 200) <= 1600u; }

// A coordinate about the cell's centre as the fraction (1/2 + rel / w) 2^64
// of the cell, inv = 1 / w; only where |rel| <= w / 2 (in_cell).
__device__ __forceinline__ uint64_t magnitude_bits(double x) { return soft::bits_of(x) & 0x7fffffffffffffffull; }
__device__ __forceinline__ bool in_cell(const Geom& g, const double (&rel)[3]) {
    return magnitude_bits(rel[0]) <= soft::bits_of(g.half_w[0]) &&
           magnitude_bits(rel[1]) <= soft::bits_of(g.half_w[1]) &&
           magnitude_bits(rel[2]) <= soft::bits_of(g.half_w[2]);
}
__device__ __forceinline__ uint64_t fraction(double rel, double inv) {
    const soft::Num n = soft::unpack(rel), w = soft::unpack(inv);
    const uint64_t p = __umul64hi(n.m << 11, w.m << 11);
    const int sh = 2044 - n.e - w.e;  // |rel| / w 2^64 = p 2^-sh, sh >= -1
    constexpr uint64_t kHalf = 1ull << 63;
    uint64_t t = n.e == 0 || sh > 63 ? 0 : sh >= 0 ? p >> sh : p << 1;
    t = min(t, kHalf);  // (the rounding of 1 / w)
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

// Component q of E, B at (rx, ry, rz) from the centre of a cell, by one
// thread in FP64: the positions outside the cell (a particle that crossed
// more than a cell) and the values out of the fixed-point range.
__device__ __noinline__ double gather_fp64(const Geom& g, int cx, int cy, int cz, double scale, double rx, double ry,
                                           double rz, int q) {
    const double x = rx * g.inv_w[0], y = ry * g.inv_w[1], z = rz * g.inv_w[2];
    double f = 0.0;
    for (int k = 0; k < 8; ++k) {
        const double w = ((k & 1) ? 0.5 + x : 0.5 - x) * ((k & 2) ? 0.5 + y : 0.5 - y) *
                         ((k & 4) ? 0.5 + z : 0.5 - z);
        f = __fma_rn(corner_field(g, cx, cy, cz, k)[q], w, f);
    }
    return f * scale;
}

// ---- mover ----------------------------------------------------------------------

// Boris rotations and positions (particle.h:24-49), fused: ns sub-cycles of
// dts, k = q/m dts / 2. The rotation v- + (v- + v- x t) x s, s = t f, is
// taken as v- + f (w + w x t), w = v- x t: three roundings of the velocity's
// size per sub-cycle and no s.
__device__ __forceinline__ void boris64(const double (&F)[6], double k, double dts, int ns, PState<double>& p) {
    const double tx = __dmul_rn(k, F[3]), ty = __dmul_rn(k, F[4]), tz = __dmul_rn(k, F[5]);
    const double den = __fma_rn(tx, tx, __fma_rn(ty, ty, __fma_rn(tz, tz, 1.0)));
    const double y = reciprocal(den), f = __dadd_rn(y, y);
#pragma unroll 1
    for (int s = 0; s < ns; ++s) {
        const double mx = __fma_rn(k, F[0], p.u), my = __fma_rn(k, F[1], p.v), mz = __fma_rn(k, F[2], p.w);
        const double wx = __fma_rn(my, tz, -__dmul_rn(mz, ty));
        const double wy = __fma_rn(mz, tx, -__dmul_rn(mx, tz));
        const double wz = __fma_rn(mx, ty, -__dmul_rn(my, tx));
        const double qx = __fma_rn(wy, tz, __fma_rn(-wz, ty, wx));
        const double qy = __fma_rn(wz, tx, __fma_rn(-wx, tz, wy));
        const double qz = __fma_rn(wx, ty, __fma_rn(-wy, tx, wz));
        p.u = __fma_rn(k, F[0], __fma_rn(f, qx, mx));
        p.v = __fma_rn(k, F[1], __fma_rn(f, qy, my));
        p.w = __fma_rn(k, F[2], __fma_rn(f, qz, mz));
        p.x = __fma_rn(p.u, dts, p.x);
        p.y = __fma_rn(p.v, dts, p.y);
        p.z = __fma_rn(p.w, dts, p.z);
    }
}

struct SubCycles64 {
    double dts, k;
    int n;
};
// (a call: its divisions would sit in every particle's instruction stream)
__device__ __noinline__ SubCycles64 sub_cycles64(double dt, double c, double inv_pic, double qom, double bx, double by,
                                                 double bz) {
    SubCycles64 s;
    const double bmag = (bx * bx + by * by) + bz * bz;
    s.n = sub_cycles_dt(dt, c, inv_pic, qom, bmag, s.dts);
    s.k = qom * 0.5 * s.dts;
    return s;
}

// Exponent of a rotation t = k B above which 1 + |t|^2 or |t|^2 v may overflow
// in boris64, where the reference's operations stay finite.
constexpr int kLargeRotation = 1023 + 100;
__device__ __noinline__ PState<double> boris_large64(double ex, double ey, double ez, double bx, double by, double bz,
                                                     double qom, double dts, int ns, PState<double> p) {
    for (int s = 0; s < ns; ++s) {
        boris<double>(p.u, p.v, p.w, ex, ey, ez, bx, by, bz, qom, dts);
        p.x = p.x + p.u * dts;
        p.y = p.y + p.v * dts;
        p.z = p.z + p.w * dts;
    }
    return p;
}

// The field mover's step from the gathered E, B in F.
__device__ __forceinline__ void move_field64(const Geom& g, const Push64Const& pc, double qom, double (&F)[6],
                                             PState<double>& p) {
    // (without a dipole moment the dipole's field is zero at a finite distance)
    if ((g.flags & 4u /*IPIC3D_F_DIPOLE_IN_GATHER*/) && !(pc.no_field && coordinates_regular(p.x, p.y, p.z))) {
        const double r2 = __fma_rn(p.x, p.x, __fma_rn(p.y, p.y, __dmul_rn(p.z, p.z)));
        // mft / r2^2.5 on the integer pipe
        double f;
        if (pc.d.usable && soft::regular(r2, 200)) {
            bool sure;  // either neighbour will do where it is not
            f = soft::pack(soft::div(pc.d.mft, soft::divisor(soft::pow25(soft::unpack(r2), sure))));
        } else {
            f = dipole_factor(g.mft, r2);
        }
        const double z3 = __dmul_rn(3.0, p.z), zf = __dmul_rn(z3, f);
        F[3] = __fma_rn(p.x, zf, F[3]);
        F[4] = __fma_rn(p.y, zf, F[4]);
        F[5] = __fma_rn(__fma_rn(z3, p.z, -r2), f, F[5]);
    }
    // one sub-cycle is sure below an exponent; else the reference's rule
    const int e = max(max(soft::exponent_of(F[3]), soft::exponent_of(F[4])), soft::exponent_of(F[5]));
    SubCycles64 s = {g.dt, pc.k1, 1};
    if (e > pc.d.e_max) {
        s = sub_cycles64(g.dt, g.c, g.inv_pic, qom, F[3], F[4], F[5]);
        if (soft::exponent_of(s.k) + e > 1023 + kLargeRotation) {
            p = boris_large64(F[0], F[1], F[2], F[3], F[4], F[5], qom, s.dts, s.n, p);
            return;
        }
    }
    boris64(F, s.k, s.dts, s.n, p);
}

// The dipole mover's step (cell.h:939-960), rounded as the reference's.
__device__ __forceinline__ void move_dipole64(const Geom& g, const Push64Const& pc, double qom, PState<double>& p) {
    if (pc.d.usable && coordinates_regular(p.x, p.y, p.z) &&
        dipole_rotate(pc.d, p.x, p.y, p.z, squared_position(p.x, p.y, p.z), p.u, p.v, p.w)) {
        advance_position(p.x, p.y, p.z, p.u, p.v, p.w, g.dt);
        return;
    }
    // No dipole (the host's pc.no_field): every component of the field is a
    // zero of some sign, one sub-cycle is enough, and the rotation adds zeros
    // to velocities, which changes them only if they are zero (the sign)
    // or no finite numbers: those take the operations below. (33.6M
    // particles of the reference's own benchmark mode, which has no dipole:
    // 11.5 -> 0.90 ms a step, half the copy bandwidth.)
    if (pc.no_field && coordinates_regular(p.x, p.y, p.z) && coordinates_regular(p.u, p.v, p.w)) {
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
// The same rounded once, for the weights of gather and deposit (the three
// roundings above show in both on widths that are no powers of two).
__device__ __forceinline__ double cell_middle(const Geom& g, int a, int pos) {
    return __fma_rn((double)pos + 0.5, g.w[a], g.origin[a]);
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
    if (!c.near_planet && in_cell(g, rel)) return kStay;
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
        const double at[3] = {p.x - cell_middle(g, 0, c.x), p.y - cell_middle(g, 1, c.y),
                              p.z - cell_middle(g, 2, c.z)};
        double F[6];
        bool fixed = in_cell(g, at);
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
            const uint64_t rx = fraction(at[0], g.inv_w[0]), ry = fraction(at[1], g.inv_w[1]),
                           rz = fraction(at[2], g.inv_w[2]);
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
#pragma unroll
            for (int q = 0; q < 6; ++q)
                F[q] = gather_fp64(g, c.x, c.y, c.z, pc.field_scale, at[0], at[1], at[2], q);
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
constexpr int kMaxItem64 = 32 * kGroup64;  // a lane's rounds fit a word
// warps per SM: 128 registers with the deposit (96 spill), 96 without
constexpr int kDepWarps64 = 16, kMoveWarps64 = 20;

// A warp's dynamic shared memory: the cells of its span, their coefficients
// per group.
struct Push64Smem {
    int64_t* start;  // [cells + 1]
    int64_t* coef;   // [groups][kCoefStride64]
    int* count;      // [cells]
    int* first;      // [cells + 1] items before the cell's
};
__host__ __device__ constexpr size_t push64_smem_bytes(int span) {
    const int cells = span * kMaxCellsPerCta;
    return (size_t)(cells + 2) / 2 * 2 * sizeof(int64_t) + (size_t)kWarpItems64 * kCoefStride64 * sizeof(double) +
           (size_t)(2 * cells + 1 + 3) / 4 * 4 * sizeof(int);
}
__device__ __forceinline__ Push64Smem push64_smem(int span, int warp) {
    extern __shared__ __align__(16) unsigned char push64_raw[];
    const int cells = span * kMaxCellsPerCta;
    Push64Smem sm;
    sm.start = reinterpret_cast<int64_t*>(push64_raw + warp * push64_smem_bytes(span));
    sm.coef = sm.start + (cells + 2) / 2 * 2;  // 16-byte aligned
    sm.count = reinterpret_cast<int*>(sm.coef + kWarpItems64 * kCoefStride64);
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

// The cloud-in-cell moments of a lane's particles in 64-bit fixed point: the
// sums of Q m for Q in {u, v, w, 1} and m in {1, x, y, xy, z, xz, yz, xyz}
// of the position in the cell, a 64-bit fraction. The values of a component
// share the exponent `top` of the largest in the group of 8 lanes; with
// `room` = log2 of the rounds, they keep 63 - room bits below it, offset by
// 2^(63 - room) so that the products are unsigned and add without overflow:
// the sum of the offsets is known from the sums of m and taken off at the end.
//
// Precision. A unit is 2^-(63 - room) of the power of two above the largest
// value (of one charge, for the density), room going by the particles of the
// cell that a lane adds up, not by the launch's items: 2^-63 for up to 8
// particles of a cell, 2^-58 for 256. Before the lanes' sums are added they
// are cut by the bits that the sum of all takes (sum_shift: 1 for a single
// particle, 6 for a warp of 1024), and nothing else rounds until the node's
// FP64 addition. RMS error over the cell's largest corner, FP64 sums before
// and this, 1 / 8 / 64 particles a cell, long items: J 3.3e-17 / 6.1e-17 /
// 8.3e-17 -> 2.0e-17 / 2.4e-17 / 2.7e-17, rho 2.7e-17 / 5.0e-17 / 6.4e-17 ->
// 2.0e-17 / 2.9e-17 / 4.0e-17 (with the unit and the cut of the longest items
// for all: rho 1.5e-16 / 1.1e-16 / 4.5e-17). Whole universes, error over the
// size of J: 33k particles 1.9e-16 -> 1.2e-16, 4.8M of 600 a cell 2.7e-16 ->
// 1.6e-16; of rho: 0.88e-16 -> 0.83e-16 and 1.62e-16 -> 0.95e-16.
// What is fine is the sum's size, not every node's share of it: a slow
// particle beside a fast one of its cell, and a node that little of the cell
// reaches, keep less than 53 bits. One particle at (0.01, 0.02, 0.03) of its
// cell: 4e-14 of the far node's share, where FP64 products have 3e-16.
//
// Cost. 25 high products of 64 x 64 bits and 32 sums per particle, about 600
// cycles of a warp on the integer pipe; in FP64 35 instructions, 2400
// cycles of the FP64 pipe, and 40 per work item for the reduction (8.4M
// particles: the deposit alone 0.70 -> 0.35 ms, the push 2.10 -> 1.82).
struct Moments64 {
    uint64_t a[32];  // Q, moment: 8 Q + m; a[24] unused (the particle count)

    __device__ __forceinline__ static int log2_up(int n) { return n > 1 ? 32 - __clz(n - 1) : 0; }
    // log2 of a lane's rounds, for items of `len` particles
    __device__ __forceinline__ static int headroom(int len) { return log2_up((len + kGroup64 - 1) / kGroup64); }
    // The shift that lets the sums of `n` particles in all, in units of
    // `room`, add up to 2^62 at most.
    __device__ __forceinline__ static int sum_shift(int n, int room) { return max(0, log2_up(n) + 1 - room); }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int l = 0; l < 32; ++l) a[l] = 0;
    }
    // the lane's particle, if `in`
    __device__ __forceinline__ void add(const Geom& g, int room, bool in, const double (&rel)[3],
                                        const double (&v)[3], const int (&top)[3]) {
        uint64_t M[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (in) {
            M[1] = fraction(rel[0], g.inv_w[0]);
            M[2] = fraction(rel[1], g.inv_w[1]);
            M[4] = fraction(rel[2], g.inv_w[2]);
        }
        M[3] = __umul64hi(M[1], M[2]);
        M[5] = __umul64hi(M[1], M[4]);
        M[6] = __umul64hi(M[2], M[4]);
        M[7] = __umul64hi(M[3], M[4]);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const soft::Num x = soft::unpack(v[q]);
            const int sh = room + 1 + top[q] - x.e;
            const uint64_t f = x.e == 0 || sh > 63 ? 0 : (x.m << 11) >> sh;
            const uint64_t Q = in ? (1ull << (63 - room)) + (x.sign ? 0 - f : f) : 0;
            a[8 * q] += Q;
#pragma unroll
            for (int m = 1; m < 8; ++m) a[8 * q + m] += __umul64hi(Q, M[m]);
        }
#pragma unroll
        for (int m = 1; m < 8; ++m) a[24 + m] += M[m] >> (room + 1);
    }
    // The moments turned into the corners' sums of weights (1 - r, r). n: the
    // lane's particles.
    __device__ __forceinline__ void corners(int room, int n) {
        a[24] = (uint64_t)n << (63 - room);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            // Products and shifts round down, by half a unit on average: what
            // is left of that (a bias grows with n) is made up for. x, y, z
            // shift without a remainder: a coordinate is a multiple of 2^-58
            // cell widths unless within 1/64 of one from zero.
            const bool exact = m == 1 || m == 2 || m == 4;
#pragma unroll
            for (int q = 0; q < 3; ++q) a[8 * q + m] += (exact ? n >> 1 : 0) - a[24 + m];
            if (m && !exact) a[24 + m] += n >> 1;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int bit = 1; bit < 8; bit <<= 1)
#pragma unroll
                for (int m = 0; m < 8; ++m)
                    if (!(m & bit)) a[8 * q + m] -= a[8 * q + (m | bit)];
    }
    // The shift that lets the velocity sums of 32 lanes add without overflow:
    // 0 for most (velocities of both signs), up to 6.
    __device__ __forceinline__ int spare_bits() const {
        uint32_t mag = 0;
#pragma unroll
        for (int l = 0; l < 24; ++l) mag |= (uint32_t)(((uint64_t)((int64_t)a[l] >> 63) ^ a[l]) >> 32);
        return max(0, 6 - __clz(__reduce_or_sync(0xffffffffu, mag)));
    }
    // A lane's sum of weights at a corner, up to 2^63 (all particles in the
    // corner): where every particle is within 2^-49 of the opposite face, the
    // sums' roundings can leave it below zero, by up to 1.5 units a particle,
    // which as an unsigned number would be 2^64 less that: zero then.
    __device__ __forceinline__ static uint64_t density_sum(uint64_t v) {
        return (uint32_t)(v >> 32) >= 0xc0000000u ? 0 : v;
    }
    // Over the group's 8 lanes: lane m is left with corner m's sums in a[0],
    // a[8], a[16] (in units 2^shift as large) and a[24] (2^rho_shift).
    __device__ __forceinline__ void reduce(int shift, int rho_shift) {
        constexpr unsigned kAll = 0xffffffffu;
        const int gl = threadIdx.x & (kGroup64 - 1);
        const uint32_t half = (1u << shift) >> 1, rho_half = (1u << rho_shift) >> 1;
#pragma unroll
        for (int l = 0; l < 32; ++l)
            a[l] = l < 24 ? (uint64_t)((int64_t)(a[l] + half) >> shift) : (density_sum(a[l]) + rho_half) >> rho_shift;
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int off = 4; off >= 1; off >>= 1) {
                const bool up = (gl & off) != 0;
#pragma unroll
                for (int m = 0; m < off; ++m) {
                    const uint64_t send = up ? a[8 * q + m] : a[8 * q + m + off];
                    const uint64_t keep = up ? a[8 * q + m + off] : a[8 * q + m];
                    a[8 * q + m] = keep + __shfl_xor_sync(kAll, send, off);
                }
            }
    }
    // The groups of one cell: the first is left with their sums (the others
    // with parts of them).
    __device__ __forceinline__ void join(bool next, bool after) {
        constexpr unsigned kAll = 0xffffffffu;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint64_t o = __shfl_down_sync(kAll, a[8 * q], kGroup64);
            if (next) a[8 * q] += o;
            o = __shfl_down_sync(kAll, a[8 * q], 2 * kGroup64);
            if (after) a[8 * q] += o;
        }
    }
    // charge times component q's sum at the lane's corner (shift: as given to
    // reduce; top = 0: every value is zero, what is left the offsets' rounding)
    __device__ __forceinline__ double velocity(int q, double charge, int top, int room, int shift) const {
        return top ? times_fixed(charge, (int64_t)a[8 * q], top + room + shift - 4) : 0.0;
    }
    __device__ __forceinline__ double density(double charge, int room, int rho_shift) const {
        return times_fixed(charge, (int64_t)a[24], 1018 + room + rho_shift);
    }
};
// a velocity component the moments take: zero, or of an exponent in fixed_range
__device__ __forceinline__ bool moment_range(double v) {
    const int e = soft::exponent_of(v);
    return fixed_range(e) && (e != 0 || (soft::bits_of(v) << 1) == 0);
}
// A particle outside its cell, or whose velocity is out of the fixed-point
// range (or no number).
__device__ __noinline__ void deposit_fp64(const Geom& g, int cell, double x, double y, double z, double u, double v,
                                          double w, double q) {
    const PState<double> p = {x, y, z, u, v, w};
    deposit_one<double>(g, cell, p, q);
}

// Blocks of four warps, where items are short (8 or 16 particles): the items'
// sums are added per cell before the nodes' atomics. Every addition to a node
// rounds, and a warp's four items are half a cell of 64 particles: with a warp
// per block rho was 5 to 10 % further from exact sums than FP64 sums of 32
// lanes of 4 slots each (8^3 cells of 64: 0.93e-16 of its size against 0.87e-16,
// 10^3 of 256: 1.23e-16 against 1.17e-16), joined it is closer (0.83e-16,
// 0.86e-16). It costs 2 to 5 % of such a push (8^3: 21.7 -> 22.8 us).
struct Joint64 {
    static constexpr int kWarps = 4;
    static constexpr int kRows = kWarps * kWarpItems64;
    double sum[kRows][32];  // [item][component * 8 + corner]
    int cell[kRows];        // -1: nothing, or joined with the item before

    // Adds the rows of every cell to its nodes, a warp per cell.
    __device__ __forceinline__ void flush(const Geom& g) const {
        const int lane = threadIdx.x & 31;
        const int mine = lane < kRows ? cell[lane] : -1;
        for (int r = threadIdx.x >> 5; r < kRows; r += kWarps) {
            const int c = __shfl_sync(0xffffffffu, mine, r);
            unsigned rows = __ballot_sync(0xffffffffu, mine == c);
            if (c < 0 || (rows & ((1u << r) - 1u))) continue;  // nothing, or the cell's first row has it
            double s = 0.0;
            for (; rows; rows &= rows - 1) s += sum[__ffs(rows) - 1][lane];
            int x, y, z;
            cell_coords(g, c, x, y, z);
            const int64_t node = node_index(g, x + (lane & 1), y + ((lane >> 1) & 1), z + ((lane >> 2) & 1));
            const int q = lane >> 3;
            atomicAdd(q < 3 ? g.J + 3 * node + q : g.rho + node, s);
        }
    }
};

// The cells of a block's span and its items.
struct Span64 {
    int base, top;  // slots
    int c0, nc;     // cells
    int total;      // items
};

// kStep: mover + export (else the deposit of the particles as they are);
// kField: field-gather mover (else the dipole mover); kDep: deposit; kWarps:
// warps of the block (more than one: their sums are joined, Joint64).
// Four items of the span from j0 < total, by one warp.
template <bool kStep, bool kField, bool kDep, int kWarps>
__device__ __forceinline__ void push64_items(const Geom& g, const Pop<double>& P, const Push64Const& pc,
                                             const Push64Smem& sm, const Span64& S, int item, int j0, float reach,
                                             Joint64* joint, uint32_t& nmig, uint32_t& nrem) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = kWarps > 1 ? threadIdx.x >> 5 : 0;
    const int gl = lane & (kGroup64 - 1), sub = lane / kGroup64;
    const int c0 = S.c0, nc = S.nc, total = S.total;
    int64_t* const coef = sm.coef + sub * kCoefStride64;
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
    span_range64(sm, i, S.base, S.top, lo, end);
    const int pieces = sm.first[i + 1] - sm.first[i];
    const int piece = ((int)(end - lo) + pieces * kGroup64 - 1) / (pieces * kGroup64) * kGroup64;
    const int a = (int)lo + (j - sm.first[i]) * piece;
    int len = max(0, min(piece, (int)end - a));
    if (j0 + sub >= total) len = 0;
    const int cell = c0 + i;
    const int64_t cstart = sm.start[i];
    Cell64 c;
    cell_coords(g, cell, c.x, c.y, c.z);
    double mid[3];
    {   // lane 0, 1, 2 of the group: the axis' centre
        const int pos = gl == 0 ? c.x : gl == 1 ? c.y : c.z;
        const double cen = gl < 3 ? cell_centre(g, gl, pos) : 0.0;
        const double middle = gl < 3 ? cell_middle(g, gl, pos) : 0.0;
        const float mine = gl < 3 ? planet_gap(g, gl, cen) : 0.f;
        float gap[3];
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            c.cen[b] = __shfl_sync(kAll, cen, b, kGroup64);
            mid[b] = __shfl_sync(kAll, middle, b, kGroup64);
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
    uint32_t adds = 0;            // bit r: the lane's particle of round r adds to the moments
    int top[3] = {0, 0, 0};       // the components' largest exponents among them
    const int rounds = __reduce_max_sync(kAll, (len + kGroup64 - 1) / kGroup64);
    for (int r = 0; r < rounds; ++r) {
        const int k = r * kGroup64 + gl;
        const bool has = k < len;
        const int slot = a + k;
        // lanes without a particle: the cell's centre at rest
        PState<double> p = {c.cen[0], c.cen[1], c.cen[2], 0.0, 0.0, 0.0};
        if (has) p = {P.x[slot], P.y[slot], P.z[slot], P.u[slot], P.v[slot], P.w[slot]};
        double rel[3];
        bool stays;
        if (kStep) {
            if (kField) {
                const double at[3] = {p.x - mid[0], p.y - mid[1], p.z - mid[2]};
                double F[6];
                if (fixed && in_cell(g, at)) {
                    const uint64_t rx = fraction(at[0], g.inv_w[0]), ry = fraction(at[1], g.inv_w[1]),
                                   rz = fraction(at[2], g.inv_w[2]);
                    // a loop, the results passing through F: unrolled, the
                    // gather alone was a third of the instruction stream
                    // (push 1.60 -> 1.43 ms)
#pragma unroll 1
                    for (int q = 0; q < 6; ++q) {
                        const uint32_t e = q < 2 ? exps[0] : q < 4 ? exps[1] : exps[2];
                        const double f = from_fixed(poly_fixed(coef + 8 * q, rx, ry, rz),
                                                    (int)(e >> (16 * (q & 1)) & 0xffffu));
#pragma unroll
                        for (int k = 0; k < 5; ++k) F[k] = F[k + 1];
                        F[5] = f;
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 6; ++q)
                        F[q] = has ? gather_fp64(g, c.x, c.y, c.z, pc.field_scale, at[0], at[1], at[2], q) : 0.0;
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
            stays = outcome == kStay;
        } else {
            rel[0] = p.x - c.cen[0];
            rel[1] = p.y - c.cen[1];
            rel[2] = p.z - c.cen[2];
            stays = has;
        }
        if (kDep && stays) {
            const int e[3] = {soft::exponent_of(p.u), soft::exponent_of(p.v), soft::exponent_of(p.w)};
            if (in_cell(g, rel) && moment_range(p.u) && moment_range(p.v) && moment_range(p.w)) {
                adds |= 1u << r;
#pragma unroll
                for (int q = 0; q < 3; ++q) top[q] = max(top[q], e[q]);
            } else {
                deposit_fp64(g, cell, p.x, p.y, p.z, p.u, p.v, p.w, P.q);
            }
        }
    }
    if (kDep && __any_sync(kAll, adds != 0)) {
        Moments64 sums;
        sums.clear();
        // groups with items of the same cell (they follow one another) add up
        // before the FP64 atomics, which round: next: the following
        // group's cell is this one's, after: the one after it too
        const int c1 = __shfl_down_sync(kAll, cell, kGroup64), c2 = __shfl_down_sync(kAll, cell, 2 * kGroup64);
        const int before = __shfl_up_sync(kAll, cell, kGroup64);
        const bool next = sub < kWarpItems64 - 1 && c1 == cell, after = sub < kWarpItems64 - 2 && c2 == cell;
        const bool first = sub == 0 || before != cell;
        const bool shared = __any_sync(kAll, next);
#pragma unroll
        for (int q = 0; q < 3; ++q) top[q] = __reduce_max_sync(0xffu << (sub * kGroup64), top[q]);
        if (shared) {
            int t[3] = {top[0], top[1], top[2]};
#pragma unroll
            for (int k = 1; k < kWarpItems64; ++k) {
                const bool same = __shfl_xor_sync(kAll, cell, k * kGroup64) == cell;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const int o = __shfl_xor_sync(kAll, t[q], k * kGroup64);
                    if (same) top[q] = max(top[q], o);
                }
            }
        }
        // at most so many of the cell's particles in an item, in the warp
        // (the same in all groups of the cell)
        const int in_item = min(item, sm.count[cell - c0]), in_warp = min(kWarpItems64 * item, sm.count[cell - c0]);
        const int room = Moments64::headroom(in_item);
        for (int r = 0; r < rounds; ++r) {
            const int slot = a + r * kGroup64 + gl;
            const bool in = (adds >> r & 1u) != 0;
            double rel[3] = {0.0, 0.0, 0.0}, v[3] = {0.0, 0.0, 0.0};
            if (in) {
                rel[0] = P.x[slot] - mid[0];
                rel[1] = P.y[slot] - mid[1];
                rel[2] = P.z[slot] - mid[2];
                v[0] = P.u[slot]; v[1] = P.v[slot]; v[2] = P.w[slot];
            }
            sums.add(g, room, in, rel, v, top);
        }
        sums.corners(room, __popc(adds));
        const int rho_shift = Moments64::sum_shift(in_warp, room), shift = min(sums.spare_bits(), rho_shift);
        sums.reduce(shift, rho_shift);
        if (shared) sums.join(next, after);
        if (kWarps > 1) {
            __syncwarp();
            if (first) {
                double* const row = joint->sum[warp * kWarpItems64 + sub];
                if (gl == 0) joint->cell[warp * kWarpItems64 + sub] = cell;
#pragma unroll
                for (int q = 0; q < 3; ++q) row[8 * q + gl] = sums.velocity(q, P.q, top[q], room, shift);
                row[24 + gl] = sums.density(P.q, room, rho_shift);
            }
        } else if (first) {
            const int64_t node = node_index(g, c.x + (gl & 1), c.y + ((gl >> 1) & 1), c.z + (gl >> 2));
#pragma unroll
            for (int q = 0; q < 3; ++q)
                atomicAdd(g.J + 3 * node + q, sums.velocity(q, P.q, top[q], room, shift));
            atomicAdd(g.rho + node, sums.density(P.q, room, rho_shift));
        }
    }
}

// The items of a span that block `part` of `parts` takes.
template <bool kStep, bool kField, bool kDep, int kWarps>
__device__ __forceinline__ void push64_body(const Geom& g, const Pop<double>& P, const Push64Const& pc, int64_t tile,
                                            int span, int part, int parts, int item, Joint64* joint) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = kWarps > 1 ? threadIdx.x >> 5 : 0;
    const Push64Smem sm = push64_smem(span, warp);
    // the cells of the span: consecutive tiles' cells follow one another
    const int base = (int)tile * kSlotsPerCta, top = (int)min(base + (int64_t)span * kSlotsPerCta, P.capacity);
    const int2 cc = __ldg(P.cta_cells + tile), ce = __ldg(P.cta_cells + (top - 1) / kSlotsPerCta);
    const int c0 = cc.x, nc = ce.x + ce.y - cc.x;
    for (int i = lane; i <= nc; i += 32) sm.start[i] = P.start[c0 + i];
    for (int i = lane; i < nc; i += 32) sm.count[i] = P.count[c0 + i];
    __syncwarp();
    {  // items before each cell
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
    __syncwarp();
    const int total = sm.first[nc];
    const float reach = planet_reach(g);
    uint32_t nmig = 0, nrem = 0;

    const Span64 S = {base, top, c0, nc, total};
    for (int jb = part * kWarps * kWarpItems64; jb < total; jb += parts * kWarps * kWarpItems64) {
        const int j0 = jb + warp * kWarpItems64;
        if (kWarps > 1 && lane < kWarpItems64) joint->cell[warp * kWarpItems64 + lane] = -1;
        if (kWarps == 1 || j0 < total)
            push64_items<kStep, kField, kDep, kWarps>(g, P, pc, sm, S, item, j0, reach, joint, nmig, nrem);
        if (kWarps > 1) {
            __syncthreads();
            joint->flush(g);
            if (jb + parts * kWarps * kWarpItems64 < total) __syncthreads();
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

template <int kWarps>
__device__ __forceinline__ Joint64* joint64() {
    if constexpr (kWarps > 1) {
        __shared__ Joint64 joint;
        return &joint;
    } else {
        return nullptr;
    }
}

// Block (span, part) of population blockIdx.z of the set.
template <bool kStep, bool kField, bool kDep, int kWarps>
__global__ void __launch_bounds__(32 * kWarps, (kDep ? kDepWarps64 : kMoveWarps64) / kWarps)
    k_push64(Geom g, const __grid_constant__ PopSet<double> S, const __grid_constant__ Push64Set pcs, int span,
             int item) {
    const Pop<double>& P = S.p[blockIdx.z];
    const int64_t tile = (int64_t)blockIdx.x * span;
    if (tile * kSlotsPerCta >= P.capacity) return;
    push64_body<kStep, kField, kDep, kWarps>(g, P, pcs.c[blockIdx.z], tile, span, blockIdx.y, gridDim.y, item,
                                             joint64<kWarps>());
}

// Batched: block b is part b % parts of cta_job[b / parts] = (job, tile of the
// job); the span starts at every span-th tile of a job, the other tiles'
// blocks end at once. The parts of a tile are consecutive blocks: with the
// tiles along x, every fourth block had work, and the SMs, which hand
// one-warp blocks to their four sub-partitions in turn, ran it all on one
// (64 universes of 34M particles: 15.3 ms a step, now 7.0).
template <bool kStep, bool kField, bool kDep, int kWarps>
__global__ void __launch_bounds__(32 * kWarps, (kDep ? kDepWarps64 : kMoveWarps64) / kWarps)
    k_push64_batch(const PopJob<double>* __restrict__ jobs, const int2* __restrict__ cta_job, int span, int item,
                   int parts) {
    __shared__ PopJob<double> job;
    const unsigned tile = blockIdx.x / (unsigned)parts;
    const int2 cj = __ldg(cta_job + tile);
    if (cj.y % span != 0) return;
    load_job(job, jobs + cj.x);
    push64_body<kStep, kField, kDep, kWarps>(job.g, job.P, job.pc, cj.y, span, (int)(blockIdx.x - tile * parts), parts,
                                             item, joint64<kWarps>());
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
