// One step of the FP64 dipole mover (moveParticles, cell.h:896-964;
// traceParticle, pic_tracer.cxx:104-127) with a single sub-cycle, bit for
// bit the reference's rounding. Shared by the tracer and the FP64 push.
//
// The FP64 pipe bounds these kernels (64 to 76 cycles per warp instruction
// and sub-partition), so the field, the squares, the quotients and the
// position's products run on the integer pipe (fp64_int.cuh) and the
// velocity's cross products and the sums that can cancel stay FP64: 35 FP64
// instructions per particle step in place of about 149, beside about 1700
// others (pipe use: FP64 78 %, integer ALU 66 %). Moving 3 or 6 products of the
// cross products over as well was slower (tracer, 16M particles x 151 steps:
// 177 and 189 ms against 163 ms; all FP64 641 ms).
#pragma once

#include "fp64_int.cuh"
#include "particle_kernels.cuh"

namespace ipg {

// |B|^2 <= 3 2^(2 (e - 1023) + 2) for components of biased exponent <= e; one
// sub-cycle is sure while the estimate of sub_cycles_dt is below 1/2.
__host__ __device__ __forceinline__ DipoleSpecies dipole_species(double mft, double qom, double dt, double inv_pic) {
    DipoleSpecies s;
    const double k = qom * 0.5 * dt;
    const double lim = (0.49 / 3.0) / ((dt * (4.0 * fabs(qom))) * inv_pic);
    s.mft = soft::unpack(mft);
    s.k = soft::unpack(k);
    s.e_max = soft::regular(lim, 1000) ? 1023 + ((soft::exponent_of(lim) - 1023 - 2) >> 1) : -1;
    s.usable = soft::regular(dt, 100) && soft::regular(mft, 200) && soft::regular(k, 100) && soft::regular(lim, 1000);
    return s;
}

// The squares of a position that the field, the planet test and the next
// step share. Filled only for regular coordinates.
struct SquaredPosition {
    soft::Num x2, y2, z2, r2;
};

__device__ __forceinline__ bool coordinates_regular(double x, double y, double z) {
    return soft::regular(x, 100) && soft::regular(y, 100) && soft::regular(z, 100);
}
__device__ __forceinline__ SquaredPosition squared_position(double x, double y, double z) {
    SquaredPosition s;
    s.x2 = soft::sqr(soft::unpack(x));
    s.y2 = soft::sqr(soft::unpack(y));
    s.z2 = soft::sqr(soft::unpack(z));
    s.r2 = soft::add_positive(soft::add_positive(s.x2, s.y2), s.z2);
    return s;
}

// updatePosition (particle.h:24-26) with the products on the integer pipe.
__device__ __forceinline__ void advance_position(double& x, double& y, double& z, double u, double v, double w,
                                                 double dt) {
    if (coordinates_regular(u, v, w)) {
        const soft::Num d = soft::unpack(dt);
        x = x + soft::pack(soft::mul(soft::unpack(u), d));
        y = y + soft::pack(soft::mul(soft::unpack(v), d));
        z = z + soft::pack(soft::mul(soft::unpack(w), d));
    } else {
        x = x + u * dt;
        y = y + v * dt;
        z = z + w * dt;
    }
}

// Advances the velocity by one Boris rotation in the dipole field at
// (x, y, z) (regular coordinates, S their squares). False, with the velocity
// unchanged, where a value leaves the range in which the integer operations
// are exact or one sub-cycle is not sure: the caller then takes the FP64
// path, which covers everything.
// Exponents: coordinates within 2^+-101, so r^5 within 2^+-510, mft / r^5
// within 2^+-711, the components within 2^+-1012.
__device__ __forceinline__ bool dipole_rotate(const DipoleSpecies& K, double x, double y, double z,
                                              const SquaredPosition& S, double& u, double& v, double& w) {
    using namespace soft;
    const Num X = unpack(x), Y = unpack(y), Z = unpack(z);
    // 2 z^2 - x^2 - y^2 can cancel
    Num zz = S.z2;
    zz.e += 1;
    const double dz = (pack(zz) - pack(S.x2)) - pack(S.y2);
    if (!regular(dz, 300)) return false;
    bool sure;
    Num r5 = pow25(S.r2, sure);
    if (!sure) r5 = unpack(pow25_core(pack(S.r2)));
    const Num f = div(K.mft, divisor(r5));
    const Num bx = mul(mul(triple(X), Z), f);
    const Num by = mul(mul(triple(Y), Z), f);
    const Num bz = mul(unpack(dz), f);
    if (max(max(bx.e, by.e), bz.e) > K.e_max) return false;
    Num tx = mul(K.k, bx), ty = mul(K.k, by), tz = mul(K.k, bz);
    constexpr int kLow = 1023 - 250, kSpan = 500;
    if ((unsigned)(tx.e - kLow) > kSpan || (unsigned)(ty.e - kLow) > kSpan || (unsigned)(tz.e - kLow) > kSpan)
        return false;
    const Num tt = add_positive(add_positive(sqr(tx), sqr(ty)), sqr(tz));
    const Num one = {1ull << 52, 1023, 0u};
    const Divisor den = divisor(add_positive(one, tt));
    const double dtx = pack(tx), dty = pack(ty), dtz = pack(tz);
    ++tx.e;
    ++ty.e;
    ++tz.e;
    const double sx = pack(div(tx, den)), sy = pack(div(ty, den)), sz = pack(div(tz, den));
    const bool kneg = K.k.sign != 0;
    const double mx = add_zero(u, kneg), my = add_zero(v, kneg), mz = add_zero(w, kneg);  // v_minus
    const double px = mx + (my * dtz - mz * dty);  // v_prime = v_minus + v_minus x t
    const double py = my + (mz * dtx - mx * dtz);
    const double pz = mz + (mx * dty - my * dtx);
    u = add_zero(mx + (py * sz - pz * sy), kneg);  // v_plus + k E
    v = add_zero(my + (pz * sx - px * sz), kneg);
    w = add_zero(mz + (px * sy - py * sx), kneg);
    return true;
}

}  // namespace ipg
