// What the FP32 and FP64 particle kernels share, templated on the storage
// type (double: absolute positions; float: positions relative to the cell
// origin in cell widths): r^2.5 and the Boris rotation as the reference
// rounds them, the sub-cycle rule, the deposit of single particles, the
// outbox and arrival lists (the TransferBuffers of transfer_buffer.h:48-95),
// and these kernels of a step of the reference's active loop
// (simulator.h:214-223):
//   k_inject          x = 0 injection (not in the reference);
//   k_place           import (cell.h:1195-1310): a warp scans a few cells and
//                     fills the holes left by leavers with arrivals;
//   k_pending_rotate  hands the particles without a slot to the next step;
//   k_relayout_copy, k_pending_place, k_pending_count  the re-layout.
// The mover, export and deposit of the bulk are in push32_pipe.cuh and
// push64.cuh, of the particles that waited in push32.cuh and push64.cuh.
#pragma once

#include <type_traits>

#include "device.cuh"

namespace ipg {

// ---- r^2.5 correctly rounded (FP64) ----------------------------------------
// The reference evaluates pow(|x|^2, 2.5) with the host libm (cell.h:940),
// whose result is the correctly rounded one in all but rare cases. CUDA's pow
// is not correctly rounded, so the FP64 path evaluates a^2.5 = a^2 * sqrt(a)
// in double-double arithmetic and rounds once at the end. sqrt(a) = s + ds
// to ~2^-100 relative comes from the reciprocal square root y (error <= 1
// ulp): s0 = a y, then s = s0 + (a - s0^2) y / 2, the correctly rounded root
// (exact when a is a square), and ds = (a - s^2) y / 2, with the residuals
// exact through fma; a^2 = p + pe and p s = h + l are Dekker's exact
// products. The result is the correctly rounded one unless a^2.5 lies within
// ~2^-100 relative of a rounding boundary (exact midpoints, from squares,
// round to even). Inputs in [2^400, 2^410) are scaled by 2^-400 (exactly)
// and the result by 2^1000; from 2^410 on a^2.5 overflows. Below 2^-400 the
// result is subnormal or zero and is rounded twice.
__device__ __forceinline__ double pow25_core(double a) {
    const double y = rsqrt(a);
    double s = __dmul_rn(a, y);
    double e = __fma_rn(-s, s, a);
    s = __dadd_rn(s, __dmul_rn(__dmul_rn(e, y), 0.5));
    e = __fma_rn(-s, s, a);
    const double ds = __dmul_rn(__dmul_rn(e, y), 0.5);
    const double p = __dmul_rn(a, a);
    const double pe = __fma_rn(a, a, -p);  // a*a = p + pe exactly
    const double h = __dmul_rn(p, s);
    double l = __fma_rn(p, s, -h);         // p*s = h + l exactly
    l = __dadd_rn(l, __dadd_rn(__dmul_rn(p, ds), __dmul_rn(pe, s)));
    return __dadd_rn(h, l);
}

__device__ __forceinline__ double pow25_rn(double a) {
    if (a >= 0x1p-400 && a < 0x1p400) return pow25_core(a);
    if (a != a) return a;
    if (a < 0.0) return __longlong_as_double(0x7ff8000000000000LL);
    if (a < 0x1p-800) return 0.0;  // a^2.5 < 2^-2000 (and a == 0)
    if (a < 0x1p-400) return __dmul_rn(pow25_core(__dmul_rn(a, 0x1p400)), 0x1p-1000);
    if (a < 0x1p410) return __dmul_rn(pow25_core(__dmul_rn(a, 0x1p-400)), 0x1p1000);
    return __longlong_as_double(0x7ff0000000000000LL);  // +inf
}

// ---- the Boris rotation (Particle::updateVelocity, particle.h:31-49) -------
template <typename T>
__device__ __forceinline__ void boris(T& u, T& v, T& w, T ex, T ey, T ez, T bx, T by, T bz, T qom, T dt) {
    T k = qom * T(0.5) * dt;
    T tx = k * bx, ty = k * by, tz = k * bz;
    T t_mag2 = tx * tx;
    t_mag2 += ty * ty;
    t_mag2 += tz * tz;
    T den = T(1.0) + t_mag2;
    T sx = (T(2.0) * tx) / den, sy = (T(2.0) * ty) / den, sz = (T(2.0) * tz) / den;
    T kex = k * ex, key = k * ey, kez = k * ez;
    T mx = u + kex, my = v + key, mz = w + kez;            // v_minus
    T px = mx + (my * tz - mz * ty);                        // v_prime = v_minus + v_minus x t
    T py = my + (mz * tx - mx * tz);
    T pz = mz + (mx * ty - my * tx);
    T qx = mx + (py * sz - pz * sy);                        // v_plus = v_minus + v_prime x s
    T qy = my + (pz * sx - px * sz);
    T qz = mz + (px * sy - py * sx);
    u = qx + kex;
    v = qy + key;
    w = qz + kez;
}

// x + z for z = k * 0 = +-0 (k finite, z negative when k is): x itself,
// except -0 + +0 = +0. Integer work in place of the FP64 addition.
__device__ __forceinline__ double add_zero(double x, bool z_negative) {
    return (!z_negative && __double_as_longlong(x) == (long long)0x8000000000000000ULL) ? 0.0 : x;
}

// Particle::updateVelocity (particle.h:31-49) in FP64 for E = 0 (the dipole
// mover, the tracer): boris<double> with the k E terms (+-0 for finite k)
// applied as add_zero, bit for bit the same velocities.
__device__ __forceinline__ void boris_e0(double& u, double& v, double& w, double bx, double by, double bz,
                                         double qom, double dt) {
    const double k = qom * 0.5 * dt;
    if (!isfinite(k)) {  // k E is NaN: the general routine
        boris<double>(u, v, w, 0.0, 0.0, 0.0, bx, by, bz, qom, dt);
        return;
    }
    const bool kneg = signbit(k);
    const double tx = k * bx, ty = k * by, tz = k * bz;
    double t_mag2 = tx * tx;
    t_mag2 += ty * ty;
    t_mag2 += tz * tz;
    const double den = 1.0 + t_mag2;
    const double sx = (2.0 * tx) / den, sy = (2.0 * ty) / den, sz = (2.0 * tz) / den;
    const double mx = add_zero(u, kneg), my = add_zero(v, kneg), mz = add_zero(w, kneg);  // v_minus
    const double px = mx + (my * tz - mz * ty);  // v_prime = v_minus + v_minus x t
    const double py = my + (mz * tx - mx * tz);
    const double pz = mz + (mx * ty - my * tx);
    u = add_zero(mx + (py * sz - pz * sy), kneg);  // v_plus + k E
    v = add_zero(my + (pz * sx - px * sz), kneg);
    w = add_zero(mz + (px * sy - py * sx), kneg);
}

// Sub-cycle count of moveParticles (cell.h:947-952): min(int(dt/dt_sub)+1,
// 100) with dt_sub = pi c / (4 |qom| |B|^2). Quotients outside the int range
// (and NaN) convert to INT_MIN on the reference's x86 build, which leaves the
// particle unmoved; that outcome is returned as 0.
template <typename T>
__device__ __forceinline__ int sub_cycles(T dt, T c, T qom, T bmag) {
    T dt_sub = T(3.14159265358979323846) * c / (T(4.0) * fabs(qom) * bmag);
    T ratio = dt / dt_sub;
    if (!(ratio >= T(-2147483648.0) && ratio < T(2147483647.0))) return 0;
    int n = (int)ratio + 1;
    return n < 100 ? n : 100;
}

// The FP64 sub-cycle count and step together: dt / dt_sub is first
// estimated from its product form dt (4 |qom| |B|^2) / (pi c), with inv_pic
// = 1 / (pi c) rounded any way; below 1/2 the reference's two roundings of
// the quotient cannot reach 1, so the count is 1 and the step dt (dt / 1.0
// == dt), without a division. Otherwise sub_cycles and dt / n.
__device__ __forceinline__ int sub_cycles_dt(double dt, double c, double inv_pic, double qom, double bmag,
                                             double& dts) {
    const double est = (dt * ((4.0 * fabs(qom)) * bmag)) * inv_pic;
    // |est| < 0.5 on the bit pattern (NaN compares above): integer work in
    // place of an FP64 comparison
    if ((__double_as_longlong(est) & 0x7fffffffffffffffLL) < 0x3fe0000000000000LL) {
        dts = dt;
        return 1;
    }
    const int ns = sub_cycles<double>(dt, c, qom, bmag);
    dts = dt / double(ns);
    return ns;
}

// Outcome of one particle's mover + export step.
enum : int { kStay = 0, kMove = 1, kDrop = 2 };

template <typename T>
struct PState {
    T x, y, z, u, v, w;
};

// ---- deposit -----------------------------------------------------------------
// Cloud-in-cell weights of projectToDensityField (cell.h:810-816): a particle
// at fractional position r in cell c adds q v fac and q fac to node c+(i,j,k)
// with fac = prod (i ? r : 1-r). Index l = corner*4 + comp, comp 3 = rho.
template <typename T>
__device__ __forceinline__ void frac_in_cell(const Geom& g, int cx, int cy, int cz, const PState<T>& p, T& rx, T& ry,
                                             T& rz) {
    if constexpr (std::is_same<T, double>::value) {
        rx = soft::quotient(p.x - (g.origin[0] + (double)cx * g.w[0]), g.w[0], g.inv_w[0], g.exact_inv[0]);
        ry = soft::quotient(p.y - (g.origin[1] + (double)cy * g.w[1]), g.w[1], g.inv_w[1], g.exact_inv[1]);
        rz = soft::quotient(p.z - (g.origin[2] + (double)cz * g.w[2]), g.w[2], g.inv_w[2], g.exact_inv[2]);
    } else {
        rx = p.x; ry = p.y; rz = p.z;
    }
}

template <typename T>
__device__ __forceinline__ T cic_weight(int corner, T rx, T ry, T rz) {
    int i = corner >> 2, j = (corner >> 1) & 1, k = corner & 1;
    return (i == 0 ? (1 - rx) : rx) * (j == 0 ? (1 - ry) : ry) * (k == 0 ? (1 - rz) : rz);
}

__device__ __forceinline__ void node_atomic_add(const Geom& g, int cx, int cy, int cz, int l, double val) {
    if (val == 0.0) return;
    int corner = l >> 2, comp = l & 3;
    int64_t n = node_index(g, cx + (corner >> 2), cy + ((corner >> 1) & 1), cz + (corner & 1));
    if (comp < 3)
        atomicAdd(g.J + 3 * n + comp, val);
    else
        atomicAdd(g.rho + n, val);
}

// Direct deposit of one particle (rare paths: migrants, pending, injected).
template <typename T>
__device__ __forceinline__ void deposit_one(const Geom& g, int c, const PState<T>& p, double q) {
    int cx, cy, cz;
    cell_coords(g, c, cx, cy, cz);
    T rx, ry, rz;
    frac_in_cell(g, cx, cy, cz, p, rx, ry, rz);
#pragma unroll
    for (int corner = 0; corner < 8; ++corner) {
        double fac = (double)cic_weight<T>(corner, rx, ry, rz);
        node_atomic_add(g, cx, cy, cz, corner * 4 + 0, (q * (double)p.u) * fac);
        node_atomic_add(g, cx, cy, cz, corner * 4 + 1, (q * (double)p.v) * fac);
        node_atomic_add(g, cx, cy, cz, corner * 4 + 2, (q * (double)p.w) * fac);
        node_atomic_add(g, cx, cy, cz, corner * 4 + 3, q * fac);
    }
}

// Deposit of the warp's leavers into their destination cells, one leaver at
// a time: lane l adds value l (corner l & 7, component l >> 3) of the leaver's
// cloud-in-cell contribution, the same values deposit_one adds one by one, so
// a leaver costs one 32-lane atomic instead of 32 serial ones. Every lane of
// the warp must call it.
template <typename T>
__device__ __forceinline__ void warp_deposit_leavers(const Geom& g, bool leave, int dest, const PState<T>& p,
                                                     double q) {
    unsigned m = __ballot_sync(0xffffffffu, leave);
    const int lane = threadIdx.x & 31, corner = lane & 7, comp = lane >> 3;
    while (m) {
        const int src = __ffs(m) - 1;
        m &= m - 1;
        const int c = __shfl_sync(0xffffffffu, dest, src);
        PState<T> s;
        s.x = __shfl_sync(0xffffffffu, p.x, src);
        s.y = __shfl_sync(0xffffffffu, p.y, src);
        s.z = __shfl_sync(0xffffffffu, p.z, src);
        s.u = __shfl_sync(0xffffffffu, p.u, src);
        s.v = __shfl_sync(0xffffffffu, p.v, src);
        s.w = __shfl_sync(0xffffffffu, p.w, src);
        int cx, cy, cz;
        cell_coords(g, c, cx, cy, cz);
        T rx, ry, rz;
        frac_in_cell(g, cx, cy, cz, s, rx, ry, rz);
        const double fac = (double)cic_weight<T>(corner, rx, ry, rz);
        const double Q = comp == 0 ? (double)s.u : (comp == 1 ? (double)s.v : (double)s.w);
        node_atomic_add(g, cx, cy, cz, corner * 4 + comp, comp < 3 ? (q * Q) * fac : q * fac);
    }
}

// Warp transpose-reduction: every lane holds 32 values; afterwards lane l
// holds the warp-wide sum of value l (31 exchanges in total).
template <typename T>
__device__ __forceinline__ T warp_transpose_sum(T (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        const bool upper = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < off; ++i) {
            T send = upper ? v[i] : v[i + off];
            T keep = upper ? v[i + off] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    return v[0];
}

// ---- slot / outbox helpers -------------------------------------------------
template <typename T>
__device__ __forceinline__ void write_slot(const Pop<T>& P, int64_t slot, const Mover<T>& m) {
    P.x[slot] = m.x; P.y[slot] = m.y; P.z[slot] = m.z;
    P.u[slot] = m.u; P.v[slot] = m.v; P.w[slot] = m.w;
    if (P.id) P.id[slot] = m.id;
}

template <typename T>
__device__ __forceinline__ void move_slot(const Pop<T>& P, int64_t from, int64_t to) {
    P.x[to] = P.x[from]; P.y[to] = P.y[from]; P.z[to] = P.z[from];
    P.u[to] = P.u[from]; P.v[to] = P.v[from]; P.w[to] = P.w[from];
    if (P.id) P.id[to] = P.id[from];
}

// Files an outbox entry as an arrival of its destination cell: slot k of the
// cell's arrival list, or the pending list when the cell's slots are short.
template <typename T>
__device__ __forceinline__ void register_arrival(const Pop<T>& P, uint32_t o, const Mover<T>& m) {
    int k = atomicAdd(P.arr_cnt + m.cell, 1);
    int64_t s = P.start[m.cell];
    if (k < (int)(P.start[m.cell + 1] - s)) {
        P.arr_list[s + k] = (int32_t)o;
    } else {
        uint32_t pi = atomicAdd(&P.ctr->pending_out, 1u);
        if (pi < P.pending_cap) P.pending_out[pi] = m;
        else atomicAdd(&P.ctr->lost, 1u);
    }
}

// ---- injection at the x = 0 face (not in the reference) ---------------------
// MurmurHash3's 64-bit finaliser (fmix64, A. Appleby, public domain) drives a
// counter-based generator keyed by (seed, step, cell, draw); the CPU oracle
// uses the same keys. Per face cell: floor(rate + u) particles, positions
// uniform in the cell, velocities drift + vth * Box-Muller normals.
__device__ __forceinline__ uint64_t fmix64(uint64_t k) {
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdULL;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ULL;
    k ^= k >> 33;
    return k;
}
__device__ __forceinline__ uint64_t inj_key(uint64_t seed, uint64_t step, uint64_t cell, uint64_t draw) {
    return fmix64(fmix64(seed ^ (step * 0x9E3779B97F4A7C15ULL)) ^ (cell * 0xD1B54A32D192ED03ULL + draw));
}
__device__ __forceinline__ double u01(uint64_t key) { return (double)(key >> 11) * (1.0 / 9007199254740992.0); }

struct InjectParams {
    double per_cell, drift[3], vth[3];
    uint64_t seed;
    const uint64_t* step;  // device step counter
};

template <typename T>
__global__ void k_inject(Geom g, Pop<T> P, InjectParams ip) {
    // one thread per face cell; the warp takes its cells' particles one round
    // at a time (warp-aggregated outbox appends, cooperative deposit)
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int j = 0, k = 0, c = 0, n = 0;
    const uint64_t step = *ip.step;
    if (f < g.sy * g.sz) {
        j = f / g.sz;
        k = f - j * g.sz;
        c = cell_id(g, 0, j, k);
        n = (int)floor(ip.per_cell + u01(inj_key(ip.seed, step, (uint64_t)c, 0)));
    }
    const int nmax = __reduce_max_sync(0xffffffffu, n);
    for (int m = 0; m < nmax; ++m) {
        const bool has = m < n;
        PState<T> p = {};
        Mover<T> mv = {};
        if (has) {
            const uint64_t d = 1 + 8 * (uint64_t)m;
            double u[7];
#pragma unroll
            for (int t = 0; t < 7; ++t) u[t] = u01(inj_key(ip.seed, step, (uint64_t)c, d + t));
            if constexpr (std::is_same<T, double>::value) {
                const double g1 = sqrt(-2.0 * log(1.0 - u[3])), th1 = 2.0 * 3.14159265358979323846 * u[4];
                const double g2 = sqrt(-2.0 * log(1.0 - u[5])), th2 = 2.0 * 3.14159265358979323846 * u[6];
                p.x = g.origin[0] + u[0] * g.w[0];
                p.y = g.origin[1] + ((double)j + u[1]) * g.w[1];
                p.z = g.origin[2] + ((double)k + u[2]) * g.w[2];
                p.u = ip.drift[0] + ip.vth[0] * (g1 * cos(th1));
                p.v = ip.drift[1] + ip.vth[1] * (g1 * sin(th1));
                p.w = ip.drift[2] + ip.vth[2] * (g2 * cos(th2));
            } else {
                // the same draws, Box-Muller in FP32 (GB300's FP64
                // transcendentals would dominate this kernel)
                const float g1 = sqrtf(-2.f * logf(1.f - (float)u[3])), g2 = sqrtf(-2.f * logf(1.f - (float)u[5]));
                float s1, c1, s2, c2;
                sincospif(2.f * (float)u[4], &s1, &c1);
                sincospif(2.f * (float)u[6], &s2, &c2);
                p.x = (float)u[0]; p.y = (float)u[1]; p.z = (float)u[2];
                p.u = (float)ip.drift[0] + (float)ip.vth[0] * (g1 * c1);
                p.v = (float)ip.drift[1] + (float)ip.vth[1] * (g1 * s1);
                p.w = (float)ip.drift[2] + (float)ip.vth[2] * (g2 * c2);
            }
            mv = {c, 0xffffffffu, p.x, p.y, p.z, p.u, p.v, p.w};
        }
        const uint32_t o = warp_append(&P.ctr->outbox, has);
        if (has) {
            if (o < P.outbox_cap) {
                P.outbox[o] = mv;
                register_arrival(P, o, mv);
            } else {
                atomicAdd(&P.ctr->lost, 1u);
            }
        }
        if (g.deposit) warp_deposit_leavers<T>(g, has, c, p, P.q);
    }
    const int tot = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0 && tot) atomicAdd(&P.ctr->injected, (uint32_t)tot);
}

// ---- import ---------------------------------------------------------------------
// Fills a cell's holes (ascending) with its arrivals; surplus arrivals append
// after the last particle, surplus holes are closed by moving the cell's last
// particles into them. Arrivals beyond the cell's slots go to the pending
// list and are pushed and placed again next step.
//
// The kernels wait on memory, and what counts is the number of round trips in
// a row. A warp looks after up to 8 consecutive cells (place_cells_per_warp:
// fewer on small grids): one round of loads fetches the hole, arrival and
// particle counts and the slot ranges of all of them; groups of kPlaceLanes
// lanes then take the cells that have holes or arrivals, four at a time: the
// two lists, then the arriving records and the cell's last particles, then
// the stores. Cells with more than kPlaceLanes holes or arrivals take the
// whole warp (place_body, whose lists are sorted in memory). Listing the
// flagged cells in a kernel of its own and placing from the list took 4 + 13
// us on the headline workload and 4 + 21 us where most cells have arrivals;
// this takes 10 us on both.
constexpr int kPlaceLanes = 8;

// The general path, by a warp on cell c.
template <typename T>
__device__ __forceinline__ void place_body(const Geom& g, const Pop<T>& P, int32_t* sort_tmp, int c) {
    constexpr int kG = 32;
    const int lane = threadIdx.x & 31;
    const int nh = P.hole_cnt[c], na_all = P.arr_cnt[c];
    const int64_t s0 = P.start[c];
    const int cap = (int)(P.start[c + 1] - s0);
    const int cnt = P.count[c];
    const int na = na_all < cap ? na_all : cap;
    const int free_slots = cap - (cnt - nh);
    const int np = na < free_slots ? na : free_slots;
    for (int i = np + lane; i < na; i += kG) {
        const Mover<T> m = P.outbox[P.arr_list[s0 + i]];
        uint32_t pi = atomicAdd(&P.ctr->pending_out, 1u);
        if (pi < P.pending_cap) P.pending_out[pi] = m;
        else atomicAdd(&P.ctr->lost, 1u);
    }
    // holes in ascending order (rank sort; hole counts are small; one hole
    // is sorted already)
    if (nh > 1) {
        for (int i = lane; i < nh; i += kG) {
            const int32_t h = P.hole_list[s0 + i];
            int r = 0;
            for (int j = 0; j < nh; ++j) r += P.hole_list[s0 + j] < h;
            sort_tmp[s0 + r] = h;
        }
        __syncwarp();
    }
    const int32_t* H = (nh > 1 ? sort_tmp : P.hole_list) + s0;
    const int m = nh < np ? nh : np;
    for (int i = lane; i < m; i += kG) write_slot(P, H[i], P.outbox[P.arr_list[s0 + i]]);
    for (int i = nh + lane; i < np; i += kG) write_slot(P, s0 + cnt + (i - nh), P.outbox[P.arr_list[s0 + i]]);
    const int newcount = cnt - nh + np;
    if (nh > np) {
        const int64_t lim = s0 + newcount, end = s0 + cnt;
        // remaining holes H[np, nh): the first L are below lim
        int lo = np, hi = nh;
        while (lo < hi) {
            int mid = (lo + hi) >> 1;
            if (H[mid] < lim) lo = mid + 1; else hi = mid;
        }
        const int L0 = lo;  // H[np, L0) < lim <= H[L0, nh)
        int filled = 0;
        for (int64_t b = lim; b < end; b += kG) {
            const int64_t t = b + lane;
            bool valid = false;
            if (t < end) {
                int a = L0, z = nh;  // is t one of the holes H[L0, nh)?
                while (a < z) {
                    int mid = (a + z) >> 1;
                    if (H[mid] < t) a = mid + 1; else z = mid;
                }
                valid = !(a < nh && H[a] == t);
            }
            const unsigned bal = __ballot_sync(0xffffffffu, valid);
            const int idx = filled + __popc(bal & ((1u << lane) - 1u));
            if (valid) move_slot(P, t, H[np + idx]);
            filled += __popc(bal);
        }
    }
    if (lane == 0) {
        P.count[c] = newcount;
        P.hole_cnt[c] = 0;
        P.arr_cnt[c] = 0;
    }
}

// The cells [c0, c0 + cells) of population P, cells <= 8, by one warp.
template <typename T>
__device__ __forceinline__ void place_cells(const Geom& g, const Pop<T>& P, int32_t* sort_tmp, int c0, int cells) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int kG = kPlaceLanes;
    const int lane = threadIdx.x & 31, gl = lane & (kG - 1), grp = lane / kG;
    cells = min(cells, g.ncells - c0);
    int v = 0;
    int64_t s = 0;
    {   // lanes 0-7 the holes, 8-15 the arrivals, 16-23 the particles of a cell each
        const int32_t* tab = lane < 8 ? P.hole_cnt : lane < 16 ? P.arr_cnt : P.count;
        if (lane < 24 && (lane & 7) < cells) v = tab[c0 + (lane & 7)];
        if (lane <= cells) s = P.start[c0 + lane];
    }
    const unsigned any = __ballot_sync(kAll, v != 0), many = __ballot_sync(kAll, v > kG);
    unsigned heavy = (many | (many >> 8)) & 0xffu;
    unsigned todo = (any | (any >> 8)) & 0xffu & ~heavy;
    for (; heavy; heavy &= heavy - 1) {
        __syncwarp();
        place_body<T>(g, P, sort_tmp, c0 + __ffs(heavy) - 1);
    }
    while (todo) {
        // group k takes the k-th cell left
        unsigned t = todo;
        for (int k = 0; k < grp; ++k) t &= t - 1;
        const bool small = t != 0;
        const int i = small ? __ffs(t) - 1 : 0;
#pragma unroll
        for (int k = 0; k < 32 / kG; ++k) todo &= todo - 1;
        const int nh = __shfl_sync(kAll, v, i), na_all = __shfl_sync(kAll, v, 8 + i);
        const int cnt = __shfl_sync(kAll, v, 16 + i);
        const int64_t s0 = __shfl_sync(kAll, s, i), s1 = __shfl_sync(kAll, s, i + 1);
        const int cap = (int)(s1 - s0);
        const int na = small ? min(na_all, cap) : 0, holes = small ? nh : 0;
        const int np = min(na, cap - (cnt - holes));  // arrivals that find a slot
        const int newcount = cnt - holes + np;
        int32_t h = gl < holes ? P.hole_list[s0 + gl] : 0x7fffffff;
        const int32_t o = gl < na ? P.arr_list[s0 + gl] : 0;
        // the arriving record and, where holes are left over, the cell's last
        // particles: issued together
        Mover<T> m = {};
        if (gl < na) m = P.outbox[o];
        const int left = holes - np;  // > 0: holes to close, as many last slots
        const int64_t tail = s0 + newcount + gl;
        const bool in_tail = gl < left;
        Mover<T> last = {};
        if (in_tail) {
            last.x = P.x[tail]; last.y = P.y[tail]; last.z = P.z[tail];
            last.u = P.u[tail]; last.v = P.v[tail]; last.w = P.w[tail];
            last.id = P.id ? P.id[tail] : 0u;
        }
        // the holes in ascending order: bitonic, 8 lanes
#pragma unroll
        for (int size = 2; size <= kG; size <<= 1)
#pragma unroll
            for (int step = size >> 1; step >= 1; step >>= 1) {
                const int32_t x = __shfl_xor_sync(kAll, h, step);
                const bool up = (gl & size) == 0, low = (gl & step) == 0;
                h = (up == low) ? min(h, x) : max(h, x);
            }
        if (gl < na && gl >= np) {  // no slot: waits a step
            const uint32_t pi = atomicAdd(&P.ctr->pending_out, 1u);
            if (pi < P.pending_cap) P.pending_out[pi] = m;
            else atomicAdd(&P.ctr->lost, 1u);
        }
        if (gl < np) write_slot(P, gl < holes ? (int64_t)h : s0 + cnt + (gl - holes), m);
        // is this lane's last slot one of the remaining holes H[np, holes)?
        bool valid = in_tail;
#pragma unroll
        for (int k = 0; k < kG; ++k) {
            const int32_t x = __shfl_sync(kAll, h, k, kG);
            valid = valid && !(k >= np && (int64_t)x == tail);
        }
        const unsigned moving = (__ballot_sync(kAll, valid) >> (grp * kG)) & 0xffu;
        const int32_t to = __shfl_sync(kAll, h, max(0, np) + __popc(moving & ((1u << gl) - 1u)), kG);
        if (valid) write_slot(P, to, last);
        if (small && gl == 0) {
            P.count[c0 + i] = newcount;
            P.hole_cnt[c0 + i] = 0;
            P.arr_cnt[c0 + i] = 0;
        }
    }
}

// Population blockIdx.y of the set, `cells` cells per warp.
template <typename T>
__global__ void __launch_bounds__(kPlaceThreads) k_place(Geom g, const __grid_constant__ PopSet<T> S, int cells) {
    const int64_t c0 = (blockIdx.x * (int64_t)kPlaceThreads + threadIdx.x) / 32 * cells;
    if (c0 < g.ncells) place_cells<T>(g, S.p[blockIdx.y], S.sort_tmp[blockIdx.y], (int)c0, cells);
}

// Moves this step's pending list to the next step's input (thread t0 = 0
// also sets the count).
template <typename T>
__device__ __forceinline__ void pending_rotate_body(const Pop<T>& P, uint32_t* pending_in_count, uint32_t t0,
                                                    uint32_t stride) {
    uint32_t n = P.ctr->pending_out;
    if (n > P.pending_cap) n = P.pending_cap;
    for (uint32_t i = t0; i < n; i += stride) P.pending_in[i] = P.pending_out[i];
    if (t0 == 0) *pending_in_count = n;
}

// Population blockIdx.y; thread 0 of population 0 also advances the device
// step counter (`step`, may be null), which keys the injection generator.
template <typename T>
__global__ void k_pending_rotate(const __grid_constant__ PopSet<T> S, uint64_t* step) {
    pending_rotate_body<T>(S.p[blockIdx.y], S.pend_count[blockIdx.y], blockIdx.x * blockDim.x + threadIdx.x,
                           gridDim.x * blockDim.x);
    if (step && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *step += 1;
}

// ---- re-layout (cells ran out of slack) ---------------------------------------
// Pending particles per cell.
template <typename T>
__global__ void k_pending_count(const Mover<T>* pend, const uint32_t* n_pend, int32_t* per_cell) {
    const uint32_t n = *n_pend;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        atomicAdd(per_cell + pend[i].cell, 1);
}

// One warp per cell: the cell's particles move to the new slot range.
template <typename T>
__global__ void k_relayout_copy(Pop<T> from, Pop<T> to, int ncells) {
    const int c = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (c >= ncells) return;
    const int64_t a = from.start[c], b = to.start[c];
    const int n = from.count[c];
    for (int i = lane; i < n; i += 32) {
        to.x[b + i] = from.x[a + i]; to.y[b + i] = from.y[a + i]; to.z[b + i] = from.z[a + i];
        to.u[b + i] = from.u[a + i]; to.v[b + i] = from.v[a + i]; to.w[b + i] = from.w[a + i];
        if (to.id) to.id[b + i] = from.id[a + i];
    }
    if (lane == 0) to.count[c] = n;
}

// Pending particles go after the copied ones (the new capacities hold them).
template <typename T>
__global__ void k_pending_place(const Mover<T>* pend, const uint32_t* n_pend, Pop<T> to) {
    const uint32_t n = *n_pend;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const Mover<T> m = pend[i];
        const int k = atomicAdd(to.count + m.cell, 1);
        write_slot(to, to.start[m.cell] + k, m);
    }
}

}  // namespace ipg
