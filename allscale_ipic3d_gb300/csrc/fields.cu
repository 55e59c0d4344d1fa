// Field-grid kernels of the GB300 path (FP64, built with -fmad=false so every
// expression rounds as the reference's does).
//
//   k_ghost        updateFieldsOnBoundaries (field.h:407-440)
//   k_leapfrog_e   solveFieldLeapfrog, E part   (field.h:359-363)
//   k_leapfrog_b   solveFieldLeapfrog, Bc part  (field.h:366-372)
//   k_forward_e/b  solveFieldForward            (field.h:294-337, curls 162-229)
//   k_interp_c2n   interpC2N                    (field.h:234-247)
//   k_j_finalize   J = (Js / vol) / 8           (cell.h:822-823) plus the
//                  periodic duplicate nodes of the gather form (cell.h:799-805)
//   k_node32       FP32 copy of node E, B for the FP32 gather
//   reductions     getFieldEnergy (field.h:443-459), particle sums
//                  (cell.h:1315-1355), Neumaier-compensated
//
// The reference's per-node solver updates E and then Bc in one in-place pass
// whose result depends on the visiting order; here E is updated everywhere
// first and Bc afterwards (the order-independent two-phase reading).
#include <algorithm>
#include <cmath>

#include "launch.h"

namespace ipg {

namespace {

__device__ __forceinline__ int64_t fidx(int n, int x, int y, int z) { return ((int64_t)x * n + y) * n + z; }

// Copies the six ghost faces of a cubic grid of n^3 records of `per` doubles:
// index (a, b) in [1, n-1)^2 of each face (edges and corners stay).
__device__ __forceinline__ void ghost_body(double* g, int n, int per, int64_t t0, int64_t stride) {
    const int end = n - 1;
    const int64_t m = (int64_t)(end - 1) * (end - 1);
    for (int64_t t = t0; t < m * per; t += stride) {
        int a, b, comp;
        split3(t, end - 1, per, a, b, comp);  // t = (a' (end - 1) + b') per + comp
        a += 1;
        b += 1;
        g[fidx(n, 0, a, b) * per + comp] = g[fidx(n, end - 1, a, b) * per + comp];
        g[fidx(n, end, a, b) * per + comp] = g[fidx(n, 1, a, b) * per + comp];
        g[fidx(n, a, 0, b) * per + comp] = g[fidx(n, a, end - 1, b) * per + comp];
        g[fidx(n, a, end, b) * per + comp] = g[fidx(n, a, 1, b) * per + comp];
        g[fidx(n, a, b, 0) * per + comp] = g[fidx(n, a, b, end - 1) * per + comp];
        g[fidx(n, a, b, end) * per + comp] = g[fidx(n, a, b, 1) * per + comp];
    }
}

struct SolverArgs {
    int s;                // cells per axis (cubic)
    double dt, c, c2;     // c2 = c^2
    double w[3];
    double iw[3];         // 1 / w
    float4* n32;          // FP32 node copy {Ex,Ey,Ez,0},{Bx,By,Bz,0} kept current (FP32 path), or null
    double* field;        // (s+3)^3 x 9
    double* bc;           // (s+2)^3 x 3
    const double* J;      // (s+1)^3 x 3
    // J as the E update reads it: jmode 0, final (folded, normalised); else
    // raw node sums of the deposit, folded over the periodic images and
    // normalised on the read exactly as k_j_finalize (jmode 1: / vol [/ 8])
    // or k_j_finalize_mul (jmode 2: * jinv) would store them
    int jmode, jdiv8;
    double jvol, jivol;   // vol, 1 / vol
    double jinv;          // 1 / vol [/ 8]
};

// Component `comp` of J at node m (per axis in [0, s]) as the J finalisation
// stores it: the sum over the node's images {0, s} on each axis where it lies
// on the boundary, in the finalisation's order, then normalised.
__device__ __forceinline__ double final_j(const SolverArgs& A, int mx, int my, int mz, int comp) {
    const int s = A.s, nd = A.s + 1;
    const int x = mx == s ? 0 : mx, y = my == s ? 0 : my, z = mz == s ? 0 : mz;
    const int nxs = x == 0 ? 2 : 1, nys = y == 0 ? 2 : 1, nzs = z == 0 ? 2 : 1;
    double a = soft::plus_zero(A.J[3 * fidx(nd, x, y, z) + comp]);
    for (int i = 0; i < nxs; ++i)
        for (int j = 0; j < nys; ++j)
            for (int k = 0; k < nzs; ++k)
                if (i + j + k) a += A.J[3 * fidx(nd, i ? s : x, j ? s : y, k ? s : z) + comp];
    if (A.jmode == 1) {
        a = soft::quotient(a, A.jvol, A.jivol, 0);
        if (A.jdiv8) a = a * 0.125;
    } else {
        a = a * A.jinv;
    }
    return a;
}

__device__ __forceinline__ double read_j(const SolverArgs& A, int mx, int my, int mz, int comp) {
    return A.jmode == 0 ? A.J[3 * fidx(A.s + 1, mx, my, mz) + comp] : final_j(A, mx, my, mz, comp);
}

// d / w of an axis: the reference's division, correctly rounded (kMul false),
// or the product with 1 / w (kMul: equal bit for bit when w is a power of two;
// the FP32 path's solver otherwise)
template <bool kMul>
__device__ __forceinline__ double over(double d, double w, double iw) {
    return kMul ? d * iw : soft::quotient(d, w, iw, 0);
}

// The leapfrog, the node refresh and the J finalisation of smaller grids run a
// thread per node and component, components fastest: neighbouring lanes read neighbouring
// doubles, and three times the threads hide the latency of grids that fill
// the SMs once. A block works on a row (x, y) of the grid, so a thread divides
// by 3 only (a flat index costs two divisions by the grid size, as much as
// the update itself). The grids' traffic (72-byte records of which a kernel
// needs 24) bounds them; taking a third of the FP64 instructions out changed
// nothing. With the L2 warm, as in a step: 0.336 -> 0.325 ms a step at 48^3,
// a thread per node before.
struct NodeComp {
    int x, y, z, a, b, c;  // (a, b, c): the component and the next two axes, cyclic
};
// item r of row (x, y), coordinates from 1
__device__ __forceinline__ NodeComp node_comp(int x, int y, int r) {
    NodeComp p;
    const unsigned z = (unsigned)r / 3u;
    p.x = x + 1;
    p.y = y + 1;
    p.z = (int)z + 1;
    p.a = r - 3 * (int)z;
    p.b = p.a == 2 ? 0 : p.a + 1;
    p.c = p.a == 0 ? 2 : p.a - 1;
    return p;
}

__device__ __forceinline__ double pick(int a, const double (&v)[3]) { return a == 0 ? v[0] : a == 1 ? v[1] : v[2]; }

// E at pos in [1, s+2)^3 from Bc(pos), Bc(pos - e_i) and J(pos - 1).
template <bool kMul>
__device__ __forceinline__ void leapfrog_e_point(const SolverArgs& A, const NodeComp& p) {
    const int nb = A.s + 2, nf = A.s + 3;
    const int64_t sx = 3 * (int64_t)nb * nb, sy = 3 * (int64_t)nb, sz = 3;
    const double* B0 = A.bc + 3 * fidx(nb, p.x, p.y, p.z);
    const double* Bb = B0 - (p.b == 0 ? sx : p.b == 1 ? sy : sz);
    const double* Bc = B0 - (p.c == 0 ? sx : p.c == 1 ? sy : sz);
    const double wb = pick(p.b, A.w), iwb = pick(p.b, A.iw), wc = pick(p.c, A.w), iwc = pick(p.c, A.iw);
    const double J = read_j(A, p.x - 1, p.y - 1, p.z - 1, p.a);
    const int64_t f = fidx(nf, p.x, p.y, p.z);
    double* E = A.field + 9 * f + p.a;
    const double e =
        *E + A.dt * (A.c2 * (over<kMul>(B0[p.c] - Bb[p.c], wb, iwb) - over<kMul>(B0[p.b] - Bc[p.b], wc, iwc)) - J);
    *E = e;
    if (A.n32) reinterpret_cast<float*>(A.n32 + 2 * f)[p.a] = (float)e;
}

// Bc at pos in [1, s+1)^3 from the new E at pos and pos + e_i.
template <bool kMul>
__device__ __forceinline__ void leapfrog_b_point(const SolverArgs& A, const NodeComp& p) {
    const int nb = A.s + 2, nf = A.s + 3;
    const int64_t sx = 9 * (int64_t)nf * nf, sy = 9 * (int64_t)nf, sz = 9;
    const double* E0 = A.field + 9 * fidx(nf, p.x, p.y, p.z);
    const double* Eb = E0 + (p.b == 0 ? sx : p.b == 1 ? sy : sz);
    const double* Ec = E0 + (p.c == 0 ? sx : p.c == 1 ? sy : sz);
    const double wb = pick(p.b, A.w), iwb = pick(p.b, A.iw), wc = pick(p.c, A.w), iwc = pick(p.c, A.iw);
    double* B = A.bc + 3 * fidx(nb, p.x, p.y, p.z) + p.a;
    *B = *B - A.dt * (over<kMul>(Eb[p.c] - E0[p.c], wb, iwb) - over<kMul>(Ec[p.b] - E0[p.b], wc, iwc));
}

// node B at pos in [1, s+2)^3 = 1/8 sum of Bc at pos - (i,j,k) (interpC2N)
__device__ __forceinline__ void interp_c2n_point(const SolverArgs& A, const NodeComp& p) {
    const int64_t nb = A.s + 2;
    const double* B0 = A.bc + 3 * fidx((int)nb, p.x, p.y, p.z) + p.a;
    double a = soft::plus_zero(B0[0]);
#pragma unroll
    for (int m = 1; m < 8; ++m) a = a + B0[-3 * (((m >> 2) * nb + ((m >> 1) & 1)) * nb + (m & 1))];
    const double b = .125 * a;
    const int64_t f = fidx(A.s + 3, p.x, p.y, p.z);
    A.field[9 * f + 3 + p.a] = b;
    if (A.n32) reinterpret_cast<float*>(A.n32 + 2 * f + 1)[p.a] = (float)b;
}

// computeCurlB (field.h:162-193) at node pos from the 8 Bc at pos - (i,j,k).
template <bool kMul>
__device__ __forceinline__ void curl_b(const SolverArgs& A, int x, int y, int z, double& cx, double& cy, double& cz) {
    const int nb = A.s + 2;
    double b[2][2][2][3];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const double* p = A.bc + 3 * fidx(nb, x - i, y - j, z - k);
                b[i][j][k][0] = p[0]; b[i][j][k][1] = p[1]; b[i][j][k][2] = p[2];
            }
    // d/dy of z: (j=0) - (j=1) over the 4 (i,k); d/dz of y: (k=0) - (k=1); ...
    double zdy = over<kMul>(.25 * (b[0][0][0][2] - b[0][1][0][2] + b[0][0][1][2] - b[0][1][1][2] + b[1][0][0][2] - b[1][1][0][2] + b[1][0][1][2] - b[1][1][1][2]), A.w[1], A.iw[1]);
    double ydz = over<kMul>(.25 * (b[0][0][0][1] - b[0][0][1][1] + b[1][0][0][1] - b[1][0][1][1] + b[0][1][0][1] - b[0][1][1][1] + b[1][1][0][1] - b[1][1][1][1]), A.w[2], A.iw[2]);
    cx = zdy - ydz;
    double xdz = over<kMul>(.25 * (b[0][0][0][0] - b[0][0][1][0] + b[1][0][0][0] - b[1][0][1][0] + b[0][1][0][0] - b[0][1][1][0] + b[1][1][0][0] - b[1][1][1][0]), A.w[2], A.iw[2]);
    double zdx = over<kMul>(.25 * (b[0][0][0][2] - b[1][0][0][2] + b[0][0][1][2] - b[1][0][1][2] + b[0][1][0][2] - b[1][1][0][2] + b[0][1][1][2] - b[1][1][1][2]), A.w[0], A.iw[0]);
    cy = xdz - zdx;
    double ydx = over<kMul>(.25 * (b[0][0][0][1] - b[1][0][0][1] + b[0][0][1][1] - b[1][0][1][1] + b[0][1][0][1] - b[1][1][0][1] + b[0][1][1][1] - b[1][1][1][1]), A.w[0], A.iw[0]);
    double xdy = over<kMul>(.25 * (b[0][0][0][0] - b[0][1][0][0] + b[0][0][1][0] - b[0][1][1][0] + b[1][0][0][0] - b[1][1][0][0] + b[1][0][1][0] - b[1][1][1][0]), A.w[1], A.iw[1]);
    cz = ydx - xdy;
}

// computeCurlE (field.h:198-229) at centre pos from the 8 node E at pos + (i,j,k).
template <bool kMul>
__device__ __forceinline__ void curl_e(const SolverArgs& A, int x, int y, int z, double& cx, double& cy, double& cz) {
    const int nf = A.s + 3;
    double e[2][2][2][3];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const double* p = A.field + 9 * fidx(nf, x + i, y + j, z + k);
                e[i][j][k][0] = p[0]; e[i][j][k][1] = p[1]; e[i][j][k][2] = p[2];
            }
    double zdy = over<kMul>(.25 * (e[0][1][0][2] - e[0][0][0][2] + e[0][1][1][2] - e[0][0][1][2] + e[1][1][0][2] - e[1][0][0][2] + e[1][1][1][2] - e[1][0][1][2]), A.w[1], A.iw[1]);
    double ydz = over<kMul>(.25 * (e[0][0][1][1] - e[0][0][0][1] + e[1][0][1][1] - e[1][0][0][1] + e[0][1][1][1] - e[0][1][0][1] + e[1][1][1][1] - e[1][1][0][1]), A.w[2], A.iw[2]);
    cx = zdy - ydz;
    double xdz = over<kMul>(.25 * (e[0][0][1][0] - e[0][0][0][0] + e[1][0][1][0] - e[1][0][0][0] + e[0][1][1][0] - e[0][1][0][0] + e[1][1][1][0] - e[1][1][0][0]), A.w[2], A.iw[2]);
    double zdx = over<kMul>(.25 * (e[1][0][0][2] - e[0][0][0][2] + e[1][0][1][2] - e[0][0][1][2] + e[1][1][0][2] - e[0][1][0][2] + e[1][1][1][2] - e[0][1][1][2]), A.w[0], A.iw[0]);
    cy = xdz - zdx;
    double ydx = over<kMul>(.25 * (e[1][0][0][1] - e[0][0][0][1] + e[1][0][1][1] - e[0][0][1][1] + e[1][1][0][1] - e[0][1][0][1] + e[1][1][1][1] - e[0][1][1][1]), A.w[0], A.iw[0]);
    double xdy = over<kMul>(.25 * (e[0][1][0][0] - e[0][0][0][0] + e[0][1][1][0] - e[0][0][1][0] + e[1][1][0][0] - e[1][0][0][0] + e[1][1][1][0] - e[1][0][1][0]), A.w[1], A.iw[1]);
    cz = ydx - xdy;
}

template <bool kMul = false>
__device__ __forceinline__ void forward_e_body(SolverArgs A, int64_t t0, int64_t stride) {
    const int n = A.s + 1;
    const int64_t total = (int64_t)n * n * n;
    for (int64_t t = t0; t < total; t += stride) {
        int x, y, z;
        split3(t, n, n, x, y, z);
        ++x; ++y; ++z;
        double cx, cy, cz;
        curl_b<kMul>(A, x, y, z, cx, cy, cz);
        double J[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) J[a] = read_j(A, x - 1, y - 1, z - 1, a);
        double* E = A.field + 9 * fidx(A.s + 3, x, y, z);
        E[0] += (A.c * cx - J[0]) * A.dt;
        E[1] += (A.c * cy - J[1]) * A.dt;
        E[2] += (A.c * cz - J[2]) * A.dt;
        if (A.n32) A.n32[2 * fidx(A.s + 3, x, y, z)] = make_float4((float)E[0], (float)E[1], (float)E[2], 0.f);
    }
}

template <bool kMul = false>
__device__ __forceinline__ void forward_b_body(SolverArgs A, int64_t t0, int64_t stride) {
    const int n = A.s;
    const int64_t total = (int64_t)n * n * n;
    for (int64_t t = t0; t < total; t += stride) {
        int x, y, z;
        split3(t, n, n, x, y, z);
        ++x; ++y; ++z;
        double cx, cy, cz;
        curl_e<kMul>(A, x, y, z, cx, cy, cz);
        double* B = A.bc + 3 * fidx(A.s + 2, x, y, z);
        B[0] -= A.c * cx * A.dt;
        B[1] -= A.c * cy * A.dt;
        B[2] -= A.c * cz * A.dt;
    }
}

// A node's sum over vol [/ 8], correctly rounded with inv = 1 / vol (kMul
// false), or its product with inv.
template <bool kMul>
__device__ __forceinline__ double j_normal(double a, double vol, double inv, int div8) {
    if (kMul) return a * inv;
    a = soft::quotient(a, vol, inv, 0);
    return div8 ? a * 0.125 : a;
}

// The gather form of the reference adds, at node index 0 and index s of an
// axis, the same two cells (periodic wrap of the cell index): the final value
// of a node is the sum of the raw deposits over its image set {0, s} on every
// axis where it lies on the boundary. Then J = (Js / vol) [/ 8], correctly
// rounded (kMul false), or the product with `inv` = 1 / vol [/ 8] (the FP32
// path, and wherever vol is a power of two: then the product equals the
// reference's quotients bit for bit). Item r of row (x, y): node z = r / 4,
// component r % 4 (rho the last); the images' loads issued together (in
// loops over the images, one after the other, 8^3 cells took 10 us, now 3.5).
template <bool kMul>
__device__ __forceinline__ void j_finalize_point(int sx, int sy, int sz, double* J, double* rho, double vol, double inv,
                                                 int div8, int x, int y, int r) {
    const int ny = sy + 1, nz = sz + 1;
    const int comp = r & 3, z = r >> 2;
    double* const base = comp < 3 ? J + comp : rho;
    const int64_t pitch = comp < 3 ? 3 : 1;
    const auto normal = [&](double a) { return j_normal<kMul>(a, vol, inv, div8); };
    if (x != 0 && y != 0 && z != 0) {
        double* p = base + pitch * (((int64_t)x * ny + y) * nz + z);
        *p = normal(soft::plus_zero(*p));
    } else {
        int64_t n[8];
        double v[8];
        bool in[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            in[k] = (!(k & 4) || x == 0) && (!(k & 2) || y == 0) && (!(k & 1) || z == 0);
            n[k] = pitch * (((int64_t)((k & 4) ? sx : x) * ny + ((k & 2) ? sy : y)) * nz + ((k & 1) ? sz : z));
            if (in[k]) v[k] = base[n[k]];
        }
        double a = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (in[k]) a += v[k];
        a = normal(a);
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (in[k]) base[n[k]] = a;
    }
}

// The same by a thread per node (larger grids, launch_j_finalize; batches).
template <bool kMul>
__device__ __forceinline__ void j_finalize_node(int sx, int sy, int sz, double* J, double* rho, double vol, double inv,
                                                int div8, int x, int y, int z) {
    const int ny = sy + 1, nz = sz + 1;
    const int nxs = x == 0 ? 2 : 1, nys = y == 0 ? 2 : 1, nzs = z == 0 ? 2 : 1;
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    for (int i = 0; i < nxs; ++i)
        for (int j = 0; j < nys; ++j)
            for (int k = 0; k < nzs; ++k) {
                const int64_t n = ((int64_t)(i ? sx : x) * ny + (j ? sy : y)) * nz + (k ? sz : z);
                a[0] += J[3 * n]; a[1] += J[3 * n + 1]; a[2] += J[3 * n + 2]; a[3] += rho[n];
            }
#pragma unroll
    for (int c = 0; c < 4; ++c) a[c] = j_normal<kMul>(a[c], vol, inv, div8);
    for (int i = 0; i < nxs; ++i)
        for (int j = 0; j < nys; ++j)
            for (int k = 0; k < nzs; ++k) {
                const int64_t n = ((int64_t)(i ? sx : x) * ny + (j ? sy : y)) * nz + (k ? sz : z);
                J[3 * n] = a[0]; J[3 * n + 1] = a[1]; J[3 * n + 2] = a[2]; rho[n] = a[3];
            }
}

__global__ void k_node32(const double* field, float4* node32, int64_t nodes) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nodes; t += (int64_t)gridDim.x * blockDim.x) {
        const double* f = field + 9 * t;
        node32[2 * t] = make_float4((float)f[0], (float)f[1], (float)f[2], 0.f);
        node32[2 * t + 1] = make_float4((float)f[3], (float)f[4], (float)f[5], 0.f);
    }
}

__device__ __forceinline__ int64_t grid_t0() { return blockIdx.x * (int64_t)blockDim.x + threadIdx.x; }
__device__ __forceinline__ int64_t grid_stride() { return (int64_t)gridDim.x * blockDim.x; }

__host__ __device__ inline SolverArgs solver_args(const Geom& g) {
    SolverArgs A;
    A.s = g.sx;
    A.dt = g.dt;
    A.c = g.c;
    A.c2 = g.c * g.c;
    for (int a = 0; a < 3; ++a) {
        A.w[a] = g.w[a];
        A.iw[a] = g.inv_w[a];
    }
    A.field = g.field;
    A.bc = g.bcfield;
    A.J = g.J;
    A.n32 = g.node32;
    A.jmode = 0;
    A.jdiv8 = 0;
    A.jvol = g.vol;
    A.jivol = 1.0;
    A.jinv = 1.0;
    return A;
}

// single-universe kernels
// both grids' ghost faces in one launch: threads [0, nf_items) the field,
// the rest the Bc grid
__global__ void k_ghost2(double* field, int nf, double* bc, int nb) {
    const int64_t mf = (int64_t)(nf - 2) * (nf - 2) * 9;
    const int64_t t = grid_t0();
    if (t < mf)
        ghost_body(field, nf, 9, t, mf);
    else
        ghost_body(bc, nb, 3, t - mf, (int64_t)(nb - 2) * (nb - 2) * 3);
}
// rows: block (., y, x), items of the row along the threads
__device__ __forceinline__ int row_item() { return blockIdx.x * blockDim.x + threadIdx.x; }
template <bool kMul>
__global__ void k_leapfrog_e(SolverArgs A) {
    const int r = row_item();
    if (r < 3 * (A.s + 1)) leapfrog_e_point<kMul>(A, node_comp(blockIdx.z, blockIdx.y, r));
}
template <bool kMul>
__global__ void k_leapfrog_b(SolverArgs A) {
    const int r = row_item();
    if (r < 3 * A.s) leapfrog_b_point<kMul>(A, node_comp(blockIdx.z, blockIdx.y, r));
}
__global__ void k_interp_c2n(SolverArgs A) {
    const int r = row_item();
    if (r < 3 * (A.s + 1)) interp_c2n_point(A, node_comp(blockIdx.z, blockIdx.y, r));
}
template <bool kMul>
__global__ void k_j_finalize(int sx, int sy, int sz, double* J, double* rho, double vol, double inv, int div8) {
    const int r = row_item();
    if (r < 4 * sz) j_finalize_point<kMul>(sx, sy, sz, J, rho, vol, inv, div8, blockIdx.z, blockIdx.y, r);
}
template <bool kMul>
__global__ void __launch_bounds__(256)
    k_j_finalize_flat(int sx, int sy, int sz, double* J, double* rho, double vol, double inv, int div8) {
    for (int64_t t = grid_t0(); t < (int64_t)sx * sy * sz; t += grid_stride()) {
        int x, y, z;
        split3(t, sy, sz, x, y, z);
        j_finalize_node<kMul>(sx, sy, sz, J, rho, vol, inv, div8, x, y, z);
    }
}
template <bool kMul>
__global__ void k_forward_e(SolverArgs A) { forward_e_body<kMul>(A, grid_t0(), grid_stride()); }
template <bool kMul>
__global__ void k_forward_b(SolverArgs A) { forward_b_body<kMul>(A, grid_t0(), grid_stride()); }
// batched kernels: blockIdx.y is the universe, blockIdx.x strides over its
// items (the grid is sized for the largest universe of the batch)
__global__ void k_ghost_batch(const InstJob* jobs) {
    const Geom& g = jobs[blockIdx.y].g;
    ghost_body(g.field, g.sx + 3, 9, grid_t0(), grid_stride());
    ghost_body(g.bcfield, g.sx + 2, 3, grid_t0(), grid_stride());
}
// item t of the rows of n x n x len: row (x, y), item r of it
__device__ __forceinline__ void row_of(int64_t t, int n, int len, int& x, int& y, int& r) { split3(t, n, len, x, y, r); }
__global__ void k_leapfrog_e_batch(const InstJob* jobs) {
    const SolverArgs A = solver_args(jobs[blockIdx.y].g);
    const int n = A.s + 1;
    for (int64_t t = grid_t0(); t < 3 * (int64_t)n * n * n; t += grid_stride()) {
        int x, y, r;
        row_of(t, n, 3 * n, x, y, r);
        leapfrog_e_point<false>(A, node_comp(x, y, r));
    }
}
__global__ void k_leapfrog_b_batch(const InstJob* jobs) {
    const SolverArgs A = solver_args(jobs[blockIdx.y].g);
    const int n = A.s;
    for (int64_t t = grid_t0(); t < 3 * (int64_t)n * n * n; t += grid_stride()) {
        int x, y, r;
        row_of(t, n, 3 * n, x, y, r);
        leapfrog_b_point<false>(A, node_comp(x, y, r));
    }
}
__global__ void k_forward_e_batch(const InstJob* jobs) {
    forward_e_body(solver_args(jobs[blockIdx.y].g), grid_t0(), grid_stride());
}
__global__ void k_forward_b_batch(const InstJob* jobs) {
    forward_b_body(solver_args(jobs[blockIdx.y].g), grid_t0(), grid_stride());
}
__global__ void k_interp_c2n_batch(const InstJob* jobs) {
    const SolverArgs A = solver_args(jobs[blockIdx.y].g);
    const int n = A.s + 1;
    for (int64_t t = grid_t0(); t < 3 * (int64_t)n * n * n; t += grid_stride()) {
        int x, y, r;
        row_of(t, n, 3 * n, x, y, r);
        interp_c2n_point(A, node_comp(x, y, r));
    }
}
__global__ void k_j_finalize_batch(const InstJob* jobs) {
    const InstJob& b = jobs[blockIdx.y];
    const Geom& g = b.g;
    const double inv = b.div8 && b.mul_vol ? b.inv_vol * 0.125 : b.inv_vol;
    for (int64_t t = grid_t0(); t < (int64_t)g.sx * g.sy * g.sz; t += grid_stride()) {
        int x, y, z;
        split3(t, g.sy, g.sz, x, y, z);
        if (b.mul_vol) j_finalize_node<true>(g.sx, g.sy, g.sz, g.J, g.rho, g.vol, inv, b.div8, x, y, z);
        else j_finalize_node<false>(g.sx, g.sy, g.sz, g.J, g.rho, g.vol, inv, b.div8, x, y, z);
    }
}

// ---- compensated reductions ----------------------------------------------------
// Neumaier's improved Kahan summation: (s, c) with s + c the running sum.
struct Neu {
    double s, c;
    __device__ void add(double x) {
        double t = s + x;
        if (fabs(s) >= fabs(x)) c += (s - t) + x;
        else c += (x - t) + s;
        s = t;
    }
    __device__ void merge(const Neu& o) {
        add(o.s);
        c += o.c;
    }
};

__device__ __forceinline__ Neu shfl_neu(Neu a, int off) {
    Neu b;
    b.s = __shfl_down_sync(0xffffffffu, a.s, off);
    b.c = __shfl_down_sync(0xffffffffu, a.c, off);
    return b;
}

// Block-level merge of kQ compensated sums; thread 0 writes 2*kQ doubles.
template <int kQ>
__device__ void block_merge(Neu (&acc)[kQ], double* out) {
    __shared__ Neu sm[32][kQ];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < kQ; ++q)
        for (int off = 16; off > 0; off >>= 1) acc[q].merge(shfl_neu(acc[q], off));
    if (lane == 0)
        for (int q = 0; q < kQ; ++q) sm[wid][q] = acc[q];
    __syncthreads();
    if (threadIdx.x == 0) {
        const int nw = (blockDim.x + 31) / 32;
        for (int q = 0; q < kQ; ++q) {
            Neu t = {0.0, 0.0};
            for (int w = 0; w < nw; ++w) t.merge(sm[w][q]);
            out[2 * q] = t.s;
            out[2 * q + 1] = t.c;
        }
    }
}

// Particle sums of one population: sum (q/qom)|v|, sum 1/2 (q/qom)|v|^2,
// sum q (cell.h:1315-1338), over the particles in slots (slots beyond
// count[c] are skipped) and those waiting in the pending list.
template <typename T>
__device__ __forceinline__ void add_particle(Neu (&acc)[3], double m, double q, T u, T v, T w) {
    const double a = (double)u, b = (double)v, d = (double)w;
    double ss = a * a;
    ss += b * b;
    ss += d * d;
    acc[0].add(m * sqrt(ss));
    acc[1].add(0.5 * m * ss);
    acc[2].add(q);
}

template <typename T>
__global__ void k_reduce_particles(const T* u, const T* v, const T* w, const int64_t* start, const int32_t* count,
                                   int ncells, const Mover<T>* pend, const uint32_t* npend, double q, double qom,
                                   double* partial) {
    Neu acc[3] = {{0, 0}, {0, 0}, {0, 0}};
    const double m = q / qom;
    for (int c = blockIdx.x; c < ncells; c += gridDim.x) {
        const int64_t s0 = start[c];
        const int n = count[c];
        for (int i = threadIdx.x; i < n; i += blockDim.x) add_particle<T>(acc, m, q, u[s0 + i], v[s0 + i], w[s0 + i]);
    }
    const uint32_t np = *npend;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x)
        add_particle<T>(acc, m, q, pend[i].u, pend[i].v, pend[i].w);
    block_merge<3>(acc, partial + 6 * blockIdx.x);
}

// Field energies over [1, s+2)^3: vol * |E|^2 / 4pi and vol * |B + Bext|^2 /
// 4pi with vol = cell volume / 2 (field.h:443-459).
__global__ void k_reduce_fields(const double* field, int s, double vol, double four_pi, double* partial) {
    Neu acc[2] = {{0, 0}, {0, 0}};
    const int n = s + 1, nf = s + 3;
    const int64_t total = (int64_t)n * n * n;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        int x, y, z;
        split3(t, n, n, x, y, z);
        ++x; ++y; ++z;
        const double* f = field + 9 * fidx(nf, x, y, z);
        double e = f[0] * f[0];
        e += f[1] * f[1];
        e += f[2] * f[2];
        const double b0 = f[3] + f[6], b1 = f[4] + f[7], b2 = f[5] + f[8];
        double b = b0 * b0;
        b += b1 * b1;
        b += b2 * b2;
        acc[0].add(vol * e / four_pi);
        acc[1].add(vol * b / four_pi);
    }
    block_merge<2>(acc, partial + 4 * blockIdx.x);
}

// Final merge of `blocks` partial records of kq (s, c) pairs: warp q merges
// quantity q, lane l the records l, l + 32, ... in order, then the lanes'
// sums in a fixed shuffle tree (the same order every call).
__global__ void k_reduce_final(const double* partial, int blocks, int kq, double* out) {
    const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
    if (blockIdx.x != 0 || q >= kq) return;
    Neu t = {0.0, 0.0};
    for (int b = lane; b < blocks; b += 32) {
        t.add(partial[2 * kq * b + 2 * q]);
        t.c += partial[2 * kq * b + 2 * q + 1];
    }
    for (int off = 16; off > 0; off >>= 1) t.merge(shfl_neu(t, off));
    if (lane == 0) out[q] = t.s + t.c;
}

inline int grid_for(int64_t n, int threads, int64_t max_blocks = 152 * 32) {
    int64_t b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > max_blocks) b = max_blocks;
    return (int)b;
}


}  // namespace

// ---- host launchers ------------------------------------------------------------

int launch_ghost(const Geom& g, cudaStream_t st) {
    const int nf = g.sx + 3, nb = g.sx + 2;
    const int64_t items = (int64_t)(nf - 2) * (nf - 2) * 9 + (int64_t)(nb - 2) * (nb - 2) * 3;
    k_ghost2<<<(unsigned)((items + 255) / 256), 256, 0, st>>>(g.field, nf, g.bcfield, nb);
    return 1;
}

// The launch of a row kernel: nx x ny rows of `items`, at most 65535 each way
// (the solvers' grids are cubes, the J finalisation takes few rows this way).
struct Rows {
    dim3 grid;
    unsigned threads;
};
static Rows rows(int nx, int ny, int items) {
    Rows r;
    // evenly: 387 items (128^3) are a block of 416 threads, not 256 and 131
    const int blocks = (items + 511) / 512, each = (items + blocks - 1) / blocks;
    r.threads = (unsigned)(each + 31) / 32 * 32;
    r.grid = dim3(blocks, ny, nx);
    return r;
}

static bool pow2(double v) {
    int e = 0;
    return std::frexp(v, &e) == 0.5;
}

// raw J: read as the J finalisation (div8 / exact as launch_j_finalize's)
// would store it
static void set_raw_j(SolverArgs& A, const Geom& g, bool div8, bool exact);

int launch_leapfrog(const Geom& g, bool refresh_node_b, bool exact, cudaStream_t st, bool raw_j, bool div8,
                    cudaEvent_t after_e) {
    SolverArgs A = solver_args(g);
    if (raw_j) set_raw_j(A, g, div8, exact);
    const bool mul = !exact || (pow2(g.w[0]) && pow2(g.w[1]) && pow2(g.w[2]));
    const Rows nodes = rows(g.sx + 1, g.sx + 1, 3 * (g.sx + 1)), cells = rows(g.sx, g.sx, 3 * g.sx);
    if (mul) k_leapfrog_e<true><<<nodes.grid, nodes.threads, 0, st>>>(A);
    else k_leapfrog_e<false><<<nodes.grid, nodes.threads, 0, st>>>(A);
    if (after_e) cudaEventRecord(after_e, st);
    if (mul) k_leapfrog_b<true><<<cells.grid, cells.threads, 0, st>>>(A);
    else k_leapfrog_b<false><<<cells.grid, cells.threads, 0, st>>>(A);
    if (refresh_node_b) {
        k_interp_c2n<<<nodes.grid, nodes.threads, 0, st>>>(A);
        return 3;
    }
    return 2;
}

int launch_forward(const Geom& g, cudaStream_t st, bool raw_j, bool div8, bool exact, cudaEvent_t after_e) {
    SolverArgs A = solver_args(g);
    if (raw_j) set_raw_j(A, g, div8, exact);
    const int64_t ne = (int64_t)(g.sx + 1) * (g.sx + 1) * (g.sx + 1);
    const int64_t nc = (int64_t)g.sx * g.sx * g.sx;
    const bool mul = pow2(g.w[0]) && pow2(g.w[1]) && pow2(g.w[2]);  // the products are the quotients
    if (mul) k_forward_e<true><<<grid_for(ne, 256), 256, 0, st>>>(A);
    else k_forward_e<false><<<grid_for(ne, 256), 256, 0, st>>>(A);
    if (after_e) cudaEventRecord(after_e, st);
    if (mul) k_forward_b<true><<<grid_for(nc, 256), 256, 0, st>>>(A);
    else k_forward_b<false><<<grid_for(nc, 256), 256, 0, st>>>(A);
    const Rows nodes = rows(g.sx + 1, g.sx + 1, 3 * (g.sx + 1));
    k_interp_c2n<<<nodes.grid, nodes.threads, 0, st>>>(A);
    return 3;
}

static void set_raw_j(SolverArgs& A, const Geom& g, bool div8, bool exact) {
    A.jdiv8 = div8 ? 1 : 0;
    A.jvol = g.vol;
    A.jivol = 1.0 / g.vol;
    A.jinv = div8 ? 1.0 / g.vol / 8.0 : 1.0 / g.vol;
    A.jmode = exact && !pow2(g.vol) ? 1 : 2;  // launch_j_finalize's choice
}

int launch_j_finalize(const Geom& g, bool div8, bool exact, cudaStream_t st) {
    const bool mul = !exact || pow2(g.vol);  // vol = 2^k: 1 / vol is exact
    const double inv = mul && div8 ? 1.0 / g.vol / 8.0 : 1.0 / g.vol;
    const int64_t nodes = (int64_t)g.sx * g.sy * g.sz;
    // Above 160,000 nodes or 16,384 rows a thread per node is faster, below a
    // row's items side by side, whose blocks are then too many and too small.
    // us, rows / nodes (in brackets with the exact quotient): 32^3 4.6 / 10
    // (6.3 / 10.5), 48^3 8.2 / 11.5 (13.3 / 13.0), 59^3 11.6 / 10.9 (23 /
    // 19), 128^3 61 / 47 (125 / 120), 70 x 70 x 16 7.4 / 11.6 (12 / 13), 256 x
    // 256 x 4 43 / 13 (83 / 22), 1024 x 1024 x 1, 4 items a row, 579 / 31
    // (895 / 66).
    const bool flat = nodes > 160000 || (int64_t)g.sx * g.sy > 16384;
    const Rows r = rows(g.sx, g.sy, 4 * g.sz);
    const auto run = [&](auto k, dim3 grid, unsigned threads) {
        k<<<grid, threads, 0, st>>>(g.sx, g.sy, g.sz, g.J, g.rho, g.vol, inv, div8 ? 1 : 0);
    };
    if (flat && mul) run(k_j_finalize_flat<true>, grid_for(nodes, 256), 256);
    else if (flat) run(k_j_finalize_flat<false>, grid_for(nodes, 256), 256);
    else if (mul) run(k_j_finalize<true>, r.grid, r.threads);
    else run(k_j_finalize<false>, r.grid, r.threads);
    return 1;
}

int launch_node32(const Geom& g, float4* node32, cudaStream_t st) {
    const int64_t nodes = (int64_t)(g.sx + 3) * (g.sy + 3) * (g.sz + 3);
    k_node32<<<grid_for(nodes, 256), 256, 0, st>>>(g.field, node32, nodes);
    return 1;
}

// batched launchers: `ninst` universes, `max_s` the largest cells per axis
int launch_ghost_batch(const InstJob* jobs, int ninst, int max_s, cudaStream_t st) {
    const int64_t m = (int64_t)(max_s + 1) * (max_s + 1) * 9;
    k_ghost_batch<<<dim3(grid_for(m, 256, 64), ninst), 256, 0, st>>>(jobs);
    return 1;
}

int launch_leapfrog_batch(const InstJob* jobs, int ninst, int max_s, bool refresh_node_b, cudaStream_t st) {
    const int64_t ne = (int64_t)(max_s + 1) * (max_s + 1) * (max_s + 1);
    const unsigned gx = grid_for(3 * ne, 256, 192);
    k_leapfrog_e_batch<<<dim3(gx, ninst), 256, 0, st>>>(jobs);
    k_leapfrog_b_batch<<<dim3(gx, ninst), 256, 0, st>>>(jobs);
    if (!refresh_node_b) return 2;
    k_interp_c2n_batch<<<dim3(gx, ninst), 256, 0, st>>>(jobs);
    return 3;
}

int launch_forward_batch(const InstJob* jobs, int ninst, int max_s, cudaStream_t st) {
    const int64_t ne = (int64_t)(max_s + 1) * (max_s + 1) * (max_s + 1);
    const unsigned gx = grid_for(ne, 256, 64);
    k_forward_e_batch<<<dim3(gx, ninst), 256, 0, st>>>(jobs);
    k_forward_b_batch<<<dim3(gx, ninst), 256, 0, st>>>(jobs);
    k_interp_c2n_batch<<<dim3(gx, ninst), 256, 0, st>>>(jobs);
    return 3;
}

int launch_j_finalize_batch(const InstJob* jobs, int ninst, int64_t max_cells, cudaStream_t st) {
    k_j_finalize_batch<<<dim3(grid_for(max_cells, 256, 64), ninst), 256, 0, st>>>(jobs);
    return 1;
}

int reduce_blocks() { return 152 * 4; }

template <typename T>
int launch_reduce_particles(const Pop<T>& P, int ncells, double* partial, cudaStream_t st) {
    k_reduce_particles<T><<<reduce_blocks(), 256, 0, st>>>(P.u, P.v, P.w, P.start, P.count, ncells, P.pending_in,
                                                            P.pending_in_count, P.q, P.qom, partial);
    return 1;
}
template int launch_reduce_particles<float>(const Pop<float>&, int, double*, cudaStream_t);
template int launch_reduce_particles<double>(const Pop<double>&, int, double*, cudaStream_t);

int launch_reduce_fields(const Geom& g, double* partial, cudaStream_t st) {
    const double vol = 0.5 * g.w[0] * g.w[1] * g.w[2];
    const double four_pi = 16.0 * atan(1.0);
    k_reduce_fields<<<reduce_blocks(), 256, 0, st>>>(g.field, g.sx, vol, four_pi, partial);
    return 1;
}

int launch_reduce_final(const double* partial, int blocks, int kq, double* out, cudaStream_t st) {
    k_reduce_final<<<1, 32 * kq, 0, st>>>(partial, blocks, kq, out);
    return 1;
}

}  // namespace ipg
