// omx_fd.cu -- the frequency-domain operator of the reference's inverse-design program on the GPU
// (src/freq_domain_inverse_design/operator_mod.f90: apply_operator_1D :293-361, _2D :364-514,
// _3D :518-710) and its BiCGStab(L) solver (bicgstab_mod.f90:76-243).
//
// Vectors are complex components (Riemann-Silberstein pl_x, pl_y, pl_z, mi_x, mi_y, mi_z; in 1D
// pl_x, pl_y, mi_x, mi_y), each an array over [1-g, n+g] along every active axis (g = n_der
// ghost cells), x fastest, FP64 as in the reference.
// The operator kernel keeps the reference's operand order with FMA contraction off (this file is
// compiled with -fmad=false), so A f equals the FP64 oracle bit for bit.  The solver's scalar
// recursion runs on the host exactly as the oracle's; its dot products are reduced on the device
// per row of cells and summed on the host in row order (deterministic, not the oracle's order).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/omx_gpu.h"

namespace omx {
void set_global_error(const std::string &msg);
}

namespace {

struct cplx {
    double re, im;
};
__host__ __device__ inline cplx cadd(cplx a, cplx b) { return {a.re + b.re, a.im + b.im}; }
__host__ __device__ inline cplx csub(cplx a, cplx b) { return {a.re - b.re, a.im - b.im}; }
__host__ __device__ inline cplx cmul(cplx a, cplx b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__host__ __device__ inline cplx cscale(cplx a, double s) { return {a.re * s, a.im * s}; }
// complex division by Smith's method (R. L. Smith, CACM 5:435, 1962), the range-reduced form
// gfortran uses for complex(dp) division under its default Fortran rules
inline cplx cdiv(cplx a, cplx b)
{
    if (std::fabs(b.re) < std::fabs(b.im)) {
        const double t = b.re / b.im, d = b.re * t + b.im;
        return {(a.re * t + a.im) / d, (a.im * t - a.re) / d};
    }
    const double t = b.im / b.re, d = b.im * t + b.re;
    return {(a.im * t + a.re) / d, (a.im - a.re * t) / d};
}

struct FdGeom {
    int dims, ncomp, nx, ny, nz, g, gy, gz, n_der;   // ny = nz = 1 in 1D, nz = 1 in 2D
    long long px, pxy, len;   // padded row and plane pitch, elements per component
    int per[3];
    double coef[9];
    double w0, w0_half, sign;
};

__device__ inline long long fd_at(const FdGeom &G, int i, int j, int k)   // 1-based interior indices
{
    return (long long)(i - 1 + G.g) + G.px * (j - 1 + G.gy) + G.pxy * (k - 1 + G.gz);
}

// periodic ghost copies (1D operator_mod.f90:316-329, 2D :389-452, 3D :549-621): axis 0 over
// interior y, z; axis 1 over interior x, z (in 3D with mi_x only into the low ghosts and mi_y only
// into the high ones); axis 2 over interior x, y.  One thread per (component, ghost cell pair).
__global__ void k_fd_ghosts(cplx *f, FdGeom G, int axis)
{
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int na = axis == 0 ? G.nx : (axis == 1 ? G.ny : G.nz);
    const int n1 = axis == 0 ? G.ny : G.nx, n2 = axis == 2 ? G.ny : G.nz;
    const long long per_c = (long long)G.g * n1 * n2;
    if (q >= G.ncomp * per_c) return;
    const int c = (int)(q / per_c);
    long long r = q % per_c;
    const int t = 1 + (int)(r % G.g);
    r /= G.g;
    const int a1 = 1 + (int)(r % n1), a2 = 1 + (int)(r / n1);
    cplx *v = f + c * G.len;
    auto at = [&](int s) {
        if (axis == 0) return fd_at(G, s, a1, a2);
        if (axis == 1) return fd_at(G, a1, s, a2);
        return fd_at(G, a1, a2, s);
    };
    const bool quirk = axis == 1 && G.dims == 3;
    const bool lo = !(quirk && c == 4), hi = !(quirk && c == 3);
    if (lo) v[at(1 - t)] = v[at(na + 1 - t)];
    if (hi) v[at(na + t)] = v[at(t)];
}

// The operator's cell functions.  fd_cell drops what is exact in finite arithmetic: the zero centre
// tap and products with the zero parts of C1..C4 and with a stretch factor of 1 (282 of 476 FP64
// operations a cell left in 3D at n_der 2, and 72 more in cells with PML on every axis).  Infinities
// and NaN spread differently through the dropped products, so a component that meets one is computed
// again by the full form below, which writes every product out as the reference's complex
// arithmetic does.
struct FdTables {
    const cplx *sx, *sy, *sz, *eps;
};

// component c of apply_operator_3D at one cell, written out
__device__ __noinline__ void fd_full3(const cplx *f, cplx *Af, const FdGeom &G, const FdTables &T, int i, int j, int k,
                                     int c)
{
    const cplx *sx = T.sx, *sy = T.sy, *sz = T.sz, *eps = T.eps;
    const long long p = fd_at(G, i, j, k);
    const cplx *plx = f, *ply = f + G.len, *plz = f + 2 * G.len, *mix = f + 3 * G.len, *miy = f + 4 * G.len,
               *miz = f + 5 * G.len;
    const int n = G.n_der;
    cplx dpydx = {0, 0}, dpzdx = {0, 0}, dmydx = {0, 0}, dmzdx = {0, 0};
    cplx dpxdy = {0, 0}, dpzdy = {0, 0}, dmxdy = {0, 0}, dmzdy = {0, 0};
    cplx dpxdz = {0, 0}, dpydz = {0, 0}, dmxdz = {0, 0}, dmydz = {0, 0};
    for (int q = -n; q <= n; ++q) {
        const double a = G.coef[n + q];
        dpydx = cadd(dpydx, cscale(ply[p + q], a));
        dpzdx = cadd(dpzdx, cscale(plz[p + q], a));
        dmydx = cadd(dmydx, cscale(miy[p + q], a));
        dmzdx = cadd(dmzdx, cscale(miz[p + q], a));
    }
    for (int q = -n; q <= n; ++q) {
        const double a = G.coef[n + q];
        const long long o = p + q * G.px;
        dpxdy = cadd(dpxdy, cscale(plx[o], a));
        dpzdy = cadd(dpzdy, cscale(plz[o], a));
        dmxdy = cadd(dmxdy, cscale(mix[o], a));
        dmzdy = cadd(dmzdy, cscale(miz[o], a));
    }
    for (int q = -n; q <= n; ++q) {
        const double a = G.coef[n + q];
        const long long o = p + q * G.pxy;
        dpxdz = cadd(dpxdz, cscale(plx[o], a));
        dpydz = cadd(dpydz, cscale(ply[o], a));
        dmxdz = cadd(dmxdz, cscale(mix[o], a));
        dmydz = cadd(dmydz, cscale(miy[o], a));
    }
    const cplx Ex = cadd(plx[p], mix[p]), Ey = cadd(ply[p], miy[p]), Ez = cadd(plz[p], miz[p]);
    const cplx sxi = sx[i - 1], syj = sy[j - 1], szk = sz[k - 1];
    dpxdy = cmul(dpxdy, syj);
    dpxdz = cmul(dpxdz, szk);
    dpydx = cmul(dpydx, sxi);
    dpydz = cmul(dpydz, szk);
    dpzdx = cmul(dpzdx, sxi);
    dpzdy = cmul(dpzdy, syj);
    dmxdy = cmul(dmxdy, syj);
    dmxdz = cmul(dmxdz, szk);
    dmydz = cmul(dmydz, szk);
    dmydx = cmul(dmydx, sxi);
    dmzdx = cmul(dmzdx, sxi);
    dmzdy = cmul(dmzdy, syj);
    // C1 = sign c0 i, C2 = -w0 i, C3 = -w0 i / (2 eps0), C4 = eps0 (c0 = eps0 = 1)
    const cplx C1 = {0.0, G.sign}, mC1 = {-0.0, -G.sign}, C2 = {0.0, -G.w0}, C3 = {0.0, -G.w0 / 2.0}, C4 = {1.0, 0.0};
    const cplx e = eps[(long long)(i - 1) + (long long)G.nx * ((j - 1) + (long long)G.ny * (k - 1))];
    const cplx m3 = cmul(C3, csub(e, C4));
    cplx out[6];
    out[0] = cadd(cadd(cmul(C1, csub(dpzdy, dpydz)), cmul(C2, plx[p])), cmul(m3, Ex));
    out[1] = cadd(cadd(cmul(C1, csub(dpxdz, dpzdx)), cmul(C2, ply[p])), cmul(m3, Ey));
    out[2] = cadd(cadd(cmul(C1, csub(dpydx, dpxdy)), cmul(C2, plz[p])), cmul(m3, Ez));
    out[3] = cadd(cadd(cmul(mC1, csub(dmzdy, dmydz)), cmul(C2, mix[p])), cmul(m3, Ex));
    out[4] = cadd(cadd(cmul(mC1, csub(dmxdz, dmzdx)), cmul(C2, miy[p])), cmul(m3, Ey));
    out[5] = cadd(cadd(cmul(mC1, csub(dmydx, dmxdy)), cmul(C2, miz[p])), cmul(m3, Ez));
    for (int y = 0; y < 6; ++y)
        if (y == c) Af[p + c * G.len] = out[y];
}

// apply_operator_1D at one cell, component c (M = 1) or all of them (M = 4); the products keep the
// reference's order C1 * d * s_inv, and the y components carry no medium term (as written in the
// reference).  A thread per component computes its own alone (all four in each: 100000 cells 225 us,
// 1000 cells 31 against 10.4 us).
template <int M> __device__ __forceinline__ void fd_cell1(const cplx *f, const FdGeom &G, const FdTables &T, int i, int c, cplx *out)
{
    const cplx *sx = T.sx, *eps = T.eps;
    const long long p = fd_at(G, i, 1, 1);
    const int n = G.n_der;
    cplx d[M] = {};
    for (int q = -n; q <= n; ++q) {
        const double a = G.coef[n + q];
#pragma unroll
        for (int m = 0; m < M; ++m)            // x and y of a half cross over
            d[m] = cadd(d[m], cscale(f[((M == 1 ? c : m) ^ 1) * G.len + p + q], a));
    }
    const cplx C1 = {0.0, G.sign}, mC1 = {-0.0, -G.sign}, C2 = {0.0, -G.w0}, C3 = {0.0, -G.w0 / 2.0}, C4 = {1.0, 0.0};
    const cplx Ex = cadd(f[p], f[p + 2 * G.len]);
    const cplx s = sx[i - 1], e = eps[i - 1];
    const cplx m3 = cmul(C3, csub(e, C4));
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int y = M == 1 ? c : m;
        out[m] = cadd(cmul(cmul(y == 0 || y == 3 ? mC1 : C1, d[m]), s), cmul(C2, f[p + y * G.len]));
        if (!(y & 1)) out[m] = cadd(out[m], cmul(m3, Ex));
    }
}

// component c of apply_operator_2D at one cell, written out; the curl terms carry the opposite sign of the 3D
// operator's (as written in the reference)
__device__ __noinline__ void fd_full2(const cplx *f, cplx *Af, const FdGeom &G, const FdTables &T, int i, int j, int c)
{
    const cplx *sx = T.sx, *sy = T.sy, *eps = T.eps;
    const long long p = fd_at(G, i, j, 1);
    const cplx *plx = f, *ply = f + G.len, *plz = f + 2 * G.len, *mix = f + 3 * G.len, *miy = f + 4 * G.len,
               *miz = f + 5 * G.len;
    const int n = G.n_der;
    cplx dpxdy = {0, 0}, dpydx = {0, 0}, dpzdx = {0, 0}, dpzdy = {0, 0};
    cplx dmxdy = {0, 0}, dmydx = {0, 0}, dmzdx = {0, 0}, dmzdy = {0, 0};
    for (int q = -n; q <= n; ++q) {
        const double a = G.coef[n + q];
        dpydx = cadd(dpydx, cscale(ply[p + q], a));
        dpzdx = cadd(dpzdx, cscale(plz[p + q], a));
        dmydx = cadd(dmydx, cscale(miy[p + q], a));
        dmzdx = cadd(dmzdx, cscale(miz[p + q], a));
    }
    for (int q = -n; q <= n; ++q) {
        const double a = G.coef[n + q];
        const long long o = p + q * G.px;
        dpxdy = cadd(dpxdy, cscale(plx[o], a));
        dpzdy = cadd(dpzdy, cscale(plz[o], a));
        dmxdy = cadd(dmxdy, cscale(mix[o], a));
        dmzdy = cadd(dmzdy, cscale(miz[o], a));
    }
    const cplx Ex = cadd(plx[p], mix[p]), Ey = cadd(ply[p], miy[p]), Ez = cadd(plz[p], miz[p]);
    const cplx sxi = sx[i - 1], syj = sy[j - 1];
    dpxdy = cmul(dpxdy, syj);
    dpydx = cmul(dpydx, sxi);
    dpzdx = cmul(dpzdx, sxi);
    dpzdy = cmul(dpzdy, syj);
    dmxdy = cmul(dmxdy, syj);
    dmydx = cmul(dmydx, sxi);
    dmzdx = cmul(dmzdx, sxi);
    dmzdy = cmul(dmzdy, syj);
    const cplx C1 = {0.0, G.sign}, mC1 = {-0.0, -G.sign}, C2 = {0.0, -G.w0}, C3 = {0.0, -G.w0 / 2.0}, C4 = {1.0, 0.0};
    const cplx e = eps[(long long)(i - 1) + (long long)G.nx * (j - 1)];
    const cplx m3 = cmul(C3, csub(e, C4));
    cplx out[6];
    out[0] = cadd(cadd(cmul(mC1, dpzdy), cmul(C2, plx[p])), cmul(m3, Ex));
    out[1] = cadd(cadd(cmul(C1, dpzdx), cmul(C2, ply[p])), cmul(m3, Ey));
    out[2] = cadd(cadd(cmul(mC1, csub(dpydx, dpxdy)), cmul(C2, plz[p])), cmul(m3, Ez));
    out[3] = cadd(cadd(cmul(C1, dmzdy), cmul(C2, mix[p])), cmul(m3, Ex));
    out[4] = cadd(cadd(cmul(mC1, dmzdx), cmul(C2, miy[p])), cmul(m3, Ey));
    out[5] = cadd(cadd(cmul(C1, csub(dmydx, dmxdy)), cmul(C2, miz[p])), cmul(m3, Ez));
    for (int y = 0; y < 6; ++y)
        if (y == c) Af[p + c * G.len] = out[y];
}

// derivative of one component along the axis of pitch o: the taps in the reference's order
template <int N> __device__ __forceinline__ cplx fd_der(const cplx *v, long long o, const double *coef)
{
    cplx d = cscale(v[-N * o], coef[0]);
#pragma unroll
    for (int q = -N + 1; q <= N; ++q)
        if (q != 0) d = cadd(d, cscale(v[q * o], coef[N + q]));
    return d;
}
// The tests and sign changes below are integer operations: the FP64 pipe is what the pass waits for.
__device__ __forceinline__ bool fd_is(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }
__device__ __forceinline__ double fd_flip(double a, bool neg)
{
    return __longlong_as_double(__double_as_longlong(a) ^ (neg ? (long long)0x8000000000000000ull : 0ll));
}
__device__ __forceinline__ cplx fd_stretch(cplx d, cplx s) { return fd_is(s.re, 1.0) && fd_is(s.im, 0.0) ? d : cmul(d, s); }
// (s i) x with s = -1 (neg) or +1, and -(w i) x
__device__ __forceinline__ cplx fd_times_i(cplx x, bool neg) { return {fd_flip(x.im, !neg), fd_flip(x.re, neg)}; }
__device__ __forceinline__ cplx fd_times_mwi(cplx x, double w) { return {w * x.im, -(w * x.re)}; }
__device__ __forceinline__ bool fd_nonfinite(cplx a)
{
    return (__double2hiint(a.re) & 0x7ff00000) == 0x7ff00000 || (__double2hiint(a.im) & 0x7ff00000) == 0x7ff00000;
}

// Component c of A f at one cell (2D, 3D).  Component 3 h + q of half h takes the curl component q of
// that half's three: the difference of the derivatives of its v1 along one axis and v2 along another.
template <int DIMS, int N>
__device__ __forceinline__ cplx fd_cell(const cplx *__restrict__ f, const FdGeom &G, const FdTables &T, int i, int j, int k,
                                        int c, bool &bad)
{
    const long long p = fd_at(G, i, j, k);
    const int h = c >= 3 ? 3 : 0, q = c - h;
    const cplx e = T.eps[(long long)(i - 1) + (long long)G.nx * ((j - 1) + (long long)G.ny * (k - 1))];
    const cplx m3 = fd_times_mwi(cplx{e.re - 1.0, e.im}, G.w0_half);
    const cplx x = f[p + c * G.len];
    const cplx med = cmul(m3, cadd(f[p + q * G.len], f[p + (q + 3) * G.len]));
    const bool neg = (h == 0) != (G.sign > 0.0);
    // 3D: z along y - y along z;  x along z - z along x;  y along x - x along y.  2D: the z terms vanish
    const cplx *v1 = f + p + (h + (q == 0 ? 2 : (q == 1 ? (DIMS == 3 ? 0 : 2) : 1))) * G.len;
    const cplx *v2 = f + p + (h + (q == 0 ? 1 : (q == 1 ? 2 : 0))) * G.len;
    cplx cu;
    bad = fd_nonfinite(v1[0]);
    if (DIMS == 3 || q == 2) {
        const long long o1 = q == 0 ? G.px : (q == 1 ? G.pxy : 1), o2 = q == 0 ? G.pxy : (q == 1 ? 1 : G.px);
        const cplx t1 = q == 0 ? T.sy[j - 1] : (q == 1 ? T.sz[k - 1] : T.sx[i - 1]);
        const cplx t2 = q == 0 ? T.sz[k - 1] : (q == 1 ? T.sx[i - 1] : T.sy[j - 1]);
        bad |= fd_nonfinite(v2[0]);
        const cplx d = csub(fd_stretch(fd_der<N>(v1, o1, G.coef), t1), fd_stretch(fd_der<N>(v2, o2, G.coef), t2));
        cu = fd_times_i(d, DIMS == 3 ? neg : !neg);
    } else {
        cu = fd_times_i(fd_stretch(fd_der<N>(v1, q == 0 ? G.px : 1, G.coef), q == 0 ? T.sy[j - 1] : T.sx[i - 1]),
                        q == 0 ? !neg : neg);
    }
    const cplx out = cadd(cadd(cu, fd_times_mwi(x, G.w0)), med);
    bad |= fd_nonfinite(out);
    return out;
}

// component c of A f at one cell, into Af
template <int DIMS, int N>
__device__ __forceinline__ void fd_apply_value(const cplx *__restrict__ f, cplx *Af, const FdGeom &G, const FdTables &T, int i,
                                               int j, int k, int c)
{
    cplx *dst = Af + fd_at(G, i, j, k) + c * G.len;
    if (DIMS == 1) {
        fd_cell1<1>(f, G, T, i, c, dst);
        return;
    }
    bool bad;
    *dst = fd_cell<DIMS == 1 ? 2 : DIMS, N>(f, G, T, i, j, k, c, bad);
    if (bad) {
        if (DIMS == 3) fd_full3(f, Af, G, T, i, j, k, c);
        else fd_full2(f, Af, G, T, i, j, c);
    }
}

// One launch of the solver between two of its dot products: A f (optional), a list of vector
// operations over the interior of every component (rs_operations_subs_mod.f90), the periodic ghost
// copies of the vector the next operator application reads, and the row partials of up to three
// dot products.  All of it but the operator's taps is local to a value, so a thread that owns
// the cells i, i + T, ... of one row (or one component of them) needs no synchronisation between
// the parts.
struct FdLin {
    cplx *v1;
    const cplx *v2;
    cplx a;
    int mode;   // 0: v1 = v1 + a v2;  1: v1 = a v1 + v2;  2: v1 = a v1
};
constexpr int FD_LIN_MAX = 26, FD_DOT_MAX = 3;
struct FdPass {
    const cplx *f;           // operator application Af = A f, or null
    cplx *Af;
    int nlin, ndot;
    FdLin lin[FD_LIN_MAX];
    const cplx *da[FD_DOT_MAX], *db[FD_DOT_MAX];   // sum conj(da) db
    cplx *ghost;             // vector whose periodic ghosts are refreshed, or null
    cplx *part;              // [ndot][rows] row partials, in host memory
    unsigned *done;          // finished blocks (device), zero between launches
    unsigned *flag, seq;     // *flag = seq once every partial is written (host memory)
};

__device__ __forceinline__ void fd_lin_value(const FdLin &o, long long q)
{
    const cplx x = o.v1[q];
    if (o.mode == 0) o.v1[q] = cadd(x, cmul(o.a, o.v2[q]));
    else if (o.mode == 1) o.v1[q] = cadd(cmul(o.a, x), o.v2[q]);
    else o.v1[q] = cmul(o.a, x);
}

// k_fd_ghosts' copies of component c of the cell (i, j, k), by the thread that owns it
__device__ __forceinline__ void fd_ghost_value(cplx *f, const FdGeom &G, int i, int j, int k, int c)
{
    const int at[3] = {i, j, k}, n[3] = {G.nx, G.ny, G.nz};
    const long long pitch[3] = {1, G.px, G.pxy};
    cplx *v = f + fd_at(G, i, j, k) + c * G.len;
    for (int a = 0; a < G.dims; ++a) {
        if (!G.per[a]) continue;
        const bool quirk = a == 1 && G.dims == 3;
        if (at[a] > n[a] - G.g && !(quirk && c == 4)) v[-n[a] * pitch[a]] = v[0];
        if (at[a] <= G.g && !(quirk && c == 3)) v[n[a] * pitch[a]] = v[0];
    }
}

// T threads (32, 64 or 128) along a row of cells.  The FP64 pipe bounds the pass; it takes a warp's
// instruction every 64 cycles per sub-partition.  SPLIT: one row per block, a thread row per
// component, for grids with few rows -- with a thread per cell a 30 x 27 x 25 grid is 675 warps on 608
// sub-partitions, two rounds of the longest chain (294 us an outer iteration of BiCGStab(2)); split, it
// is 4050 short ones (223 us).  Otherwise a thread per cell and 128 / T rows per block: the medium
// term is formed once for a component pair (60^3: 1.43 against 1.59 ms split).  Before, every dot,
// vector operation and operator was a launch of its own: 457 us and 2.00 ms.
// A row's dot partial is summed per thread over its cells (components outermost) and then over the T
// threads by halving: the order of a 128-thread block per row whose threads past nx hold zeros, for
// every T >= nx.
constexpr int fd_threads(bool split, int dims, int T) { return split ? T * (dims == 1 ? 4 : 6) : 128; }
constexpr int fd_min_blocks(bool split, int T) { return split ? (T == 32 ? 5 : (T == 64 ? 2 : 1)) : 4; }
template <int DIMS, int N, int T, bool SPLIT>
__global__ void __launch_bounds__(fd_threads(SPLIT, DIMS, T), fd_min_blocks(SPLIT, T))
    k_fd_pass(const __grid_constant__ FdPass P, const __grid_constant__ FdGeom G, const __grid_constant__ FdTables A)
{
    constexpr int NC = DIMS == 1 ? 4 : 6, RPB = SPLIT ? 1 : 128 / T;
    __shared__ cplx sh[FD_DOT_MAX][SPLIT ? NC : RPB][T];
    const int t = threadIdx.x, ty = threadIdx.y;
    const int rows = G.ny * G.nz, row = blockIdx.x * RPB + (SPLIT ? 0 : ty);
    const bool live = row < rows;
    const int j = 1 + row % G.ny, k = 1 + row / G.ny;
    // blockIdx.y: pieces of a long row (launches without dots only)
    const int i0 = 1 + t + T * blockIdx.y, i1 = live ? G.nx : 0, step = T * gridDim.y;
    if (P.f)
        for (int i = i0; i <= i1; i += step) {
            if (SPLIT) {
                fd_apply_value<DIMS, N>(P.f, P.Af, G, A, i, j, k, ty);
            } else if (DIMS == 1) {
                cplx all[4];
                fd_cell1<4>(P.f, G, A, i, 0, all);
                for (int c = 0; c < NC; ++c) P.Af[fd_at(G, i, j, k) + c * G.len] = all[c % 4];
            } else {
#pragma unroll
                for (int c = 0; c < NC; ++c) fd_apply_value<DIMS, N>(P.f, P.Af, G, A, i, j, k, c);
            }
        }
    if (P.nlin || P.ghost)
        for (int i = i0; i <= i1; i += step)
            for (int c = SPLIT ? ty : 0; c < (SPLIT ? ty + 1 : NC); ++c) {
                const long long q = fd_at(G, i, j, k) + c * G.len;
                for (int o = 0; o < P.nlin; ++o) fd_lin_value(P.lin[o], q);
                if (P.ghost) fd_ghost_value(P.ghost, G, i, j, k, c);
            }
    if (P.ndot == 0) return;
    // product of one value pair, and a thread's sum over its cells
    auto product = [&](int d, long long q) {
        const cplx va = P.da[d][q], vb = P.db[d][q];
        return cmul(cplx{va.re, -va.im}, vb);
    };
    auto row_sum = [&](int d) {
        cplx s = {0, 0};
        for (int y = 0; y < NC; ++y)
            for (int i = 1 + t; i <= i1; i += T) s = cadd(s, product(d, fd_at(G, i, j, k) + y * G.len));
        return s;
    };
    const bool one = G.nx <= T;             // a cell per thread: split, the products by component in parallel
    if (SPLIT && one) {
        const long long q = fd_at(G, min(1 + t, G.nx), j, k) + ty * G.len;
        for (int d = 0; d < P.ndot; ++d) sh[d][ty][t] = t < G.nx ? product(d, q) : cplx{0.0, 0.0};
    }
    if (SPLIT) __syncthreads();             // and the values that other components' threads wrote
    // split: thread row d sums dot d; else a row's threads sum every dot
    const int d0 = SPLIT ? ty : 0, d1 = SPLIT ? min(ty + 1, P.ndot) : P.ndot, slot = SPLIT ? 0 : ty;
    for (int d = d0; d < d1; ++d) {
        cplx s = {0, 0};
        if (SPLIT && one)
            for (int y = 0; y < NC; ++y) s = cadd(s, sh[d][y % (SPLIT ? NC : RPB)][t]);
        else
            s = row_sum(d);
        sh[d][slot][t] = s;
    }
    for (int o = T / 2; o > 0; o >>= 1) {
        if (T == 32) __syncwarp();          // a thread row is a warp
        else __syncthreads();
        if (t < o)
            for (int d = d0; d < d1; ++d) sh[d][slot][t] = cadd(sh[d][slot][t], sh[d][slot][t + o]);
    }
    if (t == 0 && live && d0 < d1) {
        for (int d = d0; d < d1; ++d) P.part[(long long)d * rows + row] = sh[d][slot][0];
        __threadfence_system();
    }
    __syncthreads();
    if (ty == 0 && t == 0 && atomicAdd(P.done, 1u) == gridDim.x - 1) {
        *P.done = 0;
        __threadfence_system();
        *(volatile unsigned *)P.flag = P.seq;
    }
}

}  // namespace

struct omx_fdop {
    FdGeom G{};
    cudaStream_t s = nullptr;
    cplx *sx = nullptr, *sy = nullptr, *sz = nullptr, *eps = nullptr;
    cplx *hpart = nullptr;      // [FD_DOT_MAX][rows] partials, then the flag word (pinned, written by the device)
    unsigned *done = nullptr;
    unsigned seq = 0;
    std::vector<cplx *> vecs;   // solver work vectors
    ~omx_fdop()
    {
        cudaFree(sx);
        cudaFree(sy);
        cudaFree(sz);
        cudaFree(eps);
        cudaFree(done);
        if (hpart) cudaFreeHost(hpart);
        for (auto *v : vecs) cudaFree(v);
        if (s) cudaStreamDestroy(s);
    }
};

namespace {

int fd_fail(int code, const std::string &m)
{
    omx::set_global_error("omx_fd: " + m);
    return code;
}

struct FdErr {
    int code;
    std::string msg;
};
void fck(cudaError_t e, const char *w)
{
    if (e != cudaSuccess) throw FdErr{OMX_ERR_CUDA, std::string(w) + ": " + cudaGetErrorString(e)};
}

template <int V> struct IntC {
    static constexpr int value = V;
};
// call fn(dimensions, n_der) with both as compile-time constants
template <class F> void by_shape(const FdGeom &G, F &&fn)
{
    auto order = [&](auto d) {
        switch (G.n_der) {
        case 1: fn(d, IntC<1>{}); break;
        case 2: fn(d, IntC<2>{}); break;
        case 3: fn(d, IntC<3>{}); break;
        default: fn(d, IntC<4>{}); break;
        }
    };
    if (G.dims == 1) fn(IntC<1>{}, IntC<1>{});   // the 1D cell reads n_der itself
    else if (G.dims == 2) order(IntC<2>{});
    else order(IntC<3>{});
}

// Rows up to this long go through one launch a pass.  Longer ones are cut into pieces for the
// operator and the vector operations, and the dots get a launch of their own: one block a row would
// leave a grid of few long rows to a handful of blocks.
constexpr int FD_ROW_MAX = 256;
// warps of one thread per cell (all pieces of a row) below which a pass takes a thread per component
// (k_fd_pass)
constexpr int FD_SPLIT_WARPS = 1024;

void fd_launch_pass(omx_fdop *op, const FdPass &P)
{
    const FdGeom &G = op->G;
    const int rows = G.ny * G.nz, T = G.nx <= 32 ? 32 : (G.nx <= 64 ? 64 : 128);
    const unsigned pieces = P.ndot > 0 ? 1u : (unsigned)std::min((G.nx + T - 1) / T, 65535);
    // the 1D operator alone: a thread per cell forms the medium term and reads the tables once (1000 and
    // 30000 cells 14.3 and 20.5 us; a thread per component 16.3 and 24.6)
    const bool whole = G.dims == 1 && P.f && P.ndot == 0;
    const bool split = !whole && (long long)rows * pieces * (T / 32) < FD_SPLIT_WARPS;
    const FdTables A{op->sx, op->sy, op->sz, op->eps};
    by_shape(G, [&](auto dc, auto nc) {
        constexpr int D = decltype(dc)::value, N = decltype(nc)::value, C = D == 1 ? 4 : 6;
        auto go = [&](auto tc) {
            constexpr int W = decltype(tc)::value, R = 128 / W;
            if (split) k_fd_pass<D, N, W, true><<<dim3((unsigned)rows, pieces), dim3(W, C), 0, op->s>>>(P, G, A);
            else k_fd_pass<D, N, W, false><<<dim3((unsigned)((rows + R - 1) / R), pieces), dim3(W, R), 0, op->s>>>(P, G, A);
        };
        if (T == 32) go(IntC<32>{});
        else if (T == 64) go(IntC<64>{});
        else go(IntC<128>{});
    });
    fck(cudaPeekAtLastError(), "launch");
}

// Af = A f for a vector whose periodic ghosts may be stale
void fd_apply_dev(omx_fdop *op, cplx *f, cplx *Af)
{
    const FdGeom &G = op->G;
    for (int a = 0; a < G.dims; ++a) {
        if (!G.per[a]) continue;
        const int n1 = a == 0 ? G.ny : G.nx, n2 = a == 2 ? G.ny : G.nz;
        const long long cnt = (long long)G.ncomp * G.g * n1 * n2;
        k_fd_ghosts<<<(unsigned)((cnt + 255) / 256), 256, 0, op->s>>>(f, G, a);
    }
    FdPass P{};
    P.f = f;
    P.Af = Af;
    fd_launch_pass(op, P);
}

// Run a pass; with dots, wait for their partials and sum them in row order into dots[0..ndot-1].
// The partials come straight into pinned memory and the host watches the flag word behind them
// (a copy and a stream synchronisation per dot cost 10 us; this about 3).  The stream's own state
// ends the wait when the launch failed.
void fd_pass(omx_fdop *op, FdPass &P, cplx *dots = nullptr)
{
    const FdGeom &G = op->G;
    const size_t rows = (size_t)G.ny * G.nz;
    const int ndot = P.ndot;
    if (ndot > 0 && G.nx > FD_ROW_MAX && (P.f || P.nlin || P.ghost)) {
        P.ndot = 0;
        fd_launch_pass(op, P);
        P.ndot = ndot;
        P.f = nullptr;
        P.nlin = 0;
        P.ghost = nullptr;
    }
    unsigned *flag = reinterpret_cast<unsigned *>(op->hpart + FD_DOT_MAX * rows);
    P.part = op->hpart;
    P.done = op->done;
    P.flag = flag;
    P.seq = ++op->seq;
    fd_launch_pass(op, P);
    if (ndot == 0) return;
    for (long long spin = 1; __atomic_load_n(flag, __ATOMIC_ACQUIRE) != P.seq; ++spin) {
        if (spin % 4096) continue;
        const cudaError_t e = cudaStreamQuery(op->s);
        if (e == cudaErrorNotReady) continue;
        fck(e, "dot");
        fck(cudaStreamSynchronize(op->s), "dot");
        if (__atomic_load_n(flag, __ATOMIC_ACQUIRE) != P.seq) throw FdErr{OMX_ERR_CUDA, "dot: the partial sums did not arrive"};
        break;
    }
    for (int d = 0; d < ndot; ++d) {
        cplx s = {0, 0};
        for (size_t b = 0; b < rows; ++b) s = cadd(s, op->hpart[d * rows + b]);
        dots[d] = s;
    }
}

}  // namespace

extern "C" {

int omx_fd_create(int dimensions, const int grid_Ndims[3], int n_pml, int n_der, const int boundaries[3], double dr,
                  double w0, const double *eps_r, omx_fdop **out)
{
    if (!grid_Ndims || !boundaries || !eps_r || !out || n_der < 1 || n_der > 4 || !(dr > 0) || !(w0 > 0) ||
        dimensions < 1 || dimensions > 3)
        return fd_fail(OMX_ERR_ARG, "bad argument (dimensions 1..3, n_der 1..4)");
    for (int a = 0; a < dimensions; ++a) {
        if (grid_Ndims[a] < 1) return fd_fail(OMX_ERR_ARG, "grid sizes must be >= 1");
        if (boundaries[a] < 1 || boundaries[a] > 3) return fd_fail(OMX_ERR_ARG, "boundaries: 1 close, 2 periodic, 3 PML");
        if (boundaries[a] == 3 && grid_Ndims[a] < 2 * n_pml) return fd_fail(OMX_ERR_ARG, "PML slabs do not fit");
        if (boundaries[a] == 2 && grid_Ndims[a] < n_der) return fd_fail(OMX_ERR_ARG, "periodic axis shorter than the stencil");
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return fd_fail(OMX_ERR_NODEV, "no CUDA device");
    }
    *out = nullptr;
    omx_fdop *op = new omx_fdop;
    try {
        FdGeom &G = op->G;
        G.dims = dimensions;
        G.ncomp = dimensions == 1 ? 4 : 6;
        G.nx = grid_Ndims[0];
        G.ny = dimensions >= 2 ? grid_Ndims[1] : 1;
        G.nz = dimensions == 3 ? grid_Ndims[2] : 1;
        G.g = n_der;
        G.gy = dimensions >= 2 ? n_der : 0;
        G.gz = dimensions == 3 ? n_der : 0;
        G.n_der = n_der;
        G.px = G.nx + 2 * G.g;
        G.pxy = G.px * (G.ny + 2 * G.gy);
        G.len = G.pxy * (G.nz + 2 * G.gz);
        for (int a = 0; a < 3; ++a) G.per[a] = a < dimensions && boundaries[a] == 2;
        G.w0 = w0;
        G.w0_half = w0 / 2.0;
        // operator_mod.f90:97-140: central-difference coefficients of order 2 n_der, / dr
        static const double C[4][9] = {{-0.5, 0.0, 0.5},
                                       {1.0 / 12.0, -2.0 / 3.0, 0.0, 2.0 / 3.0, -1.0 / 12.0},
                                       {-1.0 / 60.0, 3.0 / 20.0, -3.0 / 4.0, 0.0, 3.0 / 4.0, -3.0 / 20.0, 1.0 / 60.0},
                                       {1.0 / 280.0, -4.0 / 105.0, 1.0 / 5.0, -4.0 / 5.0, 0.0, 4.0 / 5.0, -1.0 / 5.0,
                                        4.0 / 105.0, -1.0 / 280.0}};
        for (int q = 0; q <= 2 * n_der; ++q) G.coef[q] = C[n_der - 1][q] / dr;
        // :185-232: s_inv = 1 / (kappa + sig / (i w0 eps0)) on the PML faces, 1 elsewhere
        const int n[3] = {G.nx, G.ny, G.nz};
        std::vector<cplx> s[3];
        const double m = 3.0, kmax = 5.0, sig_max = 0.8 * (m + 1.0) / (dr * std::sqrt(1.0 / 1.0));
        for (int a = 0; a < 3; ++a) {
            s[a].assign(n[a], cplx{1.0, 0.0});
            if (a >= dimensions || boundaries[a] != 3) continue;
            for (int i = 1; i <= n_pml; ++i) {
                const double r = (double)(n_pml - i + 1) / (double)n_pml;
                const double sig = sig_max * std::pow(r, m);
                const double kap = 1.0 + (kmax - 1.0) * std::pow(r, m);
                const cplx si = {kap, -(sig / w0)};
                s[a][i - 1] = cdiv(cplx{1.0, 0.0}, si);
                s[a][n[a] - n_pml + (n_pml - i)] = cdiv(cplx{1.0, 0.0}, si);
            }
        }
        fck(cudaStreamCreateWithFlags(&op->s, cudaStreamNonBlocking), "stream");
        cplx **dst[3] = {&op->sx, &op->sy, &op->sz};
        for (int a = 0; a < 3; ++a) {
            fck(cudaMalloc(dst[a], sizeof(cplx) * n[a]), "alloc");
            fck(cudaMemcpy(*dst[a], s[a].data(), sizeof(cplx) * n[a], cudaMemcpyHostToDevice), "upload");
            fck(cudaStreamSynchronize(0), "upload");   // pageable copies may return before their DMA ends
        }
        const size_t ncell = (size_t)G.nx * G.ny * G.nz;
        fck(cudaMalloc(&op->eps, sizeof(cplx) * ncell), "alloc");
        fck(cudaMemcpy(op->eps, eps_r, sizeof(cplx) * ncell, cudaMemcpyHostToDevice), "upload");
        fck(cudaStreamSynchronize(0), "upload");   // pageable copies may return before their DMA ends
        const size_t hpart = sizeof(cplx) * (FD_DOT_MAX * (size_t)G.ny * G.nz + 1);
        fck(cudaMallocHost(&op->hpart, hpart), "alloc");
        std::memset(static_cast<void *>(op->hpart), 0, hpart);
        fck(cudaMalloc(&op->done, sizeof(unsigned)), "alloc");
        fck(cudaMemset(op->done, 0, sizeof(unsigned)), "memset");
        fck(cudaStreamSynchronize(0), "memset");
    } catch (const FdErr &e) {
        delete op;
        return fd_fail(e.code, e.msg);
    }
    *out = op;
    return OMX_OK;
}

int omx_fd_set_eps(omx_fdop *op, const double *eps_r)
{
    if (!op || !eps_r) return fd_fail(OMX_ERR_ARG, "null argument");
    try {
        const size_t ncell = (size_t)op->G.nx * op->G.ny * op->G.nz;
        fck(cudaMemcpyAsync(op->eps, eps_r, sizeof(cplx) * ncell, cudaMemcpyHostToDevice, op->s), "upload");
        fck(cudaStreamSynchronize(op->s), "upload");
    } catch (const FdErr &e) {
        return fd_fail(e.code, e.msg);
    }
    return OMX_OK;
}

int omx_fd_destroy(omx_fdop *op)
{
    if (op) {
        cudaStreamSynchronize(op->s);
        delete op;
    }
    return OMX_OK;
}

long long omx_fd_vector_length(const omx_fdop *op) { return op ? (long long)op->G.ncomp * op->G.len : 0; }

int omx_fd_apply(omx_fdop *op, const double *f, double *Af, int transpose)
{
    if (!op || !f || !Af) return fd_fail(OMX_ERR_ARG, "null argument");
    cplx *df = nullptr, *dAf = nullptr;
    try {
        op->G.sign = transpose ? -1.0 : 1.0;
        const size_t bytes = sizeof(cplx) * op->G.ncomp * op->G.len;
        fck(cudaMalloc(&df, bytes), "alloc");
        fck(cudaMalloc(&dAf, bytes), "alloc");
        fck(cudaMemcpy(df, f, bytes, cudaMemcpyHostToDevice), "upload");
        fck(cudaStreamSynchronize(0), "upload");   // pageable copies may return before their DMA ends
        fck(cudaMemsetAsync(dAf, 0, bytes, op->s), "memset");
        fd_apply_dev(op, df, dAf);
        fck(cudaStreamSynchronize(op->s), "apply");
        fck(cudaMemcpy(Af, dAf, bytes, cudaMemcpyDeviceToHost), "download");
    } catch (const FdErr &e) {
        cudaFree(df);
        cudaFree(dAf);
        return fd_fail(e.code, e.msg);
    }
    cudaFree(df);
    cudaFree(dAf);
    return OMX_OK;
}

// Mean time of `reps` operator applications on device-resident vectors (random interior values),
// CUDA events on the operator's stream.
int omx_fd_time_apply(omx_fdop *op, int reps, double *ms_per_apply)
{
    if (!op || reps < 1 || !ms_per_apply) return fd_fail(OMX_ERR_ARG, "bad argument");
    cplx *df = nullptr, *dAf = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    try {
        op->G.sign = 1.0;
        const size_t n = (size_t)op->G.ncomp * op->G.len;
        std::vector<cplx> h(n);
        unsigned long long x = 88172645463325252ull;
        for (auto &v : h) {
            x ^= x << 13;
            x ^= x >> 7;
            x ^= x << 17;
            v = {(double)(x >> 11) * (1.0 / 9007199254740992.0) - 0.5, (double)(x & 0xffff) / 65536.0 - 0.5};
        }
        fck(cudaMalloc(&df, n * sizeof(cplx)), "alloc");
        fck(cudaMalloc(&dAf, n * sizeof(cplx)), "alloc");
        fck(cudaMemcpy(df, h.data(), n * sizeof(cplx), cudaMemcpyHostToDevice), "upload");
        fck(cudaStreamSynchronize(0), "upload");   // pageable copies may return before their DMA ends
        fck(cudaEventCreate(&e0), "event");
        fck(cudaEventCreate(&e1), "event");
        for (int r = 0; r < 2; ++r) fd_apply_dev(op, df, dAf);
        fck(cudaEventRecord(e0, op->s), "event");
        for (int r = 0; r < reps; ++r) fd_apply_dev(op, df, dAf);
        fck(cudaEventRecord(e1, op->s), "event");
        fck(cudaEventSynchronize(e1), "apply");
        float ms = 0.f;
        fck(cudaEventElapsedTime(&ms, e0, e1), "event");
        *ms_per_apply = ms / reps;
    } catch (const FdErr &e) {
        cudaFree(df);
        cudaFree(dAf);
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        return fd_fail(e.code, e.msg);
    }
    cudaFree(df);
    cudaFree(dAf);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return OMX_OK;
}

// BICGStab_L (bicgstab_mod.f90:76-243), the oracle's scalar recursion on the host
int omx_fd_solve(omx_fdop *op, const double *j_vec, double *f_io, int transpose, double tol, int n_max, int L,
                 int *converged, double *abs_err, int *iterations)
{
    if (!op || !j_vec || !f_io || L < 1 || L > 8 || n_max < 0 || !(tol > 0)) return fd_fail(OMX_ERR_ARG, "bad argument");
    try {
        FdGeom &G = op->G;
        G.sign = transpose ? -1.0 : 1.0;
        const size_t bytes = sizeof(cplx) * G.ncomp * G.len;
        const size_t need = 5 + 2 * (size_t)(L + 1);
        while (op->vecs.size() < need) {
            cplx *v = nullptr;
            fck(cudaMalloc(&v, bytes), "alloc");
            op->vecs.push_back(v);
        }
        cplx *r0 = op->vecs[0], *f = op->vecs[1], *Af = op->vecs[2], *jv = op->vecs[3], *f_out = op->vecs[4];
        cplx *r[9], *u[9];
        for (int l = 0; l <= L; ++l) {
            r[l] = op->vecs[5 + l];
            u[l] = op->vecs[5 + L + 1 + l];
        }
        for (size_t q = 0; q < need; ++q) fck(cudaMemsetAsync(op->vecs[q], 0, bytes, op->s), "memset");
        fck(cudaMemcpyAsync(f, f_io, bytes, cudaMemcpyHostToDevice, op->s), "upload");
        fck(cudaMemcpyAsync(jv, j_vec, bytes, cudaMemcpyHostToDevice, op->s), "upload");
        fck(cudaMemcpyAsync(f_out, f_io, bytes, cudaMemcpyHostToDevice, op->s), "upload");
        cplx tau[9][9] = {}, gam[9] = {}, gam_p[9] = {}, gam_pp[9] = {}, sig[9] = {};
        cplx rho0 = {1, 0}, rho1 = {1, 0}, alpha = {1, 0}, omega = {1, 0}, beta, dot[FD_DOT_MAX];
        const bool per = G.per[0] || G.per[1] || G.per[2];
        FdPass P{};
        auto begin = [&]() {
            P.f = nullptr;
            P.nlin = P.ndot = 0;
            P.ghost = nullptr;
        };
        auto lin = [&](cplx *v1, const cplx *v2, cplx a, int mode) { P.lin[P.nlin++] = FdLin{v1, v2, a, mode}; };
        auto dots = [&](const cplx *v1, const cplx *v2) {
            P.da[P.ndot] = v1;
            P.db[P.ndot++] = v2;
        };
        // A x with the ghosts of x refreshed by the pass that wrote x
        auto apply = [&](const cplx *x, cplx *Ax) {
            P.f = x;
            P.Af = Ax;
        };
        fd_apply_dev(op, f, Af);
        fck(cudaMemcpyAsync(r0, jv, bytes, cudaMemcpyDeviceToDevice, op->s), "copy");
        begin();
        lin(r0, Af, cplx{-1.0, 0.0}, 0);                        // r0 = j - A f
        dots(r0, r0);
        dots(jv, jv);
        fd_pass(op, P, dot);
        fck(cudaMemcpyAsync(r[0], r0, bytes, cudaMemcpyDeviceToDevice, op->s), "copy");
        double norm_t = std::sqrt(dot[0].re);
        const double norm_j = std::sqrt(dot[1].re);
        begin();
        lin(r0, nullptr, cplx{1.0 / norm_t, 0.0}, 2);           // r0 = r0 / |r0|
        dots(r0, r[0]);                                         // the first iteration's rho1
        cplx next_rho = {0, 0};
        fd_pass(op, P, dot);
        next_rho = dot[0];
        norm_t = norm_j;
        double err_r = 1.0;
        int n = 0, conv = 0;
        // each pass ends with every dot product that its vectors already allow: (r0, r[l]) after the
        // application that makes r[l], the first minimal-residual products after the last one, the
        // next iteration's (r0, r[0]) with the residual norm
        while (n <= n_max && !conv) {
            rho0 = cmul(cscale(omega, -1.0), rho0);
            for (int l = 0; l <= L - 1; ++l) {
                rho1 = next_rho;
                beta = cdiv(cmul(alpha, rho1), rho0);
                rho0 = rho1;
                begin();
                for (int i = 0; i <= l; ++i) lin(u[i], r[i], cscale(beta, -1.0), 1);
                if (per) P.ghost = u[l];
                fd_pass(op, P);
                begin();
                apply(u[l], u[l + 1]);
                dots(r0, u[l + 1]);
                fd_pass(op, P, dot);
                alpha = cdiv(rho0, dot[0]);
                begin();
                for (int i = 0; i <= l; ++i) lin(r[i], u[i + 1], cscale(alpha, -1.0), 0);
                lin(f_out, u[0], alpha, 0);
                if (per) P.ghost = r[l];
                fd_pass(op, P);
                begin();
                apply(r[l], r[l + 1]);
                if (l < L - 1) {
                    dots(r0, r[l + 1]);
                    fd_pass(op, P, dot);
                    next_rho = dot[0];
                }
            }
            // the last application's pass takes the minimal-residual part's first products along
            for (int l = 1; l <= L; ++l) {
                if (l == 1) {
                    dots(r[1], r[1]);
                    dots(r[1], r[0]);
                    if (L > 1) dots(r[1], r[2]);
                    fd_pass(op, P, dot);
                    sig[1] = dot[0];
                    gam_p[1] = cdiv(dot[1], sig[1]);
                    if (L > 1) dot[0] = dot[2];
                    continue;
                }
                for (int i = 1; i <= l - 1; ++i) {              // dot[0] = (r[i], r[l])
                    tau[i][l] = cdiv(dot[0], sig[i]);
                    begin();
                    lin(r[l], r[i], cscale(tau[i][l], -1.0), 0);
                    if (i < l - 1) {
                        dots(r[i + 1], r[l]);
                    } else {
                        dots(r[l], r[l]);
                        dots(r[l], r[0]);
                        if (l < L) dots(r[1], r[l + 1]);
                    }
                    fd_pass(op, P, dot);
                }
                sig[l] = dot[0];
                gam_p[l] = cdiv(dot[1], sig[l]);
                if (l < L) dot[0] = dot[2];
            }
            gam[L] = gam_p[L];
            omega = gam[L];
            for (int l = L - 1; l >= 1; --l) {
                gam[l] = gam_p[l];
                for (int i = l + 1; i <= L; ++i) gam[l] = csub(gam[l], cmul(tau[l][i], gam[i]));
            }
            for (int l = 1; l <= L - 1; ++l) {
                gam_pp[l] = gam[l + 1];
                for (int i = l + 1; i <= L - 1; ++i) gam_pp[l] = cadd(gam_pp[l], cmul(tau[l][i], gam[i + 1]));
            }
            begin();
            lin(f_out, r[0], gam[1], 0);
            lin(r[0], r[L], cscale(gam_p[L], -1.0), 0);
            lin(u[0], u[L], cscale(gam[L], -1.0), 0);
            for (int l = 1; l <= L - 1; ++l) {
                lin(u[0], u[l], cscale(gam[l], -1.0), 0);
                lin(f_out, r[l], gam_pp[l], 0);
                lin(r[0], r[l], cscale(gam_p[l], -1.0), 0);
            }
            dots(r[0], r[0]);
            dots(r0, r[0]);
            fd_pass(op, P, dot);
            next_rho = dot[1];
            err_r = std::sqrt(dot[0].re);
            n = n + 1;
            if (err_r <= tol * norm_t) conv = 1;
        }
        fck(cudaMemcpyAsync(f_io, f_out, bytes, cudaMemcpyDeviceToHost, op->s), "download");
        fck(cudaStreamSynchronize(op->s), "solve");
        if (converged) *converged = conv;
        if (abs_err) *abs_err = err_r / norm_t;
        if (iterations) *iterations = n;
    } catch (const FdErr &e) {
        return fd_fail(e.code, e.msg);
    }
    return OMX_OK;
}

}  // extern "C"
