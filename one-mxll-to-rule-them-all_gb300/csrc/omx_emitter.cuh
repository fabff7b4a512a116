// omx_emitter.cuh -- few-level density-matrix emitter arithmetic shared by the emitter kernels.
#pragma once

namespace omx {

// ---- few-level density-matrix emitters (new model behind TQ_sys_base%td_propagate) --------
// State (FP64): 2-level [p_e, Re rho_eg, Im rho_eg]; 3-level (V system)
// [p1, p2, Re r10, Im r10, Re r20, Im r20, Re r21, Im r21].  d rho/dt = -i[H0 - E_u V, rho]
// + T1 population decay to the ground state + T2 coherence decay, RK4 with E_u held over dt;
// the rates 1/T1, 1/T2 are formed once per step (FP64 division is expensive on this part).
__device__ __forceinline__ void rhs2(const double *pr, double E_u, double g1, double g2, const double *rho, double *d)
{
    const double w0 = pr[0], mu = pr[1];
    const double pe = rho[0], a = rho[1], b = rho[2];
    const double pg = 1.0 - pe;
    const double muE = mu * E_u;
    d[0] = 2.0 * muE * b - pe * g1;
    d[1] = w0 * b - a * g2;
    d[2] = -(w0 * a) + muE * (pg - pe) - b * g2;
}

__device__ __forceinline__ void rhs3(const double *pr, double E_u, double g1r, double g2r, const double *rho, double *d)
{
    const double e1 = pr[0], e2 = pr[1], mu1 = pr[2], mu2 = pr[3];
    const double p1 = rho[0], p2 = rho[1];
    const double a10 = rho[2], b10 = rho[3], a20 = rho[4], b20 = rho[5], a21 = rho[6], b21 = rho[7];
    const double p0 = 1.0 - p1 - p2;
    const double g1 = mu1 * E_u, g2 = mu2 * E_u;
    d[0] = 2.0 * g1 * b10 - p1 * g1r;
    d[1] = 2.0 * g2 * b20 - p2 * g1r;
    d[2] = e1 * b10 - g2 * b21 - a10 * g2r;
    d[3] = -(e1 * a10) + g1 * (p0 - p1) - g2 * a21 - b10 * g2r;
    d[4] = e2 * b20 + g1 * b21 - a20 * g2r;
    d[5] = -(e2 * a20) + g2 * (p0 - p2) - g1 * a21 - b20 * g2r;
    const double de = e2 - e1;
    d[6] = de * b21 + g2 * b10 + g1 * b20 - a21 * g2r;
    d[7] = -(de * a21) + g2 * a10 - g1 * a20 - b21 * g2r;
}

// One RK4 step with the decay rates g1 = 1/T1, g2 = 1/T2 and the step fractions h2 = dt/2,
// h6 = dt/6 supplied by the caller (formed once, not per emitter and step).
template <int NST>
__device__ __forceinline__ void rk4r(int model, const double *pr, double *rho, double E_u, double dt, double h2,
                                     double h6, double g1, double g2)
{
    double k1[NST], k2[NST], k3[NST], k4[NST], t[NST];
    if (model == 1) rhs2(pr, E_u, g1, g2, rho, k1); else rhs3(pr, E_u, g1, g2, rho, k1);
#pragma unroll
    for (int q = 0; q < NST; ++q) t[q] = rho[q] + h2 * k1[q];
    if (model == 1) rhs2(pr, E_u, g1, g2, t, k2); else rhs3(pr, E_u, g1, g2, t, k2);
#pragma unroll
    for (int q = 0; q < NST; ++q) t[q] = rho[q] + h2 * k2[q];
    if (model == 1) rhs2(pr, E_u, g1, g2, t, k3); else rhs3(pr, E_u, g1, g2, t, k3);
#pragma unroll
    for (int q = 0; q < NST; ++q) t[q] = rho[q] + dt * k3[q];
    if (model == 1) rhs2(pr, E_u, g1, g2, t, k4); else rhs3(pr, E_u, g1, g2, t, k4);
#pragma unroll
    for (int q = 0; q < NST; ++q)   // 2 k2 and 2 k3 are exact: fma(2, k, x) rounds as x + 2 k
        rho[q] = rho[q] + h6 * (__fma_rn(2.0, k3[q], __fma_rn(2.0, k2[q], k1[q])) + k4[q]);
}

// The same RK4 step with one lane per state word: LANES = 8 lanes hold the 3-level state, 4 the 2-level
// one (lane 3 idles along).  Every derivative is a sum of at most four products taken in rhs3 / rhs2's
// order, c0 s0 + c1 s1 + c2 s2 - own * rate, with the subtracted products as products of a negated
// coefficient (the same value), so each lane evaluates its own word's derivative with operand words
// fetched by shuffles and the results are rk4r's bit for bit.  The FP64 pipe takes a warp's
// instruction every 64 cycles per sub-partition whatever its lanes do, so this is 51 (39) instructions
// in a row for eight (four) times the warps, instead of about 270 (95).
struct EmitLane {
    double c0, c1, c2, rate;     // coefficients; rate negated
    int s0, s1, s2;              // lanes of the operand words
    bool has1, has2, pop;        // terms present; c1's operand is the population difference
};

template <int LANES>
__device__ __forceinline__ EmitLane emit_lane(int l, const double *pr, double E_u, double g1r, double g2r)
{
    EmitLane q{0.0, 0.0, 0.0, -g2r, 0, 0, 0, false, false, false};
    if (LANES == 4) {
        const double w0 = pr[0], muE = pr[1] * E_u;
        if (l == 0) { q.c0 = 2.0 * muE; q.s0 = 2; q.rate = -g1r; }
        else if (l == 1) { q.c0 = w0; q.s0 = 2; }
        else { q.c0 = -w0; q.s0 = 1; q.c1 = muE; q.has1 = q.pop = true; }
        return q;
    }
    const double e1 = pr[0], e2 = pr[1], g1 = pr[2] * E_u, g2 = pr[3] * E_u, de = e2 - e1;
    switch (l) {
    case 0: q.c0 = 2.0 * g1; q.s0 = 3; q.rate = -g1r; break;
    case 1: q.c0 = 2.0 * g2; q.s0 = 5; q.rate = -g1r; break;
    case 2: q.c0 = e1; q.s0 = 3; q.c1 = -g2; q.s1 = 7; q.has1 = true; break;
    case 3: q.c0 = -e1; q.s0 = 2; q.c1 = g1; q.has1 = q.pop = true; q.c2 = -g2; q.s2 = 6; q.has2 = true; break;
    case 4: q.c0 = e2; q.s0 = 5; q.c1 = g1; q.s1 = 7; q.has1 = true; break;
    case 5: q.c0 = -e2; q.s0 = 4; q.c1 = g2; q.has1 = q.pop = true; q.c2 = -g1; q.s2 = 6; q.has2 = true; break;
    case 6: q.c0 = de; q.s0 = 7; q.c1 = g2; q.s1 = 3; q.has1 = true; q.c2 = g1; q.s2 = 5; q.has2 = true; break;
    default: q.c0 = -de; q.s0 = 6; q.c1 = g2; q.s1 = 2; q.has1 = true; q.c2 = -g1; q.s2 = 4; q.has2 = true; break;
    }
    return q;
}

// derivative of this lane's word x; all lanes of the warp take part
template <int LANES> __device__ __forceinline__ double emit_rhs(const EmitLane &q, int l, double x)
{
    constexpr unsigned FULL = 0xffffffffu;
    double d = q.c0 * __shfl_sync(FULL, x, q.s0, LANES);
    if (LANES == 4) {
        const double pe = __shfl_sync(FULL, x, 0, LANES);
        const double t = d + q.c1 * ((1.0 - pe) - pe);
        d = q.has1 ? t : d;
    } else {
        const double p1 = __shfl_sync(FULL, x, 0, LANES), p2 = __shfl_sync(FULL, x, 1, LANES);
        const double pd = (1.0 - p1 - p2) - (l == 3 ? p1 : p2);
        const double s1 = __shfl_sync(FULL, x, q.s1, LANES), s2 = __shfl_sync(FULL, x, q.s2, LANES);
        const double t = d + q.c1 * (q.pop ? pd : s1);
        d = q.has1 ? t : d;
        const double v = d + q.c2 * s2;
        d = q.has2 ? v : d;
    }
    return d + q.rate * x;
}

template <int LANES>
__device__ __forceinline__ double rk4_lane(const EmitLane &q, int l, double x, double dt, double h2, double h6)
{
    const double k1 = emit_rhs<LANES>(q, l, x);
    const double k2 = emit_rhs<LANES>(q, l, x + h2 * k1);
    const double k3 = emit_rhs<LANES>(q, l, x + h2 * k2);
    const double k4 = emit_rhs<LANES>(q, l, x + dt * k3);
    return x + h6 * (__fma_rn(2.0, k3, __fma_rn(2.0, k2, k1)) + k4);
}

// Same step forming the rates and fractions itself.
template <int NST>
__device__ __forceinline__ void rk4(int model, const double *pr, double *rho, double E_u, double dt)
{
    const double g1 = 1.0 / pr[model == 1 ? 2 : 4], g2 = 1.0 / pr[model == 1 ? 3 : 5];
    rk4r<NST>(model, pr, rho, E_u, dt, 0.5 * dt, dt / 6.0, g1, g2);
}

}  // namespace omx
