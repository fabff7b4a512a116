// omx_run1d.cuh -- the whole time loop of a 1D grid in one launch: a cluster of eight blocks keeps
// stepping (H, sources, ADE and E with CPML, emitter current, emitters, detectors) with cluster
// barriers between the phases, instead of eight launches a step that each wait for the one before.
// A 1D step is latency alone (1500 FP64 cells, a Drude film, 16 emitters and 16 detectors: 24.7 us
// in launches of a few microseconds each, 6.5 us here); what is left is the FP64 chain of an emitter
// and of a cell (64 cycles an instruction) and two barriers.
//
// Block r owns a contiguous piece of the cells and holds their fields, coefficients and psi in shared
// memory: a cluster barrier's acquire empties L1, so every word read from memory in a phase costs an
// L2 round trip (all of it through memory: 9.0 us).  Through memory go E (the emitters and detectors
// read it, and the block before the piece's first word), the last H of a piece, ADE state and emitter
// current, each written by the thread that owns the cell; words of other threads are read past L1,
// ordered by the barriers' release / acquire.  The last SIDE threads of every block own no cells:
// they advance the emitters and take the samples (1D E: one word each) of step s while the others
// update H of step s + 1, both reading E only.  The arithmetic is k_h1 / k_e1's, k_ade's,
// k_emit_lanes', k_scatter's, inject_point's and sample_point's, in their order.
#pragma once
#include <cooperative_groups.h>
#include "omx_stencil.cuh"
#include "omx_sparse.cuh"

namespace omx {

constexpr int RUN1_CLUSTER = 8, RUN1_THREADS = 512, RUN1_SIDE = 128, RUN1_ROWS = 64;

template <class R> __device__ __forceinline__ R ld_cg(const R *p) { return __ldcg(p); }

// A lane's part of an emitter: constants, state word and dipole component
struct Run1Emitter {
    double pr[4], u[3], ul, g1, g2, x, dipole;
    long long cell;
    int n;
    bool live;
};
template <int LANES> __device__ __forceinline__ Run1Emitter run1_load(const Lay &L, const EmitArgs &A, int n0, int l)
{
    constexpr int NST = LANES == 8 ? 8 : 3;
    Run1Emitter e;
    e.live = n0 < A.n;
    e.n = e.live ? n0 : A.n - 1;          // lanes past the end follow the last emitter, without writes
    const double *pr = A.par + (long long)e.n * A.npar;
    const double *u = pr + (A.npar - 3);
#pragma unroll
    for (int q = 0; q < 4; ++q) e.pr[q] = LANES == 8 || q < 2 ? pr[q] : 0.0;
#pragma unroll
    for (int q = 0; q < 3; ++q) e.u[q] = u[q];
    e.ul = u[min(l, 2)];
    e.g1 = A.rates[2 * e.n];
    e.g2 = A.rates[2 * e.n + 1];
    e.x = A.rho[(long long)e.n * NST + min(l, NST - 1)];
    e.dipole = A.dipole[3 * e.n + min(l, 2)];
    e.cell = L.off + A.ci[e.n];
    return e;
}
template <class R, int LANES>
__device__ __forceinline__ void run1_step(const R *Ex, const EmitArgs &A, int l, Run1Emitter &e)
{
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int NST = LANES == 8 ? 8 : 3;
    const double E = (double)ld_cg(Ex + e.cell);
    const double E_u = e.u[0] * E + e.u[1] * 0.0 + e.u[2] * 0.0;
    const int w = min(l, NST - 1), n = e.n;
    const EmitLane q = emit_lane<LANES>(w, e.pr, E_u, e.g1, e.g2);
    e.x = rk4_lane<LANES>(q, w, e.x, A.dt, A.h2, A.h6);
    if (e.live && l < NST) A.rho[(long long)n * NST + l] = e.x;
    double d;
    if (LANES == 4) {
        d = 2.0 * e.pr[1] * __shfl_sync(FULL, e.x, 1, LANES);
    } else {
        const double x2 = __shfl_sync(FULL, e.x, 2, LANES), x4 = __shfl_sync(FULL, e.x, 4, LANES);
        d = 2.0 * e.pr[2] * x2 + 2.0 * e.pr[3] * x4;
    }
    const double nw = d * e.ul;
    if (e.live && l < 3) {
        A.dipole[3 * n + l] = nw;
        __stcg(A.dPdt + 3 * n + l, over_dt(nw - e.dipole, A.over));
        A.E[3 * n + l] = l == 0 ? E : 0.0;
    }
    e.dipole = nw;
}
// the emitters of one group from `from` on, LANES lanes each
template <class R, int LANES>
__device__ __forceinline__ void run1_emit(const R *Ex, const Lay &L, const EmitArgs &A, int t, int nt, int from)
{
    const int l = t % LANES;
    for (int base = from; base < A.n; base += nt / LANES) {
        Run1Emitter e = run1_load<LANES>(L, A, base + t / LANES, l);
        __syncwarp();                       // every lane has read its word
        run1_step<R, LANES>(Ex, A, l, e);
    }
}

// k_scatter at J point p for every group in turn; the point's J_old and dJ
__device__ __forceinline__ void run1_scatter(const Run1Args &A, int p, double &jo, double &dj)
{
    double j = A.J.J[0][p];
    for (int g = 0; g < A.n_grp; ++g) {
        const ScatArgs &S = A.scat[g];
        const int w = S.win[p];
        jo = j;
        j = w >= 0 ? S.wk[p] * __ldcg(S.dPdt + 3 * w) : jo;
        dj = over_dt(j - jo, S.over);
    }
    A.J.Jo[0][p] = jo;
    A.J.J[0][p] = j;
    A.J.dJ[0][p] = dj;
}

// a cell's word: its J point (RUN1_NOJ: none) and whether it has CPML terms and takes the current
constexpr int RUN1_ABS_E = 1 << 30, RUN1_ABS_H = 1 << 29, RUN1_INJ = 1 << 28, RUN1_NOJ = RUN1_INJ - 1;

template <class R, bool EXACT>
__global__ void __launch_bounds__(RUN1_THREADS) k_run1(const __grid_constant__ FieldPtrs<R> F,
                                                       const __grid_constant__ GridArgs<R> G,
                                                       const __grid_constant__ Run1Args A)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ double run1_smem[];
    const Lay &L = G.L;
    R *Ex = F.f[0] + L.off, *Hy = F.f[4] + L.off;
    const int n = L.nx, piece = (n + RUN1_CLUSTER - 1) / RUN1_CLUSTER, rank = (int)blockIdx.x;
    const int c0 = 1 + rank * piece, cells = max(0, min(piece, n - c0 + 1));
    constexpr int CELLT = RUN1_THREADS - RUN1_SIDE;
    const int t = (int)threadIdx.x;
    const bool side = t >= CELLT;
    // side thread of the cluster: warps numbered over the blocks first, so that a few emitters' warps
    // sit on several SMs (an SM issues one FP64 warp instruction in 16 cycles), and in a block from
    // the last on, away from the cells of a short piece
    const int st = ((RUN1_THREADS / 32 - 1 - t / 32) * RUN1_CLUSTER + rank) * 32 + t % 32;
    const int nst = RUN1_CLUSTER * RUN1_SIDE;

    double *rows = run1_smem;                                  // the row before and the next RUN1_ROWS
    R *sE = (R *)(rows + (RUN1_ROWS + 1) * (4 + RUN1_SOURCES)), *sH = sE + piece, *denE = sH + piece, *denH = denE + piece,
      *coef = denH + piece, *bE = coef + piece, *cE = bE + piece, *psE = cE + piece, *bH = psE + piece,
      *cH = bH + piece, *psH = cH + piece;
    int *cls = (int *)(psH + piece), *jpt = cls + piece;       // class of a dispersive cell (or -1), the cell's word
    for (int x = t; x < cells; x += RUN1_THREADS) {
        const int i = c0 + x;
        sE[x] = Ex[i];
        sH[x] = Hy[i];
        denE[x] = G.den_e[0][i];
        denH[x] = i < n ? G.den_h[0][i] : (R)0;
        coef[x] = G.dt_eps0;
        cls[x] = -1;
        if (i >= 2 && i <= n - 1 && i >= G.bb0[0] && i <= G.bb1[0]) {
            const int m = G.mat[0][i - G.bb0[0]];
            if (G.cls[m].type == CLS_PLAIN) coef[x] = G.cls[m].coef;
            else cls[x] = m;
        }
        const int le = i >= 2 && i <= n - 1 ? G.lE[0][i] : -1, lh = i <= n - 1 ? G.lH[0][i] : -1;
        bE[x] = le >= 0 ? G.bE[0][i] : (R)0;
        cE[x] = le >= 0 ? G.cE[0][i] : (R)0;
        psE[x] = le >= 0 ? G.psiE[0][0][le] : (R)0;
        bH[x] = lh >= 0 ? G.bH[0][i] : (R)0;
        cH[x] = lh >= 0 ? G.cH[0][i] : (R)0;
        psH[x] = lh >= 0 ? G.psiH[0][0][lh] : (R)0;
        int j = A.jp_at ? A.jp_at[i] : -1;
        j = j < 0 ? RUN1_NOJ : j;
        if (A.jp_at && A.inj_at[i]) j |= RUN1_INJ;
        if (le >= 0) j |= RUN1_ABS_E;
        if (lh >= 0) j |= RUN1_ABS_H;
        jpt[x] = j;
    }

    // the first group's first emitters stay in registers (read again each step: 7.2 us); warps past them
    // hold none
    Run1Emitter mine{};
    bool held = false;
    if (side && A.n_grp > 0) {
        const EmitArgs &G0 = A.grp[0];
        const int lanes = G0.model == 1 ? 4 : 8;
        held = st / 32 * 32 / lanes < G0.n;
        if (held) mine = lanes == 4 ? run1_load<4>(L, G0, st / 4, st % 4) : run1_load<8>(L, G0, st / 8, st % 8);
    }

    // emitters and samples of the step whose table row is given; side threads
    auto side_work = [&](const double *row) {
        if (row[2] != 0.0)
            for (int g = 0; g < A.n_grp; ++g) {
                if (A.grp[g].model == 1) {
                    if (held && g == 0) run1_step<R, 4>(F.f[0], A.grp[0], st % 4, mine);
                    run1_emit<R, 4>(F.f[0], L, A.grp[g], st, nst, g == 0 ? nst / 4 : 0);
                } else {
                    if (held && g == 0) run1_step<R, 8>(F.f[0], A.grp[0], st % 8, mine);
                    run1_emit<R, 8>(F.f[0], L, A.grp[g], st, nst, g == 0 ? nst / 8 : 0);
                }
            }
        const int slot = A.has_det ? (int)row[3] : -1;
        if (slot >= 0) {
            if (st == nst - 1) A.det.times[slot] = row[0];
            for (int s = nst - 1 - st; s < A.det.n; s += nst)
                A.det.rec[(long long)slot * A.det.n + s] = (double)ld_cg(F.f[A.det.field[s]] + A.det.t0[s]);
        }
    };

    const int W = A.W;
    for (int s = 0; s < A.nsteps; ++s) {
        const int r = s % RUN1_ROWS;
        if (r == 0) {                          // every thread is past the rows of the last barrier
            for (int q = t; q < (RUN1_ROWS + 1) * W; q += RUN1_THREADS) {
                const long long at = (long long)(s - 1) * W + q;
                if (at >= 0 && at < (long long)A.nsteps * W) rows[q] = A.tab[at];
            }
            __syncthreads();
        }
        const double *row = rows + (r + 1) * W, *prev = row - W;
        if (side) {
            if (s > 0) side_work(prev);
        } else {
            for (int x = t; x < cells; x += CELLT) {
                if (c0 + x > n - 1) continue;
                const R e1 = x + 1 < cells ? sE[x + 1] : ld_cg(Ex + (c0 + x + 1));
                const R d = sE[x] - e1;
                R hy = h1_bulk<R, EXACT>(G, d, denH[x], sH[x]);
                if (jpt[x] & RUN1_ABS_H) hy = h1_absorb<R, EXACT>(G, d, bH[x], cH[x], psH[x], hy);
                sH[x] = hy;
                if (x + 1 == cells) Hy[c0 + x] = hy;
            }
        }
        __syncwarp();
        cluster.sync();
        if (!side) {
            // sources (source_interactions before the E update), one after the other: the owner of a
            // source point's cell adds it (a thread that looked through every point for its own cells
            // took 57 us a step for a source of 513 points, 8.3 us in launches)
            for (int q = 0; q < A.n_src; ++q) {
                const double amp = row[4 + q];
                if (A.src_kind[q] == 1) {
                    const int x = (int)(A.plane_e[q] - L.off) - c0;
                    if (amp != 0.0 && x >= 0 && x < cells && x % CELLT == t) {
                        sE[x] = (R)__dadd_rn((double)sE[x], __dmul_rn(A.plane_c[q], amp));
                        Ex[c0 + x] = sE[x];
                    }
                    continue;
                }
                const SrcArgs &S = A.src[q];
                for (int x = t; x < cells; x += CELLT) {
                    const int k = c0 + x - A.src_first[q];
                    if (k < 0 || k >= S.n) continue;
                    const double ja = amp * S.ka[k];
                    const double jav = S.avg ? 0.5 * (ja + amp * S.kb[k]) : ja;
                    sE[x] = (R)((double)sE[x] + S.c_src * jav);
                    Ex[c0 + x] = sE[x];
                }
            }
            for (int x = t; x < cells; x += CELLT) {
                const int i = c0 + x, flags = jpt[x], p = flags & RUN1_NOJ;
                double jo = 0.0, dj = 0.0;
                if (p != RUN1_NOJ) {
                    if (s > 0 && prev[2] != 0.0) run1_scatter(A, p, jo, dj);
                    else jo = A.J.Jo[0][p], dj = A.J.dJ[0][p];
                }
                if (i < 2 || i > n - 1) continue;
                const R h0 = x > 0 ? sH[x - 1] : ld_cg(Hy + (i - 1));
                const R d = h0 - sH[x];
                const R rot = d * denE[x];
                R e = sE[x];
                const int m = cls[x];
                if (m < 0) {
                    e = fma1<R, EXACT>(coef[x], rot, e);
                } else {
                    const ClsR<R> cl = G.cls[m];
                    const long long b = i - G.bb0[0];
                    if constexpr (EXACT) e = ade_update<R>(e, rot, cl, 0, b, G);
                    else e = f3t_ade(e, rot, cl.type, G.med + cl.medium, G.ade + b, G.bbV, G.P);
                }
                if (flags & RUN1_ABS_E) e = e1_absorb<R, EXACT>(G, d, bE[x], cE[x], psE[x], e);
                if (flags & RUN1_INJ) {
                    const double jav = __dadd_rn(jo, __dmul_rn(row[0] - row[1], dj));
                    e = (R)__dsub_rn((double)e, __dmul_rn(A.dt_eps0, jav));
                }
                sE[x] = e;
                Ex[i] = e;
            }
        }
        __syncwarp();
        cluster.sync();
    }
    // the last step's emitters, samples and current; fields and psi back to memory
    const double *last = rows + ((A.nsteps - 1) % RUN1_ROWS + 1) * W;
    if (side) side_work(last);
    __syncwarp();
    cluster.sync();
    for (int x = t; x < cells && !side; x += CELLT) {
        const int i = c0 + x, p = jpt[x] & RUN1_NOJ;
        double jo, dj;
        if (p != RUN1_NOJ && last[2] != 0.0) run1_scatter(A, p, jo, dj);
        Hy[i] = sH[x];
        if (jpt[x] & RUN1_ABS_E) G.psiE[0][0][G.lE[0][i]] = psE[x];
        if (jpt[x] & RUN1_ABS_H) G.psiH[0][0][G.lH[0][i]] = psH[x];
    }
}

template <class R, bool EXACT>
cudaError_t launch_run1_impl(const FieldPtrs<R> &F, const GridArgs<R> &G, const Run1Args &A, void *s)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(RUN1_CLUSTER);
    cfg.blockDim = dim3(RUN1_THREADS);
    cfg.stream = (cudaStream_t)s;
    const size_t piece = (size_t)(G.L.nx + RUN1_CLUSTER - 1) / RUN1_CLUSTER;
    cfg.dynamicSmemBytes = (RUN1_ROWS + 1) * (4 + RUN1_SOURCES) * sizeof(double) + piece * (11 * sizeof(R) + 2 * sizeof(int));
    const cudaError_t e = cudaFuncSetAttribute((const void *)k_run1<R, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)(227 * 1024));
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = RUN1_CLUSTER;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_run1<R, EXACT>, F, G, A);
}

}  // namespace omx
