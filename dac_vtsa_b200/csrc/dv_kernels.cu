// dv_kernels.cu -- residual, matvec, diagnostics, accumulator and FD-Jacobian kernels.
// Compiled with -fmad=false (see dv_physics.cuh).
#include "dv_internal.h"
#include "dv_residual.cuh"

#include <algorithm>
#include <mutex>
#include <utility>

namespace dv {

RecLayout rec_layout(const dv_step_params& p) {
    RecLayout r;
    const int64_t nc = (int64_t)p.Nr * p.Nth * p.Nz, nf = (int64_t)p.Nr * p.Nth, nw = (int64_t)p.Nth * p.Nz;
    int64_t o = 0;
    r.T = o; o += nc;
    r.P = o; o += nc;
    r.y = o; o += 3 * nc;
    r.qstar = o; o += 2 * nc;
    r.uz = o; o += nf * (p.Nz - 1);
    r.ur = o; o += (int64_t)(p.Nr - 1) * p.Nth * p.Nz;
    r.uth = o; o += nc;
    r.bnd = o; o += 2 * BR_N * nf;
    r.Qj = o; o += nw;
    r.Qa = o; o += nw;
    r.Qw = o; o += nw;
    r.Rb = o; o += nw;
    r.Qhx = o; o += nc;
    r.total = o;
    return r;
}

static Rec make_rec(const RecLayout& l, double* base) {
    Rec r;
    r.T = base + l.T;
    r.P = base + l.P;
    r.y = base + l.y;
    r.qstar = base + l.qstar;
    r.uz = base + l.uz;
    r.ur = base + l.ur;
    r.uth = base + l.uth;
    r.bnd = base + l.bnd;
    r.Qj = base + l.Qj;
    r.Qa = base + l.Qa;
    r.Qw = base + l.Qw;
    r.Rb = base + l.Rb;
    r.Qhx = base + l.Qhx;
    return r;
}

static __device__ __forceinline__ void cell_ijk(const dv_step_params& p, int64_t c, int& i, int& j, int& k) {
    k = (int)(c % p.Nz);
    int64_t r = c / p.Nz;
    j = (int)(r % p.Nth);
    i = (int)(r / p.Nth);
}

enum { M_RHS = 0, M_STAGE = 1, M_MATVEC = 2 };

// One thread per cell.  MODE selects the epilogue:
//  M_RHS    out = f                                   (core/residual.py:361-365)
//  M_STAGE  out = y - gh f - rhs_known                (core/residual.py:420-423)
//  M_MATVEC out = (v - dh (f(z+sig v) - f0)/sig)/s    (core/solver.py:196-203)
template <int MODE, bool REC>
__global__ void __launch_bounds__(128) k_cells(dv_step_params p, Aux aux, Rec rec, double t, const double* __restrict__ y,
                                               const double* __restrict__ u, const double* __restrict__ sc,
                                               const double* __restrict__ f0, const double* __restrict__ scal,
                                               double gh, double* __restrict__ out) {
    const int64_t nc = (int64_t)p.Nr * p.Nth * p.Nz;
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    int i, j, k;
    cell_ijk(p, c, i, j, k);
    double f[DV_NV], fw = 0.0;
    const bool outer_wall = (i == p.Nr - 1) && p.wall_on;
    const int64_t iw = (int64_t)DV_NV * nc + (int64_t)j * p.Nz + k;
    if (MODE == M_MATVEC) {
        const double un = scal[0];
        if (un == 0.0) {            // matvec of a zero direction is zero
#pragma unroll
            for (int v = 0; v < DV_NV; ++v) out[v * nc + c] = 0.0;
            if (outer_wall) out[iw] = 0.0;
            return;
        }
        const double sig = 1.4901161193847656e-08 * scal[1] / un;
        LoadDir ld{y, u, sc, sig};
        cell_eval(p, aux, ld, t, i, j, k, f, outer_wall ? &fw : nullptr, REC ? &rec : nullptr);
#pragma unroll
        for (int v = 0; v < DV_NV; ++v) {
            const int64_t ix = v * nc + c;
            const double vv = u[ix] * sc[ix];
            out[ix] = (vv - gh * (f[v] - f0[ix]) / sig) / sc[ix];
        }
        if (outer_wall) {
            const double vv = u[iw] * sc[iw];
            out[iw] = (vv - gh * (fw - f0[iw]) / sig) / sc[iw];
        }
        return;
    }
    LoadPlain ld{y};
    cell_eval(p, aux, ld, t, i, j, k, f, outer_wall ? &fw : nullptr, REC ? &rec : nullptr);
    if (MODE == M_RHS) {
#pragma unroll
        for (int v = 0; v < DV_NV; ++v) out[v * nc + c] = f[v];
        if (outer_wall) out[iw] = fw;
    } else {
#pragma unroll
        for (int v = 0; v < DV_NV; ++v) {
            const int64_t ix = v * nc + c;
            out[ix] = y[ix] - gh * f[v] - u[ix];
        }
        if (outer_wall) out[iw] = y[iw] - gh * fw - u[iw];
    }
}

// Sums over the 256 threads of cnt values per thread, in the order of a tree that halves the threads
// (t + 128, 64, .. 1): the values go through shared memory, a warp takes a value and adds its eight
// entries per lane and then the lanes.  All of a batch at once: two barriers instead of nine for each
// value (the 36 rates of an 8x8x32 bed: 14.9 -> 5.7 us).
constexpr int ACC_T = 256, ACC_MAX = 10;
__device__ void block_sums(const double* v, int cnt, double (*sh)[ACC_T], double* out) {
    const int t = threadIdx.x, lane = t & 31;
#pragma unroll
    for (int q = 0; q < ACC_MAX; ++q)
        if (q < cnt) sh[q][t] = v[q];
    __syncthreads();
    for (int q = t >> 5; q < cnt; q += ACC_T / 32) {
        const double* a = sh[q] + lane;
        double s = ((a[0] + a[128]) + (a[64] + a[192])) + ((a[32] + a[160]) + (a[96] + a[224]));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s = s + __shfl_down_sync(0xffffffffu, s, off);
        if (lane == 0) out[q] = s;
    }
    __syncthreads();
}

// The 36 accumulator rates from the end-face and wall records (core/residual.py:371-417).
__global__ void __launch_bounds__(ACC_T) k_accumulators(dv_step_params p, const double* __restrict__ rec_bnd,
                                                        const double* __restrict__ Qj, const double* __restrict__ Qa,
                                                        const double* __restrict__ Qw, const double* __restrict__ Qhx,
                                                        double* __restrict__ acc) {
    __shared__ double sh[ACC_MAX][ACC_T], a[DV_NACC], sums[ACC_MAX];
    const int t = threadIdx.x;
    const int nf = p.Nr * p.Nth, nw = p.Nth * p.Nz;
    const int64_t nc = (int64_t)p.Nr * p.Nth * p.Nz;
    if (t < DV_NACC) a[t] = 0.0;
    const double ex = (p.gam - 1.0) / p.gam;
    const double pre = p.gam / (p.gam - 1.0) * DV_R;
    for (int e = 0; e < 2; ++e) {
        const dv_end& E = p.ends[e];
        if (E.valve < 0) continue;
        const double* b = rec_bnd + (int64_t)e * BR_N * nf;
        const bool parts = (E.kind == DV_END_VALVE);
        const int base = E.valve * (2 * DV_NG + 4);
        double s_in[DV_NG] = {0, 0, 0}, s_out[DV_NG] = {0, 0, 0}, h_in = 0, h_out = 0, wp = 0, wf = 0;
        for (int f = t; f < nf; f += blockDim.x) {
            const bool inflow = b[BR_UOUT * nf + f] < 0.0;
            double Fin[DV_NG];
            for (int q = 0; q < DV_NG; ++q) {
                Fin[q] = b[(BR_FIN + q) * nf + f];
                s_in[q] += parts ? b[(BR_FINP + q) * nf + f] : (inflow ? Fin[q] : 0.0);
                s_out[q] += parts ? b[(BR_FOUTP + q) * nf + f] : (inflow ? 0.0 : -Fin[q]);
            }
            const double H = b[BR_HIN * nf + f];
            h_in += parts ? b[BR_HINP * nf + f] : (inflow ? H : 0.0);
            h_out += parts ? b[BR_HOUTP * nf + f] : (inflow ? 0.0 : -H);
            const double Pf = b[BR_PFACE * nf + f];
            if (E.is_vacuum) {
                double Fo[DV_NG];
                for (int q = 0; q < DV_NG; ++q) Fo[q] = inflow ? 0.0 : -Fin[q];
                double Ft = p.pump_water ? (Fo[0] + Fo[1] + Fo[2]) : (Fo[0] + Fo[2]);
                double ratio = npmax(p.P_amb / npmax(Pf, 1.0), 1.0);
                double eta = p.eta_vac;
                if (p.vac_krishnamurthy) {
                    double pb = Pf / 1e5;
                    eta = npmax(0.8 * 19.55 * pb / (1.0 + 19.55 * pb), 1e-3);
                }
                wp += pre * b[BR_TLAY * nf + f] * Ft * (pow(ratio, ex) - 1.0) / eta;
            }
            if (E.is_feed) {
                double Ft;
                if (parts) Ft = b[(BR_FINP + 0) * nf + f] + b[(BR_FINP + 1) * nf + f] + b[(BR_FINP + 2) * nf + f];
                else Ft = (inflow ? Fin[0] : 0.0) + (inflow ? Fin[1] : 0.0) + (inflow ? Fin[2] : 0.0);
                double ratio = npmax(Pf / p.P_amb, 1.0);
                wf += pre * E.T_ext * Ft * (pow(ratio, ex) - 1.0) / p.eta_bl;
            }
        }
        const double v[ACC_MAX] = {s_in[0], s_in[1], s_in[2], s_out[0], s_out[1], s_out[2], h_in, h_out, wp, wf};
        block_sums(v, ACC_MAX, sh, sums);                // (no vacuum, no feed: sums of zeros)
        if (t < ACC_MAX) a[base + t] = sums[t];
        __syncthreads();
    }
    double jp = 0, jn = 0, qa = 0, qw = 0, hp = 0, hn = 0;
    for (int w = t; w < nw; w += blockDim.x) {
        jp += npmax(Qj[w], 0.0);
        jn += npmin(Qj[w], 0.0);
        qa += Qa[w];
        qw += Qw[w];
    }
    if (p.hx_on) {
        for (int64_t c = t; c < nc; c += blockDim.x) {
            hp += npmax(Qhx[c], 0.0);
            hn += npmin(Qhx[c], 0.0);
        }
    }
    const double v[ACC_MAX] = {jp, jn, qa, qw, hp, hn};
    block_sums(v, 6, sh, sums);
    if (t < 6) a[30 + t] = sums[t];
    __syncthreads();
    if (t < DV_NACC) acc[t] = a[t];
}

// ---------------------------------------------------------------- split residual
// The residual as three launches with short per-thread chains: per-cell properties and uptake
// (k_cprops), the flux through every face once (k_faces), divergence and sources of each row
// (k_assemble).  Each step evaluates the same expressions on the same inputs
// as cell_eval, so the results are the same bits; the thread-per-cell kernel computes the
// properties of every cell seven times and every face twice.
enum { SP_C0 = 0, SP_T = 3, SP_P, SP_CPOS, SP_Y0, SP_MU = SP_Y0 + 3, SP_KG, SP_RHO, SP_CPM, SP_DM, SP_LAM0,
       SP_RATE0, SP_QS0 = SP_RATE0 + 2, SP_NCELL = SP_QS0 + 2 };

struct Split {
    double* cell;          // [SP_NCELL][nc]
    double* zf;            // [4][ncol (Nz+1)]: +z flux through face kf of a column (kf 0 = top end, Nz = bottom end)
    double* rf;            // [4][(Nr-1) Nth Nz]: +r flux between rings i and i+1 at (j, k)
    double* tf;            // [4][Nr Nth Nz]: +theta flux between sectors j and j+1 (periodic) at (i, k)
    double* wall;          // [Nth Nz]: wall rows of a call whose result replaces its state
    int64_t nc, nzf, nrf, ntf;
};

int64_t split_doubles(const dv_step_params& p) {
    const int64_t nc = (int64_t)p.Nr * p.Nth * p.Nz, ncol = (int64_t)p.Nr * p.Nth;
    return SP_NCELL * nc + 4 * (ncol * (p.Nz + 1) + (int64_t)(p.Nr - 1) * p.Nth * p.Nz + nc) +
           (int64_t)p.Nth * p.Nz;
}

static Split split_of(const dv_step_params& p, double* base) {
    Split S;
    S.nc = (int64_t)p.Nr * p.Nth * p.Nz;
    S.nzf = (int64_t)p.Nr * p.Nth * (p.Nz + 1);
    S.nrf = (int64_t)(p.Nr - 1) * p.Nth * p.Nz;
    S.ntf = S.nc;
    S.cell = base;
    S.zf = S.cell + SP_NCELL * S.nc;
    S.rf = S.zf + 4 * S.nzf;
    S.tf = S.rf + 4 * S.nrf;
    S.wall = S.tf + 4 * S.ntf;
    return S;
}

static __device__ __forceinline__ void sp_get(const Split& S, int64_t c, Cell& s, Props& o) {
    const double* a = S.cell;
    const int64_t nc = S.nc;
#pragma unroll
    for (int q = 0; q < DV_NG; ++q) {
        s.c[q] = a[(SP_C0 + q) * nc + c];
        o.y[q] = a[(SP_Y0 + q) * nc + c];
    }
    s.q[0] = s.q[1] = s.e = 0.0;            // not read by the face and wall terms
    o.T = a[SP_T * nc + c];
    o.P = a[SP_P * nc + c];
    o.Tp = 0.0;                             // only the uptake reads it (done in k_cprops)
    o.Cpos = a[SP_CPOS * nc + c];
    o.mu = a[SP_MU * nc + c];
    o.kg = a[SP_KG * nc + c];
    o.rho = a[SP_RHO * nc + c];
    o.cpm = a[SP_CPM * nc + c];
    o.Dm = a[SP_DM * nc + c];
    o.lam0 = a[SP_LAM0 * nc + c];
}

static __device__ __forceinline__ void flux_put(double* base, int64_t stride, int64_t ix, const Flux& F) {
#pragma unroll
    for (int q = 0; q < DV_NG; ++q) base[q * stride + ix] = F.F[q];
    base[DV_NG * stride + ix] = F.H;
}

static __device__ __forceinline__ void flux_get(const double* base, int64_t stride, int64_t ix, Flux& F) {
#pragma unroll
    for (int q = 0; q < DV_NG; ++q) F.F[q] = base[q * stride + ix];
    F.H = base[DV_NG * stride + ix];
}

// Direction scale of the finite-difference matvec: sig = sqrt(eps) ||z|| / ||v|| (core/solver.py:196-203).
static __device__ __forceinline__ double matvec_sig(const double* scal) {
    return 1.4901161193847656e-08 * scal[1] / scal[0];
}

// Two warps per 32 cells: warp 0 evaluates the transport properties of its cells, warp 1 the
// temperature, isotherms and LDF rates of the same cells (the two halves of the per-cell chain run
// side by side; uptake reads only the clipped temperature of the properties).
// The work of one 64-thread block `vb` (cells vb*32 .. vb*32 + 31).  Used by the cooperative FD
// matvec (k_matvec_coop, whose phases share 64-thread blocks); k_cprops runs the eight-warp form
// below, which gives the same bits.
template <int MODE>
__device__ __forceinline__ void cprops_block(const dv_step_params& p, const Split& S, const double* __restrict__ y,
                                             const double* __restrict__ u, const double* __restrict__ sc,
                                             const double* __restrict__ scal, int64_t vb) {
    const int64_t nc = S.nc;
    const int64_t c = vb * 32 + (threadIdx.x & 31);
    const bool half = (threadIdx.x >> 5) != 0;             // warp-uniform
    if (c >= nc) return;
    Cell s;
    if (MODE == M_MATVEC) {
        if (scal[0] == 0.0) return;         // zero direction: k_assemble writes zeros
        LoadDir ld{y, u, sc, matvec_sig(scal)};
        load_cell(ld, nc, c, s);
    } else {
        LoadPlain ld{y};
        load_cell(ld, nc, c, s);
    }
    double* a = S.cell;
    if (!half) {
        Props o;
        cell_props(p, s, o);
#pragma unroll
        for (int q = 0; q < DV_NG; ++q) {
            a[(SP_C0 + q) * nc + c] = s.c[q];
            a[(SP_Y0 + q) * nc + c] = o.y[q];
        }
        a[SP_T * nc + c] = o.T;
        a[SP_P * nc + c] = o.P;
        a[SP_CPOS * nc + c] = o.Cpos;
        a[SP_MU * nc + c] = o.mu;
        a[SP_KG * nc + c] = o.kg;
        a[SP_RHO * nc + c] = o.rho;
        a[SP_CPM * nc + c] = o.cpm;
        a[SP_DM * nc + c] = o.Dm;
        a[SP_LAM0 * nc + c] = o.lam0;
    } else {
        Props o;                            // uptake reads o.Tp only (same expression as cell_props)
        o.Tp = npclip(cell_T(p, s), 150.0, 1500.0);
        double rate[DV_NA], qstar[DV_NA];
        uptake(p, s, o, rate, qstar);
#pragma unroll
        for (int q = 0; q < DV_NA; ++q) {
            a[(SP_RATE0 + q) * nc + c] = rate[q];
            a[(SP_QS0 + q) * nc + c] = qstar[q];
        }
    }
}

// Eight warps per 32 cells.  The transcendental terms of a cell's properties and uptake that do not
// depend on one another (each power is a called routine, so one thread evaluates them strictly one
// after another) are spread over the warps of its block, then combined after one barrier:
//   warp 0: viscosities and the CO2-air Fuller diffusivity     warps 1-3: conductivity of gas 0-2
//   warp 4: the CO2-water Fuller diffusivity                    warp 5: water saturation and GAB loading
//   warp 6: the dry CO2 Toth term                               warp 7: the wet CO2 Toth term (wadst)
// then warp 0 mixes the transport properties and warp 1 finishes the loadings and LDF rates.  Every
// value is the same expression on the same operands as in cell_props / uptake, so the results are
// bit-identical to the one-thread-per-cell evaluation.
#define CP_WARPS 8
static_assert(DV_NG == 3 && CP_WARPS == 8, "the warp roles assume three gases");
template <class L>
__device__ __forceinline__ void cprops_split(const dv_step_params& p, const Split& S, const L& ld, int64_t vb) {
    __shared__ double xk[DV_NG][32], xdcw[32], xqw[32], xqd[32], xqwet[32];
    const int64_t nc = S.nc;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t c = vb * 32 + lane;
    const bool in = c < nc;
    Cell s;
    if (in) load_cell(ld, nc, c, s);
    else s = Cell{};
    Props o;
    double ycl[DV_NG];
    props_state(p, s, o, ycl);
    const double T = o.Tp, T3 = T / 300.0;
    const double pp = npmax(s.c[0] * DV_R * o.Tp, 0.0);
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    double mu[DV_NG], sq[DV_NG], D_ca = 0.0;
    if (w == 0) {
#pragma unroll
        for (int s2 = 0; s2 < DV_NG; ++s2) {
            mu[s2] = gas_mu(p, s2, T);
            sq[s2] = sqrt(mu[s2]);
        }
        D_ca = fuller(p, 0, T, npmax(o.P, 1.0));
    } else if (w <= DV_NG) {
        xk[w - 1][lane] = gas_k(p, w - 1, T3);
    } else if (w == 4) {
        xdcw[lane] = fuller(p, 1, T, npmax(o.P, 1.0));
    } else if (w == 5) {
        xqw[lane] = q_h2o(p, s.c[1] * DV_R * o.Tp, o.Tp, psat_h2o(o.Tp));
    } else if (w == 6) {
        xqd[lane] = co2_needs_qw(p) ? nan : co2_toth_dry(p, pp, o.Tp);
    } else {
        xqwet[lane] = (p.coads == DV_COADS_WADST) ? co2_toth_wet(p, pp, o.Tp) : nan;
    }
    __syncthreads();
    if (!in || w > 1) return;
    double* a = S.cell;
    if (w == 0) {
        double kk[DV_NG];
#pragma unroll
        for (int s2 = 0; s2 < DV_NG; ++s2) kk[s2] = xk[s2][lane];
        double mu_m, k_m;
        wilke_mix(p, ycl, mu, kk, sq, mu_m, k_m);
        o.mu = mu_m;
        o.kg = k_m;
        o.rho = o.Cpos * wsum3(p.M, ycl);
        o.cpm = wsum3(p.cpg, ycl);
        o.Dm = blanc_Dm(ycl, D_ca, xdcw[lane]);
        o.lam0 = stagnant(p, o.kg);
#pragma unroll
        for (int q = 0; q < DV_NG; ++q) {
            a[(SP_C0 + q) * nc + c] = s.c[q];
            a[(SP_Y0 + q) * nc + c] = o.y[q];
        }
        a[SP_T * nc + c] = o.T;
        a[SP_P * nc + c] = o.P;
        a[SP_CPOS * nc + c] = o.Cpos;
        a[SP_MU * nc + c] = o.mu;
        a[SP_KG * nc + c] = o.kg;
        a[SP_RHO * nc + c] = o.rho;
        a[SP_CPM * nc + c] = o.cpm;
        a[SP_DM * nc + c] = o.Dm;
        a[SP_LAM0 * nc + c] = o.lam0;
    } else {
        double rate[DV_NA], qstar[DV_NA];
        const double qw_eq = xqw[lane];
        const double basis = p.basis_state ? s.q[1] : qw_eq;
        qstar[0] = q_co2_raw(p, pp, o.Tp, basis, xqd[lane], xqwet[lane]) * (pp / (pp + p.p_reg));
        qstar[1] = qw_eq;
        ldf_rates(p, s, o.Tp, qstar, rate);
#pragma unroll
        for (int q = 0; q < DV_NA; ++q) {
            a[(SP_RATE0 + q) * nc + c] = rate[q];
            a[(SP_QS0 + q) * nc + c] = qstar[q];
        }
    }
}

template <int MODE>
__global__ void __launch_bounds__(CP_WARPS * 32) k_cprops(dv_step_params p, Split S, const double* __restrict__ y,
                                                          const double* __restrict__ u, const double* __restrict__ sc,
                                                          const double* __restrict__ scal) {
    pdl_wait();                             // (launched programmatically inside the GMRES graph)
    pdl_trigger();
    if (MODE == M_MATVEC) {
        if (scal[0] == 0.0) return;         // zero direction (grid-uniform): k_assemble writes zeros
        cprops_split(p, S, LoadDir{y, u, sc, matvec_sig(scal)}, blockIdx.x);
    } else {
        cprops_split(p, S, LoadPlain{y}, blockIdx.x);
    }
}

// MUSCL slope of cell kk of a column starting at cell index base (zero next to the ends).
static __device__ __forceinline__ void sp_slope(const dv_step_params& p, const Split& S, int64_t base, int kk,
                                                bool muscl, double s[4]) {
    s[0] = s[1] = s[2] = s[3] = 0.0;
    if (!muscl || kk < 1 || kk > p.Nz - 2) return;
    const double* a = S.cell;
    const int64_t nc = S.nc, c = base + kk;
#pragma unroll
    for (int q = 0; q < DV_NG; ++q) {
        const double* cq = a + (SP_C0 + q) * nc;
        s[q] = limited_slope(p.limiter, cq[c] - cq[c - 1], cq[c + 1] - cq[c]);
    }
    const double* T = a + SP_T * nc;
    s[3] = limited_slope(p.limiter, T[c] - T[c - 1], T[c + 1] - T[c]);
}

// One thread per face: interior z faces, r faces, theta faces, the two end faces of every column
// (kept last so the warps of each range run one kind of face); then the wall resistance of each outer-ring
// cell, into rec.Rb (the longest chain of a cell's balances, two powers: here beside the faces).
// The face of index g (all kinds in the order above).
template <bool REC>
__device__ __forceinline__ void faces_at(const dv_step_params& p, const Aux& aux, const Split& S, const Rec& rec,
                                         double t, const double* __restrict__ scal,
                                         const double* __restrict__ dargs, int64_t g) {
    if (scal && scal[0] == 0.0) return;
    if (dargs) t = dargs[0];
    const int Nr = p.Nr, Nth = p.Nth, Nz = p.Nz;
    const int64_t ncol = (int64_t)Nr * Nth;
    const int64_t nzi = ncol * (Nz - 1);
    const int64_t nr = (Nr > 1) ? S.nrf : 0;
    const int64_t nt = (Nth > 1) ? S.ntf : 0;
    if (g < nzi) {
        const int64_t col = g / (Nz - 1);
        const int k = (int)(g % (Nz - 1));
        const int i = (int)(col / Nth);
        const int64_t base = col * Nz;
        const bool muscl = (Nz >= 3 && p.limiter != DV_LIM_UPWIND);
        double sL[4], sR[4];
        sp_slope(p, S, base, k, muscl, sL);
        sp_slope(p, S, base, k + 1, muscl, sR);
        Cell a, b;
        Props L, R;
        sp_get(S, base + k, a, L);
        sp_get(S, base + k + 1, b, R);
        Flux F;
        double uz;
        zface(p, i, L, R, a, b, sL, sR, muscl, aux.n_nom[col], F, &uz);
        flux_put(S.zf, S.nzf, col * (Nz + 1) + k + 1, F);
        if (REC) rec.uz[col * (Nz - 1) + k] = uz;
        return;
    }
    g -= nzi;
    if (g < nr) {                       // between (i, j, k) and (i+1, j, k); g = that first cell's index
        const int i = (int)(g / ((int64_t)Nth * Nz));
        Cell a, b;
        Props A, B;
        sp_get(S, g, a, A);
        sp_get(S, g + (int64_t)Nth * Nz, b, B);
        Flux F;
        double ur;
        tface(p, A, B, a, b, p.drc[i], p.Ar[i], F, &ur);
        flux_put(S.rf, S.nrf, g, F);
        if (REC) rec.ur[g] = ur;
        return;
    }
    g -= nr;
    if (g < nt) {                       // between (i, j, k) and (i, j+1 mod Nth, k); g = the first cell
        const int k = (int)(g % Nz);
        const int64_t r = g / Nz;
        const int j = (int)(r % Nth);
        const int i = (int)(r / Nth);
        const int jp = (j == Nth - 1) ? 0 : j + 1;
        Cell a, b;
        Props A, B;
        sp_get(S, g, a, A);
        sp_get(S, ((int64_t)i * Nth + jp) * Nz + k, b, B);
        Flux F;
        double ut;
        tface(p, A, B, a, b, p.arc[i], p.Ath[i], F, &ut);
        flux_put(S.tf, S.ntf, g, F);
        if (REC) rec.uth[g] = ut;
        return;
    }
    g -= nt;
    if (g < 2 * ncol) {
        const int e = (int)(g / ncol);
        const int64_t col = g % ncol;
        const int i = (int)(col / Nth);
        const int64_t c = col * Nz + (e == 0 ? 0 : Nz - 1);
        Cell s;
        Props o;
        sp_get(S, c, s, o);
        double F_in[DV_NG], H_in;
        end_face(p, p.ends[e], t, i, s, o, aux.feed_flux[col], F_in, H_in,
                 REC ? rec.bnd + (int64_t)e * BR_N * ncol + col : nullptr, ncol);
        Flux F;                           // stored as the +z flux through the face
#pragma unroll
        for (int q = 0; q < DV_NG; ++q) F.F[q] = (e == 0) ? F_in[q] : -F_in[q];
        F.H = (e == 0) ? H_in : -H_in;
        flux_put(S.zf, S.nzf, col * (Nz + 1) + (e == 0 ? 0 : Nz), F);
        return;
    }
    g -= 2 * ncol;
    if (g < (int64_t)Nth * Nz) {
        Cell s;
        Props o;
        sp_get(S, (int64_t)(Nr - 1) * Nth * Nz + g, s, o);
        rec.Rb[g] = wall_R_bed(p, o);
    }
}

template <bool REC>
__global__ void __launch_bounds__(64) k_faces(dv_step_params p, Aux aux, Split S, Rec rec, double t,
                                              const double* __restrict__ scal, const double* __restrict__ dargs) {
    pdl_wait();
    pdl_trigger();
    faces_at<REC>(p, aux, S, rec, t, scal, dargs, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

// Row v (0..5, or 6: the wall node) of cell c: true, its index and value where the cell has one.
template <int MODE, bool REC, class L>
__device__ __forceinline__ bool assemble_row(const dv_step_params& p, const Aux& aux, const Split& S, const Rec& rec,
                                             double t, const L& ld, const double* __restrict__ y,
                                             const double* __restrict__ u, const double* __restrict__ sc,
                                             const double* __restrict__ f0, double sig, double gh, int64_t c, int v,
                                             int64_t& ix, double& r) {
    const int64_t nc = S.nc;
    if (c >= nc) return false;
    int i, j, k;
    cell_ijk(p, c, i, j, k);
    const int Nr = p.Nr, Nth = p.Nth, Nz = p.Nz;
    const int64_t wn = (int64_t)j * Nz + k;
    if (v == DV_NV && !(i == Nr - 1 && p.wall_on)) return false;
    ix = v < DV_NV ? v * nc + c : (int64_t)DV_NV * nc + wn;
    double f;
    if (v == 3 || v == 4) {
        f = S.cell[(SP_RATE0 + v - 3) * nc + c];
    } else if (v == DV_NV) {
        wall_terms(p, aux, ld, jacket_T(p, t), j, k, S.cell[SP_T * nc + c], rec.Rb[wn], &f);
    } else {
        const int q = v < DV_NG ? v : DV_NG;
        const double* z = S.zf + q * S.nzf + ((int64_t)i * Nth + j) * (Nz + 1) + k;
        double rm = 0.0, rp = 0.0, tm = 0.0, tp = 0.0;
        if (Nr > 1) {
            if (i > 0) rm = S.rf[q * S.nrf + c - (int64_t)Nth * Nz];
            if (i < Nr - 1) rp = S.rf[q * S.nrf + c];
        }
        if (Nth > 1) {
            tm = S.tf[q * S.ntf + ((int64_t)i * Nth + (j == 0 ? Nth - 1 : j - 1)) * Nz + k];
            tp = S.tf[q * S.ntf + c];
        }
        const double div = face_div(p, i, z[0], z[1], rm, rp, tm, tp);
        f = v < DV_NG ? row_mass(p, i, div, (v < DV_NA) ? S.cell[(SP_RATE0 + v) * nc + c] : 0.0)
                      : row_energy(p, aux, ld, t, i, j, k, S.cell[SP_T * nc + c], i == Nr - 1 ? rec.Rb[wn] : 0.0, div,
                                   nullptr, REC ? &rec : nullptr);
    }
    if (MODE == M_RHS) {
        r = f;
    } else if (MODE == M_STAGE) {
        r = y[ix] - gh * f - u[ix];
    } else {
        const double vv = u[ix] * sc[ix];
        r = (vv - gh * (f - f0[ix]) / sig) / sc[ix];
    }
    if (REC && v == 3) {
        rec.T[c] = S.cell[SP_T * nc + c];
        rec.P[c] = S.cell[SP_P * nc + c];
#pragma unroll
        for (int q = 0; q < DV_NG; ++q) rec.y[q * nc + c] = S.cell[(SP_Y0 + q) * nc + c];
        rec.qstar[c] = S.cell[SP_QS0 * nc + c];
        rec.qstar[nc + c] = S.cell[(SP_QS0 + 1) * nc + c];
    }
    return true;
}

// A warp per row, 32 cells per block.  Bound by latency: a balance is two divisions, three more in a matvec, and a
// thread with a whole cell took them and the wall's resistance in turn with 3.5 warps an SM (16x16x64:
// 5.4 -> 3.7 us, in a matvec 9.4 -> 4.5).  A block stores its rows when all of them have been read, so out may be
// an input that is read by its own rows alone.  The wall rows also read the wall temperatures of other blocks, so
// they go to `wall`: their place in out, or scratch where out holds those temperatures.
constexpr int AS_CELLS = 32;
template <int MODE, bool REC>
__global__ void __launch_bounds__(DV_NB * AS_CELLS) k_assemble(dv_step_params p, Aux aux, Split S, Rec rec, double t,
                                                 const double* __restrict__ y, const double* __restrict__ u,
                                                 const double* __restrict__ sc, const double* __restrict__ f0,
                                                 const double* __restrict__ scal, double gh, double* __restrict__ out,
                                                 double* __restrict__ wall, const double* __restrict__ dargs) {
    pdl_wait();
    const int64_t c = (int64_t)blockIdx.x * AS_CELLS + (threadIdx.x & 31);
    const int v = threadIdx.x >> 5;
    if (dargs) {                  // launched from a CUDA graph: time and step factor live on the device
        t = dargs[0];
        gh = dargs[1];
    }
    int64_t ix = 0;
    double r = 0.0;
    bool has;
    if (MODE == M_MATVEC) {
        const double sig = matvec_sig(scal);
        has = assemble_row<MODE, REC>(p, aux, S, rec, t, LoadDir{y, u, sc, sig}, y, u, sc, f0, sig, gh, c, v, ix, r);
        if (scal[0] == 0.0) r = 0.0;      // matvec of a zero direction is zero
    } else {
        has = assemble_row<MODE, REC>(p, aux, S, rec, t, LoadPlain{y}, y, u, sc, f0, 1.0, gh, c, v, ix, r);
    }
    __syncthreads();
    if (has) (v < DV_NV ? out[ix] : wall[ix - (int64_t)DV_NV * S.nc]) = r;
}

// The FD matvec of the GMRES graph in one cooperative launch: the blocks of k_cprops, k_faces and
// k_assemble (the same per-index code, in 64-thread blocks) taken in grid-stride order, the three phases separated by two bounded grid barriers (bar[0..1]; bit 4 of *err
// on a timeout).  Saves two kernel boundaries per Arnoldi step; results are bit-identical.
__global__ void __launch_bounds__(64) k_matvec_coop(dv_step_params p, Aux aux, Split S, Rec rec,
                                                    const double* __restrict__ z, const double* __restrict__ u,
                                                    const double* __restrict__ sc, const double* __restrict__ f0,
                                                    const double* __restrict__ scal, double* __restrict__ out,
                                                    const double* __restrict__ dargs, unsigned* bar, int* err,
                                                    int64_t nb_props, int64_t nb_faces, int64_t nb_cells) {
    for (int64_t vb = blockIdx.x; vb < nb_props; vb += gridDim.x)
        cprops_block<M_MATVEC>(p, S, z, u, sc, scal, vb);
    grid_sync_bounded(bar, bar + 1, err);
    for (int64_t vb = blockIdx.x; vb < nb_faces; vb += gridDim.x)
        faces_at<false>(p, aux, S, rec, 0.0, scal, dargs, vb * 64 + threadIdx.x);
    grid_sync_bounded(bar, bar + 1, err);
    for (int64_t vb = blockIdx.x; vb < nb_cells; vb += gridDim.x)
        for (int v = 0; v < DV_NB; ++v) {
            const double sig = matvec_sig(scal);
            int64_t ix;
            double r;
            if (assemble_row<M_MATVEC, false>(p, aux, S, rec, dargs ? dargs[0] : 0.0, LoadDir{z, u, sc, sig}, z, u, sc, f0, sig,
                                              dargs ? dargs[1] : 0.0, vb * 64 + threadIdx.x, v, ix, r))
                out[ix] = scal[0] == 0.0 ? 0.0 : r;
        }
}

// ---------------------------------------------------------------- finite-difference Jacobian
// Forward differences of every column (core/jacobian.py:71-86).  With a distance-2
// colouring every row sees exactly one perturbed column of each colour, so a row evaluated with that
// single column perturbed reproduces the coloured evaluation (core/jacobian.py:78-84).  Perturbing one
// unknown of cell n changes the properties of n alone, and through them at most two of the six faces of
// a row cell, so nothing else is evaluated again:
//   k_jac_props  properties and uptake of every cell, unperturbed and with each of its six unknowns
//                perturbed (seven variants)
//   k_jac_faces  the flux of every face, unperturbed and for each unknown of each cell it depends on, and
//                the wall resistance of the outer cells' variants
//   k_jac_rows   per (row cell, neighbour slot, column): the row's six fluxes, the balances, the
//                difference quotients
// Every expression has the operands it has in an evaluation of the whole row (cell_eval), so the entries
// are the same bits.  One thread evaluating its whole row for each of the 63 (slot, column) pairs took
// 441 property evaluations and 378 faces a cell against 7 and 51 here: 155 -> 34 us at 8x8x32 and
// 1270 -> 172 us at 16x16x64 (props 50, faces 63, rows 59; 58 MB of entries, 9 us at the copy bandwidth).
// (Faces evaluated by the row threads, 99 a cell at one 224-thread block per SM: 56 and 374 us.)  What
// bounds it: FP64 latency at 2 instructions per cycle (FP64 pipe 15-32 % busy), divisions first.
constexpr int JAC_VAR = DV_NV + 1;          // unperturbed + the six cell unknowns

// y with one unknown `v` of every cell perturbed by the step of core/jacobian.py:75-76 (v < 0: none)
static __device__ __forceinline__ double fd_step(const dv_step_params& p, double yv, int v) {
    const double h = 1.5e-8 * npmax(fabs(yv), p.typ[v]);
    return (yv + h) - yv;
}
struct LoadVar {
    const dv_step_params& p;
    const double* y;
    int64_t nc;
    int v;
    __device__ __forceinline__ double operator()(int64_t i) const {
        const double x = y[i];
        return (v >= 0 && i >= v * nc && i < (v + 1) * nc) ? x + fd_step(p, x, v) : x;
    }
};

// Scratch of the Jacobian: the split residual's layout with seven variants of the cell properties
// (variant-major); the wall resistances [JAC_VAR][Nth Nz]; the perturbed fluxes: z faces
// [rel 0..3][var][4][nzf], cell kf - 2 + rel of the column perturbed at face kf, then r and theta faces
// [side][var][4][..], the face's lower or upper cell perturbed.
struct JacScratch {
    Split S;
    double *rbed, *zp, *rp, *tp;
};
constexpr int JAC_ZREL = 4;
int64_t jac_scratch_doubles(const dv_step_params& p) {
    const int64_t nc = (int64_t)p.Nr * p.Nth * p.Nz, nzf = (int64_t)p.Nr * p.Nth * (p.Nz + 1);
    const int64_t nrf = (int64_t)(p.Nr - 1) * p.Nth * p.Nz;
    return split_doubles(p) + (JAC_VAR - 1) * SP_NCELL * nc + JAC_VAR * (int64_t)p.Nth * p.Nz +
           4 * DV_NV * (JAC_ZREL * nzf + 2 * nrf + 2 * nc);
}
static JacScratch jac_scratch_of(const dv_step_params& p, double* base) {
    const int64_t nc = (int64_t)p.Nr * p.Nth * p.Nz;
    JacScratch j;
    j.S = split_of(p, base + (JAC_VAR - 1) * SP_NCELL * nc);
    j.S.cell = base;
    j.rbed = j.S.tf + 4 * j.S.ntf;
    j.zp = j.rbed + JAC_VAR * (int64_t)p.Nth * p.Nz;
    j.rp = j.zp + 4 * DV_NV * JAC_ZREL * j.S.nzf;
    j.tp = j.rp + 4 * DV_NV * 2 * j.S.nrf;
    return j;
}
static __device__ __forceinline__ Split jac_variant(const Split& S, int var) {
    Split V = S;
    V.cell = S.cell + (int64_t)var * SP_NCELL * S.nc;
    return V;
}

__global__ void __launch_bounds__(CP_WARPS * 32) k_jac_props(dv_step_params p, Split S, const double* __restrict__ y) {
    const int var = blockIdx.y;
    cprops_split(p, jac_variant(S, var), LoadVar{p, y, S.nc, var - 1}, blockIdx.x);
}

// Flux through the interior z face between cells kL and kL + 1 of a column with cell kp of that column
// taken from V (the perturbed variant) and all others from S.
static __device__ __forceinline__ void jac_zface(const dv_step_params& p, const Split& S, const Split& V, int i,
                                                 int64_t base, int kL, int kp, bool muscl, double N_nom, Flux& F) {
    const int64_t nc = S.nc;
    auto at = [&](int row, int kk) { return ((kk == kp) ? V.cell : S.cell)[row * nc + base + kk]; };
    double s[2][4];
#pragma unroll
    for (int e = 0; e < 2; ++e) {           // the slopes of sp_slope
        const int kk = kL + e;
        s[e][0] = s[e][1] = s[e][2] = s[e][3] = 0.0;
        if (!muscl || kk < 1 || kk > p.Nz - 2) continue;
#pragma unroll
        for (int q = 0; q < DV_NG; ++q) {
            const double x = at(SP_C0 + q, kk);
            s[e][q] = limited_slope(p.limiter, x - at(SP_C0 + q, kk - 1), at(SP_C0 + q, kk + 1) - x);
        }
        const double T = at(SP_T, kk);
        s[e][3] = limited_slope(p.limiter, T - at(SP_T, kk - 1), at(SP_T, kk + 1) - T);
    }
    Cell a, b;
    Props L, R;
    sp_get(kL == kp ? V : S, base + kL, a, L);
    sp_get(kL + 1 == kp ? V : S, base + kL + 1, b, R);
    double uz;
    zface(p, i, L, R, a, b, s[0], s[1], muscl, N_nom, F, &uz);
}

// blockIdx.y: 0..3 z faces with cell kf - 2 + y perturbed; 4, 5 r faces and 6, 7 theta faces with the
// lower / upper cell perturbed; 8 the unperturbed faces (the index space of faces_at), then (variant,
// wall node).  y < 8: a block takes 32 faces, its warps the six unknowns, so a block runs one kind of
// face and its warps share the unperturbed cells through L1.
constexpr int JF_THREADS = DV_NV * 32;
__global__ void __launch_bounds__(JF_THREADS, 3) k_jac_faces(dv_step_params p, Aux aux, JacScratch X, double t,
                                                             int64_t nfaces) {
    const Split& S = X.S;
    const int Nr = p.Nr, Nth = p.Nth, Nz = p.Nz;
    const int64_t nw = (int64_t)Nth * Nz;
    const int kind = blockIdx.y;
    if (kind == 8) {
        int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
        if (g < nfaces) {
            faces_at<false>(p, aux, S, Rec{}, t, nullptr, nullptr, g);
            return;
        }
        g -= nfaces;
        if (g >= JAC_VAR * nw) return;
        const int var = (int)(g / nw);
        Cell s;
        Props o;
        sp_get(jac_variant(S, var), (int64_t)(Nr - 1) * nw + (g - var * nw), s, o);
        X.rbed[g] = wall_R_bed(p, o);
        return;
    }
    const int v = threadIdx.x >> 5;
    const int64_t g = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
    const Split V = jac_variant(S, v + 1);
    Flux F;
    if (kind < JAC_ZREL) {
        if (g >= S.nzf) return;
        const int64_t col = g / (Nz + 1);
        const int kf = (int)(g - col * (Nz + 1)), kp = kf - 2 + kind;
        if (kp < 0 || kp >= Nz) return;
        const int i = (int)(col / Nth);
        if (kf > 0 && kf < Nz) {
            const bool muscl = (Nz >= 3 && p.limiter != DV_LIM_UPWIND);
            jac_zface(p, S, V, i, col * Nz, kf - 1, kp, muscl, aux.n_nom[col], F);
        } else {                            // a column end: depends on its own cell only
            if (kp != (kf == 0 ? 0 : Nz - 1)) return;
            Cell s;
            Props o;
            sp_get(V, col * Nz + kp, s, o);
            double F_in[DV_NG], H_in;
            end_face(p, p.ends[kf == 0 ? 0 : 1], t, i, s, o, aux.feed_flux[col], F_in, H_in, nullptr, 0);
#pragma unroll
            for (int q = 0; q < DV_NG; ++q) F.F[q] = (kf == 0) ? F_in[q] : -F_in[q];
            F.H = (kf == 0) ? H_in : -H_in;
        }
        flux_put(X.zp + (int64_t)(kind * DV_NV + v) * 4 * S.nzf, S.nzf, g, F);
        return;
    }
    const bool theta = kind >= 6, upper = kind & 1;
    if (g >= (theta ? (Nth > 1 ? S.ntf : 0) : (Nr > 1 ? S.nrf : 0))) return;
    int i, j, k;
    cell_ijk(p, g, i, j, k);                // the face's lower cell
    const int jp = (j == Nth - 1) ? 0 : j + 1;
    const int64_t gb = theta ? ((int64_t)i * Nth + jp) * Nz + k : g + nw;
    Cell a, b;
    Props A, B;
    sp_get(upper ? S : V, g, a, A);
    sp_get(upper ? V : S, gb, b, B);
    double u;
    tface(p, A, B, a, b, theta ? p.arc[i] : p.drc[i], theta ? p.Ath[i] : p.Ar[i], F, &u);
    const int64_t nf = theta ? S.ntf : S.nrf;
    flux_put((theta ? X.tp : X.rp) + (int64_t)((upper ? 1 : 0) * DV_NV + v) * 4 * nf, nf, g, F);
}

// A row difference over the step: rows the column does not reach difference to an exact zero, which is
// the quotient (h is positive and finite wherever the unknown is), without the division.
static __device__ __forceinline__ double jac_quot(double d, double h) {
    return (d == 0.0 && h > 0.0 && h < 1e300) ? d : d / h;
}

// Cell (ni, nj, nk) in neighbour slot `slot` of row cell (i, j, k); false where the grid has none, or where
// column variable cv is a wall temperature and that cell has no wall node.
static __device__ __forceinline__ bool jac_neighbour(const dv_step_params& p, int slot, int cv, int i, int j, int k,
                                                     int& ni, int& nj, int& nk) {
    ni = i, nj = j, nk = k;
    bool ok = true;
    switch (slot) {
        case 0: break;
        case 1: nk = k - 1; ok = nk >= 0; break;
        case 2: nk = k + 1; ok = nk < p.Nz; break;
        case 3: nk = k - 2; ok = nk >= 0; break;
        case 4: nk = k + 2; ok = nk < p.Nz; break;
        case 5: ni = i - 1; ok = ni >= 0; break;
        case 6: ni = i + 1; ok = ni < p.Nr; break;
        case 7: ok = p.Nth > 1; nj = (j == 0) ? p.Nth - 1 : j - 1; break;
        default: ok = p.Nth > 1; nj = (j == p.Nth - 1) ? 0 : j + 1; break;
    }
    return cv == DV_NV ? ok && p.wall_on && ni == p.Nr - 1 : ok;
}

// One warp per column variable cv (0..6) of a tile of 32 row cells, blockIdx.y = neighbour slot: the
// seven warps read the same unperturbed fluxes and properties (one of them from L2, the others from L1)
// and each (row, column) plane of J is written coalesced.
template <class TJ>
__global__ void __launch_bounds__(DV_NB * 32, 3) k_jac_rows(dv_step_params p, Aux aux, JacScratch X, double t,
                                                            const double* __restrict__ y,
                                                            const double* __restrict__ f0, TJ* __restrict__ J) {
    const Split& S = X.S;
    const int64_t nc = S.nc;
    const int cv = threadIdx.x >> 5, slot = blockIdx.y;
    const int64_t c = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
    if (c >= nc) return;
    int i, j, k;
    cell_ijk(p, c, i, j, k);
    const int Nr = p.Nr, Nth = p.Nth, Nz = p.Nz;
    const int jm = (j == 0) ? Nth - 1 : j - 1;
    int ni, nj, nk;
    TJ* Jb = J + ((int64_t)slot * DV_NB * DV_NB + cv) * nc + c;         // row stride DV_NB*nc
    if (!jac_neighbour(p, slot, cv, i, j, k, ni, nj, nk)) {
#pragma unroll
        for (int rv = 0; rv < DV_NB; ++rv) Jb[(int64_t)rv * DV_NB * nc] = (TJ)0.0;
        return;
    }
    const int64_t n = ((int64_t)ni * Nth + nj) * Nz + nk;               // the column's cell
    const int64_t col = (cv < DV_NV) ? (int64_t)cv * nc + n : (int64_t)DV_NV * nc + (int64_t)nj * Nz + nk;
    const double h = fd_step(p, y[col], cv);
    const LoadPert ld{y, col, h};
    const bool own = slot == 0, cellv = cv < DV_NV;      // (a wall column changes no flux and no property)
    const int var = (own && cellv) ? cv + 1 : 0;         // variant of the row cell's properties
    const double* cell = S.cell + (int64_t)var * SP_NCELL * nc;
    Props P0;
    P0.T = cell[SP_T * nc + c];                          // (all that the balances read with R_bed given)
    double rate[DV_NA], qstar[DV_NA] = {0.0, 0.0};       // (qstar goes to the records only)
#pragma unroll
    for (int q = 0; q < DV_NA; ++q) rate[q] = cell[(SP_RATE0 + q) * nc + c];
    const int64_t ccol = (int64_t)i * Nth + j;
    // the row's fluxes: the perturbed ones of the faces the column reaches.  z: the own cell and its z
    // neighbours reach both faces (k +- 1 through the own slope), the cells two planes away the nearer one
    auto face = [&](const double* f, const double* fp, bool pert, int which, int64_t nf, int64_t g, Flux& F) {
        flux_get(pert ? fp + (int64_t)(which * DV_NV + cv) * 4 * nf : f, nf, g, F);
    };
    Flux Fzm, Fzp, Frm, Frp, Ftm, Ftp;
    face(S.zf, X.zp, cellv && (own || (k > 0 && slot <= 3)), nk - k + 2, S.nzf, ccol * (Nz + 1) + k, Fzm);
    face(S.zf, X.zp, cellv && (own || (k < Nz - 1 && (slot <= 2 || slot == 4))), nk - k + 1, S.nzf,
         ccol * (Nz + 1) + k + 1, Fzp);
    if (Nr > 1) {
        if (i > 0) face(S.rf, X.rp, cellv && (own || slot == 5), own ? 1 : 0, S.nrf, c - (int64_t)Nth * Nz, Frm);
        if (i < Nr - 1) face(S.rf, X.rp, cellv && (own || slot == 6), own ? 0 : 1, S.nrf, c, Frp);
    }
    if (Nth > 1) {
        face(S.tf, X.tp, cellv && (own || slot == 7), own ? 1 : 0, S.ntf, ((int64_t)i * Nth + jm) * Nz + k, Ftm);
        face(S.tf, X.tp, cellv && (own || slot == 8), own ? 0 : 1, S.ntf, c, Ftp);
    }
    const bool outer_wall = (i == Nr - 1) && p.wall_on;
    const int64_t nw = (int64_t)Nth * Nz;
    const double R_bed = (i == Nr - 1) ? X.rbed[var * nw + (int64_t)j * Nz + k] : 0.0;
    double f[DV_NV], fw = 0.0;
    cell_tail(p, aux, ld, t, i, j, k, P0, rate, qstar, Fzm, Fzp, Frm, Frp, Ftm, Ftp, f, outer_wall ? &fw : nullptr,
              (const Rec*)nullptr, &R_bed);
#pragma unroll
    for (int rv = 0; rv < DV_NV; ++rv) Jb[(int64_t)rv * DV_NB * nc] = (TJ)jac_quot(f[rv] - f0[rv * nc + c], h);
    Jb[(int64_t)DV_NV * DV_NB * nc] =
        (TJ)(outer_wall ? jac_quot(fw - f0[(int64_t)DV_NV * nc + (int64_t)j * Nz + k], h) : 0.0);
}

// The same entries without scratch: a thread evaluates its whole row for one (neighbour slot, column) pair,
// blockIdx.y = slot * 7 + cv.  155 us at 8x8x32, 1270 at 16x16x64 (above: 34, 172): for calls that may not use
// the model's scratch.
template <class TJ>
__global__ void __launch_bounds__(128) k_jac_cells(dv_step_params p, Aux aux, double t, const double* __restrict__ y,
                                                   const double* __restrict__ f0, TJ* __restrict__ J) {
    const int64_t nc = (int64_t)p.Nr * p.Nth * p.Nz;
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    const int slot = blockIdx.y / DV_NB, cv = blockIdx.y % DV_NB;
    int i, j, k, ni, nj, nk;
    cell_ijk(p, c, i, j, k);
    TJ* Jb = J + ((int64_t)slot * DV_NB * DV_NB + cv) * nc + c;         // row stride DV_NB*nc
    if (!jac_neighbour(p, slot, cv, i, j, k, ni, nj, nk)) {
#pragma unroll
        for (int rv = 0; rv < DV_NB; ++rv) Jb[(int64_t)rv * DV_NB * nc] = (TJ)0.0;
        return;
    }
    const int64_t n = ((int64_t)ni * p.Nth + nj) * p.Nz + nk;           // the column's cell
    const int64_t col = (cv < DV_NV) ? (int64_t)cv * nc + n : (int64_t)DV_NV * nc + (int64_t)nj * p.Nz + nk;
    const double h = fd_step(p, y[col], cv);
    const bool outer_wall = (i == p.Nr - 1) && p.wall_on;
    double f[DV_NV], fw = 0.0;
    cell_eval(p, aux, LoadPert{y, col, h}, t, i, j, k, f, outer_wall ? &fw : nullptr, (const Rec*)nullptr);
#pragma unroll
    for (int rv = 0; rv < DV_NV; ++rv) Jb[(int64_t)rv * DV_NB * nc] = (TJ)jac_quot(f[rv] - f0[rv * nc + c], h);
    Jb[(int64_t)DV_NV * DV_NB * nc] =
        (TJ)(outer_wall ? jac_quot(fw - f0[(int64_t)DV_NV * nc + (int64_t)j * p.Nz + k], h) : 0.0);
}

// ---------------------------------------------------------------- residual of a tile in one launch
// The residual of a tile of TL_R x TL_T x TL_Z cells in one block, everything in between in shared memory.
// The block evaluates the transport properties of its cells and of the neighbours their faces need; the
// halo's properties (and the faces between tiles) are evaluated by each of the tiles that need them -- 56
// property evaluations for 16 cells -- so no block waits for another.  The same expressions on the same
// operands as the split residual, so the same bits.
// The work is cut into many small items per phase, so that the warps of a phase run the same short code:
// what bounds a tile is the chain of its phases, and in them the latency of FP64 operations (23 cycles) and
// of fetching code that runs once (the first form, a role per warp and whole faces per thread, spent 28 000
// cycles, half of its instruction fetches missing the SM's cache).  Phases, a barrier between each:
//   load     the six unknowns of the tile's cells, the r / theta / z neighbours and the next z neighbours
//   state    temperature, pressure, concentration of a cell
//   terms    every power of the properties (cell, term); mole fractions and viscosities (cell, gas); the two
//            Toth terms and the water loading of the own cells
//   mix      Wilke's quotients (cell, gas); diffusivities; slopes (cell, variable); loadings and LDF rates
//   flux     velocities, species fluxes and the enthalpy they carry (z, r, theta faces, column ends);
//            stagnant conductivity (cell); the wall's Nusselt number
//   heat     conduction through a face; wall resistance
//   rows     the balances (row, cell)
// 8x8x32 (128 tiles): 12.5 us, against 21.6 us for properties, faces and assembly in three launches.
constexpr int TL_R = 2, TL_T = 2, TL_Z = 4, TL_COL = TL_R * TL_T, TL_OWN = TL_COL * TL_Z, TL_PROP = 56, TL_ALL = 64;
constexpr int TL_WARPS = 14, TL_THREADS = 32 * TL_WARPS;
static_assert(TL_PROP == TL_OWN + 2 * TL_T * TL_Z + 2 * TL_R * TL_Z + 2 * TL_COL && TL_ALL == TL_PROP + 2 * TL_COL,
              "tile, r / theta / z neighbours, next z neighbours");
constexpr int TL_ZF = TL_COL * (TL_Z + 1), TL_RF = (TL_R + 1) * TL_T * TL_Z, TL_TF = (TL_T + 1) * TL_R * TL_Z;
constexpr int TL_F = TL_ZF + TL_RF + TL_TF;            // faces: z (column, face), r (face, 8), theta (face, 8)

// Local cells: the own ones id = (ii TL_T + jj) TL_Z + kk, then the neighbours: 16, 24 below / above in r
// (jj TL_Z + kk), 32, 40 in theta (ii TL_Z + kk), 48, 52 in z and 56, 60 two away in z (ii TL_T + jj).
// Along z of own column cl = ii TL_T + jj, kk = -2 .. TL_Z + 1:
static __device__ __forceinline__ int tl_zid(int cl, int kk) {
    const int own = cl * TL_Z + kk, near = 48 + (kk > 0 ? 4 : 0) + cl, far = 56 + (kk > 0 ? 4 : 0) + cl;
    return (unsigned)kk < TL_Z ? own : (kk == -1 || kk == TL_Z) ? near : far;
}
static __device__ __forceinline__ void tl_cell(int id, int& ii, int& jj, int& kk) {
    const int g = id >> 3, e = id & 7;
    if (id < 16) { ii = id >> 3; jj = (id >> 2) & 1; kk = id & 3; }
    else if (id < 32) { ii = g == 2 ? -1 : TL_R; jj = e >> 2; kk = e & 3; }
    else if (id < 48) { jj = g == 4 ? -1 : TL_T; ii = e >> 2; kk = e & 3; }
    else { ii = (e >> 1) & 1; jj = e & 1; kk = id < 52 ? -1 : id < 56 ? TL_Z : id < 60 ? -2 : TL_Z + 1; }
}

struct TileShared {
    double c[DV_NV][TL_ALL];                               // the unknowns
    double T[TL_ALL], Tp[TL_ALL], P[TL_ALL], Cpos[TL_ALL];
    double y[DV_NG][TL_PROP], mu[DV_NG][TL_PROP], sq[DV_NG][TL_PROP];
    double pw[7][TL_PROP];                                 // powers: gas 0, 1, 2 first terms, gas 2's second, T^1.75, the others
    double mt[DV_NG][TL_PROP], kt[DV_NG][TL_PROP];         // Wilke's quotients
    double Dm[TL_PROP], lam0[TL_PROP];
    double sl[4][TL_COL][TL_Z + 2];                        // slopes of cells -1 .. TL_Z of a column
    double qw[TL_OWN], qt[2][TL_OWN], rate[DV_NA][TL_OWN], qs[DV_NA][TL_OWN], dyn[TL_OWN], Rb[TL_OWN];
    double F[DV_NG + 1][TL_F], lx[TL_F], dist[TL_F], area[TL_F];      // species fluxes, enthalpy; conduction's inputs
    int ida[TL_F], idb[TL_F];                              // cells of the face (-1: no conduction, H is final)
};

template <int MODE, bool REC, class L>
static __device__ __forceinline__ void tile_residual(const dv_step_params& p, const Aux& aux, const Rec& rec, double t,
                                                     const L& ld, const double* __restrict__ y,
                                                     const double* __restrict__ u, const double* __restrict__ sc,
                                                     const double* __restrict__ f0, double sig, double gh,
                                                     double* __restrict__ out, TileShared& X) {
    const int Nr = p.Nr, Nth = p.Nth, Nz = p.Nz;
    const int64_t nc = (int64_t)Nr * Nth * Nz;
    const int tid = threadIdx.x, lane = tid & 31;
    const int w = tid >> 5;
    const int nzt = (Nz + TL_Z - 1) / TL_Z, ntt = (Nth + TL_T - 1) / TL_T;
    const int k0 = (int)(blockIdx.x % nzt) * TL_Z;
    const int rt = blockIdx.x / nzt;
    const int j0 = (rt % ntt) * TL_T, i0 = (rt / ntt) * TL_R;
    // theta wraps (a slot beyond the last sector holds the first one)
    auto sector = [&](int jj) {
        int j = j0 + jj;
        if (j < 0) j += Nth;
        while (j >= Nth) j -= Nth;
        return j;
    };
    auto own = [&](int ii, int jj, int kk) { return i0 + ii < Nr && j0 + jj < Nth && (unsigned)kk < TL_Z && k0 + kk < Nz; };
    auto get = [&](int id, Cell& s) {
#pragma unroll
        for (int q = 0; q < DV_NG; ++q) s.c[q] = X.c[q][id];
        s.q[0] = X.c[3][id];
        s.q[1] = X.c[4][id];
        s.e = X.c[5][id];
    };
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    const bool muscl = (Nz >= 3 && p.limiter != DV_LIM_UPWIND);
    // ---- load
    for (int q = tid; q < DV_NV * TL_ALL; q += TL_THREADS) {
        const int v = q / TL_ALL, id = q - v * TL_ALL;
        int ii, jj, kk;
        tl_cell(id, ii, jj, kk);
        // (a neighbour outside the grid is never read; the nearest cell inside stands in for it)
        const int i = min(max(i0 + ii, 0), Nr - 1), k = min(max(k0 + kk, 0), Nz - 1);
        X.c[v][id] = ld(v * nc + ((int64_t)i * Nth + sector(jj)) * Nz + k);
    }
    __syncthreads();
    // ---- state (as props_state)
    if (tid < TL_ALL) {
        Cell s;
        get(tid, s);
        const double Ctot = s.c[0] + s.c[1] + s.c[2];
        const double T = cell_T(p, s);
        X.T[tid] = T;
        X.P[tid] = Ctot * DV_R * T;
        X.Tp[tid] = npclip(T, 150.0, 1500.0);
        X.Cpos[tid] = npmax(Ctot, 1e-9);
    }
    __syncthreads();
    // ---- terms
    if (w < 9) {                               // powers: slots of X.pw
        for (int it = tid; it < 7 * TL_PROP; it += 9 * 32) {
            const int slot = it / TL_PROP, id = it - slot * TL_PROP;
            const int gas = slot < 3 ? slot : slot == 3 ? 2 : slot == 4 ? -1 : slot - 5, e = slot < 3 ? 0 : 1;
            if (gas >= 0 && e == 1 && p.k_nt[gas] == 1) continue;
            const double Tp = X.Tp[id];
            X.pw[slot][id] = pow(gas >= 0 ? Tp / 300.0 : Tp, gas >= 0 ? p.k_n[gas][e] : 1.75);
        }
    } else if (w == 9) {                       // the two Toth terms of the own cells, side by side
        const int id = lane & 15;
        const bool wet = lane >= 16;
        const double Tp = X.Tp[id], pp = npmax(X.c[0][id] * DV_R * Tp, 0.0);
        double v = nan;
        if (wet ? p.coads == DV_COADS_WADST : !co2_needs_qw(p)) {
            const double qi = wet ? p.wadst_q_inf0 : p.co2_q_inf0, chi = wet ? p.wadst_chi : p.co2_chi;
            const double b0 = wet ? p.wadst_b0 : p.co2_b0, dH = wet ? p.wadst_dH : p.co2_dH0;
            const double tau = wet ? p.wadst_tau0 : p.co2_tau0, al = wet ? p.wadst_alpha : p.co2_alpha;
            v = toth(pp, Tp, qi, chi, b0, dH, tau, al, p.co2_T0);
        }
        X.qt[wet ? 1 : 0][id] = v;
    } else if (w == 10) {                      // water: saturation and GAB
        if (lane < TL_OWN) {
            const double Tp = X.Tp[lane], pw = X.c[1][lane] * DV_R * Tp;
            X.qw[lane] = q_h2o(p, pw, Tp, psat_h2o(Tp));
        }
    } else {                                   // mole fractions, viscosities and their roots
        for (int it = tid - 11 * 32; it < DV_NG * TL_PROP; it += 3 * 32) {
            const int q = it / TL_PROP, id = it - q * TL_PROP;
            const double mu = gas_mu(p, q, X.Tp[id]);
            X.y[q][id] = X.c[q][id] / X.Cpos[id];
            X.sq[q][id] = sqrt(mu);
            X.mu[q][id] = mu;
        }
    }
    __syncthreads();
    // ---- mix
    if (w < 6) {                               // Wilke & Mason-Saxena, gas q of a cell (as wilke_mix)
        if (tid < DV_NG * TL_PROP) {
            const int q = tid / TL_PROP, id = tid - q * TL_PROP;
            const double sqi = X.sq[q][id];
            const double pk = p.k_nt[q] == 1 ? p.k_0[q][0] * X.pw[q][id]
                                             : p.k_w[q][0] * p.k_0[q][0] * X.pw[q][id] +
                                                   p.k_w[q][1] * p.k_0[q][1] * X.pw[q == 2 ? 3 : q + 5][id];
            const double yq = npclip(X.y[q][id], 0.0, 1.0), mu = X.mu[q][id];
            double den = 0.0;
#pragma unroll 1
            for (int j = 0; j < DV_NG; ++j) {
                const double yj = npclip(X.y[j][id], 0.0, 1.0);
                const double t1 = 1.0 + sqi / X.sq[j][id] * p.mass_q[q][j];
                const double m = t1 * t1 / p.wilke_den[q][j];
                den = den + (j == q ? yj : yj * m);
            }
            den = npmax(den, 1e-30);
            X.mt[q][id] = yq * mu / den;
            X.kt[q][id] = yq * pk / den;
        }
    } else if (w < 8) {
        const int id = tid - 6 * 32;
        if (id < TL_PROP) {
            double ycl[DV_NG];
#pragma unroll
            for (int q = 0; q < DV_NG; ++q) ycl[q] = npclip(X.y[q][id], 0.0, 1.0);
            const double tp = 1.43e-7 * X.pw[4][id], Pc = npmax(X.P[id], 1.0);
            X.Dm[id] = blanc_Dm(ycl, fuller_of(p, 0, tp, Pc), fuller_of(p, 1, tp, Pc));
        }
    } else if (w < 11) {                       // slopes of the cells next to the tile's z faces (as sp_slope)
        const int it = tid - 8 * 32, v = it / (TL_COL * (TL_Z + 2)), r = it - v * (TL_COL * (TL_Z + 2));
        const int cl = r / (TL_Z + 2), kk = r - cl * (TL_Z + 2) - 1, k = k0 + kk;
        const double* a = v < DV_NG ? X.c[v] : X.T;
        double s = 0.0;
        if (muscl && k >= 1 && k <= Nz - 2) {
            const double x = a[tl_zid(cl, kk)], dm = x - a[tl_zid(cl, kk - 1)], dp = a[tl_zid(cl, kk + 1)] - x;
            s = limited_slope(p.limiter, dm, dp);
        }
        X.sl[v][cl][kk + 1] = s;
    } else if (w == 11 && lane < TL_OWN) {     // loadings and LDF rates
        Cell s;
        get(lane, s);
        const double Tp = X.Tp[lane], pp = npmax(s.c[0] * DV_R * Tp, 0.0), qw_eq = X.qw[lane];
        const double dry = X.qt[0][lane], wet = X.qt[1][lane];
        double rate[DV_NA], qstar[DV_NA];
        qstar[0] = q_co2_raw(p, pp, Tp, p.basis_state ? s.q[1] : qw_eq, dry, wet) * (pp / (pp + p.p_reg));
        qstar[1] = qw_eq;
        ldf_rates(p, s, Tp, qstar, rate);
#pragma unroll
        for (int q = 0; q < DV_NA; ++q) {
            X.rate[q][lane] = rate[q];
            X.qs[q][lane] = qstar[q];
        }
    }
    __syncthreads();
    static_assert(4 * TL_COL * (TL_Z + 2) == 3 * 32, "slopes fill three warps");
    // ---- flux
    auto props = [&](int id, Cell& s, Props& o) {          // all but lam0
        double ycl[DV_NG];
        o.mu = o.kg = 0.0;
#pragma unroll
        for (int q = 0; q < DV_NG; ++q) {
            s.c[q] = X.c[q][id];
            o.y[q] = X.y[q][id];
            ycl[q] = npclip(o.y[q], 0.0, 1.0);
            o.mu = o.mu + X.mt[q][id];
            o.kg = o.kg + X.kt[q][id];
        }
        s.q[0] = s.q[1] = s.e = 0.0;
        o.T = X.T[id];
        o.P = X.P[id];
        o.Tp = 0.0;
        o.Cpos = X.Cpos[id];
        o.rho = o.Cpos * wsum3(p.M, ycl);
        o.cpm = wsum3(p.cpg, ycl);
        o.Dm = X.Dm[id];
        o.lam0 = 0.0;
    };
    auto put = [&](int f, const FluxPart& F, int a, int b, double dist, double area) {
#pragma unroll
        for (int q = 0; q < DV_NG; ++q) X.F[q][f] = F.F[q];
        X.F[DV_NG][f] = F.He;
        X.lx[f] = F.lx;
        X.ida[f] = a;
        X.idb[f] = b;
        X.dist[f] = dist;
        X.area[f] = area;
    };
    if (w == 0) {                              // z faces between k0 + kf - 1 and k0 + kf
        const int cl = lane / (TL_Z + 1), kf = lane - cl * (TL_Z + 1), ii = cl >> 1, jj = cl & 1, K = k0 + kf;
        if (lane < TL_ZF && i0 + ii < Nr && j0 + jj < Nth && K > 0 && K < Nz) {
            const int a = tl_zid(cl, kf - 1), b = tl_zid(cl, kf);
            Cell ca, cb;
            Props Lp, Rp;
            props(a, ca, Lp);
            props(b, cb, Rp);
            double sL[4], sR[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                sL[v] = X.sl[v][cl][kf];
                sR[v] = X.sl[v][cl][kf + 1];
            }
            const int64_t col = (int64_t)(i0 + ii) * Nth + j0 + jj;
            const double nn = aux.n_nom[col];
            FluxPart F;
            double uz;
            zface_part(p, i0 + ii, Lp, Rp, ca, cb, sL, sR, muscl, nn, F, &uz);
            put(lane, F, a, b, p.dz, p.Az[i0 + ii]);
            if (REC && kf > 0) rec.uz[col * (Nz - 1) + K - 1] = uz;      // (the tile of the lower cell)
        }
    } else if (w < 3) {                        // r faces between rings ii - 1, ii; theta faces between jj - 1, jj (periodic)
        const bool th = w == 2;
        const int n = lane >> 3, e = lane & 7, kk = e & 3;           // n: the face along r (theta)
        const int ii = th ? e >> 2 : n, jj = th ? n : e >> 2, i = i0 + ii, j = j0 + jj;
        const bool ok = lane < 24 && k0 + kk < Nz && i < Nr && (th ? Nth > 1 && j <= Nth : j < Nth && i > 0);
        if (ok) {
            const int a = th ? (n == 0 ? 32 + e : ii * 8 + (n - 1) * 4 + kk) : (n == 0 ? 16 + e : (n - 1) * 8 + e);
            const int b = th ? (n == TL_T ? 40 + e : ii * 8 + n * 4 + kk) : (n == TL_R ? 24 + e : n * 8 + e);
            Cell ca, cb;
            Props A, B;
            props(a, ca, A);
            props(b, cb, B);
            const double dist = th ? p.arc[i] : p.drc[i - 1], area = th ? p.Ath[i] : p.Ar[i - 1];
            FluxPart F;
            double ut;
            tface_part(p, A, B, ca, cb, dist, area, F, &ut);
            put(TL_ZF + (th ? TL_RF : 0) + lane, F, a, b, dist, area);
            if (REC && n > 0) {       // (the tile of the lower cell)
                if (th) rec.uth[((int64_t)i * Nth + j - 1) * Nz + k0 + kk] = ut;
                else rec.ur[((int64_t)(i - 1) * Nth + j) * Nz + k0 + kk] = ut;
            }
        }
    } else if (w == 3) {                       // the column ends
        const int e = lane >> 2, cl = lane & 3, ii = cl >> 1, jj = cl & 1, kk = e == 0 ? 0 : Nz - 1 - k0;
        if (lane < 2 * TL_COL && own(ii, jj, kk) && (e == 1 || k0 == 0)) {
            const int64_t col = (int64_t)(i0 + ii) * Nth + j0 + jj;
            Cell s;
            Props o;
            props(cl * TL_Z + kk, s, o);
            double F_in[DV_NG], H_in;
            const double ff = aux.feed_flux[col];
            end_face(p, p.ends[e], t, i0 + ii, s, o, ff, F_in, H_in,
                     REC ? rec.bnd + (int64_t)e * BR_N * Nr * Nth + col : nullptr, (int64_t)Nr * Nth);
            FluxPart F;                        // stored as the +z flux through the face
#pragma unroll
            for (int q = 0; q < DV_NG; ++q) F.F[q] = (e == 0) ? F_in[q] : -F_in[q];
            F.He = (e == 0) ? H_in : -H_in;
            F.lx = 0.0;
            put(cl * (TL_Z + 1) + (e == 0 ? 0 : kk + 1), F, -1, -1, 1.0, 0.0);
        }
    } else if (w < 6) {                        // stagnant conductivity
        const int id = tid - 4 * 32;
        if (id < TL_PROP) {
            double kg = 0.0;
#pragma unroll
            for (int q = 0; q < DV_NG; ++q) kg = kg + X.kt[q][id];
            X.lam0[id] = stagnant(p, kg);
        }
    } else if (w == 6) {                       // wall: the flow part of the Nusselt number
        if (lane < TL_OWN && i0 + (lane >> 3) == Nr - 1) {
            Cell s;
            Props o;
            props(lane, s, o);
            X.dyn[lane] = wall_dyn(p, o);
        }
    }
    __syncthreads();
    // ---- heat
    if (w < 3) {
        // (the faces put above: the same conditions)
        bool ok = false;
        int f = 0;
        if (w == 0) {
            const int cl = lane / (TL_Z + 1), K = k0 + lane - cl * (TL_Z + 1);
            ok = lane < TL_ZF && i0 + (cl >> 1) < Nr && j0 + (cl & 1) < Nth && K > 0 && K < Nz;
            f = lane;
        } else {
            const bool th = w == 2;
            const int n = lane >> 3, e = lane & 7, i = i0 + (th ? e >> 2 : n), j = j0 + (th ? n : e >> 2);
            ok = lane < 24 && k0 + (e & 3) < Nz && i < Nr && (th ? Nth > 1 && j <= Nth : j < Nth && i > 0);
            f = TL_ZF + (th ? TL_RF : 0) + lane;
        }
        if (ok) {
            const int a = X.ida[f], b = X.idb[f];
            const double He = X.F[DV_NG][f];
            X.F[DV_NG][f] = face_H(He, X.lx[f], X.lam0[a], X.lam0[b], X.T[a], X.T[b], X.dist[f], X.area[f]);
        }
    } else if (w == 3) {
        if (lane < TL_OWN && i0 + (lane >> 3) == Nr - 1) {
            Cell s;
            Props o;
            props(lane, s, o);
            o.lam0 = X.lam0[lane];
            const double dyn = X.dyn[lane];
            X.Rb[lane] = wall_R_rest(p, o, dyn);
        }
    }
    __syncthreads();
    // ---- rows: (row, own cell)
    if (tid < DV_NB * TL_OWN) {
        const int v = tid >> 4, id = tid & 15, ii = id >> 3, jj = (id >> 2) & 1, kk = id & 3;
        const int i = i0 + ii, j = j0 + jj, k = k0 + kk;
        if (own(ii, jj, kk) && (v < DV_NV || (i == Nr - 1 && p.wall_on))) {
            const int64_t c0 = ((int64_t)i * Nth + j) * Nz + k;
            const int64_t ix = v < DV_NV ? v * nc + c0 : (int64_t)DV_NV * nc + (int64_t)j * Nz + k;
            const int cl = ii * TL_T + jj, zf = cl * (TL_Z + 1) + kk, rf = TL_ZF + ii * 8 + jj * TL_Z + kk;
            const int tf = TL_ZF + TL_RF + jj * 8 + ii * TL_Z + kk;
            const double T = X.T[id], Rb = X.Rb[id];
            double r = 0.0;
            const double yo = MODE == M_STAGE ? y[ix] : 0.0, uo = MODE != M_RHS ? u[ix] : 0.0;
            const double so = MODE == M_MATVEC ? sc[ix] : 0.0, fo = MODE == M_MATVEC ? f0[ix] : 0.0;
            double f;
            if (v == 3 || v == 4) {
                f = X.rate[v - 3][id];
            } else if (v == DV_NV) {
                wall_terms(p, aux, ld, jacket_T(p, t), j, k, T, Rb, &f);
            } else {
                const double* F = X.F[v < DV_NG ? v : DV_NG];
                const double div = face_div(p, i, F[zf], F[zf + 1], F[rf], F[rf + 8], F[tf], F[tf + 8]);
                f = v < DV_NG ? row_mass(p, i, div, (v < DV_NA) ? X.rate[v][id] : 0.0)
                              : row_energy(p, aux, ld, t, i, j, k, T, Rb, div, nullptr, REC ? &rec : nullptr);
            }
            if (MODE == M_RHS) r = f;
            else if (MODE == M_STAGE) r = yo - gh * f - uo;
            else r = (uo * so - (gh * (f - fo) / sig)) / so;
            out[ix] = r;
            if (REC && v == 3) {
                rec.T[c0] = T;
                rec.P[c0] = X.P[id];
#pragma unroll
                for (int q = 0; q < DV_NG; ++q) rec.y[q * nc + c0] = X.y[q][id];
                rec.qstar[c0] = X.qs[0][id];
                rec.qstar[nc + c0] = X.qs[1][id];
            }
        }
    }
}

template <int MODE, bool REC>
__global__ void __launch_bounds__(TL_THREADS, 1) k_tile(dv_step_params p, Aux aux, Rec rec, double t,
                                                     const double* __restrict__ y, const double* __restrict__ u,
                                                     const double* __restrict__ sc, const double* __restrict__ f0,
                                                     const double* __restrict__ scal, double gh,
                                                     double* __restrict__ out, const double* __restrict__ dargs) {
    __shared__ TileShared X;
    pdl_wait();                   // (launched programmatically inside the GMRES graph)
    if (dargs) {                  // launched from a CUDA graph: time and step factor live on the device
        t = dargs[0];
        gh = dargs[1];
    }
    if (MODE == M_MATVEC) {
        if (scal[0] == 0.0) {     // matvec of a zero direction is zero
            const int64_t n = (int64_t)DV_NV * p.Nr * p.Nth * p.Nz + (p.wall_on ? (int64_t)p.Nth * p.Nz : 0);
            for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
                out[i] = 0.0;
            return;
        }
        const double sig = matvec_sig(scal);
        tile_residual<MODE, REC>(p, aux, rec, t, LoadDir{y, u, sc, sig}, y, u, sc, f0, sig, gh, out, X);
    } else {
        tile_residual<MODE, REC>(p, aux, rec, t, LoadPlain{y}, y, u, sc, f0, 1.0, gh, out, X);
    }
}

static int64_t tile_blocks(const dv_step_params& p) {
    return (int64_t)((p.Nr + TL_R - 1) / TL_R) * ((p.Nth + TL_T - 1) / TL_T) * ((p.Nz + TL_Z - 1) / TL_Z);
}

static Aux aux_of(const dv_model* m) { return Aux{m->aux.feed_flux, m->aux.n_nom, m->aux.cov}; }

static unsigned nblk(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

// Tiles up to two waves of blocks (one block per SM): up to there a tile launch is the shorter path --
// residual of 8x8x12 (48 tiles) 21.5 -> 10.2 us, 8x8x32 (128) 21.6 -> 12.5, 12x8x32 (192) 22.9 -> 18.6, 9x9x33
// (225) 22.7 -> 19.9 -- and beyond it the halo work repeats: 12x12x48 (432) 25.8 against 30.0, 16x16x64
// (1024) 25.9 against 60.7.
static bool use_tiles(const dv_step_params& p) { return tile_blocks(p) <= 296; }

// The residual: tiles, or properties, faces and assembly (one or three launches counted under `kind`).
template <int MODE, bool REC>
static int split_residual(dv_model* m, const Rec& rec, double t, const double* y, const double* u, const double* sc,
                          const double* f0, const double* scal, double gh, double* out, cudaStream_t s, int kind) {
    const dv_step_params& p = m->p;
    // out is one of the inputs that LoadPlain / LoadDir read: a tile reads its neighbours' (the right-hand side of
    // a stage residual, M_STAGE's u, is read by its own rows alone, but keeps the split path it has always taken)
    const bool over = out == y || (MODE == M_MATVEC && (out == u || out == sc));
    if (use_tiles(p) && !over && out != u) {
        DV_LAUNCH(kind, s, k_tile<MODE, REC><<<(unsigned)tile_blocks(p), TL_THREADS, 0, s>>>(p, aux_of(m), rec, t, y, u, sc, f0,
                                                                                            scal, gh, out, nullptr));
        m->nfev += 1;
        DV_CUDA(cudaGetLastError());
        return DV_OK;
    }
    const Split S = split_of(p, m->d_split);
    double* const wall = out + (int64_t)DV_NV * m->nc;
    const int64_t ncol = (int64_t)p.Nr * p.Nth;
    const int64_t nfaces = ncol * (p.Nz - 1) + (p.Nr > 1 ? S.nrf : 0) + (p.Nth > 1 ? S.ntf : 0) + 2 * ncol + p.Nth * p.Nz;
    DV_LAUNCH(kind, s, k_cprops<MODE><<<nblk(m->nc, 32), CP_WARPS * 32, 0, s>>>(p, S, y, u, sc, scal));
    DV_LAUNCH(kind, s, k_faces<REC><<<nblk(nfaces, 64), 64, 0, s>>>(p, aux_of(m), S, rec, t,
                                                                  MODE == M_MATVEC ? scal : nullptr, nullptr));
    DV_LAUNCH(kind, s, k_assemble<MODE, REC><<<nblk(m->nc, AS_CELLS), DV_NB * AS_CELLS, 0, s>>>(p, aux_of(m), S, rec, t, y, u, sc, f0,
                                                                           scal, gh, out, over ? S.wall : wall, nullptr));
    if (over && p.wall_on)
        DV_CUDA(cudaMemcpyAsync(wall, S.wall, sizeof(double) * p.Nth * p.Nz, cudaMemcpyDeviceToDevice, s));
    m->nfev += 1;
    DV_CUDA(cudaGetLastError());
    return DV_OK;
}

int launch_rhs(dv_model* m, double t, const double* y, double* f, double* acc, cudaStream_t s) {
    Rec rec = make_rec(m->rl, m->d_rec);
    if (acc) {
        int rc = split_residual<M_RHS, true>(m, rec, t, y, nullptr, nullptr, nullptr, nullptr, 0.0, f, s,
                                             dv::K_RESIDUAL);
        if (rc != DV_OK) return rc;
        DV_LAUNCH(dv::K_RESIDUAL, s, k_accumulators<<<1, 256, 0, s>>>(m->p, rec.bnd, rec.Qj, rec.Qa, rec.Qw, rec.Qhx, acc));
        DV_CUDA(cudaGetLastError());
        return DV_OK;
    }
    return split_residual<M_RHS, false>(m, rec, t, y, nullptr, nullptr, nullptr, nullptr, 0.0, f, s, dv::K_RESIDUAL);
}

int launch_stage_residual(dv_model* m, double t, const double* y, double gamma_h, const double* rhs_known,
                          double* R, cudaStream_t s) {
    Rec rec = make_rec(m->rl, m->d_rec);
    return split_residual<M_STAGE, false>(m, rec, t, y, rhs_known, nullptr, nullptr, nullptr, gamma_h, R, s,
                                          dv::K_RESIDUAL);
}

int launch_diag(dv_model* m, double t, const double* y, double* diag, cudaStream_t s) {
    Rec rec = make_rec(m->rl, diag);      // f is discarded into the model's record scratch
    return split_residual<M_RHS, true>(m, rec, t, y, nullptr, nullptr, nullptr, nullptr, 0.0, m->d_rec, s,
                                       dv::K_RESIDUAL);
}

int launch_matvec(dv_model* m, double t, const double* z, const double* u, const double* sc, const double* f0,
                  double dh, const double* scal, double* out, cudaStream_t s) {
    Rec rec = make_rec(m->rl, m->d_rec);
    return split_residual<M_MATVEC, false>(m, rec, t, z, u, sc, f0, scal, dh, out, s, dv::K_MATVEC);
}

// Launch with programmatic stream serialisation (the kernel must begin with pdl_wait()).
template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl(void (*kern)(KArgs...), unsigned grid, unsigned block, cudaStream_t s, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

// co-resident 64-thread blocks of k_matvec_coop (-1: not asked yet; 0: refused)
static int g_matvec_coop_cap = -1;

// DVTSA_MATVEC_COOP=1 runs the FD matvec inside the GMRES graph as one cooperative launch (read
// once; off by default: bit-identical, but measured 5 % slower on the 8x8x32 heating window, the
// two grid barriers costing more than the two kernel boundaries they replace).
static bool matvec_coop_enabled() {
    static int v = -1;
    if (v < 0) {
        const char* e = getenv("DVTSA_MATVEC_COOP");
        v = (e && e[0] == '1') ? 1 : 0;
    }
    return v == 1;
}

int matvec_capture_kernels(const dv_model* m) {
    return ((g_matvec_coop_cap > 0 && matvec_coop_enabled()) || use_tiles(m->p)) ? 1 : 3;
}

int matvec_capture(dv_model* m, const double* dargs, const double* z, const double* u, const double* sc,
                   const double* f0, const double* scal, double* out, cudaStream_t s, unsigned* bar) {
    const dv_step_params& p = m->p;
    const Split S = split_of(p, m->d_split);
    const Rec rec = make_rec(m->rl, m->d_rec);
    const int64_t ncol = (int64_t)p.Nr * p.Nth;
    const int64_t nfaces = ncol * (p.Nz - 1) + (p.Nr > 1 ? S.nrf : 0) + (p.Nth > 1 ? S.ntf : 0) + 2 * ncol + p.Nth * p.Nz;
    int& coop_cap = g_matvec_coop_cap;
    if (coop_cap < 0) {
        int dev = 0, nsm = 0, bps = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_matvec_coop, 64, 0) != cudaSuccess) bps = 0;
        coop_cap = bps * nsm;
        cudaGetLastError();
    }
    if (bar && coop_cap > 0 && matvec_coop_enabled()) {
        const int64_t nbp = nblk(m->nc, 32), nbf = nblk(nfaces, 64), nbc = nblk(m->nc, 64);
        const int64_t want = std::max(nbp, std::max(nbf, nbc));
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)std::min<int64_t>(want, coop_cap));
        cfg.blockDim = dim3(64);
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        if (cudaLaunchKernelEx(&cfg, k_matvec_coop, p, aux_of(m), S, rec, z, u, sc, f0, scal, out, dargs, bar,
                               m->d_err, nbp, nbf, nbc) == cudaSuccess)
            return DV_OK;
        cudaGetLastError();                   // a driver that refuses the cooperative node: three kernels
        coop_cap = 0;
    }
    if (use_tiles(p)) {
        if (pdl_enabled())
            DV_CUDA(launch_pdl(k_tile<M_MATVEC, false>, (unsigned)tile_blocks(p), TL_THREADS, s, p, aux_of(m), rec, 0.0, z, u,
                               sc, f0, scal, 0.0, out, dargs));
        else
            k_tile<M_MATVEC, false><<<(unsigned)tile_blocks(p), TL_THREADS, 0, s>>>(p, aux_of(m), rec, 0.0, z, u, sc, f0, scal,
                                                                                 0.0, out, dargs);
        DV_CUDA(cudaGetLastError());
        return DV_OK;
    }
    if (pdl_enabled()) {       // each kernel may start while its predecessor drains (pdl_wait in the kernel)
        DV_CUDA(launch_pdl(k_cprops<M_MATVEC>, nblk(m->nc, 32), CP_WARPS * 32, s, p, S, z, u, sc, scal));
        DV_CUDA(launch_pdl(k_faces<false>, nblk(nfaces, 64), 64, s, p, aux_of(m), S, rec, 0.0, scal, dargs));
        DV_CUDA(launch_pdl(k_assemble<M_MATVEC, false>, nblk(m->nc, AS_CELLS), DV_NB * AS_CELLS, s, p, aux_of(m), S, rec, 0.0, z, u, sc, f0,
                           scal, 0.0, out, out + (int64_t)DV_NV * m->nc, dargs));
        return DV_OK;
    }
    k_cprops<M_MATVEC><<<nblk(m->nc, 32), CP_WARPS * 32, 0, s>>>(p, S, z, u, sc, scal);
    k_faces<false><<<nblk(nfaces, 64), 64, 0, s>>>(p, aux_of(m), S, rec, 0.0, scal, dargs);
    k_assemble<M_MATVEC, false><<<nblk(m->nc, AS_CELLS), DV_NB * AS_CELLS, 0, s>>>(p, aux_of(m), S, rec, 0.0, z, u, sc, f0, scal, 0.0,
                                                             out, out + (int64_t)DV_NV * m->nc, dargs);
    DV_CUDA(cudaGetLastError());
    return DV_OK;
}

template <class TJ>
static int fd_jacobian(dv_model* m, double t, const double* y, const double* f0, TJ* J, cudaStream_t s) {
    const dv_step_params& p = m->p;
    // The scratch belongs to one Jacobian at a time: a call on another stream waits for the last one (jac_ev).  A
    // captured call cannot: its graph runs later, and nothing orders it against other calls.  So it takes the
    // form without scratch, as does a model whose scratch did not fit on the device.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    DV_CUDA(cudaStreamIsCapturing(s, &cap));
    if (cap != cudaStreamCaptureStatusNone || !m->d_jac) {
        DV_LAUNCH(dv::K_FDJAC, s, k_jac_cells<TJ><<<dim3(nblk(m->nc, 128), DV_NSLOT * DV_NB), 128, 0, s>>>(p, aux_of(m), t, y,
                                                                                                         f0, J));
        DV_CUDA(cudaGetLastError());
        return DV_OK;
    }
    const JacScratch X = jac_scratch_of(p, m->d_jac);
    const Split& S = X.S;
    const int64_t ncol = (int64_t)p.Nr * p.Nth, nw = (int64_t)p.Nth * p.Nz;
    const int64_t nfaces = ncol * (p.Nz - 1) + (p.Nr > 1 ? S.nrf : 0) + (p.Nth > 1 ? S.ntf : 0) + 2 * ncol;
    if (m->jac_used) DV_CUDA(cudaStreamWaitEvent(s, m->jac_ev, 0));
    DV_LAUNCH(dv::K_FDJAC, s, k_jac_props<<<dim3(nblk(m->nc, 32), JAC_VAR), CP_WARPS * 32, 0, s>>>(p, S, y));
    // x covers the z faces (the most of the perturbed kinds) and the unperturbed index space
    const unsigned gx = std::max(nblk(S.nzf, 32), nblk(nfaces + JAC_VAR * nw, JF_THREADS));
    DV_LAUNCH(dv::K_FDJAC, s, k_jac_faces<<<dim3(gx, 9), JF_THREADS, 0, s>>>(p, aux_of(m), X, t, nfaces));
    DV_LAUNCH(dv::K_FDJAC, s, k_jac_rows<TJ><<<dim3(nblk(m->nc, 32), DV_NSLOT), DV_NB * 32, 0, s>>>(p, aux_of(m), X, t, y,
                                                                                                 f0, J));
    DV_CUDA(cudaGetLastError());
    DV_CUDA(cudaEventRecord(m->jac_ev, s));
    m->jac_used = 1;
    return DV_OK;
}

int launch_fd_jacobian(dv_model* m, double t, const double* y, const double* f0, double* J, cudaStream_t s) {
    return fd_jacobian<double>(m, t, y, f0, J, s);
}

int launch_fd_jacobian32(dv_model* m, double t, const double* y, const double* f0, float* J, cudaStream_t s) {
    return fd_jacobian<float>(m, t, y, f0, J, s);
}

// ---------------------------------------------------------------- outlet record
// The summary of one accepted step that the step runner records (the columns of the outlet time
// series, steps/_runner.py:50-84,104-121), reduced on the device from the diagnostics record so that
// only DV_OUTLET_N doubles leave the GPU per step.  Per end: the net outflow (minus the summed inflow
// records), the area-weighted face pressure, and the composition and temperature of the gas leaving
// (weighted by each face's outflow, over the faces with outflow; valve ends use their outflow part)
// or, with no outflow, the area-weighted layer averages.  Fixed-order block reductions.
constexpr int OUTLET_THREADS = 256;

__device__ double outlet_sum(double v, double* red) {
    const int tid = threadIdx.x;
    red[tid] = v;
    __syncthreads();
    for (int st = OUTLET_THREADS / 2; st > 0; st >>= 1) {
        if (tid < st) red[tid] += red[tid + st];
        __syncthreads();
    }
    const double r = red[0];
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(OUTLET_THREADS) k_outlet(dv_step_params p, Rec rec, const double* __restrict__ y,
                                                           double c_feed, double* __restrict__ out) {
    __shared__ double red[OUTLET_THREADS];
    const int tid = threadIdx.x;
    const int64_t nc = (int64_t)p.Nr * p.Nth * p.Nz;
    const int nf = p.Nr * p.Nth;
    double a[5] = {0.0, 0.0, 0.0, 0.0, 0.0};          // V T, V P, V q_CO2, V q_H2O, V
    for (int64_t c = tid; c < nc; c += OUTLET_THREADS) {
        const double V = p.V[c / ((int64_t)p.Nth * p.Nz)];
        a[0] += rec.T[c] * V;
        a[1] += rec.P[c] * V;
        a[2] += y[3 * nc + c] * V;
        a[3] += y[4 * nc + c] * V;
        a[4] += V;
    }
    double bed[5];
    for (int q = 0; q < 5; ++q) bed[q] = outlet_sum(a[q], red);
    if (tid == 0) {
        out[24] = bed[0] / bed[4];
        out[25] = bed[1] / bed[4];
        out[26] = bed[2] / bed[4];
        out[27] = bed[3] / bed[4];
    }
    for (int e = 0; e < 2; ++e) {
        const int klay = e == 0 ? 0 : p.Nz - 1;
        const double* b = rec.bnd + (int64_t)e * BR_N * nf;
        const bool part = p.ends[e].kind == DV_END_VALVE;
        // A, P A, net outflow, leaving flow, leaving species (3), T leaving flow, y A (3), T A,
        // net outflow and its CO2 over the faces with net outflow, loading q_CO2 of the layer
        double sm[15];
        for (int q = 0; q < 15; ++q) sm[q] = 0.0;
        for (int f = tid; f < nf; f += OUTLET_THREADS) {
            const double A = p.Az[f / p.Nth];
            const int64_t cell = (int64_t)f * p.Nz + klay;
            double Fo[DV_NG], tot = 0.0, tot2 = 0.0;
            for (int k = 0; k < DV_NG; ++k) tot += -b[(BR_FIN + k) * nf + f];
            for (int k = 0; k < DV_NG; ++k) {
                Fo[k] = part ? b[(BR_FOUTP + k) * nf + f] : -b[(BR_FIN + k) * nf + f];
                tot2 += Fo[k];
            }
            const bool leaving = tot2 > 0.0;
            const double Tl = rec.T[cell];
            sm[0] += A;
            sm[1] += b[BR_PFACE * nf + f] * A;
            sm[2] += tot;
            if (leaving) {
                sm[3] += tot2;
                for (int k = 0; k < DV_NG; ++k) sm[4 + k] += Fo[k];
                sm[7] += Tl * tot2;
            }
            for (int k = 0; k < DV_NG; ++k) sm[8 + k] += rec.y[(int64_t)k * nc + cell] * A;
            sm[11] += Tl * A;
            if (tot > 0.0) {
                sm[12] += tot;
                sm[13] += -b[BR_FIN * nf + f];
            }
            sm[14] += y[(int64_t)DV_NG * nc + cell];
        }
        double r[15];
        for (int q = 0; q < 15; ++q) r[q] = outlet_sum(sm[q], red);
        if (tid == 0) {
            double* o = out + 12 * e;
            const double Pf = r[1] / r[0];
            double ys[DV_NG], Tg;
            if (r[3] > 1e-14) {
                for (int k = 0; k < DV_NG; ++k) ys[k] = r[4 + k] / r[3];
                Tg = r[7] / r[3];
            } else {
                for (int k = 0; k < DV_NG; ++k) ys[k] = r[8 + k] / r[0];
                Tg = r[11] / r[0];
            }
            o[0] = r[2];
            o[1] = Pf;
            o[2] = Tg;
            for (int k = 0; k < DV_NG; ++k) o[3 + k] = ys[k];
            const double cco2 = ys[0] * Pf / (DV_R * Tg);
            o[6] = cco2;
            o[7] = c_feed > 0.0 ? cco2 / c_feed : __longlong_as_double(0x7ff8000000000000LL);
            o[8] = r[3];
            o[9] = r[12] > 0.0 ? r[13] / r[12] : 0.0;
            o[10] = r[14] / nf;
            o[11] = 0.0;
        }
    }
    if (tid == 0)
        for (int q = 28; q < DV_OUTLET_N; ++q) out[q] = 0.0;
}

int launch_outlet(dv_model* m, double t, const double* y, double c_feed, double* row, cudaStream_t s) {
    DV_TRY(launch_diag(m, t, y, m->d_diag, s));
    Rec rec = make_rec(m->rl, m->d_diag);
    DV_LAUNCH(dv::K_RESIDUAL, s, k_outlet<<<1, OUTLET_THREADS, 0, s>>>(m->p, rec, y, c_feed, row));
    return launch_ok("k_outlet");
}

}  // namespace dv

// ---------------------------------------------------------------- allocation-free residual + accumulators
// dv_rhs_acc_noalloc evaluates f = dy/dt and the accumulator rates without a dv_model, so without
// any device allocation.  It exists for callers that may not allocate device memory once they are
// running: a plant controller or state estimator that reserves its device memory at start-up and
// forbids allocation inside its loop, or a host framework whose allocator owns the device and
// does not let plugins call cudaMalloc.  dv_model_create allocates the model's workspaces, so
// those callers cannot use dv_rhs.  The face and wall records that dv_rhs keeps in the model live
// here in one file-scope device array instead, shared by every call on the device.

namespace {

constexpr size_t kNoAllocScratchBytes = 2u << 20;    // 2 MiB per device, held until process exit
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) double g_noalloc_scratch[kNoAllocScratchBytes / sizeof(double)];

// Device address of g_noalloc_scratch per device, looked up once with that device current (in
// host code the symbol names a host-side shadow, never a device address).
static double* g_noalloc_ptr[kNoAllocMaxDevices] = {};
static std::mutex g_noalloc_mu;

}  // namespace

extern "C" int dv_rhs_acc_noalloc(const dv_step_params* p, const double* feed_flux, const double* n_nom,
                                  const double* coverage, double t, const double* y, double* f, double* acc,
                                  void* stream) {
    using namespace dv;
    if (!p || !feed_flux || !n_nom || !coverage || !y || !f || !acc) {
        set_error("dv_rhs_acc_noalloc: null argument");
        return DV_ERR_ARG;
    }
    if (p->Nr < 1 || p->Nth < 1 || p->Nz < 1 || p->Nr > DV_MAX_NR) {
        set_error("dv_rhs_acc_noalloc: bad grid size");
        return DV_ERR_ARG;
    }
    const RecLayout rl = rec_layout(*p);
    const size_t need = sizeof(double) * (size_t)rl.total;
    if (need > kNoAllocScratchBytes) {
        set_error("dv_rhs_acc_noalloc: the grid needs " + std::to_string(need) + " bytes of record scratch; the "
                  "static scratch holds " + std::to_string(kNoAllocScratchBytes) + " (use dv_model_create + dv_rhs)");
        return DV_ERR_ARG;
    }
    int dev = 0;
    DV_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) {
        set_error("dv_rhs_acc_noalloc: device index out of range");
        return DV_ERR_ARG;
    }
    double* base = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!g_noalloc_ptr[dev]) {                   // first call on this device: look up the address
            void* ptr = nullptr;
            DV_CUDA(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
            g_noalloc_ptr[dev] = (double*)ptr;
        }
        base = g_noalloc_ptr[dev];
    }
    cudaStream_t s = (cudaStream_t)stream;
    // The array keeps the previous call's records; records that this grid and step never write
    // (ends without a valve, the wall of a wall-less column) must read as zero.
    DV_CUDA(cudaMemsetAsync(base, 0, need, s));
    Rec rec = make_rec(rl, base);
    const int64_t nc = (int64_t)p->Nr * p->Nth * p->Nz;
    count_launch(K_RESIDUAL);
    k_cells<M_RHS, true><<<nblk(nc, 128), 128, 0, s>>>(*p, Aux{feed_flux, n_nom, coverage}, rec, t, y, nullptr,
                                                      nullptr, nullptr, nullptr, 0.0, f);
    count_launch(K_RESIDUAL);
    k_accumulators<<<1, 256, 0, s>>>(*p, rec.bnd, rec.Qj, rec.Qa, rec.Qw, rec.Qhx, acc);
    DV_CUDA(cudaGetLastError());
    return DV_OK;
}
