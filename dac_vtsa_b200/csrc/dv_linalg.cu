// dv_linalg.cu -- preconditioner: block-pentadiagonal LU of I - dh J along z, and its sweep.
//
// The reference preconditions GMRES with a SuperLU factorisation of M = I - d h J restricted to
// theta sectors (+ the innermost rings fully coupled), core/solver.py:334-337 and
// core/jacobian.py:50-69,88-91.  Here M is partitioned into z-planes: a partition is either one
// theta sector (mode 0: cells (i, j, k) for all rings i of sector j, plus the wall node (j, k)),
// a whole cross-section (mode 1), or, in mode 2, the innermost ring of every sector as one
// partition plus rings 1.. of each sector (with its wall node) as the others: the inner ring's
// theta couplings stay in the preconditioner, which the reference keeps for its innermost rings.
// Inside a partition every coupling of the
// stencil is kept: within a plane (r, and theta in full mode) and between planes k-2..k+2 (the
// MUSCL z+-2 reach).  The partition matrix is block-pentadiagonal in z with dense nb x nb blocks
// (row-major, leading dimension ld >= nb, zero padded), factorised by block Gaussian elimination:
//   L2_k = A(k,k-2) Uinv_{k-2}
//   L1_k = (A(k,k-1) - L2_k U1_{k-2}) Uinv_{k-1}
//   D_k  = A(k,k) - L1_k U1_{k-1} - L2_k U2_{k-2},      Uinv_k = D_k^-1 (Gauss-Jordan, partial pivoting)
//   U1_k = A(k,k+1) - L1_k U2_{k-1},                    U2_k = A(k,k+2)
// Stored per plane k: slot 0 L2_k, slot 1 L1_k, slot 2 Uinv_k, slot 3 -Uinv_k U1_k, slot 4 -Uinv_k U2_k,
// so that both sweeps are one fused GEMV per plane:
//   forward  z_k = b_k - L1_k z_{k-1} - L2_k z_{k-2}
//   backward x_k = Uinv_k z_k + (-Uinv_k U1_k) x_{k+1} + (-Uinv_k U2_k) x_{k+2}
// Twisted form (Nz >= 8, both kernels in shared memory): the same recurrences run top-down over
// planes 0..zs-1 and, mirrored, bottom-up over planes Nz-1..zs+2 at the same time (a cluster of
// two CTAs per partition); the separator planes zs, zs+1 (zs = (Nz-2)/2) take the Schur
// contributions of both sides, and their 2 nb x 2 nb system is inverted by blocks.  Half the
// sequential plane chain of the one-directional form, for the same matrix.
#include <algorithm>
#include <vector>
#include <type_traits>
#include "dv_internal.h"
#include "dv_physics.cuh"

namespace dv {

struct PcGeom {
    int Nr, Nth, Nz, wall, mode, nb, nparts, ld;
    int rg, tg;            // mode 3: ring groups per sector (rings 1..Nr-1), theta groups of the core ring
    int zs;                // twisted factorisation: separator planes zs, zs+1 (0: one direction, top-down)
    int ncv;               // cell unknowns (6 per cell) of the partition; nb - ncv wall nodes follow
    int64_t nc, bs;        // bs: block stride in doubles (nb*ld rounded up to even: 16-byte multiple)
    // self-checks of the kernels: factor storage (entries; < 0: unchecked), state length, error word
    int64_t cap, nstate;
    int* err;
};

// Error word bit of an index that fell outside its storage (the access is skipped, not made).
#define PC_ERR_RANGE 32
static __device__ __forceinline__ bool pc_range_ok(const PcGeom& g, int64_t first, int64_t count) {
    if (g.cap < 0 || (first >= 0 && first + count <= g.cap)) return true;
    if (g.err) atomicOr(g.err, PC_ERR_RANGE);
    return false;
}

// Mode 3 (mode 2 split for large cross-sections): contiguous groups of n items in G groups, the
// first n % G groups one item larger.  Ring groups cover rings 1..Nr-1 of a sector (the wall node
// goes with the outermost, smallest group); theta groups cover the sectors of the core ring.
static __host__ __device__ __forceinline__ void pc_group(int n, int G, int gi, int& a0, int& a1) {
    const int base = n / G, extra = n % G;
    a0 = gi * base + (gi < extra ? gi : extra);
    a1 = a0 + base + (gi < extra ? 1 : 0);
}
static __host__ __device__ __forceinline__ int pc_group_of(int n, int G, int t) {
    const int base = n / G, extra = n % G;
    return (t < extra * (base + 1)) ? t / (base + 1) : extra + (t - extra * (base + 1)) / base;
}

// Geometry as seen by one partition: nb and ncv of that partition (ld, bs and strides stay the
// largest partition's).  Mode 2: parts 0..Nth-1 are sectors (rings 1..Nr-1 + wall), part Nth the core.
// Mode 3: part j*rg + gi is ring group gi of sector j (+ the wall in the last group), part
// Nth*rg + h theta group h of the core ring.
static __host__ __device__ __forceinline__ PcGeom pc_part(const PcGeom& g, int part) {
    PcGeom q = g;
    if (g.mode == 2) {
        if (part == g.Nth) { q.ncv = DV_NV * g.Nth; q.nb = q.ncv; }
        else { q.ncv = DV_NV * (g.Nr - 1); q.nb = q.ncv + (g.wall ? 1 : 0); }
    } else if (g.mode == 3) {
        int a0, a1;
        if (part >= g.Nth * g.rg) {
            pc_group(g.Nth, g.tg, part - g.Nth * g.rg, a0, a1);
            q.ncv = DV_NV * (a1 - a0);
            q.nb = q.ncv;
        } else {
            const int gi = part % g.rg;
            pc_group(g.Nr - 1, g.rg, gi, a0, a1);
            q.ncv = DV_NV * (a1 - a0);
            q.nb = q.ncv + ((g.wall && gi == g.rg - 1) ? 1 : 0);
        }
    }
    return q;
}

// partition of the cell unknowns of cell (i, j)
static __host__ __device__ __forceinline__ int pc_part_of(const PcGeom& g, int i, int j) {
    if (g.mode == 0) return j;
    if (g.mode == 2) return (i == 0) ? g.Nth : j;
    if (g.mode == 3)
        return (i == 0) ? g.Nth * g.rg + pc_group_of(g.Nth, g.tg, j) : j * g.rg + pc_group_of(g.Nr - 1, g.rg, i - 1);
    return 0;
}

#define PC_SMEM_NB 56      // largest block the shared-memory factorisation keeps resident (9 blocks)

// leading dimension of the stored blocks: nb rounded up to 16, so a row is a whole number of
// 16-column groups that the sweep's 8 lanes read as 16-byte column pairs
static inline int pc_ld(int nb) { return (nb + 15) / 16 * 16; }

// leading dimension of the blocks the factorisation keeps in shared memory: nb rounded up to 4 and
// made == 4 (mod 8), so the 8 rows of a DMMA A fragment (and the 4 rows of a B fragment) start on
// different 8-bank groups; without that padding when nine blocks would not fit
static inline int pc_lds(int nb, size_t budget) {
    const int l4 = (nb + 3) / 4 * 4;
    const int l = (l4 % 8 == 0) ? l4 + 4 : l4;
    return (size_t)9 * nb * l * sizeof(double) <= budget ? l : l4;
}

static __host__ __device__ __forceinline__ int64_t pc_glob(const PcGeom& g, int part, int k, int l) {
    const int64_t offw = (int64_t)DV_NV * g.nc;
    if (g.mode == 3) {
        int a0, a1;
        if (part >= g.Nth * g.rg) {             // core theta group: (sector j, var v) of ring 0
            pc_group(g.Nth, g.tg, part - g.Nth * g.rg, a0, a1);
            const int j = a0 + l / DV_NV, v = l % DV_NV;
            return (int64_t)v * g.nc + (int64_t)j * g.Nz + k;
        }
        const int j = part / g.rg, gi = part % g.rg;
        pc_group(g.Nr - 1, g.rg, gi, a0, a1);
        if (l < DV_NV * (a1 - a0)) {            // rings 1 + a0 .. 1 + a1 - 1 of sector j
            const int i = 1 + a0 + l / DV_NV, v = l % DV_NV;
            return (int64_t)v * g.nc + ((int64_t)i * g.Nth + j) * g.Nz + k;
        }
        return offw + (int64_t)j * g.Nz + k;
    }
    if (g.mode == 2) {
        if (part == g.Nth) {                    // core: (sector j, var v) of ring 0
            const int j = l / DV_NV, v = l % DV_NV;
            return (int64_t)v * g.nc + (int64_t)j * g.Nz + k;
        }
        if (l < DV_NV * (g.Nr - 1)) {           // sector `part`, rings 1..Nr-1
            const int i = 1 + l / DV_NV, v = l % DV_NV;
            return (int64_t)v * g.nc + ((int64_t)i * g.Nth + part) * g.Nz + k;
        }
        return offw + (int64_t)part * g.Nz + k;
    }
    if (g.mode == 0) {   // theta sector `part`
        if (l < DV_NV * g.Nr) {
            int i = l / DV_NV, v = l % DV_NV;
            return (int64_t)v * g.nc + ((int64_t)i * g.Nth + part) * g.Nz + k;
        }
        return offw + (int64_t)part * g.Nz + k;
    }
    if (l < DV_NV * g.Nr * g.Nth) {
        int pos = l / DV_NV, v = l % DV_NV;
        return (int64_t)v * g.nc + (int64_t)pos * g.Nz + k;
    }
    return offw + (int64_t)(l - DV_NV * g.Nr * g.Nth) * g.Nz + k;
}

// local index of (cell (i, j), var v) / wall (j) inside its partition
static __host__ __device__ __forceinline__ int pc_local(const PcGeom& g, int i, int j, int v) {
    if (g.mode == 3) {
        int a0, a1;
        if (v == DV_NV) {                       // the wall node follows the cells of the outer group
            pc_group(g.Nr - 1, g.rg, g.rg - 1, a0, a1);
            return DV_NV * (a1 - a0);
        }
        if (i == 0) {
            pc_group(g.Nth, g.tg, pc_group_of(g.Nth, g.tg, j), a0, a1);
            return (j - a0) * DV_NV + v;
        }
        pc_group(g.Nr - 1, g.rg, pc_group_of(g.Nr - 1, g.rg, i - 1), a0, a1);
        return (i - 1 - a0) * DV_NV + v;
    }
    if (g.mode == 2) {
        if (v == DV_NV) return DV_NV * (g.Nr - 1);
        return (i == 0) ? j * DV_NV + v : (i - 1) * DV_NV + v;
    }
    if (g.mode == 0) return (v < DV_NV) ? i * DV_NV + v : DV_NV * g.Nr;
    return (v < DV_NV) ? (i * g.Nth + j) * DV_NV + v : DV_NV * g.Nr * g.Nth + j;
}

// The z-couplings A(k, k+-1), A(k, k+-2) only connect a cell to itself in another plane: they are
// block diagonal with 6x6 cell blocks (and 1x1 wall entries).  First index / size of the block of l:
static __device__ __forceinline__ void pc_cellblock(const PcGeom& g, int l, int& b0, int& bsz) {
    if (l < g.ncv) { b0 = (l / DV_NV) * DV_NV; bsz = DV_NV; }
    else { b0 = l; bsz = 1; }
}

// ---------------------------------------------------------------- assembly of I - dh J
// blocks: [part][Nz][5][bs] row-major (B[row*ld + col]); slot d+2 holds A(k, k+d).
__global__ void k_pc_zero(double* __restrict__ A, int64_t n) {
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
        A[q] = 0.0;
}

__global__ void k_pc_to_f32(const double* __restrict__ A, float* __restrict__ B, int64_t n) {
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
        B[q] = (float)A[q];
}

__global__ void k_pc_scatter(PcGeom g, const double* __restrict__ J, double dh, double* __restrict__ A) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.nc) return;
    const int slot = blockIdx.y;
    const int k = (int)(c % g.Nz);
    const int64_t rj = c / g.Nz;
    const int j = (int)(rj % g.Nth), i = (int)(rj / g.Nth);
    int ni = i, nj = j, nk = k;
    bool ok = true;
    switch (slot) {
        case 0: break;
        case 1: nk = k - 1; ok = nk >= 0; break;
        case 2: nk = k + 1; ok = nk < g.Nz; break;
        case 3: nk = k - 2; ok = nk >= 0; break;
        case 4: nk = k + 2; ok = nk < g.Nz; break;
        case 5: ni = i - 1; ok = ni >= 0; break;
        case 6: ni = i + 1; ok = ni < g.Nr; break;
        case 7: ok = g.Nth > 1 && g.mode != 0; nj = (j == 0) ? g.Nth - 1 : j - 1; break;
        default: ok = g.Nth > 1 && g.mode != 0; nj = (j == g.Nth - 1) ? 0 : j + 1; break;
    }
    const int part = pc_part_of(g, i, j);
    if (!ok || pc_part_of(g, ni, nj) != part) return;      // coupling across partitions: dropped
    const int d = nk - k;
    const int64_t boff = (((int64_t)part * g.Nz + k) * 5 + (d + 2)) * g.bs;
    if (part >= g.nparts || !pc_range_ok(g, boff, g.bs)) {
        if (part >= g.nparts && g.err) atomicOr(g.err, PC_ERR_RANGE);
        return;
    }
    double* B = A + boff;
    const int pnb = pc_part(g, part).nb;
    const bool row_wall_ok = g.wall && i == g.Nr - 1;
    const bool col_wall_ok = g.wall && ni == g.Nr - 1;
    for (int rv = 0; rv < DV_NB; ++rv) {
        if (rv == DV_NV && !row_wall_ok) continue;
        const int lr = pc_local(g, i, j, rv);
        for (int cv = 0; cv < DV_NB; ++cv) {
            if (cv == DV_NV && !col_wall_ok) continue;
            const int lc = pc_local(g, ni, nj, cv);
            const double jv = J[((int64_t)(slot * DV_NB + rv) * DV_NB + cv) * g.nc + c];
            double val = -dh * jv;
            if (slot == 0 && rv == cv) val += 1.0;
            if (lr >= pnb || lc >= pnb) {
                if (g.err) atomicOr(g.err, PC_ERR_RANGE);
                continue;
            }
            B[(int64_t)lr * g.ld + lc] = val;
        }
    }
}

// ---------------------------------------------------------------- shared-memory dense kernels (row-major)
// Each works with a team of whole warps of the block, so that teams can work side by side.  Functions of
// their own, not inlined: the factorisation calls them from many places, and its code then stays in the
// instruction cache while two teams run different parts of it.
struct Team {
    int tid, n, bar;                              // thread of the team, its threads, its barrier
    __device__ __forceinline__ int lane() const { return tid & 31; }
    __device__ __forceinline__ int warp() const { return tid >> 5; }
    __device__ __forceinline__ int warps() const { return n >> 5; }
    __device__ __forceinline__ void sync() const {
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(n) : "memory");
    }
};

// D = A B + D on the FP64 tensor cores: one 8x8x4 product per warp instruction.  Fragments
// (lane = 4 g + t): a = A[g][t], b = B[t][g], d = D[g][2t .. 2t+1].
static __device__ __forceinline__ void dmma_884(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// C = Cin + S A B, S = +-1 (Cin null: C = S A B); A and B in shared memory (row-major, leading
// dimension ld), Cin and C in any space (ldi, ldc).  8x8 output tiles spread over the warps, each
// accumulated by DMMA over k in steps of 4, three tiles of a warp at a time (a dependent DMMA takes 29
// cycles, three independent ones 10 each).  Rows and columns past nb read the last one (they enter no
// entry that is written); past k = nb both operands are zero.
static __device__ __noinline__ void tm_gemm(Team T, int nb, int ld, int S, const double* A, const double* B,
                                            const double* Cin, int ldi, double* C, int ldc) {
    __builtin_assume(__isShared(A));
    __builtin_assume(__isShared(B));
    constexpr int U = 4;
    const int lane = T.lane(), g = lane >> 2, t4 = lane & 3;
    const int nt = (nb + 7) >> 3, nt2 = nt * nt, full = nb & ~3;
    for (int t0 = T.warp(); t0 < nt2; t0 += U * T.warps()) {
        const double *ap[U], *bp[U];
        double d0[U], d1[U], e0[U], e1[U];
        int r[U], c0[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int tile = t0 + u * T.warps(), ti = tile / nt, tj = tile - ti * nt;
            r[u] = tile < nt2 ? 8 * ti + g : nb;  // row of A and C held by this lane (nb: no tile)
            c0[u] = 8 * tj + 2 * t4;              // columns of C in the d fragment
            ap[u] = A + min(r[u], nb - 1) * ld + t4;
            bp[u] = B + t4 * ld + min(8 * tj + g, nb - 1);
            d0[u] = d1[u] = e0[u] = e1[u] = 0.0;
            if (Cin && r[u] < nb) {
                if (c0[u] < nb) e0[u] = Cin[r[u] * ldi + c0[u]];
                if (c0[u] + 1 < nb) e1[u] = Cin[r[u] * ldi + c0[u] + 1];
            }
        }
#pragma unroll 2
        for (int kk = 0; kk < full; kk += 4) {
#pragma unroll
            for (int u = 0; u < U; ++u) dmma_884(d0[u], d1[u], ap[u][kk], bp[u][kk * ld]);
        }
        if (full < nb) {
            const bool in = full + t4 < nb;
#pragma unroll
            for (int u = 0; u < U; ++u) dmma_884(d0[u], d1[u], in ? ap[u][full] : 0.0, in ? bp[u][full * ld] : 0.0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (r[u] >= nb) continue;
            const double f0 = S < 0 ? 0.0 - d0[u] : d0[u], f1 = S < 0 ? 0.0 - d1[u] : d1[u];
            if (c0[u] < nb) C[r[u] * ldc + c0[u]] = Cin ? e0[u] + f0 : f0;
            if (c0[u] + 1 < nb) C[r[u] * ldc + c0[u] + 1] = Cin ? e1[u] + f1 : f1;
        }
    }
}

// C = Bd X with Bd block diagonal (cell blocks; any space, leading dimension ldb): a cell per warp
static __device__ __noinline__ void tm_bd_left(Team T, int nb, int ncv, int ld, const double* Bd, int ldb,
                                               const double* X, double* C) {
    __builtin_assume(__isShared(X));
    __builtin_assume(__isShared(C));
    const int lane = T.lane();
    const int ncell = ncv / DV_NV, nblk = ncell + (nb - ncv);
    for (int cell = T.warp(); cell < nblk; cell += T.warps()) {
        const int b0 = cell < ncell ? cell * DV_NV : ncv + cell - ncell, bsz = cell < ncell ? DV_NV : 1;
        double x[2][DV_NV];
#pragma unroll
        for (int q = 0; q < DV_NV; ++q) {
            x[0][q] = (q < bsz && lane < nb) ? X[(b0 + q) * ld + lane] : 0.0;
            x[1][q] = (q < bsz && lane + 32 < nb) ? X[(b0 + q) * ld + lane + 32] : 0.0;
        }
        for (int r = b0; r < b0 + bsz; ++r) {
            double acc[2] = {0.0, 0.0};
#pragma unroll
            for (int q = 0; q < DV_NV; ++q) {
                if (q < bsz) {
                    const double v = Bd[r * ldb + b0 + q];
                    acc[0] += v * x[0][q];
                    acc[1] += v * x[1][q];
                }
            }
            if (lane < nb) C[r * ld + lane] = acc[0];
            if (lane + 32 < nb) C[r * ld + lane + 32] = acc[1];
        }
    }
}

// Block-diagonal right factors in shared memory by columns: u2[q][c] is entry (first row of c's block + q, c),
// zero past the block.  One entry per thread of a team of 64 DV_NV.
constexpr int BD_LD = 64;
static __device__ __forceinline__ double bd_entry(const PcGeom& g, int tid, const double* Bd, int ldb) {
    const int q = tid / BD_LD, c = tid - q * BD_LD;
    int b0, bsz;
    pc_cellblock(g, c, b0, bsz);
    return (c < g.nb && q < bsz) ? Bd[(b0 + q) * ldb + c] : 0.0;
}

// C = Cin - X Bd (Cin null: C = -X Bd), Bd block diagonal as above; X in shared memory, Cin and C in any space
static __device__ __noinline__ void tm_bd_right(Team T, int nb, int ncv, int ld, const double* X, const double* u2,
                                                const double* Cin, int ldi, double* C, int ldc) {
    __builtin_assume(__isShared(X));
    __builtin_assume(__isShared(u2));
    const int lane = T.lane();
    const int ca = lane, cb = lane + 32;
    const int ba = ca < ncv ? ca / DV_NV * DV_NV : ca, bb = cb < ncv ? cb / DV_NV * DV_NV : cb;
    const int na = ca >= nb ? 0 : ca < ncv ? DV_NV : 1, nbb = cb >= nb ? 0 : cb < ncv ? DV_NV : 1;
    double va[DV_NV], vb[DV_NV];
#pragma unroll
    for (int q = 0; q < DV_NV; ++q) {
        va[q] = u2[q * BD_LD + ca];
        vb[q] = u2[q * BD_LD + cb];
    }
    constexpr int U = 4;                          // rows together, their inputs loaded first
    for (int r0 = T.warp(); r0 < nb; r0 += U * T.warps()) {
        double ia[U], ib[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int r = r0 + u * T.warps();
            ia[u] = (Cin && r < nb && na) ? Cin[r * ldi + ca] : 0.0;
            ib[u] = (Cin && r < nb && nbb) ? Cin[r * ldi + cb] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int r = r0 + u * T.warps();
            if (r >= nb) break;
            double acc0 = 0.0, acc1 = 0.0;
#pragma unroll
            for (int q = 0; q < DV_NV; ++q) {
                if (q < na) acc0 += X[r * ld + ba + q] * va[q];
                if (q < nbb) acc1 += X[r * ld + bb + q] * vb[q];
            }
            if (na) C[r * ldc + ca] = Cin ? ia[u] - acc0 : -acc0;
            if (nbb) C[r * ldc + cb] = Cin ? ib[u] - acc1 : -acc1;
        }
    }
}

// D = S, entries of nb x nb, any spaces
static __device__ __noinline__ void tm_copy(Team T, int nb, const double* S, int lds, double* D, int ldd) {
    const int lane = T.lane();
    constexpr int U = 4;
    for (int r0 = T.warp(); r0 < nb; r0 += U * T.warps()) {
        double v0[U], v1[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int r = r0 + u * T.warps();
            v0[u] = (r < nb && lane < nb) ? S[r * lds + lane] : 0.0;
            v1[u] = (r < nb && lane + 32 < nb) ? S[r * lds + lane + 32] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int r = r0 + u * T.warps();
            if (r < nb && lane < nb) D[r * ldd + lane] = v0[u];
            if (r < nb && lane + 32 < nb) D[r * ldd + lane + 32] = v1[u];
        }
    }
}

// Gauss-Jordan inverse with partial pivoting of the nb x nb block *A (shared memory, nb <= 32, a team
// of 128 threads), ping-ponging between *A and *B (same size).  Thread t updates column t % 32 on
// the rows congruent to t / 32 modulo 4 (coalesced row accesses, broadcast column-k reads); the
// threads of column k+1 also keep the running maxima of its new entries (rows > k), so the next
// pivot is known after the one barrier of the step.  The pivot is the largest |entry|, the
// smallest row index among equal ones.  The row interchanges are undone at the end by a single
// column gather.  On return *A holds the inverse (the pointers may have been exchanged).
static __device__ __noinline__ int tm_inverse_unb(Team T, int nb, int ld, double* A, double* B, int* perm, int* idx,
                                                  double* pv, int* pi) {
    __builtin_assume(__isShared(A));
    __builtin_assume(__isShared(B));
    __builtin_assume(__isShared(perm));
    __builtin_assume(__isShared(idx));
    __builtin_assume(__isShared(pv));
    __builtin_assume(__isShared(pi));
    const int tid = T.tid;
    const int cc = tid & 31, rq = tid >> 5;
    constexpr int RPT = 8;                        // rows per thread for nb <= 32
    int bad = 0;
    if (cc == 0) {                                // column 0: partial maxima per row group
        double best = -1.0;
        int bi = nb;
        for (int i = rq; i < nb; i += 4) {
            const double v = fabs(A[i * ld]);
            if (v > best) { best = v; bi = i; }
        }
        pv[rq] = best;
        pi[rq] = bi;
    }
    T.sync();
    for (int k = 0; k < nb; ++k) {
        const double* cpv = pv + 4 * (k & 1);
        const int* cpi = pi + 4 * (k & 1);
        double best = cpv[0];
        int p = cpi[0];
#pragma unroll
        for (int q = 1; q < 4; ++q)
            if (cpv[q] > best || (cpv[q] == best && cpi[q] < p)) { best = cpv[q]; p = cpi[q]; }
        if (p >= nb) p = k;                       // (a column of NaN has no largest entry)
        if (tid == 0) perm[k] = p;
        double piv = A[p * ld + k];
        if (!(fabs(piv) > 0.0) || !isfinite(piv)) { bad = 1; piv = 1.0; }
        const double inv = 1.0 / piv;
        if (cc < nb) {
            const double pr = ((cc == k) ? 1.0 : A[p * ld + cc]) * inv;     // scaled pivot row
            const bool nextcol = (cc == k + 1);
            double nbest = -1.0;
            int nbi = nb;
#pragma unroll
            for (int a = 0; a < RPT; ++a) {
                const int i = rq + 4 * a;
                if (i >= nb) break;
                double val;
                if (i == k) {
                    val = pr;
                } else {
                    const int src = (i == p) ? k : i;                      // rows k and p exchanged
                    const double fc = A[src * ld + k];                     // old column k
                    val = ((cc == k) ? 0.0 : A[src * ld + cc]) - fc * pr;
                }
                B[i * ld + cc] = val;
                if (nextcol && i > k) {
                    const double v = fabs(val);
                    if (v > nbest) { nbest = v; nbi = i; }
                }
            }
            if (nextcol) {
                pv[4 * ((k + 1) & 1) + rq] = nbest;
                pi[4 * ((k + 1) & 1) + rq] = nbi;
            }
        }
        T.sync();
        double* t = A; A = B; B = t;
    }
    if (tid == 0) {                               // the row interchanges, undone as column interchanges
        for (int c = 0; c < nb; ++c) idx[c] = c;
        for (int k = nb - 1; k >= 0; --k) {
            const int q = perm[k], t = idx[k];
            idx[k] = idx[q];
            idx[q] = t;
        }
    }
    T.sync();
    if (cc < nb)
        for (int i = rq; i < nb; i += 4) B[i * ld + cc] = A[i * ld + idx[cc]];
    T.sync();
    double* t = A; A = B; B = t;
    return bad;
}

// One panel of the blocked inverse: Gauss-Jordan steps on columns j0 .. j0 + jb - 1 of A by one warp, the
// panel in its registers (rows lane and lane + 32).  Rows keep their place in memory; pos0 / pos1 are
// the positions that row interchanges give them, which decide ties: the pivot is the largest |entry| of the rows
// that are no pivot yet (done0 / done1), at the smallest position among equal ones.  Returns 1 on a zero or
// non-finite pivot (replaced by 1 so the factors stay finite).  Pan: the panel again, [row][PAN_LD]; prow: its
// pivots' rows in memory, pmask: the same as bits.
// A step works on x[0], and the columns move down by one with it, so that the loop need not be unrolled (its code
// is fetched once).  A step's chain is the search and the quotient, the next column's update and again: the
// lanes divide by their own larger entry, magnitudes are ordered by their upper words (integers; FP64 comparisons
// took half of a step), and the other columns' updates (pivot row q, factors g) follow while the next
// division runs.  All lanes take the same branches; one lane storing by itself would leave the warp in two
// parts, each of which issues the rest of the step.
constexpr int PAN_LD = 12;                        // (a DMMA fragment's 8 rows on different banks)
static __device__ __forceinline__ int inv_panel(int nb, int ld, double* A, int j0, int jb, int lane, int& pos0, int& pos1,
                                                bool& done0, bool& done1, double* Pan, int* prow, unsigned* pmask) {
    const unsigned all = 0xffffffffu;
    const int r0 = min(lane, nb - 1), r1 = min(lane + 32, nb - 1);
    double x0[9], x1[9];                          // from the second on shifted: see the updates below
    if (jb == 8) {                                // (rows of 16-byte pairs: ld and j0 are even)
#pragma unroll
        for (int c = 0; c < 8; c += 2) {
            const double2 a = *reinterpret_cast<const double2*>(A + r0 * ld + j0 + c);
            const double2 b = *reinterpret_cast<const double2*>(A + r1 * ld + j0 + c);
            x0[c ? c + 1 : 0] = a.x;
            x0[c + 2] = a.y;
            x1[c ? c + 1 : 0] = b.x;
            x1[c + 2] = b.y;
        }
    } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int cc = j0 + min(c, jb - 1);
            x0[c ? c + 1 : 0] = (c < jb) ? A[r0 * ld + cc] : 0.0;
            x1[c ? c + 1 : 0] = (c < jb) ? A[r1 * ld + cc] : 0.0;
        }
    }
    int bad = 0;
    unsigned m0 = 0u, m1 = 0u;
    double q[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, g0 = 0.0, g1 = 0.0;
    bool w0 = false, w1 = false;                  // this lane's row is the last step's pivot row
#pragma unroll 1
    for (int kq = 0; kq < jb; ++kq) {
        const double f0 = x0[0], f1 = x1[0];
        const unsigned h0 = done0 ? 0u : ((unsigned)__double2hiint(f0) & 0x7fffffffu) + 1u;      // 0: no candidate
        const unsigned h1 = done1 ? 0u : ((unsigned)__double2hiint(f1) & 0x7fffffffu) + 1u;
        const bool up = h1 > h0;                  // the lane's larger entry: row lane + 32
        const unsigned hm = up ? h1 : h0;
        const unsigned best = __reduce_max_sync(all, hm);
        double xc = (hm > 0x100000u && hm <= 0x7ff00000u) ? (up ? f1 : f0) : 1.0;   // (normal numbers: no branch in the quotient)
        asm("" : "+d"(xc));                       // (or the quotient of a zero is taken, and not used: 150 cycles)
#pragma unroll
        for (int c = 1; c < 8; ++c) {
            x0[c] = w0 ? q[c] : __fma_rn(-g0, q[c], x0[c + 1]);
            x1[c] = w1 ? q[c] : __fma_rn(-g1, q[c], x1[c + 1]);
        }
        const unsigned b0 = __ballot_sync(all, h0 == best), b1 = __ballot_sync(all, h1 == best);
        int src = __ffs(b0 | b1) - 1;
        bool srcup = b1 != 0u;
        const bool odd = __popc(b0) + __popc(b1) != 1 || best <= 0x100000u || best > 0x7ff00000u;
        double inv = 1.0 / xc;
        if (odd) {
            // equal upper words, zero, subnormal, infinite, NaN: whole magnitudes, then positions
            constexpr unsigned long long INF = 0x7ff0000000000000ull, MAG = 0x7fffffffffffffffull;
            const unsigned long long a0 = (unsigned long long)__double_as_longlong(f0) & MAG;
            const unsigned long long a1 = (unsigned long long)__double_as_longlong(f1) & MAG;
            const unsigned long long k0 = (!done0 && a0 <= INF) ? a0 + 1 : 0, k1 = (!done1 && a1 <= INF) ? a1 + 1 : 0;
            bool u = k1 > k0 || (k1 == k0 && k1 != 0 && pos1 < pos0);
            const unsigned long long kk = u ? k1 : k0;
            unsigned pc = (unsigned)(u ? pos1 : pos0);
            const unsigned mh = __reduce_max_sync(all, (unsigned)(kk >> 32));
            const bool c1 = (unsigned)(kk >> 32) == mh;
            const unsigned ml = __reduce_max_sync(all, c1 ? (unsigned)kk : 0u);
            bool c2 = c1 && (unsigned)kk == ml;
            if ((mh | ml) == 0u) {                // a column of NaN: the row in the smallest place
                u = done0 || (!done1 && pos1 < pos0);
                pc = (unsigned)(u ? pos1 : pos0);
                c2 = !(done0 && done1);
            }
            const unsigned mp = __reduce_min_sync(all, c2 ? pc : all);
            c2 = c2 && pc == mp;
            src = __ffs(__ballot_sync(all, c2)) - 1;
            srcup = (__ballot_sync(all, u) >> src) & 1u;
            const bool ok = (__ballot_sync(all, kk > 1 && kk <= INF) >> src) & 1u;
            inv = 1.0 / (ok ? (srcup ? f1 : f0) : 1.0);
            if (!ok) bad = 1;
        }
        inv = __shfl_sync(all, inv, src);
        const double p1 = __shfl_sync(all, srcup ? x1[1] : x0[1], src) * inv;
        const int k = j0 + kq, pp = __shfl_sync(all, srcup ? pos1 : pos0, src);
#pragma unroll
        for (int c = 2; c < 8; ++c) q[c - 1] = __shfl_sync(all, srcup ? x1[c] : x0[c], src) * inv;
        q[7] = inv;
        w0 = lane == src && !srcup;
        w1 = lane == src && srcup;
        x0[0] = w0 ? p1 : __fma_rn(-f0, p1, x0[1]);
        x1[0] = w1 ? p1 : __fma_rn(-f1, p1, x1[1]);
        x0[8] = x1[8] = 0.0;
        g0 = f0;
        g1 = f1;
        pos0 = w0 ? k : pos0 == k ? pp : pos0;
        pos1 = w1 ? k : pos1 == k ? pp : pos1;
        done0 = done0 || w0;
        done1 = done1 || w1;
        if (srcup) m1 |= 1u << src;
        else m0 |= 1u << src;
        prow[kq] = src + (srcup ? 32 : 0);
    }
#pragma unroll
    for (int c = 1; c < 8; ++c) {
        x0[c] = w0 ? q[c] : __fma_rn(-g0, q[c], x0[c + 1]);
        x1[c] = w1 ? q[c] : __fma_rn(-g1, q[c], x1[c + 1]);
    }
    pmask[0] = m0;
    pmask[1] = m1;
    if (jb == 8) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int r = lane + 32 * e;
            if (r < nb) {
#pragma unroll
                for (int c = 0; c < 8; c += 2) {
                    const double2 v = make_double2(e ? x1[c] : x0[c], e ? x1[c + 1] : x0[c + 1]);
                    *reinterpret_cast<double2*>(A + r * ld + j0 + c) = v;
                    *reinterpret_cast<double2*>(Pan + r * PAN_LD + c) = v;
                }
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int c = (i + jb) & 7;           // the column in x[i] now
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = lane + 32 * e;
                const double v = e ? x1[i] : x0[i];
                if (r < nb && c < jb) A[r * ld + j0 + c] = v;
                if (r < nb) Pan[r * PAN_LD + c] = (c < jb) ? v : 0.0;
            }
        }
    }
    __syncwarp();
    return bad;
}

// Columns 8 tb .. 8 tb + 7 of A after a panel of jb pivots,
//   x <- [x with the pivot rows zeroed] + Panel * x(pivot rows), a rank-8 DMMA update:
// by one warp, or (`shared`) by all of the team, each a part of the rows.
static __device__ __forceinline__ void inv_update(const Team& T, bool shared, int nb, int ld, double* A, int tb, int jb,
                                                  const double* Pan, const int* prow, const unsigned* pmask) {
    const int lane = T.lane(), g = lane >> 2, t4 = lane & 3, nt = (nb + 7) >> 3;
    const int cb = min(8 * tb + g, nb - 1), c0 = 8 * tb + 2 * t4;
    const double b0 = (t4 < jb) ? A[prow[t4] * ld + cb] : 0.0, b1 = (t4 + 4 < jb) ? A[prow[t4 + 4] * ld + cb] : 0.0;
    const unsigned m0 = pmask[0], m1 = pmask[1];
    if (shared) T.sync();                         // (every pivot row has been read)
    else __syncwarp();
    const int first = shared ? T.warp() : 0, step = shared ? T.warps() : 1;
#pragma unroll 1
    for (int t0 = first; t0 < nt; t0 += 4 * step) {
        double d0[4], d1[4], e0[4], e1[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int r = 8 * (t0 + u * step) + g;
            const double* pp = Pan + min(r, nb - 1) * PAN_LD + t4;
            const bool live = r < nb && !(((r < 32 ? m0 : m1) >> (r & 31)) & 1u);      // (a pivot row counts as zero)
            e0[u] = (live && c0 < nb) ? A[r * ld + c0] : 0.0;
            e1[u] = (live && c0 + 1 < nb) ? A[r * ld + c0 + 1] : 0.0;
            d0[u] = d1[u] = 0.0;
            dmma_884(d0[u], d1[u], pp[0], b0);
            dmma_884(d0[u], d1[u], pp[4], b1);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int r = 8 * (t0 + u * step) + g;
            if (r >= nb) continue;
            if (c0 < nb) A[r * ld + c0] = e0[u] + d0[u];
            if (c0 + 1 < nb) A[r * ld + c0 + 1] = e1[u] + d1[u];
        }
    }
}

// Blocked Gauss-Jordan inverse with partial pivoting of the nb x nb block A (shared memory, nb <= 64) into
// X, by a team of 4 warps; A is overwritten.  Panels of 8 columns: warp 0 takes a panel's pivot steps, the
// others meanwhile update the columns that the next panel does not need with the panel before.  The pivot steps are a serial chain (a division and a search for the largest entry, 48 times
// for nb = 48); with the panel in one warp's registers a step has no barrier and no trip through shared
// memory: 79 000 -> 32 000 cycles an inverse (nb = 43; before, steps by eight warps with a barrier each).
static __device__ __noinline__ int tm_inverse_blk(Team T, int nb, int ld, double* A, double* X, int* pos, int* prow,
                                                  unsigned* pmask) {
    __builtin_assume(__isShared(A));
    __builtin_assume(__isShared(X));
    __builtin_assume(__isShared(pos));
    __builtin_assume(__isShared(prow));
    __builtin_assume(__isShared(pmask));
    const int lane = T.lane(), warp = T.warp(), nt = (nb + 7) >> 3;
    int pos0 = lane, pos1 = lane + 32, bad = 0;
    bool done0 = lane >= nb, done1 = lane + 32 >= nb;       // (rows past nb are never pivots)
    for (int j = 0; j < nt; ++j) {
        const int b = j & 1, jb = min(8, nb - 8 * j);
        double* Pan = X + b * nb * PAN_LD;
        if (warp == 0) {
            bad |= inv_panel(nb, ld, A, 8 * j, jb, lane, pos0, pos1, done0, done1, Pan, prow + 8 * b, pmask + 2 * b);
            if (j == nt - 1) {
                if (lane < nb) pos[lane] = pos0;
                if (lane + 32 < nb) pos[lane + 32] = pos1;
            }
        }
        T.sync();
        // the next panel's columns by all warps, the other columns by warps 1 to 3 (after the last panel by all)
        const bool end = j == nt - 1;
        if (!end) {
            inv_update(T, true, nb, ld, A, j + 1, jb, Pan, prow + 8 * b, pmask + 2 * b);
            T.sync();
        }
        for (int e = end ? warp : warp == 0 ? nt : warp - 1; e < (end ? nt - 1 : nt - 2); e += end ? 4 : 3)
            inv_update(T, false, nb, ld, A, (end || e < j) ? e : e + 2, jb, Pan, prow + 8 * b, pmask + 2 * b);
        __syncwarp();
    }
    T.sync();
    for (int r = warp; r < nb; r += 4) {          // the rows in their positions, the interchanges undone on the columns
        double* xp = X + pos[r] * ld;
        if (lane < nb) xp[lane] = A[r * ld + pos[lane]];
        if (lane + 32 < nb) xp[lane + 32] = A[r * ld + pos[lane + 32]];
    }
    T.sync();
    return bad;
}

// Inverse of the block A into X, by a team of 4 warps (the pointers may have been exchanged in all
// threads of the block: `odd`); blocked when X can hold two panels (24 nb doubles of nb ld) and the block is large
// enough for panels to pay (nb >= 21 in its own ld; smaller ones where the partition's largest block sets ld).
struct InvWork {
    double pv[8];
    int pi[8], perm[64], idx[64], pos[64], prow[16];
    unsigned pmask[4];
};
static __device__ __forceinline__ bool inv_blocked(int nb, int ld) {
    return 2 * PAN_LD <= ld && 16 * nb + 8 * ld <= nb * ld;
}
static __device__ __forceinline__ int tm_inverse(const Team& T, int nb, int ld, double* A, double* X, InvWork& W) {
    if (inv_blocked(nb, ld)) return tm_inverse_blk(T, nb, ld, A, X, W.pos, W.prow, W.pmask);
    return tm_inverse_unb(T, nb, ld, A, X, W.perm, W.idx, W.pv, W.pi);
}
// after tm_inverse, in every thread: X the inverse, A free (an odd number of unblocked steps ends in A)
static __device__ __forceinline__ void inv_swap(int nb, int ld, double*& A, double*& X) {
    if (!inv_blocked(nb, ld) && (nb & 1)) { double* t = A; A = X; X = t; }
}

// ---------------------------------------------------------------- clusters of two CTAs
static __device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
static __device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// a value in the shared memory of CTA `rank` of this cluster, at the address of *p in this CTA
static __device__ __forceinline__ double ld_peer_cta(const double* p, uint32_t rank) {
    uint32_t ra;
    double v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(ra) : "memory");
    return v;
}
static __device__ __forceinline__ int ld_peer_cta(const int* p, uint32_t rank) {
    uint32_t ra;
    int v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(ra) : "memory");
    return v;
}

// One CTA per partition (TW: per direction of a partition, a cluster of two), every working block
// resident in shared memory (nb <= PC_SMEM_NB).  The elimination runs in the CTA's local plane
// frame: rank 0 top-down over planes 0..zs-1, rank 1 bottom-up over planes Nz-1..zs+2, local
// slot sl of local plane t being global slot 4 - sl of plane Nz-1-t for rank 1.  TW: after its n
// planes each rank also forms the multipliers of the separator planes n, n+1 and their Schur contributions Q = -(couplings through
// the eliminated planes); rank 0 adds both ranks' Q to the separator blocks (read through
// distributed shared memory) and stores the inverse of the 2 nb x 2 nb separator matrix
// S = [S11 S12; S21 S22] by blocks (Dm = S11^-1, Dn = (S22 - S21 Dm S12)^-1):
//   plane zs:   slot 2 Sinv11 = Dm + Dm S12 Dn S21 Dm,  slot 3 Sinv12 = -Dm S12 Dn
//   plane zs+1: slot 1 Sinv21 = -Dn S21 Dm,             slot 2 Sinv22 = Dn
// so that the sweep solves the separator in two independent stages.
//
// What bounds it is the chain through the planes: L1 = (..) Uinv_{k-1}, D -= L1 U1_{k-1}, the inverse of D
// (a serial chain itself).  Four warps take the inverse; the other twelve do meanwhile what plane k's
// inverse does not need -- U1_k, the products of plane k-1 that are only stored, and from plane k+1
// L2 = A(k+1,k-1) Uinv_{k-1}, A(k+1,k) - L2 U1_{k-1}, A(k+1,k+1) - L2 U2_{k-1} -- with results that are only
// stored written from registers, so that nine blocks are enough.  The warps that share the panel warp's scheduler
// stay out of it: their DMMAs would keep its FP64 unit busy (514 us with them, 488 without).
// 8x8x32 (18 CTAs): 1190 -> 449 us; 16x16x64 (68): 2440 -> 861.  Of a plane's 135 000 cycles before, 79 000 were
// the inverse and the rest products and copies in turn with it; now the inverse is two thirds of 50 000.
constexpr int FAC_T = 512, FAC_INV = 128, FAC_HELP = 288;
static_assert(2 * FAC_HELP >= DV_NV * BD_LD, "two entries of U2 per thread");
static __device__ __forceinline__ void pc_prefetch(const double* b, int64_t n, int tid, int nt) {
    for (int64_t e = (int64_t)tid * 16; e < n; e += (int64_t)nt * 16) asm volatile("prefetch.global.L2 [%0];" ::"l"(b + e));
}
template <bool TW>
__global__ void __launch_bounds__(FAC_T) k_pc_factor_smem(PcGeom gin, double* __restrict__ Af, int* __restrict__ info, int lds) {
    const int rank = TW ? (int)(blockIdx.x & 1u) : 0;
    const int part = TW ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const PcGeom g = pc_part(gin, part);
    extern __shared__ __align__(128) double dsm[];
    __shared__ InvWork W;
    __shared__ double u2[DV_NV * BD_LD];       // U2_{k-1} = A(k-1, k+1) during plane k
    __shared__ int qoff[4], sbad;
    const int nb = g.nb, ld = g.ld;
    const int n2 = nb * lds;                   // one shared-memory block
    const int Nz = g.Nz;
    const int n = TW ? (rank == 0 ? g.zs : Nz - g.zs - 2) : Nz;
    const int tid = threadIdx.x;
    const bool inverts = tid < FAC_INV;
    const Team all{tid, FAC_T, 0};
    const int hw = ((tid >> 7) - 1) * 3 + ((tid >> 5) & 3) - 1;          // helping warp
    const bool helps = !inverts && ((tid >> 5) & 3) != 0;
    const Team mine{inverts ? tid : hw * 32 + (tid & 31), inverts ? FAC_INV : FAC_HELP, inverts ? 1 : 2};
    // D of the plane and of the next, (A(k,k-1) - ..), L1, L2 of the next, U1, Uinv_{k-1}, U1_{k-1}, Uinv
    double *S2 = dsm, *S2n = dsm + n2, *S1 = dsm + 2 * n2, *L1 = dsm + 3 * n2, *S0 = dsm + 4 * n2, *S3 = dsm + 5 * n2;
    double *Ui = dsm + 6 * n2, *U1 = dsm + 7 * n2, *X = dsm + 8 * n2;
    double* base = Af + (int64_t)part * Nz * 5 * g.bs;
    // block (local plane t, local slot sl)
    auto B = [&](int t, int sl) -> double* {
        const int P = (rank == 0) ? t : Nz - 1 - t;
        const int64_t off = ((int64_t)P * 5 + ((rank == 0) ? sl : 4 - sl)) * g.bs;
        // outside the partition's planes or the storage: recorded, and the partition's first block
        // stands in (the factors are then wrong and the error word says so)
        if (P < 0 || P >= Nz || !pc_range_ok(g, (int64_t)part * Nz * 5 * g.bs + off, g.bs)) return base;
        return base + off;
    };
    auto swap = [](double*& a, double*& b) { double* t = a; a = b; b = t; };
    int bad = 0;
    tm_copy(all, nb, B(0, 2), ld, S2, lds);
    all.sync();
    for (int k = 0; k < n; ++k) {
        if (k >= 1) {
            if (k == 1) tm_bd_left(all, nb, g.ncv, lds, S1, lds, Ui, L1);                    // L1 = A(1,0) Uinv_0
            else tm_gemm(all, nb, lds, 1, S1, Ui, nullptr, 0, L1, lds);              // L1 = (...) Uinv_{k-1}
            all.sync();
            tm_gemm(all, nb, lds, -1, L1, U1, S2, lds, S2, lds);                     // D -= L1 U1_{k-1}
            all.sync();
        }
        if (inverts) {
            bad |= tm_inverse(mine, nb, lds, S2, X, W);
            double *a = S2, *x = X;
            inv_swap(nb, lds, a, x);
            tm_copy(mine, nb, x, lds, B(k, 2), ld);
        } else if (helps) {
            const bool next = k + 1 < n || TW;
            const double u2a = bd_entry(g, mine.tid, B(k, 4), ld);                   // U2_k, for the next plane
            const double u2b = mine.tid + FAC_HELP < DV_NV * BD_LD ? bd_entry(g, mine.tid + FAC_HELP, B(k, 4), ld) : 0.0;
            if (k + 2 < Nz) pc_prefetch(B(k + 2, rank == 0 ? 0 : 4), 5 * g.bs, mine.tid, mine.n);
            if (k >= 1) {
                if (next) tm_bd_left(mine, nb, g.ncv, lds, B(k + 1, 0), ld, Ui, S0);         // L2 = A(k+1,k-1) Uinv_{k-1}
                tm_bd_right(mine, nb, g.ncv, lds, L1, u2, B(k, 3), ld, S3, lds);            // U1 = A(k,k+1) - L1 U2_{k-1}
                tm_gemm(mine, nb, lds, -1, Ui, U1, nullptr, 0, B(k - 1, 3), ld);     // -Uinv_{k-1} U1_{k-1}
                tm_copy(mine, nb, L1, lds, B(k, 1), ld);
            } else {
                tm_copy(mine, nb, B(0, 3), ld, S3, lds);
                if (next) {
                    tm_copy(mine, nb, B(1, 1), ld, S1, lds);
                    tm_copy(mine, nb, B(1, 2), ld, S2n, lds);
                }
            }
            if (next && k >= 1) {
                mine.sync();                                                         // L2 complete, U2 and A(k+1,k-1) read
                tm_gemm(mine, nb, lds, -1, S0, U1, B(k + 1, 1), ld, S1, lds);        // A(k+1,k) - L2 U1_{k-1}
                // A(k+1,k+1) - L2 U2_{k-1}; of a separator plane the Schur contribution alone
                tm_bd_right(mine, nb, g.ncv, lds, S0, u2, k + 1 < n ? B(k + 1, 2) : nullptr, ld, S2n, lds);
                tm_copy(mine, nb, S0, lds, B(k + 1, 0), ld);
                tm_bd_right(mine, nb, g.ncv, lds, Ui, u2, nullptr, 0, B(k - 1, 4), ld);     // -Uinv_{k-1} U2_{k-1}
            }
            mine.sync();
            u2[mine.tid] = u2a;
            if (mine.tid + FAC_HELP < DV_NV * BD_LD) u2[mine.tid + FAC_HELP] = u2b;
        }
        all.sync();
        inv_swap(nb, lds, S2, X);
        swap(Ui, X);
        swap(U1, S3);
        swap(S2, S2n);
    }
    tm_gemm(all, nb, lds, -1, Ui, U1, nullptr, 0, B(n - 1, 3), ld);                  // -Uinv_{n-1} U1_{n-1}
    if constexpr (!TW) {
        // slot 4 of the last two planes: U2_k = A(k, k+2) = 0 for k >= Nz-2 (zeroed at assembly)
        if (tid == 0) info[part] = bad;
    } else {
        // separator plane n (L2_n, A(n,n-1) - L2 U1_{n-2} and -L2 U2_{n-2} are there), plane n+1: coupled to n-1 only
        tm_gemm(all, nb, lds, 1, S1, Ui, nullptr, 0, L1, lds);                       // L1_n = (...) Uinv_{n-1}
        tm_bd_left(all, nb, g.ncv, lds, B(n + 1, 0), ld, Ui, S0);                            // L2_{n+1} = A(n+1,n-1) Uinv_{n-1}
        all.sync();
        double *Q00 = S2, *Q01 = S3, *Q10 = X, *Q11 = S2n;
        tm_gemm(all, nb, lds, -1, L1, U1, Q00, lds, Q00, lds);                       // Q(n,n) -= L1 U1_{n-1}
        tm_bd_right(all, nb, g.ncv, lds, L1, u2, nullptr, 0, Q01, lds);                     // Q(n,n+1) = -L1 U2_{n-1}
        tm_gemm(all, nb, lds, -1, S0, U1, nullptr, 0, Q10, lds);                     // Q(n+1,n) = -L2 U1_{n-1}
        tm_bd_right(all, nb, g.ncv, lds, S0, u2, nullptr, 0, Q11, lds);                     // Q(n+1,n+1) = -L2 U2_{n-1}
        tm_bd_right(all, nb, g.ncv, lds, Ui, u2, nullptr, 0, B(n - 1, 4), ld);              // -Uinv_{n-1} U2_{n-1}
        tm_copy(all, nb, L1, lds, B(n, 1), ld);
        tm_copy(all, nb, S0, lds, B(n + 1, 0), ld);
        if (tid == 0) {
            qoff[0] = (int)(Q00 - dsm);
            qoff[1] = (int)(Q01 - dsm);
            qoff[2] = (int)(Q10 - dsm);
            qoff[3] = (int)(Q11 - dsm);
            sbad = bad;
        }
        __syncthreads();
        cluster_sync_all();                                                    // both ranks hold Q
        // rank 0: S = A_sep + Q(rank 0) + Q(rank 1); rank 1's local block (a, b) is separator (1-a, 1-b)
        double* Sb[4] = {Q00, Q01, Q10, Q11};                                  // separator (0,0) (0,1) (1,0) (1,1)
        if (rank == 0) {
            const double* Ab[4] = {B(n, 2), B(n, 3), B(n + 1, 1), B(n + 1, 2)};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int ro = ld_peer_cta(&qoff[3 - q], 1u);
#pragma unroll 2
                for (int r = tid >> 5; r < nb; r += FAC_T / 32)
                    for (int c = tid & 31; c < nb; c += 32) {
                        const int es = r * lds + c;
                        Sb[q][es] = (Ab[q][r * ld + c] + Sb[q][es]) + ld_peer_cta(dsm + ro + es, 1u);
                    }
            }
            if (tid == 0) bad |= ld_peer_cta(&sbad, 1u);
        }
        __syncthreads();
        cluster_sync_all();                                                    // rank 1's blocks have been read
        if (rank == 0) {
            double *S11 = Sb[0], *S12 = Sb[1], *S21 = Sb[2], *S22 = Sb[3];
            double *Xn = S0, *Y = S1, *T = L1;                                 // free: S0, S1, L1, Ui, U1
            if (inverts) bad |= tm_inverse(mine, nb, lds, S11, T, W);          // Dm = S11^-1
            all.sync();
            inv_swap(nb, lds, S11, T);
            swap(S11, T);
            tm_gemm(all, nb, lds, -1, S11, S12, nullptr, 0, Xn, lds);          // Xn = -Dm S12
            tm_gemm(all, nb, lds, 1, S21, S11, nullptr, 0, Y, lds);            // Y = S21 Dm
            all.sync();
            tm_gemm(all, nb, lds, 1, S21, Xn, S22, lds, S22, lds);             // S22 - S21 Dm S12
            all.sync();
            if (inverts) bad |= tm_inverse(mine, nb, lds, S22, T, W);          // Dn = Sinv22
            all.sync();
            inv_swap(nb, lds, S22, T);
            swap(S22, T);
            tm_gemm(all, nb, lds, 1, Xn, S22, nullptr, 0, S12, lds);           // Sinv12 = Xn Dn
            tm_gemm(all, nb, lds, -1, S22, Y, nullptr, 0, S21, lds);           // Sinv21 = -Dn Y
            all.sync();
            tm_gemm(all, nb, lds, -1, S12, Y, S11, lds, B(n, 2), ld);          // Sinv11 = Dm - Sinv12 Y
            tm_copy(all, nb, S12, lds, B(n, 3), ld);
            tm_copy(all, nb, S21, lds, B(n + 1, 1), ld);
            tm_copy(all, nb, S22, lds, B(n + 1, 2), ld);
            if (tid == 0) info[part] = bad;
        }
    }
}

// ---------------------------------------------------------------- global-memory fallback (large blocks)
// C = beta C + alpha A B, row-major (leading dimension ld) in global memory; 256 threads, 32x32 tiles.
static __device__ void cta_gemm(int nb, int ld, double alpha, const double* A, const double* B, double beta,
                                double* C, double* shA, double* shB) {
    const int tid = threadIdx.x;
    const int tc = tid % 32, tr4 = (tid / 32) * 4;
    for (int ti = 0; ti < nb; ti += 32) {
        for (int tj = 0; tj < nb; tj += 32) {
            double acc[4] = {0.0, 0.0, 0.0, 0.0};
            for (int kk = 0; kk < nb; kk += 32) {
                for (int q = tid; q < 1024; q += blockDim.x) {
                    int r = q / 32, cc = q % 32;
                    int gr = ti + r, gk = kk + cc;
                    shA[r * 32 + cc] = (gr < nb && gk < nb) ? A[(int64_t)gr * ld + gk] : 0.0;
                    int gk2 = kk + r, gc = tj + cc;
                    shB[r * 32 + cc] = (gk2 < nb && gc < nb) ? B[(int64_t)gk2 * ld + gc] : 0.0;
                }
                __syncthreads();
#pragma unroll 8
                for (int q = 0; q < 32; ++q) {
                    double b = shB[q * 32 + tc];
#pragma unroll
                    for (int u = 0; u < 4; ++u) acc[u] += shA[(tr4 + u) * 32 + q] * b;
                }
                __syncthreads();
            }
            const int gc = tj + tc;
            if (gc < nb) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    int gr = ti + tr4 + u;
                    if (gr < nb) {
                        double* cp = C + (int64_t)gr * ld + gc;
                        *cp = (beta == 0.0) ? alpha * acc[u] : beta * (*cp) + alpha * acc[u];
                    }
                }
            }
        }
    }
    __syncthreads();
}

static __device__ void cta_copy(int64_t n, const double* src, double* dst) {
    for (int64_t q = threadIdx.x; q < n; q += blockDim.x) dst[q] = src[q];
    __syncthreads();
}

// Gauss-Jordan inverse of the row-major D (leading dimension ld) through an augmented scratch W
// (nb x 2nb, column-major over the augmented matrix).  Reading D column-major inverts D^T; the
// inverse of the transpose is the transpose of the inverse, so writing back the same way yields
// the row-major inverse.
static __device__ int cta_inverse(int nb, int ld, double* D, double* W, double* red_v, int* red_i) {
    const int tid = threadIdx.x;
    const int64_t n2 = (int64_t)nb * nb;
    for (int64_t q = tid; q < 2 * n2; q += blockDim.x) {
        int64_t col = q / nb, row = q % nb;
        W[q] = (col < nb) ? D[col * ld + row] : ((col - nb) == row ? 1.0 : 0.0);
    }
    __syncthreads();
    int bad = 0;
    for (int pc = 0; pc < nb; ++pc) {
        double best = -1.0;
        int bi = pc;
        for (int r = pc + tid; r < nb; r += blockDim.x) {
            double v = fabs(W[(int64_t)pc * nb + r]);
            if (v > best || (v == best && r < bi)) { best = v; bi = r; }
        }
        red_v[tid] = best;
        red_i[tid] = bi;
        __syncthreads();
        for (int s = blockDim.x / 2; s > 0; s >>= 1) {
            if (tid < s) {
                double ov = red_v[tid + s];
                int oi = red_i[tid + s];
                if (ov > red_v[tid] || (ov == red_v[tid] && oi < red_i[tid])) { red_v[tid] = ov; red_i[tid] = oi; }
            }
            __syncthreads();
        }
        const int pr = red_i[0];
        const double pmax = red_v[0];
        __syncthreads();
        if (pr != pc) {
            for (int c = pc + tid; c < 2 * nb; c += blockDim.x) {
                double a = W[(int64_t)c * nb + pc];
                W[(int64_t)c * nb + pc] = W[(int64_t)c * nb + pr];
                W[(int64_t)c * nb + pr] = a;
            }
        }
        __syncthreads();
        double piv = W[(int64_t)pc * nb + pc];
        if (!(pmax > 0.0) || !isfinite(piv)) {
            bad = 1;
            piv = 1.0;
        }
        const double inv = 1.0 / piv;
        __syncthreads();
        for (int c = pc + 1 + tid; c < 2 * nb; c += blockDim.x) W[(int64_t)c * nb + pc] *= inv;
        __syncthreads();
        const int64_t ncols = 2 * nb - (pc + 1);
        for (int64_t q = tid; q < ncols * nb; q += blockDim.x) {
            int c = pc + 1 + (int)(q / nb);
            int r = (int)(q % nb);
            if (r == pc) continue;
            double fr = W[(int64_t)pc * nb + r];
            if (fr != 0.0) W[(int64_t)c * nb + r] -= fr * W[(int64_t)c * nb + pc];
        }
        __syncthreads();
    }
    for (int64_t q = tid; q < n2; q += blockDim.x) {
        int64_t col = q / nb, row = q % nb;
        D[col * ld + row] = W[n2 + q];
    }
    __syncthreads();
    return bad;
}

__global__ void __launch_bounds__(256) k_pc_factor_glob(PcGeom gin, double* __restrict__ A, double* __restrict__ work,
                                                        int* __restrict__ info, int use_smem) {
    const PcGeom g = pc_part(gin, (int)blockIdx.x);
    extern __shared__ double dsm[];
    __shared__ double shA[1024], shB[1024];
    __shared__ double red_v[256];
    __shared__ int red_i[256];
    const int part = blockIdx.x;
    const int nb = g.nb, ld = g.ld;
    const int64_t n2 = (int64_t)nb * ld;
    const int64_t bs = g.bs;
    if (!pc_range_ok(g, (int64_t)part * g.Nz * 5 * bs, (int64_t)g.Nz * 5 * bs)) return;   // geometry beyond the storage
    double* base = A + (int64_t)part * g.Nz * 5 * bs;
    const int64_t n2w = (int64_t)gin.nb * ld;          // workspace stride: the largest partition's block
    double* T = work + (int64_t)part * 4 * n2w;
    double* W = use_smem ? dsm : (T + n2w);
    int bad = 0;
    for (int k = 0; k < g.Nz; ++k) {
        double* Ak = base + (int64_t)k * 5 * bs;
        double* Am2 = Ak;
        double* Am1 = Ak + bs;
        double* A0 = Ak + 2 * bs;
        double* Ap1 = Ak + 3 * bs;
        double* Uinv_1 = (k >= 1) ? base + ((int64_t)(k - 1) * 5 + 2) * bs : nullptr;
        double* U1_1 = (k >= 1) ? base + ((int64_t)(k - 1) * 5 + 3) * bs : nullptr;
        double* U2_1 = (k >= 1) ? base + ((int64_t)(k - 1) * 5 + 4) * bs : nullptr;
        double* Uinv_2 = (k >= 2) ? base + ((int64_t)(k - 2) * 5 + 2) * bs : nullptr;
        double* U1_2 = (k >= 2) ? base + ((int64_t)(k - 2) * 5 + 3) * bs : nullptr;
        double* U2_2 = (k >= 2) ? base + ((int64_t)(k - 2) * 5 + 4) * bs : nullptr;
        if (k >= 2) {
            cta_gemm(nb, ld, 1.0, Am2, Uinv_2, 0.0, T, shA, shB);
            cta_copy(n2, T, Am2);
            cta_gemm(nb, ld, -1.0, Am2, U1_2, 1.0, Am1, shA, shB);
            cta_gemm(nb, ld, -1.0, Am2, U2_2, 1.0, A0, shA, shB);
        }
        if (k >= 1) {
            cta_gemm(nb, ld, 1.0, Am1, Uinv_1, 0.0, T, shA, shB);
            cta_copy(n2, T, Am1);
            cta_gemm(nb, ld, -1.0, Am1, U1_1, 1.0, A0, shA, shB);
            cta_gemm(nb, ld, -1.0, Am1, U2_1, 1.0, Ap1, shA, shB);
        }
        bad |= cta_inverse(nb, ld, A0, W, red_v, red_i);
    }
    // fused-sweep form: slot 3 <- -Uinv_k U1_k, slot 4 <- -Uinv_k U2_k
    for (int k = 0; k < g.Nz; ++k) {
        double* Ak = base + (int64_t)k * 5 * bs;
        for (int slot = 3; slot <= 4; ++slot) {
            cta_gemm(nb, ld, -1.0, Ak + 2 * bs, Ak + slot * bs, 0.0, T, shA, shB);
            cta_copy(n2, T, Ak + slot * bs);
        }
    }
    if (threadIdx.x == 0) info[part] = bad;
}

// ---------------------------------------------------------------- sweeps
// Plane frame of one elimination direction.  TW = false: planes 0..Nz-1 top-down (the whole
// partition).  TW = true (twisted factorisation, a cluster of two CTAs per partition): rank 0
// eliminates planes 0..zs-1 top-down, rank 1 planes Nz-1..zs+2 bottom-up, and the separator
// planes zs, zs+1 take both ranks' contributions and an explicit inverse of their own.  In its
// local frame each rank sees planes
// t = 0, 1, .. (global gp(t)) with slot sl holding the coupling to local plane t + sl - 2, which is
// global slot gs(sl): bottom-up, A(t, t-1) local is A(p, p+1) global, and so on.  The local
// eliminated planes are 0..n-1; local n and n+1 are the separator planes.
struct PcFrame {
    int rank, n, Nz;
    __device__ __forceinline__ int gp(int t) const { return rank == 0 ? t : Nz - 1 - t; }
    __device__ __forceinline__ int gs(int sl) const { return rank == 0 ? sl : 4 - sl; }
};

// x = diag(1/sc) M^-1 diag(sc) b for all partitions: one CTA per partition, or per direction of a
// partition (TW).  Eight lanes take two rows of a plane's blocks; NJ = ld / 16: lane l holds the column
// pairs (2l + 16j, 2l + 16j + 1), j < NJ, of its rows.  The factors go from global memory (L2) straight
// into registers, two stages ahead of their use, and only the solution planes live in shared memory:
// nothing of a stage but its newest plane is read after the barrier, and the plane before it stays in
// registers.  Padding columns hold zeros.
// Stages of one CTA (local frame):
//   F(t), t = 1..n-1:   z_t = b_t - L1_t z_{t-1} - L2_t z_{t-2}                  (slots 0, 1)
//   TW only:
//   X:                  p_n = b_n - L1_n z_{n-1} - L2_n z_{n-2},  p_{n+1} = b_{n+1} - L2_{n+1} z_{n-1}
//                       (b of the separator read by rank 0 only); the two ranks' p are summed
//                       through distributed shared memory into r
//   C0, C1:             the separator (both ranks; r_m, r_m1: global planes zs, zs+1)
//                       x of local plane n + i = [Sinv blocks of that plane] [r_m; r_m1]
//   B(t), t = n-1..0:   x_t = Uinv_t z_t + (-Uinv_t U1_t) x_{t+1} + (-Uinv_t U2_t) x_{t+2}  (slots 2..4)
// Without TW the backward stages run t = Nz-1..0 (couplings beyond the last plane are absent).
// A row's sum runs over its blocks in the order written above, then over the lanes by a butterfly.
// What bounds it: 8x8x32 (18 CTAs, 26.5 MB in L2) 19.3 us a launch, 0.46 us a stage: the stage's 37 to 55
// KB come from L2 at 50 bytes a cycle and SM, 4.5 us are before the first stage and after the last.  A
// three-deep ring of bulk copies in shared memory, whose blocks then crossed shared memory twice more,
// took 30.6 us; one row per lane group (twice the shared-memory reads of the planes) 23.6 us.  8x8x12: 15.3
// -> 10.0 us, 16x16x64: 57.3 -> 46.4 us (182 MB at 4.0 TB/s).
#define PA_LANES 8
#define PA_DEPTH 2         // stages whose factors are in flight ahead of their use
// Factors that do not stay in L2 (126 MB) from one sweep to the next are also prefetched into it, PA_AHEAD
// stages ahead.  The line lies between 86 MB, where prefetching what is already there costs 4 % (12x12x48:
// 27.4 -> 28.6 us), and 94 MB, where it gains 23 % (4x64x48 in sectors: 33.4 -> 25.8 us; 16x16x64 in FP32, 100 MB:
// 50.5 -> 47.4); at 162 MB 50.8 -> 36.8 us (5x64x64 in sectors), at 182 MB 57.6 -> 46.5 us (16x16x64; 8 stages
// ahead: 46.9, 16: 55.6).
#define PA_AHEAD 4
#define PA_L2_BYTES (90ll << 20)
#define PA_IO 4            // entries per thread whose loads the prologue / epilogue batch
#define PA_SUM 256         // the result's sum of squares is taken over this many strided parts, warp by warp
constexpr int pa_threads(int NJ) { return NJ <= 2 ? 128 : 64 * NJ; }       // 8 NJ row pairs of 8 lanes

// stages of a CTA that holds np planes, at most (both ranks)
constexpr int pa_stages(int np, bool tw) { return tw ? 2 * np - 2 : 2 * np - 1; }
// The kernel's last parameter ALT.  Twisted: prefetch into L2 as above.  Top-down: a stage's blocks are worked out
// when they are fetched, instead of looked up in a table in shared memory -- only where small blocks in a long
// column leave no room for the table beside the planes (1x1x806 in FP64 and beyond), as it is slower (1x1x700:
// 324 -> 368 us, 4x1x200: 143 -> 154).

template <int NJ, typename TS, bool TW, bool ALT>
__global__ void __launch_bounds__(pa_threads(NJ), 1) k_pc_apply(PcGeom gin, const TS* __restrict__ A,
                                                                const double* __restrict__ b,
                                                                const double* __restrict__ sc, double* __restrict__ x,
                                                                PaFuse F) {
    pdl_wait();                                // (launched programmatically inside the GMRES graph)
    pdl_trigger();
    extern __shared__ __align__(128) double dsm[];
    constexpr int LD = NJ * 2 * PA_LANES, NT = pa_threads(NJ), DEPTH = PA_DEPTH;
    constexpr bool AH = TW && ALT, TABLE = TW || !ALT;
    using TS2 = typename std::conditional<std::is_same<TS, float>::value, float2, double2>::type;
    const int rank = TW ? (int)(blockIdx.x & 1u) : 0;
    const int part = TW ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const PcGeom g = pc_part(gin, part);
    const int nb = g.nb, Nz = g.Nz;
    const int tid = threadIdx.x;
    const int bs = (int)g.bs;
    const PcFrame fr{rank, TW ? (rank == 0 ? g.zs : Nz - g.zs - 2) : Nz, Nz};
    const int n = fr.n;
    // local planes held (the same on both ranks: each reads the other's xch at its own address)
    const int np = TW ? max(g.zs, Nz - g.zs - 2) + 2 : Nz;
    const int S = TW ? 2 * n + 2 : 2 * Nz - 1;
    double* xs = dsm;                          // [np][LD] local planes: b, then z (forward, in place); r on the separator
    double* xb = xs + np * LD;                 // [np][LD]: x (backward sweep); padding columns zero
    double* xch = xb + np * LD;                // [2][LD]: this rank's partial right-hand sides of the separator (TW)
    int4* desc = reinterpret_cast<int4*>(xch + 2 * LD);     // [S + DEPTH] (table): offsets of a stage's blocks (-1: none)
    int* gl = reinterpret_cast<int*>(desc + (TABLE ? pa_stages(np, TW) + DEPTH : 0));     // [LD]: state index of row l at plane 0
    const int stopped = F.stop ? *F.stop : 0;
    const int fcol = F.V ? *F.col : 0;
    const double fscale = F.V ? *F.scale : 0.0;
    // a geometry beyond the storage is recorded and x is left untouched (the same on every CTA of a partition)
    if (!pc_range_ok(g, (int64_t)part * Nz * 5 * bs, (int64_t)Nz * 5 * bs)) return;
    const TS* base = A + (int64_t)part * Nz * 5 * bs;
    // a stage's blocks, in the order their products are added
    auto blocks = [&](int s, int (&o)[3]) {
        o[0] = o[1] = o[2] = -1;
        auto blk = [&](int t, int sl) { return (fr.gp(t) * 5 + fr.gs(sl)) * bs; };
        if (s >= S) {
        } else if (s < n - 1) {                            // F(t), t = s + 1
            o[0] = blk(s + 1, 1);
            if (s >= 1) o[1] = blk(s + 1, 0);
        } else if (TW && s == n - 1) {                     // X
            o[0] = blk(n, 1);
            o[1] = blk(n, 0);
            o[2] = blk(n + 1, 0);
        } else if (TW && s <= n + 1) {                     // C(i): the separator plane's two Sinv blocks
            const int P = fr.gp(s);
            o[0] = (P * 5 + (P == g.zs ? 2 : 1)) * bs;
            o[1] = o[0] + bs;
        } else {                                           // B(t)
            const int t = TW ? 2 * n + 1 - s : 2 * Nz - 2 - s;
            o[0] = blk(t, 2);
            if (TW || t + 1 < Nz) o[1] = blk(t, 3);
            if (TW || t + 2 < Nz) o[2] = blk(t, 4);
        }
    };
    for (int s = TABLE ? tid : S + DEPTH; s < S + DEPTH; s += NT) {
        int o[3];
        blocks(s, o);
        // (the blocks of a stage are one run of slots, but for X's third: the run's first and its blocks)
        const bool x3 = TW && s == n - 1;
        const int first = o[1] < 0 ? o[0] : (o[2] < 0 || x3) ? min(o[0], o[1]) : min(o[0], o[2]);
        const int cnt = o[0] < 0 ? 0 : o[1] < 0 ? 1 : (o[2] < 0 || x3) ? 2 : 3;
        desc[s] = make_int4(o[0], o[1], o[2], s < S ? (first / bs) * 4 + cnt : 0);
    }
    if (tid < LD) {
        int64_t gi = -1;
        if (tid < nb) {
            gi = pc_glob(g, part, 0, tid);                 // (plane k of the row: gi + k)
            if (gi < 0 || gi + Nz > g.nstate) {
                if (g.err) atomicOr(g.err, PC_ERR_RANGE);
                gi = -1;
            }
        }
        gl[tid] = (int)gi;
    }
    __syncthreads();
    const int lane = tid % PA_LANES, rh = (nb + 1) >> 1;
    const int r0 = tid / PA_LANES, r1 = r0 + rh;            // rows of this group
    const bool put0 = r0 < rh && lane == 0, put1 = put0 && r1 < nb;
    // this lane's first pair of its rows in slot 0, plane 0 (a row beyond the plane reads row 0 and is not stored)
    const TS* mine0 = base + (r0 < rh ? r0 : 0) * LD + 2 * lane;
    const TS* mine1 = base + (r0 < rh && r1 < nb ? r1 : 0) * LD + 2 * lane;
    struct Blk {
        TS2 a[NJ], b[NJ];
    };
    Blk R[DEPTH][3];
    auto load = [&](int s, Blk (&M)[3]) {
        int o[3];
        if constexpr (TABLE) {
            const int4 d = desc[s];
            o[0] = d.x, o[1] = d.y, o[2] = d.z;
        } else {
            blocks(s, o);
        }
#pragma unroll
        for (int e = 0; e < 3; ++e)
            if (o[e] >= 0) {
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    M[e].a[j] = __ldg(reinterpret_cast<const TS2*>(mine0 + o[e]) + PA_LANES * j);
                    M[e].b[j] = __ldg(reinterpret_cast<const TS2*>(mine1 + o[e]) + PA_LANES * j);
                }
            }
    };
    // stages beyond the ones in registers, into L2 (factors larger than L2)
    auto prefetch = [&](int s) {
        if (s >= S) return;
        const int w = desc[s].w;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;"
                     ::"l"(base + (int64_t)(w >> 2) * bs), "r"((uint32_t)((w & 3) * bs * (int)sizeof(TS))) : "memory");
    };
    if (AH && tid >= DEPTH && tid < PA_AHEAD) prefetch(tid);
    // buffer u serves the stages congruent to rem + u, so that X (without TW the first backward stage) is 0's
    const int nf = n - 1;                      // forward stages
    const int rem = nf % DEPTH;
#pragma unroll
    for (int u = 0; u < DEPTH; ++u) load(min((rem + u) % DEPTH, S), R[u]);
    // an Arnoldi step after the solve stopped: a zero direction (every CTA of the grid returns here)
    if (stopped) {
        if (blockIdx.x == 0 && tid == 0 && F.out) *F.out = 0.0;
        return;
    }
    const double* __restrict__ src = F.V ? ((F.src0 == F.src1 || fcol != 0) ? F.src1 : F.src0) : b;
    // b (or the basis vector to normalise) into xs: PA_IO entries per thread at a time, all their
    // loads issued before the first use; rank 1 leaves the separator's b to rank 0
    const int nio = TW ? (rank == 0 ? n + 2 : n) : Nz;
    for (int q0 = tid; q0 < np * LD; q0 += PA_IO * NT) {
        int gi[PA_IO];
        double bv[PA_IO], sv[PA_IO];
#pragma unroll
        for (int u = 0; u < PA_IO; ++u) {
            const int q = q0 + u * NT;
            const int t = q / LD, l = q - t * LD;
            gi[u] = (t < nio && gl[l] >= 0) ? gl[l] + fr.gp(t) : -1;
            bv[u] = gi[u] >= 0 ? src[gi[u]] : 0.0;
            sv[u] = (gi[u] >= 0 && sc) ? sc[gi[u]] : 1.0;
        }
#pragma unroll
        for (int u = 0; u < PA_IO; ++u) {
            const int q = q0 + u * NT;
            if (q >= np * LD) break;
            double v = 0.0;
            if (gi[u] >= 0) {
                double x0 = bv[u];
                if (F.V) {                       // normalise the basis vector on the way in
                    x0 = fscale * x0;
                    F.V[(int64_t)fcol * F.ldv + gi[u]] = x0;
                }
                v = sc ? x0 * sv[u] : x0;
            }
            xs[q] = v;
            xb[q] = 0.0;
        }
    }
    __syncthreads();
    // a plane's entries at this lane's columns
    struct Vec {
        double2 v[NJ];
    };
    auto plane = [&](const double* p, Vec& o) {
        const double2* vp = reinterpret_cast<const double2*>(p) + lane;
#pragma unroll
        for (int j = 0; j < NJ; ++j) o.v[j] = vp[PA_LANES * j];
    };
    auto dot = [&](const Blk& M, const Vec& o, double& a0, double& a1) {
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            a0 += (double)M.a[j].x * o.v[j].x;
            a1 += (double)M.b[j].x * o.v[j].x;
            a0 += (double)M.a[j].y * o.v[j].y;
            a1 += (double)M.b[j].y * o.v[j].y;
        }
    };
    auto reduce = [&](double& a0, double& a1) {
#pragma unroll
        for (int off = PA_LANES / 2; off > 0; off >>= 1) {
            a0 += __shfl_xor_sync(0xffffffffu, a0, off, PA_LANES);
            a1 += __shfl_xor_sync(0xffffffffu, a1, off, PA_LANES);
        }
    };
    auto store = [&](double* p, double a0, double a1) {
        if (put0) p[r0] = a0;
        if (put1) p[r1] = a1;
    };
    // One barrier per stage: it publishes the previous stage's rows.  Forward rows overwrite b_t by z_t in
    // xs (each row reads and writes only its own entry of plane t); backward rows go to xb.  V[u] takes the
    // newest plane of a stage served by buffer u, so V[u ^ 1] still holds the one before it.  The code of
    // both loops is kept small: a launch runs through it once, from a cold instruction cache.
    static_assert(DEPTH == 2, "V alternates with the buffers");
    Vec V[2];
#pragma unroll 1
    for (int s0 = rem ? rem - DEPTH : 0; s0 < nf; s0 += DEPTH) {
#pragma unroll
        for (int u = 0; u < DEPTH; ++u) {
            const int s = s0 + u;
            if (s < 0) continue;
            double* o = xs + (s + 1) * LD;
            const double b0 = put0 ? o[r0] : 0.0, b1 = put1 ? o[r1] : 0.0;
            __syncthreads();
            plane(xs + s * LD, V[u]);
            double a0 = 0.0, a1 = 0.0;
            dot(R[u][0], V[u], a0, a1);
            if (s >= 1) dot(R[u][1], V[u ^ 1], a0, a1);
            load(s + DEPTH, R[u]);
            if (AH && tid == 0) prefetch(s + PA_AHEAD);
            reduce(a0, a1);
            store(o, b0 - a0, b1 - a1);
        }
    }
    if constexpr (TW) {
        {                                        // X: partial right-hand sides of the separator
            __syncthreads();
            plane(xs + (n - 1) * LD, V[0]);
            double a0 = 0.0, a1 = 0.0, c0 = 0.0, c1 = 0.0;
            dot(R[0][0], V[0], a0, a1);
            dot(R[0][1], V[1], a0, a1);
            dot(R[0][2], V[0], c0, c1);
            load(n - 1 + DEPTH, R[0]);
            if (AH && tid < 3) prefetch(n - 1 + tid + PA_AHEAD);      // (and C0's and C1's)
            reduce(a0, a1);
            reduce(c0, c1);
            const double* p = xs + n * LD;
            store(xch, (put0 ? p[r0] : 0.0) - a0, (put1 ? p[r1] : 0.0) - a1);
            store(xch + LD, (put0 ? p[LD + r0] : 0.0) - c0, (put1 ? p[LD + r1] : 0.0) - c1);
        }
        cluster_sync_all();                      // both ranks' partials are in xch (both always arrive)
        const uint32_t other = (uint32_t)(fr.rank ^ 1);
        for (int q = tid; q < 2 * LD; q += NT) {
            const int c = q / LD, l = q - c * LD;       // separator plane zs + c, row l
            if (l >= nb) continue;
            // plane zs + c is slot c of rank 0's xch and slot 1 - c of rank 1's; the sum is
            // taken in the same order on both ranks, so both hold the same r
            const double* q0 = xch + c * LD + l;
            const double* q1 = xch + (1 - c) * LD + l;
            const double p0 = (fr.rank == 0) ? *q0 : ld_peer_cta(q0, other);
            const double p1 = (fr.rank == 0) ? ld_peer_cta(q1, other) : *q1;
            xs[(n + ((fr.rank == 0) ? c : 1 - c)) * LD + l] = p0 + p1;
        }
        __syncthreads();
        {                                        // C0, C1: both ranks solve the separator
            const int lz0 = (fr.rank == 0) ? n : n + 1;     // local plane of global zs
            plane(xs + lz0 * LD, V[0]);
            plane(xs + (2 * n + 1 - lz0) * LD, V[1]);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                Blk (&M)[3] = R[(1 + e) % DEPTH];
                double a0 = 0.0, a1 = 0.0;
                dot(M[0], V[0], a0, a1);
                dot(M[1], V[1], a0, a1);
                load(n + e + DEPTH, M);
                reduce(a0, a1);
                store(xb + (n + e) * LD, a0, a1);
            }
        }
    }
    __syncthreads();                             // planes read ahead of the first barrier below
    if (TW) plane(xb + (n + 1) * LD, V[1]);
    constexpr int B0 = TW ? 3 : 0;               // buffer of the first backward stage
    const int lim = TW ? n + 2 : Nz;
#pragma unroll 1
    for (int s0 = TW ? n + 2 : Nz - 1; s0 < S; s0 += DEPTH) {
#pragma unroll
        for (int u = 0; u < DEPTH; ++u) {
            const int s = s0 + u;
            if (s >= S) break;
            Blk (&M)[3] = R[(B0 + u) % DEPTH];
            const int t = TW ? 2 * n + 1 - s : 2 * Nz - 2 - s;
            Vec zt;
            plane(xs + t * LD, zt);
            double a0 = 0.0, a1 = 0.0;
            dot(M[0], zt, a0, a1);
            __syncthreads();
            if (TW || t + 1 < lim) {
                plane(xb + (t + 1) * LD, V[u]);
                dot(M[1], V[u], a0, a1);
            }
            if (TW || t + 2 < lim) dot(M[2], V[u ^ 1], a0, a1);
            load(s + DEPTH, M);
            if (AH && tid == 0) prefetch(s + PA_AHEAD);
            reduce(a0, a1);
            store(xb + t * LD, a0, a1);
        }
    }
    __syncthreads();                             // the last stage's rows
    // x out, and its sum of squares: part vt takes the entries congruent to vt, in order
    __shared__ double wsum[PA_SUM / 32];
    for (int vt = tid; vt < PA_SUM; vt += NT) {
        double ss = 0.0;
        for (int q0 = vt; q0 < nio * LD; q0 += PA_IO * PA_SUM) {     // PA_IO entries at a time
            int gi[PA_IO];
            double sv[PA_IO];
#pragma unroll
            for (int u = 0; u < PA_IO; ++u) {
                const int q = q0 + u * PA_SUM;
                const int t = q / LD, l = q - t * LD;
                gi[u] = (t < nio && gl[l] >= 0) ? gl[l] + fr.gp(t) : -1;
                sv[u] = (gi[u] >= 0 && sc) ? sc[gi[u]] : 1.0;
            }
#pragma unroll
            for (int u = 0; u < PA_IO; ++u) {
                if (gi[u] < 0) continue;
                const int q = q0 + u * PA_SUM;
                const double xv = sc ? xb[q] / sv[u] : xb[q];
                x[gi[u]] = xv;
                ss += xv * xv;
            }
        }
        if (F.out) {                             // (vt's warp is whole: PA_SUM and NT are multiples of 32)
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
            if ((vt & 31) == 0) wsum[vt >> 5] = ss;
        }
    }
    if (F.out) {                                 // rms of the result: per-CTA partial, last CTA finishes
        __shared__ bool last;
        __syncthreads();
        if (tid == 0) {
            double t = 0.0;
            for (int w = 0; w < PA_SUM / 32; ++w) t += wsum[w];
            F.part[blockIdx.x] = t;
            __threadfence();
            last = (atomicAdd(F.ticket, 1u) == gridDim.x - 1);
        }
        __syncthreads();
        if (last && tid == 0) {
            __threadfence();
            *F.out = sqrt(sum_partials(F.part, (int)gridDim.x, 1) / (double)F.n);
            *F.ticket = 0u;
        }
    }
    if constexpr (TW) cluster_sync_all();        // the other rank has finished reading this CTA's xch
}

// Sweep for partitions too large for the shared-memory pipeline: same fused stages, operands read
// from global memory (L2).
template <typename TS>
__global__ void __launch_bounds__(512) k_pc_apply_glob(PcGeom gin, const TS* __restrict__ A,
                                                       const double* __restrict__ b, const double* __restrict__ sc,
                                                       double* __restrict__ x, double* __restrict__ xs_all) {
    __shared__ double tv[512];
    const int part = blockIdx.x;
    const PcGeom g = pc_part(gin, part);
    const int nb = g.nb, ld = g.ld;
    const int tid = threadIdx.x;
    const int64_t bs = g.bs;
    double* xs = xs_all + (int64_t)part * g.Nz * ld;
    if (!pc_range_ok(g, (int64_t)part * g.Nz * 5 * bs, (int64_t)g.Nz * 5 * bs)) return;   // geometry beyond the storage
    const TS* base = A + (int64_t)part * g.Nz * 5 * bs;
    for (int64_t q = tid; q < (int64_t)g.Nz * nb; q += blockDim.x) {
        int k = (int)(q / nb), l = (int)(q % nb);
        int64_t gi = pc_glob(g, part, k, l);
        xs[(int64_t)k * ld + l] = sc ? b[gi] * sc[gi] : b[gi];
    }
    __syncthreads();
    const int S = 2 * g.Nz - 1;
    for (int s = 0; s < S; ++s) {
        const bool fwd = s < g.Nz - 1;
        const int k = fwd ? s + 1 : g.Nz - 1 - (s - (g.Nz - 1));
        const TS* Ak = base + (int64_t)k * 5 * bs;
        const TS* M0 = fwd ? Ak + bs : Ak + 2 * bs;
        const double* v0 = fwd ? xs + (int64_t)(k - 1) * ld : xs + (int64_t)k * ld;
        const TS* M1 = fwd ? ((k >= 2) ? Ak : nullptr) : ((k + 1 < g.Nz) ? Ak + 3 * bs : nullptr);
        const double* v1 = fwd ? ((k >= 2) ? xs + (int64_t)(k - 2) * ld : nullptr)
                               : ((k + 1 < g.Nz) ? xs + (int64_t)(k + 1) * ld : nullptr);
        const TS* M2 = (!fwd && k + 2 < g.Nz) ? Ak + 4 * bs : nullptr;
        const double* v2 = (!fwd && k + 2 < g.Nz) ? xs + (int64_t)(k + 2) * ld : nullptr;
        for (int r = tid; r < nb; r += blockDim.x) {
            double acc = 0.0;
            for (int c = 0; c < nb; ++c) acc += (double)M0[(int64_t)r * ld + c] * v0[c];
            if (M1) for (int c = 0; c < nb; ++c) acc += (double)M1[(int64_t)r * ld + c] * v1[c];
            if (M2) for (int c = 0; c < nb; ++c) acc += (double)M2[(int64_t)r * ld + c] * v2[c];
            tv[r] = fwd ? xs[(int64_t)k * ld + r] - acc : acc;
        }
        __syncthreads();
        for (int r = tid; r < nb; r += blockDim.x) xs[(int64_t)k * ld + r] = tv[r];
        __syncthreads();
    }
    for (int64_t q = tid; q < (int64_t)g.Nz * nb; q += blockDim.x) {
        int k = (int)(q / nb), l = (int)(q % nb);
        int64_t gi = pc_glob(g, part, k, l);
        x[gi] = sc ? xs[(int64_t)k * ld + l] / sc[gi] : xs[(int64_t)k * ld + l];
    }
}

// Largest partition of mode 3 the shared-memory kernels take at their tuned size.
#define PC_SPLIT_NB 48

static PcGeom geom_of_params(const dv_step_params& p, int mode) {
    PcGeom g;
    g.Nr = p.Nr;
    g.Nth = p.Nth;
    g.Nz = p.Nz;
    g.wall = p.wall_on;
    g.rg = g.tg = 1;
    g.cap = -1;
    g.nstate = (int64_t)DV_NV * p.Nr * p.Nth * p.Nz + (p.wall_on ? (int64_t)p.Nth * p.Nz : 0);
    g.err = nullptr;
    // mode 3 is the split form of mode 2 (a factorisation records it as the mode it used): derive it again
    if (mode == 3) mode = 2;
    // mode 2 needs a second ring and a second sector; below that it is mode 0 (or 1 for one sector)
    if (mode == 2 && (p.Nr < 2 || p.Nth < 2)) mode = 0;
    g.mode = (p.Nth > 1 && (mode == 0 || mode == 2)) ? mode : 1;
    g.nc = (int64_t)p.Nr * p.Nth * p.Nz;
    static const bool split_ok = [] {
        const char* e = getenv("DVTSA_PC_SPLIT");
        return !(e && e[0] == '0');
    }();
    if (g.mode == 2 && split_ok && std::max(DV_NV * (g.Nr - 1) + (g.wall ? 1 : 0), DV_NV * g.Nth) > PC_SMEM_NB) {
        // too large for the shared-memory kernels: split the sectors into ring groups and the core
        // ring into theta groups of at most PC_SPLIT_NB unknowns (mode 3)
        g.mode = 3;
        auto nb_ring = [&](int G) {
            int worst = 0;
            for (int gi = 0; gi < G; ++gi) {
                int a0, a1;
                pc_group(g.Nr - 1, G, gi, a0, a1);
                worst = std::max(worst, DV_NV * (a1 - a0) + ((g.wall && gi == G - 1) ? 1 : 0));
            }
            return worst;
        };
        g.rg = 1;
        while (g.rg < g.Nr - 1 && nb_ring(g.rg) > PC_SPLIT_NB) ++g.rg;
        g.tg = 1;
        while (g.tg < g.Nth && DV_NV * ((g.Nth + g.tg - 1) / g.tg) > PC_SPLIT_NB) ++g.tg;
        g.nb = std::max(nb_ring(g.rg), DV_NV * ((g.Nth + g.tg - 1) / g.tg));
        g.ncv = g.nb;
        g.nparts = g.Nth * g.rg + g.tg;
        g.ld = pc_ld(g.nb);
        g.bs = (((int64_t)g.nb * g.ld + 1) / 2) * 2;
        g.zs = 0;
        return g;
    }
    if (g.mode == 0) {
        g.nb = DV_NV * g.Nr + (g.wall ? 1 : 0);
        g.ncv = DV_NV * g.Nr;
        g.nparts = g.Nth;
    } else if (g.mode == 2) {
        const int nb_sector = DV_NV * (g.Nr - 1) + (g.wall ? 1 : 0), nb_core = DV_NV * g.Nth;
        g.nb = std::max(nb_sector, nb_core);
        g.ncv = g.nb;                       // per-partition values come from pc_part
        g.nparts = g.Nth + 1;
    } else {
        g.nb = DV_NV * g.Nr * g.Nth + (g.wall ? g.Nth : 0);
        g.ncv = DV_NV * g.Nr * g.Nth;
        g.nparts = 1;
    }
    g.ld = pc_ld(g.nb);
    g.bs = (((int64_t)g.nb * g.ld + 1) / 2) * 2;
    g.zs = 0;
    return g;
}

static PcGeom geom_of(const dv_model* m, int mode) {
    PcGeom g = geom_of_params(m->p, mode);
    g.cap = m->pc_doubles;
    g.err = m->d_err;
    return g;
}

void precond_capacity(const dv_step_params& p, int* cap_nb, int* cap_parts, int64_t* pc_need, int64_t* work_need) {
    int nb = 0, parts = 0;
    int64_t need = 0;
    for (int mode : {0, 1, 2}) {
        const PcGeom g = geom_of_params(p, mode);
        if (g.mode == 1 && g.nb > 512) continue;       // whole cross-sections only up to 512 unknowns
        nb = std::max(nb, g.nb);
        parts = std::max(parts, g.nparts);
        need = std::max(need, precond_doubles(g.nb, g.nparts, g.Nz));
    }
    *cap_nb = nb;
    *cap_parts = parts;
    *pc_need = need;
    *work_need = precond_work_doubles(nb, parts, p.Nz);
}

// Host check of the partition maps of a geometry (tests): every (partition, plane, local index) maps
// to an unknown inside the state, each unknown exactly once, and the inverse map (cell / wall ->
// partition, local index) agrees.  Returns the number of violations.
int64_t precond_check_maps(const dv_step_params& p, int mode, int* nparts_out, int* nb_out) {
    const PcGeom g = geom_of_params(p, mode);
    const int64_t nc = g.nc, offw = (int64_t)DV_NV * nc, n = offw + (g.wall ? (int64_t)g.Nth * g.Nz : 0);
    std::vector<int> seen(n, 0);
    int64_t bad = 0;
    for (int part = 0; part < g.nparts; ++part) {
        const PcGeom q = pc_part(g, part);
        if (q.nb > g.nb || q.ncv > q.nb || q.nb < 1) ++bad;
        for (int k = 0; k < g.Nz; ++k)
            for (int l = 0; l < q.nb; ++l) {
                const int64_t gi = pc_glob(q, part, k, l);
                if (gi < 0 || gi >= n) { ++bad; continue; }
                seen[gi] += 1;
            }
    }
    for (int64_t u = 0; u < n; ++u)
        if (seen[u] != 1) ++bad;
    for (int i = 0; i < g.Nr; ++i)
        for (int j = 0; j < g.Nth; ++j)
            for (int k = 0; k < g.Nz; ++k) {
                const int part = pc_part_of(g, i, j);
                if (part < 0 || part >= g.nparts) { ++bad; continue; }
                const PcGeom q = pc_part(g, part);
                const int64_t cell = ((int64_t)i * g.Nth + j) * g.Nz + k;
                for (int v = 0; v < DV_NV; ++v) {
                    const int l = pc_local(g, i, j, v);
                    if (l < 0 || l >= q.ncv || pc_glob(q, part, k, l) != v * nc + cell) ++bad;
                }
                if (g.wall && i == g.Nr - 1) {
                    const int l = pc_local(g, i, j, DV_NV);
                    if (l < q.ncv || l >= q.nb || pc_glob(q, part, k, l) != offw + (int64_t)j * g.Nz + k) ++bad;
                }
            }
    *nparts_out = g.nparts;
    *nb_out = g.nb;
    return bad;
}

int precond_partitions(const dv_model* m, int* mode, int* zs, int* nb_out, int cap) {
    if (!m->pc_ready) return 0;
    const PcGeom g = geom_of(m, m->pc_mode);
    *mode = g.mode;
    *zs = m->pc_zs;
    for (int q = 0; q < g.nparts && q < cap; ++q) nb_out[q] = pc_part(g, q).nb;
    return g.nparts;
}

// the geometry the current factors were computed with
static PcGeom geom_factored(const dv_model* m) {
    PcGeom g = geom_of(m, m->pc_mode);
    g.zs = m->pc_zs;
    return g;
}

static int smem_optin() {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return v;
}

int64_t precond_doubles(int nb, int nparts, int Nz) {
    const int ld = pc_ld(nb);
    return (int64_t)nparts * Nz * 5 * ((((int64_t)nb * ld + 1) / 2) * 2);
}

int64_t precond_work_doubles(int nb, int nparts, int Nz) {
    const int ld = pc_ld(nb);
    return std::max((int64_t)nparts * 4 * (int64_t)nb * ld, (int64_t)nparts * Nz * (int64_t)ld);
}

// a launch of `kern` as clusters of two CTAs (grid = 2 x partitions)
template <typename... KArgs, typename... Args>
static cudaError_t launch_pair(void (*kern)(KArgs...), unsigned grid, unsigned block, size_t dyn, cudaStream_t s,
                               bool pdl, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = dyn;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

static bool apply_fusable(const PcGeom& g, size_t tsize);
static size_t pc_tsize(const dv_model* m);

// Twisted factorisation: the top-down and bottom-up eliminations run at the same time and meet at
// the separator planes zs, zs+1, which halves the sequential plane chain of the factorisation and
// of both sweeps.  Taken when each direction keeps at least three planes and both kernels run from
// shared memory; DVTSA_PC_TWIST=0 keeps the one-directional form.
static int pc_twist_zs(const PcGeom& g, size_t tsize, bool factor_smem) {
    const char* e = getenv("DVTSA_PC_TWIST");
    if (e && e[0] == '0') return 0;
    if (g.Nz < 8 || !factor_smem || !apply_fusable(g, tsize)) return 0;
    return (g.Nz - 2) / 2;
}

int precond_factor(dv_model* m, const double* J, double dh, int mode, cudaStream_t s) {
    PcGeom g = geom_of(m, mode);
    if (g.nb > m->pc_cap_nb || g.nparts > m->pc_cap_parts) {
        set_error("preconditioner partition larger than the workspace allocated at model creation");
        return DV_ERR_ARG;
    }
    if (g.nb > 512) {
        set_error("preconditioner block size above the supported 512 (use theta_block)");
        return DV_ERR_UNSUPPORTED;
    }
    const int64_t total = (int64_t)g.nparts * g.Nz * 5 * g.bs;
    DV_LAUNCH(dv::K_PC_FACTOR, s, k_pc_zero<<<std::min<int64_t>((total + 255) / 256, 4096), 256, 0, s>>>(m->d_pc, total));
    dim3 grid((unsigned)((m->nc + 127) / 128), DV_NSLOT);
    DV_LAUNCH(dv::K_PC_FACTOR, s, k_pc_scatter<<<grid, 128, 0, s>>>(g, J, dh, m->d_pc));
    const int optin = smem_optin();
    constexpr size_t own = 6144;                            // static shared memory of the kernel (at most)
    const size_t budget = (size_t)optin - own;
    const int lds = pc_lds(g.nb, budget);
    const size_t dyn = (size_t)9 * g.nb * lds * sizeof(double);
    const bool factor_smem = g.nb <= PC_SMEM_NB && dyn <= budget;
    g.zs = pc_twist_zs(g, pc_tsize(m), factor_smem);
    if (factor_smem && g.zs > 0) {
        if (dyn + own > 48 * 1024)
            DV_CUDA(allow_dyn_smem((const void*)k_pc_factor_smem<true>));
        DV_LAUNCH(dv::K_PC_FACTOR, s,
                  DV_CUDA(launch_pair(k_pc_factor_smem<true>, 2u * g.nparts, (unsigned)FAC_T, dyn, s, false, g, m->d_pc, m->d_pc_info,
                                      lds)));
    } else if (factor_smem) {
        if (dyn + own > 48 * 1024)
            DV_CUDA(allow_dyn_smem((const void*)k_pc_factor_smem<false>));
        DV_LAUNCH(dv::K_PC_FACTOR, s, k_pc_factor_smem<false><<<g.nparts, FAC_T, dyn, s>>>(g, m->d_pc, m->d_pc_info, lds));
    } else {
        const size_t static_smem = (2 * 1024 + 256) * sizeof(double) + 256 * sizeof(int);
        size_t need = (size_t)2 * g.nb * g.nb * sizeof(double);
        int use_smem = (need + static_smem) <= (size_t)optin ? 1 : 0;
        size_t dyn = use_smem ? need : 0;
        if (use_smem && dyn > 48 * 1024)
            DV_CUDA(allow_dyn_smem((const void*)k_pc_factor_glob));
        DV_LAUNCH(dv::K_PC_FACTOR, s, k_pc_factor_glob<<<g.nparts, 256, dyn, s>>>(g, m->d_pc, m->d_pc_work, m->d_pc_info, use_smem));
    }
    if (m->pc_fp32) {               // the sweep streams an FP32 copy of the factors
        const int64_t tot = (int64_t)g.nparts * g.Nz * 5 * g.bs;
        DV_LAUNCH(dv::K_PC_FACTOR, s, k_pc_to_f32<<<std::min<int64_t>((tot + 255) / 256, 4096), 256, 0, s>>>(m->d_pc, m->d_pc32, tot));
    }
    DV_CUDA(cudaGetLastError());
    m->pc_mode = g.mode;
    m->pc_nb = g.nb;
    m->pc_nparts = g.nparts;
    m->pc_zs = g.zs;
    m->pc_ready = 1;
    return DV_OK;
}

// The rule for the register-streamed sweep, and with it for the twisted factorisation: two sets of
// solution planes, the exchange planes and 2 x 3 factor blocks of `tsize`-byte values within the shared
// memory of a CTA.  (The sweep itself needs the planes only; the line stays where it was because moving
// it would change which shapes are factorised from both ends, and so their results.)
static size_t apply_smem(const PcGeom& g, size_t tsize) {
    return sizeof(double) * (size_t)(2 * (int64_t)g.Nz * g.ld + 2 * g.ld) + tsize * (size_t)(2 * 3 * g.bs);
}

static size_t pc_tsize(const dv_model* m) { return m->pc_fp32 ? sizeof(float) : sizeof(double); }

template <int NJ, typename TS, bool TW>
static void launch_apply_tw(const PcGeom& g, dv_model* m, const TS* A, const double* b, const double* sc, double* x,
                            cudaStream_t s, const PaFuse& F, bool count) {
    const int np = TW ? std::max(g.zs, g.Nz - g.zs - 2) + 2 : g.Nz;
    const size_t planes = sizeof(double) * (size_t)(2 * np + 2) * g.ld + sizeof(int) * (size_t)g.ld;
    const size_t table = sizeof(int4) * (size_t)(pa_stages(np, TW) + PA_DEPTH);
    size_t dyn = planes + table;
    auto kern = k_pc_apply<NJ, TS, TW, false>;
    if constexpr (TW) {
        const int64_t bytes = (int64_t)sizeof(TS) * g.nparts * g.Nz * 5 * g.bs;
        if (m->tune.sweep_nbuf == 3 || (m->tune.sweep_nbuf != 2 && bytes > PA_L2_BYTES)) kern = k_pc_apply<NJ, TS, TW, true>;
    }
    if constexpr (!TW && NJ <= 2) {             // (larger blocks: the rule's six are more than a table for its planes)
        constexpr size_t own = 256;             // static shared memory of the kernel (at most)
        if (dyn + own > (size_t)smem_optin()) {
            kern = k_pc_apply<NJ, TS, TW, true>;
            dyn = planes;
        }
    }
    if (dyn > 48 * 1024) allow_dyn_smem((const void*)kern);
    if (count) prof_begin(dv::K_PC_APPLY, s);
    if (TW) launch_pair(kern, 2u * g.nparts, pa_threads(NJ), dyn, s, F.pdl, g, A, b, sc, x, F);
    else kern<<<g.nparts, pa_threads(NJ), dyn, s>>>(g, A, b, sc, x, F);
    if (count) prof_end(dv::K_PC_APPLY, s);
}

template <int NJ, typename TS>
static void launch_apply_k(const PcGeom& g, dv_model* m, const TS* A, const double* b, const double* sc, double* x,
                           cudaStream_t s, const PaFuse& F, bool count) {
    if (g.zs > 0) launch_apply_tw<NJ, TS, true>(g, m, A, b, sc, x, s, F, count);
    else launch_apply_tw<NJ, TS, false>(g, m, A, b, sc, x, s, F, count);
}

template <int NJ>
static void launch_apply_nj(const PcGeom& g, dv_model* m, const double* b, const double* sc, double* x, cudaStream_t s,
                            const PaFuse& F, bool count) {
    if (m->pc_fp32) launch_apply_k<NJ, float>(g, m, m->d_pc32, b, sc, x, s, F, count);   // FP32 factors, products in FP64
    else launch_apply_k<NJ, double>(g, m, m->d_pc, b, sc, x, s, F, count);
}

static void launch_apply(const PcGeom& g, dv_model* m, const double* b, const double* sc, double* x, cudaStream_t s,
                         const PaFuse& F, bool count) {
    switch (g.ld / (2 * PA_LANES)) {
        case 1: launch_apply_nj<1>(g, m, b, sc, x, s, F, count); break;
        case 2: launch_apply_nj<2>(g, m, b, sc, x, s, F, count); break;
        case 3: launch_apply_nj<3>(g, m, b, sc, x, s, F, count); break;
        default: launch_apply_nj<4>(g, m, b, sc, x, s, F, count); break;
    }
}

int precond_apply(dv_model* m, const double* b, const double* sc, double* x, cudaStream_t s) {
    if (!m->pc_ready) {
        set_error("preconditioner applied before it was factorised");
        return DV_ERR_ARG;
    }
    PcGeom g = geom_factored(m);
    if (precond_apply_fusable(m)) {
        launch_apply(g, m, b, sc, x, s, PaFuse(), true);
    } else {
        if (m->pc_fp32) {
            DV_LAUNCH(dv::K_PC_APPLY, s, k_pc_apply_glob<float><<<g.nparts, 512, 0, s>>>(g, m->d_pc32, b, sc, x, m->d_pc_work));
        } else {
            DV_LAUNCH(dv::K_PC_APPLY, s, k_pc_apply_glob<double><<<g.nparts, 512, 0, s>>>(g, m->d_pc, b, sc, x, m->d_pc_work));
        }
    }
    DV_CUDA(cudaGetLastError());
    return DV_OK;
}

static bool apply_fusable(const PcGeom& g, size_t tsize) {
    return g.nb <= 64 && g.ld % (2 * PA_LANES) == 0 && apply_smem(g, tsize) <= (size_t)smem_optin();
}

bool precond_apply_fusable(dv_model* m) { return apply_fusable(geom_factored(m), pc_tsize(m)); }

int precond_apply_capture(dv_model* m, const double* b, const double* sc, double* x, cudaStream_t s,
                          const PaFuse& F) {
    PcGeom g = geom_factored(m);
    if (precond_apply_fusable(m)) {
        launch_apply(g, m, b, sc, x, s, F, false);    // attributes were set by an earlier precond_apply
    } else {
        if (F.V || F.out) {
            set_error("fused sweep requested for a partition the shared-memory sweep does not take");
            return DV_ERR_ARG;
        }
        if (m->pc_fp32) k_pc_apply_glob<float><<<g.nparts, 512, 0, s>>>(g, m->d_pc32, b, sc, x, m->d_pc_work);
        else k_pc_apply_glob<double><<<g.nparts, 512, 0, s>>>(g, m->d_pc, b, sc, x, m->d_pc_work);
    }
    DV_CUDA(cudaGetLastError());
    return DV_OK;
}

// ---------------------------------------------------------------- FP32 assembled-Jacobian operator
// Mixed-precision Krylov: the GMRES operator u -> (v - dh J v)/s, v = u s, with J the FP32 block
// Jacobian (the same difference quotients as the FD Jacobian, rounded), products and sums in FP32;
// replaces the FP64 finite-difference matvec (core/solver.py:196-203) inside GMRES.  One thread per
// cell computes its six rows and, for an outer-ring cell, its wall node's row.  Blocks known to be
// structurally zero (loading rows of neighbour slots, the wall row of inner cells) are not read.
__global__ void __launch_bounds__(256) k_spmv32(int Nr, int Nth, int Nz, int wall, const float* __restrict__ J,
                                                const double* __restrict__ u, const double* __restrict__ sc,
                                                double dh, const double* __restrict__ dh_dev, double* __restrict__ out) {
    const int64_t nc = (int64_t)Nr * Nth * Nz;
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    const double dhv = dh_dev ? dh_dev[1] : dh;
    const int k = (int)(c % Nz);
    const int64_t rr = c / Nz;
    const int j = (int)(rr % Nth);
    const int i = (int)(rr / Nth);
    const bool outer_wall = wall && i == Nr - 1;
    const int64_t offw = (int64_t)DV_NV * nc;
    float acc[DV_NB];
#pragma unroll
    for (int r = 0; r < DV_NB; ++r) acc[r] = 0.0f;
#pragma unroll
    for (int slot = 0; slot < DV_NSLOT; ++slot) {
        int ni = i, nj = j, nk = k;
        bool ok = true;
        switch (slot) {
            case 0: break;
            case 1: nk = k - 1; ok = nk >= 0; break;
            case 2: nk = k + 1; ok = nk < Nz; break;
            case 3: nk = k - 2; ok = nk >= 0; break;
            case 4: nk = k + 2; ok = nk < Nz; break;
            case 5: ni = i - 1; ok = ni >= 0; break;
            case 6: ni = i + 1; ok = ni < Nr; break;
            case 7: ok = Nth > 1; nj = (j == 0) ? Nth - 1 : j - 1; break;
            default: ok = Nth > 1; nj = (j == Nth - 1) ? 0 : j + 1; break;
        }
        if (!ok) continue;
        const int64_t cn = ((int64_t)ni * Nth + nj) * Nz + nk;
        const float* Js = J + (int64_t)slot * DV_NB * DV_NB * nc + c;
#pragma unroll
        for (int cv = 0; cv < DV_NV; ++cv) {
            const int64_t q = (int64_t)cv * nc + cn;
            const float x = (float)(u[q] * sc[q]);
#pragma unroll
            for (int rv = 0; rv < DV_NV; ++rv) {
                if ((rv == 3 || rv == 4) && slot != 0) continue;
                acc[rv] = fmaf(Js[(int64_t)(rv * DV_NB + cv) * nc], x, acc[rv]);
            }
            if (outer_wall && slot == 0) acc[DV_NV] = fmaf(Js[(int64_t)(DV_NV * DV_NB + cv) * nc], x, acc[DV_NV]);
        }
        if (wall && ni == Nr - 1) {      // the neighbour's wall node (column 6)
            const int64_t q = offw + (int64_t)nj * Nz + nk;
            const float x = (float)(u[q] * sc[q]);
            if (slot == 0) {
#pragma unroll
                for (int rv = 0; rv < DV_NV; ++rv) {
                    if (rv == 3 || rv == 4) continue;
                    acc[rv] = fmaf(Js[(int64_t)(rv * DV_NB + DV_NV) * nc], x, acc[rv]);
                }
            }
            if (outer_wall && (slot == 0 || slot == 1 || slot == 2 || slot == 7 || slot == 8))
                acc[DV_NV] = fmaf(Js[(int64_t)(DV_NV * DV_NB + DV_NV) * nc], x, acc[DV_NV]);
        }
    }
#pragma unroll
    for (int rv = 0; rv < DV_NV; ++rv) {
        const int64_t q = (int64_t)rv * nc + c;
        out[q] = (u[q] * sc[q] - dhv * (double)acc[rv]) / sc[q];
    }
    if (outer_wall) {
        const int64_t q = offw + (int64_t)j * Nz + k;
        out[q] = (u[q] * sc[q] - dhv * (double)acc[DV_NV]) / sc[q];
    }
}

int launch_spmv32(dv_model* m, const double* u, const double* sc, double dh, const double* dh_dev, double* out,
                  cudaStream_t s, bool count) {
    const dv_step_params& p = m->p;
    const int bl = (m->tune.spmv_block == 64 || m->tune.spmv_block == 256) ? m->tune.spmv_block : 128;
    const unsigned grid = (unsigned)((m->nc + bl - 1) / bl);
    if (count) {
        DV_LAUNCH(dv::K_SPMV, s, k_spmv32<<<grid, bl, 0, s>>>(p.Nr, p.Nth, p.Nz, p.wall_on, m->d_J32, u, sc, dh, dh_dev, out));
    } else {
        k_spmv32<<<grid, bl, 0, s>>>(p.Nr, p.Nth, p.Nz, p.wall_on, m->d_J32, u, sc, dh, dh_dev, out);
    }
    DV_CUDA(cudaGetLastError());
    return DV_OK;
}

}  // namespace dv
