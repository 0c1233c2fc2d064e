// dv_mlp.cu -- the learned Newton predictor: a per-cell network whose BF16 products run on the sm_100a
// tensor cores (tcgen05.mma, FP32 accumulation in tensor memory), with its own forward, backward and
// Adam kernels.
//
// The reference starts every implicit stage from an extrapolation (core/solver.py:420 for stage 1,
// :432/:435 for stage 2): a straight line through the two latest states to the stage's time.  The
// network adds a per-cell correction to that line, predicted from the cell's and its six face
// neighbours' states at those two levels, the right-hand side at the latest level, the step-size
// ratio, the stage and the cycle step.  It is trained on stage solutions the plain solver itself
// produced; the integrator starts Newton from whichever of the two guesses has the smaller scaled
// residual, so the unchanged Newton tolerance decides the converged state in both cases.
//
// Products (all M = 128 rows per CTA, N <= 128 columns, operands staged in shared memory by cp.async, one
// elected thread issuing the MMAs and committing to an mbarrier):
//   forward   H1 = tanh(X W1^T + b1), H2, H3 likewise, O = H3 W4^T + b4
//   backward  D4 = dL/dO, D3 = (D4 W4) * (1 - H3^2), D2 = (D3 W3) * (1 - H2^2), D1 = (D2 W2) * (1 - H1^2)
//             dW4^T = H3^T D4, dW3 = D3^T H2, dW2 = D2^T H1, dW1 = D1^T X (K = samples, split over CTAs)
// Forward and backward of 128 rows are one launch (k_chain): activations and gradients stay in shared memory
// with rows = samples and are written with rows = features for the weight-gradient products (k_gemm).
#include <cmath>
#include <cstdio>
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>
#include "dv_internal.h"
#include "dv_mlp.h"
#include "dv_umma.cuh"

using bf16 = __nv_bfloat16;

namespace dv {
namespace mlp {

using namespace dv::umma;

__device__ __forceinline__ float bf2f(bf16 x) { return __bfloat162float(x); }

constexpr int GT = 512;                        // threads of a product: the epilogue has 4 warps per 32 rows,
                                               // each a quarter of the 16-column groups

// ------------------------------------------------------------------------------------ products
// D [128 nb][N] = A B^T, block x of nb its rows 128 x (split 0), or a part of K to an FP32 partial sum of its
// own, D [x][128][N] (split 1: the weight gradients).  Up to four products in one launch, `per` blocks each.
struct GemmP {
    const bf16* A;
    int64_t ra;           // rows of A's panel layout
    const bf16* B;
    int64_t rb;           // rows of B's panel layout (rows 0..N-1 used)
    int N;                // 16..128, multiple of 16
    float* of;
};
struct GemmBatch {
    GemmP p[4];
    int per;              // blocks of a product
    int kpanels;          // K / 8 of a block (even)
    int split;
    int* err;
};

constexpr int KCH = 8;                         // panels per staged K chunk (64 columns)
constexpr int RING = 6;                        // staged chunks
constexpr uint32_t STAGE_A = KCH * 128 * 16;   // 16 KB
constexpr uint32_t STAGE_B = KCH * 128 * 16;   // 16 KB (N <= 128)
constexpr uint32_t GEMM_SMEM = RING * (STAGE_A + STAGE_B);

// Bound by latency: six of a block's chunks are in flight before its first product (two in flight and a
// launch for each weight gradient: 74 us a training step; the four together now 11.6).
__global__ void __launch_bounds__(GT) k_gemm(GemmBatch gb) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[RING];
    __shared__ uint32_t tmem_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int which = blockIdx.x / gb.per, x = blockIdx.x - which * gb.per;
    const GemmP g = gb.p[which];
    const int N = g.N;
    const int64_t m0 = gb.split ? 0 : (int64_t)x * 128;
    const int64_t kp0 = gb.split ? (int64_t)x * gb.kpanels : 0;
    const int nch = (gb.kpanels + KCH - 1) / KCH;
    const uint32_t sb = smem_u32(smem);
    const uint32_t ncols = N <= 32 ? 32u : (N <= 64 ? 64u : 128u);
    if (warp == 0) tmem_alloc(smem_u32(&tmem_s), ncols);
    if (tid == 0) {
        for (int q = 0; q < RING; ++q) mbar_init(smem_u32(&bars[q]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    auto load = [&](int c) {                   // a (possibly empty) group of copies per chunk
        if (c < nch) {
            const uint32_t sA = sb + (c % RING) * (STAGE_A + STAGE_B), sB = sA + STAGE_A;
            const int pc = min(KCH, gb.kpanels - c * KCH);
            const int64_t kp = kp0 + (int64_t)c * KCH;
            for (int idx = tid; idx < pc * 128; idx += GT) {
                const int p = idx >> 7, r = idx & 127;
                cp_async16(sA + p * 2048 + r * 16, g.A + ((kp + p) * g.ra + m0 + r) * 8);
            }
            for (int idx = tid; idx < pc * N; idx += GT) {
                const int p = idx / N, r = idx - p * N;
                cp_async16(sB + p * (N * 16) + r * 16, g.B + ((kp + p) * g.rb + r) * 8);
            }
        }
        cp_async_commit();
    };
    for (int c = 0; c < RING; ++c) load(c);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_s;
    const uint32_t idesc = idesc_bf16_m128(N);
    bool ok = true;
    for (int c = 0; c < nch; ++c) {
        cp_async_wait<RING - 1>();
        fence_proxy_async();
        __syncthreads();
        const uint32_t bar = smem_u32(&bars[c % RING]);
        if (tid == 0) {
            fence_after_sync();
            const uint32_t sA = sb + (c % RING) * (STAGE_A + STAGE_B), sB = sA + STAGE_A;
            const int pc = min(KCH, gb.kpanels - c * KCH);
            for (int q = 0; q < pc / 2; ++q) {
                const uint64_t da = sdesc(sA + q * 2 * 2048, 2048, 128);
                const uint64_t db = sdesc(sB + q * 2 * (N * 16), N * 16, 128);
                mma_bf16(tmem, da, db, idesc, (c > 0 || q > 0) ? 1u : 0u);
            }
            mma_commit(bar);
        }
        if (c + RING < nch && !mbar_wait(bar, (uint32_t)((c / RING) & 1))) ok = false;     // its buffer is free
        load(c + RING);
    }
    const uint32_t bar = smem_u32(&bars[(nch - 1) % RING]);
    const uint32_t par = (uint32_t)(((nch - 1) / RING) & 1);
    if (!mbar_wait(bar, par)) ok = false;
    cp_async_wait<0>();
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    fence_after_sync();
    if (!ok) {
        atomicOr(gb.err, 8);
        mbar_wait(bar, par);                   // the products may still run: one more bounded wait before the memory is released
    }
    const int row = (warp & 3) * 32 + lane;
    const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    for (int c0 = (warp >> 2) * 16; c0 < N && ok; c0 += 64) {
        float v[16];
        tmem_ld16(trow + c0, v);
        float4* o = reinterpret_cast<float4*>(g.of + ((int64_t)x * 128 + row) * N + c0);
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, ncols);
}

// Self-test of the products' bounded wait: an mbarrier that nothing arrives at, waited on by one warp with
// `polls` polls; the timeout sets bit 1 of *err, and the kernel returns.
__global__ void k_selftest_mbar(int polls, int* err) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    const bool arrived = mbar_wait(smem_u32(&bar), 0u, polls);
    __syncwarp();
    if (threadIdx.x == 0) {
        if (!arrived) atomicOr(err, 1);
        asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(&bar)) : "memory");
    }
}

static int gemm(const GemmBatch& g, int products, cudaStream_t s) {
    DV_CUDA(dv::allow_dyn_smem((const void*)k_gemm));
    DV_LAUNCH(dv::K_MLP, s, k_gemm<<<products * g.per, GT, GEMM_SMEM, s>>>(g));
    return launch_ok("k_gemm");
}

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
    x ^= x >> 30;
    x *= 0xbf58476d1ce4e5b9ull;
    x ^= x >> 27;
    x *= 0x94d049bb133111ebull;
    x ^= x >> 31;
    return x;
}

// ------------------------------------------------------------------------------------ the chain of a row tile
// The whole chain of 128 rows in one block: forward (TRAIN 0: X -> O), or forward, loss and backward down to D1.
// Nothing in it crosses rows, so an activation stays in shared memory as the next product's operand
// (and for 1 - H^2), weights arrive two products ahead, and a training step's products leave only what the weight
// gradients read: H and D with rows = features, written 128 bytes at a time while the next product runs.
// Bound by latency, seven times product, epilogue, barrier, on 32 SMs for 4096 rows: 34 us with the drawing of the
// batch, where a launch for each product with 128 threads and every activation through L2 in both layouts took 97
// and the drawing another 6.
enum { E_TANH = 0, E_OUT = 1, E_LOSS = 2, E_DTANH = 3 };
struct ChainP {
    const bf16* X;        // rows x NIN, panel layout of xr rows
    int64_t xr;
    // a batch drawn from the recorded samples (else null): row j is sample hash(seed, step, j) mod count of X, its
    // targets Ts scaled and clipped by nrm, X^T written for the first weight gradient
    const float* Ts;
    const double* nrm;
    int64_t count, seed, step;
    bf16* Xbt;
    const bf16 *W1, *W2, *W3, *W4, *W4t, *W3t, *W2t;
    const float* P;       // parameters (biases)
    int64_t rows_valid;   // rows at or beyond this: no loss, zero activations and gradients; O is not written there
    float* out;           // O [rows][NOUT] (forward)
    const float* tgt;     // targets [rows][8]
    float dscale;         // dL/dO = dscale * (O - target)
    float* lossp;         // per-block sum of squared errors
    float* bsum;          // per-block column sums of D1, D2, D3, D4, each [blocks][its width], TB * 128 apart
    bf16 *H1t, *H2t, *H3t, *D4t, *D3t, *D2t, *D1t;      // rows = features, K = samples
    int* err;
};
constexpr uint32_t ACT = 16 * 128 * 16;        // an activation of 128 rows x 128 columns
constexpr uint32_t D4_AT = 4 * ACT, WBUF_AT = D4_AT + 2 * 128 * 16, CHAIN_SMEM = WBUF_AT + 2 * ACT;

template <bool TRAIN>
__global__ void __launch_bounds__(GT) k_chain(ChainP g) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t bar_s;
    __shared__ uint32_t tmem_s;
    __shared__ int64_t sample[128];
    __shared__ float red[2][4][4][16];         // (group of columns, column group's warps, quarter of the rows, column)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quarter = warp & 3, cg = warp >> 2;
    constexpr int STAGES = TRAIN ? 7 : 4;
    const int64_t m0 = (int64_t)blockIdx.x * 128;
    const uint32_t sb = smem_u32(smem), bar = smem_u32(&bar_s);
    if (warp == 0) tmem_alloc(smem_u32(&tmem_s), 128);
    if (tid == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // stage s: X W1^T, H1 W2^T, H2 W3^T, H3 W4^T, D4 W4, D3 W3, D2 W2.  Operand and result places (multiples of ACT; 4: D4):
    // D3 takes X's, D2 H3's, D1 D3's
    const uint32_t a_at = 0x3043210u, o_at = 0x0304321u;
    auto place = [&](uint32_t code, int st) { return ((code >> (4 * st)) & 15u) * ACT; };
    auto panels = [](int st) { return st == 0 ? NIN / 8 : st == 4 ? NOUT / 8 : NH / 8; };
    auto width = [](int st) { return st == 3 ? NOUT : NH; };
    auto load_w = [&](int st) {                // (a group of copies per stage, empty past the last)
        if (st < STAGES) {
            const bf16* w = st == 0 ? g.W1 : st == 1 ? g.W2 : st == 2 ? g.W3 : st == 3 ? g.W4 : st == 4 ? g.W4t : st == 5 ? g.W3t : g.W2t;
            const uint32_t dst = sb + WBUF_AT + (st & 1) * ACT;
            for (int q = tid; q < panels(st) * width(st); q += GT) cp_async16(dst + q * 16, w + (int64_t)q * 8);
        }
        cp_async_commit();
    };
    const bool drawn = TRAIN && g.Ts != nullptr;
    if (drawn) {
        if (tid < 128)
            sample[tid] = (int64_t)(mix64((uint64_t)g.seed * 0x9e3779b97f4a7c15ull + (uint64_t)g.step * 1000003ull +
                                          (uint64_t)(m0 + tid)) % (uint64_t)g.count);
        __syncthreads();
    }
    for (int q = tid; q < NIN / 8 * 128; q += GT)
        cp_async16(sb + q * 16, g.X + ((int64_t)(q >> 7) * g.xr + (drawn ? sample[q & 127] : m0 + (q & 127))) * 8);
    load_w(0);
    load_w(1);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_s, trow = tmem + ((uint32_t)(quarter * 32) << 16);
    const int64_t row = m0 + quarter * 32 + lane;
    const bool live = row < g.rows_valid;
    // columns of the result at `at` as rows: 8 x 8 blocks (panel, eight rows), transposed by the load, 128 bytes each
    auto transpose_out = [&](uint32_t at, int np, bf16* dst) {
        for (int b = warp * 4; b < np * 16; b += GT / 32 * 4) {
            const int q = b + (lane >> 3);
            uint32_t r[4];
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                         : "r"(sb + at + (q >> 4) * 2048 + ((q & 15) * 8 + (lane & 7)) * 16)
                         : "memory");
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int pe = (b + e) >> 4, ge = (b + e) & 15;
                reinterpret_cast<uint32_t*>(dst + ((m0 >> 3) + ge) * (int64_t)(np * 64) + pe * 64)[lane] = r[e];
            }
        }
    };
    auto tdst = [&](int st) {
        return st == 0 ? g.H1t : st == 1 ? g.H2t : st == 2 ? g.H3t : st == 3 ? g.D4t : st == 4 ? g.D3t : st == 5 ? g.D2t : g.D1t;
    };
    bool ok = true;
#pragma unroll 1
    for (int st = 0; st < STAGES; ++st) {
        const int N = width(st), np = panels(st);
        cp_async_wait<1>();                    // this stage's weights (the next stage's may be on their way)
        fence_proxy_async();
        __syncthreads();
        if (tid == 0) {
            fence_after_sync();
            const uint32_t sA = sb + place(a_at, st), sB = sb + WBUF_AT + (st & 1) * ACT;
            const uint32_t idesc = idesc_bf16_m128(N);
            for (int q = 0; q < np / 2; ++q)
                mma_bf16(tmem, sdesc(sA + q * 2 * 2048, 2048, 128), sdesc(sB + q * 2 * (N * 16), N * 16, 128), idesc, q > 0 ? 1u : 0u);
            mma_commit(bar);
        }
        __syncwarp();
        if (drawn && st == 0) transpose_out(0, NIN / 8, g.Xbt);
        if (TRAIN && st > 0) transpose_out(place(o_at, st - 1), width(st - 1) / 8, tdst(st - 1));
        if (!mbar_wait(bar, (uint32_t)(st & 1))) ok = false;
        ok = __syncthreads_and(ok ? 1 : 0) != 0;
        fence_after_sync();
        if (!ok) {
            if (tid == 0) atomicOr(g.err, 8);
            mbar_wait(bar, (uint32_t)(st & 1));          // the product may still run: one more bounded wait
            break;
        }
        load_w(st + 2);
        const int mode = st < 3 ? E_TANH : st > 3 ? E_DTANH : TRAIN ? E_LOSS : E_OUT;
        const float* bias = g.P + (st == 0 ? OFF_B1 : st == 1 ? OFF_B2 : st == 2 ? OFF_B3 : OFF_B4);
        uint8_t* const orow = smem + place(o_at, st) + (quarter * 32 + lane) * 16;
        const uint8_t* const hrow = smem + (7 - st) * ACT + (quarter * 32 + lane) * 16;      // (H3, H2, H1 of stages 4, 5, 6)
        float lsum = 0.0f;
        int half = 0;
#pragma unroll 1
        for (int c0 = cg * 16; c0 < N; c0 += 64, half ^= 1) {
            float v[16], w[16];
            tmem_ld16(trow + c0, v);
            if (mode == E_OUT) {
                if (live) {
                    float* o = g.out + row * NOUT + c0;
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = v[i] + bias[c0 + i];
                }
                continue;
            }
            if (mode == E_TANH) {
#pragma unroll
                for (int i = 0; i < 16; ++i) w[i] = live ? tanhf(v[i] + bias[c0 + i]) : 0.0f;
            } else if (mode == E_DTANH) {
                const uint4 hv[2] = {*reinterpret_cast<const uint4*>(hrow + (c0 >> 3) * 2048),
                                     *reinterpret_cast<const uint4*>(hrow + (c0 >> 3) * 2048 + 2048)};
                const bf16* hb = reinterpret_cast<const bf16*>(hv);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float h = bf2f(hb[i]);
                    w[i] = live ? v[i] * (1.0f - h * h) : 0.0f;
                }
            } else {
                const int64_t sj = drawn ? sample[quarter * 32 + lane] : row;
                const double clip = drawn ? g.nrm[19] : 0.0;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int n = c0 + i;
                    float d = 0.0f;
                    if (live && n < NOUT_USED) {
                        const float tgt = drawn ? (float)fmax(-clip, fmin(clip, (double)g.Ts[sj * 8 + n] / g.nrm[13 + n]))
                                                : g.tgt[row * 8 + n];
                        d = (v[i] + bias[n]) - tgt;
                    }
                    lsum += d * d;
                    w[i] = g.dscale * d;
                }
            }
            bf16 wb[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) wb[i] = __float2bfloat16_rn(w[i]);
            *reinterpret_cast<uint4*>(orow + (c0 >> 3) * 2048) = *reinterpret_cast<const uint4*>(wb);
            *reinterpret_cast<uint4*>(orow + (c0 >> 3) * 2048 + 2048) = *reinterpret_cast<const uint4*>(wb + 8);
            if (mode >= E_LOSS) {   // column sums of the bf16-rounded gradient, in a fixed order
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float x = bf2f(wb[i]);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                    if (lane == 0) red[half][cg][quarter][i] = x;
                }
            }
        }
        if (mode == E_LOSS && cg == 0) {
            float x = lsum;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            if (lane == 0) red[1][0][quarter][0] = x;
        }
        fence_before_sync();
        if (mode >= E_LOSS) {
            __syncthreads();
            float* bs = g.bsum + (int64_t)(6 - st) * gridDim.x * 128 + (int64_t)blockIdx.x * N;
            if (tid < N) {
                const float (*r)[16] = red[tid >> 6][(tid >> 4) & 3];
                const int i = tid & 15;
                bs[tid] = ((r[0][i] + r[1][i]) + r[2][i]) + r[3][i];
            }
            if (mode == E_LOSS && tid == 0)
                g.lossp[blockIdx.x] = ((red[1][0][0][0] + red[1][0][1][0]) + red[1][0][2][0]) + red[1][0][3][0];
        }
    }
    cp_async_wait<0>();
    fence_before_sync();
    __syncthreads();
    if (TRAIN && ok) transpose_out(place(o_at, 6), NH / 8, g.D1t);
    if (warp == 0) {
        fence_after_sync();
        tmem_dealloc(tmem, 128);
    }
}

template <bool TRAIN>
static int chain(const ChainP& g, int blocks, cudaStream_t s) {
    DV_CUDA(dv::allow_dyn_smem((const void*)k_chain<TRAIN>));
    DV_LAUNCH(dv::K_MLP, s, k_chain<TRAIN><<<blocks, GT, CHAIN_SMEM, s>>>(g));
    return launch_ok("k_chain");
}

// ------------------------------------------------------------------------------------ features
__device__ __forceinline__ double fasinh(double x) { return asinh(x); }

// Feature row of cell c (see the file comment): levels, spatial differences at A, changes A - B at the
// seven stencil points and dt_tgt f(A) in the solver's error-scale units of the cell, the extrapolation
// ratio, log10 h, the stage, the cycle step one-hot and a constant 1.
__device__ void cell_features(const StageInputs& in, const double* __restrict__ nrm, int64_t c, float* f) {
    const int k = (int)(c % in.Nz);
    const int64_t rr = c / in.Nz;
    const int j = (int)(rr % in.Nth);
    const int i = (int)(rr / in.Nth);
    const int64_t nc = in.nc;
    int64_t nb[7];
    nb[0] = c;
    nb[1] = k > 0 ? c - 1 : c;
    nb[2] = k < in.Nz - 1 ? c + 1 : c;
    nb[3] = i > 0 ? c - (int64_t)in.Nth * in.Nz : c;
    nb[4] = i < in.Nr - 1 ? c + (int64_t)in.Nth * in.Nz : c;
    const int jm = j > 0 ? j - 1 : in.Nth - 1, jp = j < in.Nth - 1 ? j + 1 : 0;
    nb[5] = ((int64_t)i * in.Nth + jm) * in.Nz + k;
    nb[6] = ((int64_t)i * in.Nth + jp) * in.Nz + k;
    const double ts = nrm[12];
#pragma unroll
    for (int v = 0; v < 6; ++v) {
        const double a0 = in.A[v * nc + c];
        const double sc = in.atol7[v] + in.rtol * fabs(a0);
        f[v] = (float)fasinh(a0 / nrm[v]);
#pragma unroll
        for (int p = 1; p < 7; ++p) f[6 + (p - 1) * 6 + v] = (float)fasinh((in.A[v * nc + nb[p]] - a0) / nrm[6 + v]);
#pragma unroll
        for (int p = 0; p < 7; ++p) {
            const int64_t q = v * nc + nb[p];
            f[42 + p * 6 + v] = (float)fasinh((in.A[q] - in.B[q]) / sc / ts);
        }
        f[84 + v] = (float)fasinh(in.dt_tgt * in.fA[v * nc + c] / sc / ts);
    }
    f[90] = (float)fmin(in.dt_tgt / in.dt_ab, 10.0);
    f[91] = (float)(log10(in.h) / 4.0);
    f[92] = (float)in.stage;
#pragma unroll
    for (int q = 0; q < 4; ++q) f[93 + q] = in.step_code == q ? 1.0f : 0.0f;
}

__global__ void k_features(StageInputs in, const double* __restrict__ nrm, int64_t first, int64_t stride,
                           int64_t cnt, bf16* __restrict__ X, int64_t xr, int64_t row0) {
    const int64_t jj = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (jj >= cnt) return;
    const int64_t c = first + jj * stride;
    float f[NIN];
#pragma unroll
    for (int q = 0; q < NIN; ++q) f[q] = 0.0f;
    cell_features(in, nrm, c, f);
    const int64_t row = row0 + jj;
#pragma unroll
    for (int p = 0; p < NIN / 8; ++p) {
        bf16 wb[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) wb[q] = __float2bfloat16_rn(f[p * 8 + q]);
        *reinterpret_cast<uint4*>(X + pidx(row, p * 8, xr)) = *reinterpret_cast<const uint4*>(wb);
    }
}

// The network's correction of the extrapolated start, per cell and variable, in units of that
// cell's extrapolated increment |z_ext - A| plus 1 % of the error scale s: the extrapolation error
// grows with the local rate of change (fronts, blowdown) and vanishes in quiet stages, so a target
// in fixed error-scale units would give the network a constant error floor that quiet stages, where
// the extrapolation is already close, cannot afford.
__device__ __forceinline__ double increment_unit(double zext, double a, double sc) { return fabs(zext - a) + 1e-2 * sc; }

// pred[v][c] = max(pred + out * oscale_v * unit, 0.1 max(ytr, 0)) (the floor for c and q only).
// Corrections smaller than nrm[20] increment units are not applied: where the extrapolation is
// already close (most cells of most stages, within a few percent of the increment) the network's
// own error is of the same size, and leaving those cells alone keeps its gain at the fronts.
__global__ void k_apply(StageInputs in, const double* __restrict__ nrm, const float* __restrict__ O,
                        const double* __restrict__ ytr, double* __restrict__ pred) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= in.nc) return;
    const double gate = nrm[20];
#pragma unroll
    for (int v = 0; v < 6; ++v) {
        const int64_t q = v * in.nc + c;
        const double sc = in.atol7[v] + in.rtol * fabs(in.A[q]);
        const double corr = (double)O[c * NOUT + v] * nrm[13 + v];
        if (fabs(corr) < gate) continue;
        double z = pred[q] + corr * increment_unit(pred[q], in.A[q], sc);
        if (v < 5) z = fmax(z, 0.1 * fmax(ytr[q], 0.0));
        pred[q] = z;
    }
}

__global__ void k_targets(StageInputs in, const double* __restrict__ zs, const double* __restrict__ ze, int64_t first,
                          int64_t stride, int64_t cnt, float* __restrict__ T, int64_t row0) {
    const int64_t jj = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (jj >= cnt) return;
    const int64_t c = first + jj * stride;
    float* t = T + (row0 + jj) * 8;
#pragma unroll
    for (int v = 0; v < 6; ++v) {
        const int64_t q = v * in.nc + c;
        const double sc = in.atol7[v] + in.rtol * fabs(in.A[q]);
        t[v] = (float)((zs[q] - ze[q]) / increment_unit(ze[q], in.A[q], sc));
    }
    t[6] = 1.0f;
    t[7] = 0.0f;
}

// ------------------------------------------------------------------------------------ training
// Gradient of parameter q: the weight-gradient partials (or the bias column sums) summed in CTA order.
__device__ float param_grad(int64_t q, const float* __restrict__ part, const float* __restrict__ bsum) {
    // part: [4 products][NSPLIT][128][128] ; bsum: [4 layers][NB/128][128]
    const int64_t PS = (int64_t)NSPLIT * 128 * 128, TB = NB / 128;
    float g = 0.0f;
    int layer = -1, m = 0, n = 0, nn = 0;
    bool bias = false;
    if (q < OFF_B1) { layer = 0; m = (int)(q / NIN); n = (int)(q % NIN); nn = NIN; }
    else if (q < OFF_W2) { layer = 0; bias = true; n = (int)(q - OFF_B1); nn = NH; }
    else if (q < OFF_B2) { layer = 1; m = (int)((q - OFF_W2) / NH); n = (int)((q - OFF_W2) % NH); nn = NH; }
    else if (q < OFF_W3) { layer = 1; bias = true; n = (int)(q - OFF_B2); nn = NH; }
    else if (q < OFF_B3) { layer = 2; m = (int)((q - OFF_W3) / NH); n = (int)((q - OFF_W3) % NH); nn = NH; }
    else if (q < OFF_W4) { layer = 2; bias = true; n = (int)(q - OFF_B3); nn = NH; }
    else if (q < OFF_B4) {   // W4[o][h] = dW4^T[h][o]
        layer = 3;
        const int o = (int)((q - OFF_W4) / NH), h = (int)((q - OFF_W4) % NH);
        m = h; n = o; nn = NOUT;
    } else { layer = 3; bias = true; n = (int)(q - OFF_B4); nn = NOUT; }
    if (bias) {
        const int w = layer == 3 ? NOUT : NH;
        for (int64_t b = 0; b < TB; ++b) g += bsum[layer * TB * 128 + b * w + n];
    } else {
        for (int sp = 0; sp < NSPLIT; ++sp) g += part[layer * PS + ((int64_t)sp * 128 + m) * nn + n];
    }
    return g;
}

__global__ void k_collect_grad(const float* __restrict__ part, const float* __restrict__ bsum, float* __restrict__ G) {
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < NPARAM) G[q] = param_grad(q, part, bsum);
}

// bf16 operand copies of parameter q: W (rows = outputs) and W^T (rows = inputs) panels
struct Packed {
    bf16 *W1, *W2, *W3, *W4, *W2t, *W3t, *W4t;
};
__device__ __forceinline__ void pack_param(const Packed& k, int64_t q, float p) {
    const bf16 w = __float2bfloat16_rn(p);
    if (q < OFF_B1) {
        k.W1[pidx(q / NIN, q % NIN, NH)] = w;
    } else if (q >= OFF_W2 && q < OFF_B2) {
        const int m = (int)((q - OFF_W2) / NH), n = (int)((q - OFF_W2) % NH);
        k.W2[pidx(m, n, NH)] = w;
        k.W2t[pidx(n, m, NH)] = w;
    } else if (q >= OFF_W3 && q < OFF_B3) {
        const int m = (int)((q - OFF_W3) / NH), n = (int)((q - OFF_W3) % NH);
        k.W3[pidx(m, n, NH)] = w;
        k.W3t[pidx(n, m, NH)] = w;
    } else if (q >= OFF_W4 && q < OFF_B4) {
        const int o = (int)((q - OFF_W4) / NH), h = (int)((q - OFF_W4) % NH);
        k.W4[pidx(o, h, NOUT)] = w;
        k.W4t[pidx(h, o, NH)] = w;
    }
}

// A training step's end: gradient, Adam and operand copies of each parameter.
__global__ void k_update(const float* __restrict__ part, const float* __restrict__ bsum, float* __restrict__ P,
                         float* __restrict__ Mo, float* __restrict__ Vo, float lr, float b1, float b2, float eps, float c1,
                         float c2, Packed k) {
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= NPARAM) return;
    const float g = param_grad(q, part, bsum);
    const float m = b1 * Mo[q] + (1.0f - b1) * g;
    const float v = b2 * Vo[q] + (1.0f - b2) * g * g;
    Mo[q] = m;
    Vo[q] = v;
    const float p = P[q] - lr * (m / c1) / (sqrtf(v / c2) + eps);
    P[q] = p;
    pack_param(k, q, p);
}

__global__ void k_pack_weights(const float* __restrict__ P, Packed k) {
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < NPARAM) pack_param(k, q, P[q]);
}

static unsigned g1(int64_t n, int b = 256) { return (unsigned)((n + b - 1) / b); }

static Packed packed(const dv_mlp* net) { return Packed{net->W1, net->W2, net->W3, net->W4, net->W2t, net->W3t, net->W4t}; }

static int pack(dv_mlp* net, cudaStream_t s) {
    DV_LAUNCH(dv::K_MLP, s, k_pack_weights<<<g1(NPARAM), 256, 0, s>>>(net->P, packed(net)));
    return launch_ok("k_pack_weights");
}

static ChainP chain_of(dv_mlp* net, const bf16* X, int64_t xr, int64_t rows_valid) {
    ChainP g;
    memset(&g, 0, sizeof g);
    g.X = X; g.xr = xr; g.rows_valid = rows_valid; g.P = net->P; g.err = net->d_err;
    g.W1 = net->W1; g.W2 = net->W2; g.W3 = net->W3; g.W4 = net->W4; g.W4t = net->W4t; g.W3t = net->W3t; g.W2t = net->W2t;
    return g;
}

// Forward + backward of one batch (draw < 0: the rows of Xb/Xbt/Tb; else step `draw` of the batches drawn from
// the recorded samples with `seed`); leaves the weight-gradient partials in net->part, the bias sums in
// net->bpart and the loss partials in lossp.
static int grad_batch(dv_mlp* net, int64_t rows_valid, int64_t seed, int64_t draw, float* lossp, cudaStream_t s) {
    ChainP g = draw < 0 ? chain_of(net, net->Xb, NB, rows_valid) : chain_of(net, net->Xs, net->cap, rows_valid);
    if (draw >= 0) {
        g.Ts = net->Ts; g.nrm = net->norm; g.count = net->count; g.seed = seed; g.step = draw;
    }
    g.Xbt = net->Xbt; g.tgt = net->Tb; g.dscale = 2.0f / (float)((double)rows_valid * NOUT_USED);
    g.lossp = lossp; g.bsum = net->bpart;
    g.H1t = net->H1t; g.H2t = net->H2t; g.H3t = net->H3t; g.D4t = net->D4t; g.D3t = net->D3t; g.D2t = net->D2t; g.D1t = net->D1t;
    DV_TRY(chain<true>(g, NB / 128, s));
    // weight gradients: K = samples split over NSPLIT CTAs each
    const int64_t PS = (int64_t)NSPLIT * 128 * 128;
    GemmBatch w;
    w.per = NSPLIT; w.kpanels = NB / 8 / NSPLIT; w.split = 1; w.err = net->d_err;
    w.p[0] = GemmP{net->D1t, NH, net->Xbt, NIN, NIN, net->part};
    w.p[1] = GemmP{net->D2t, NH, net->H1t, NH, NH, net->part + PS};
    w.p[2] = GemmP{net->D3t, NH, net->H2t, NH, NH, net->part + 2 * PS};
    w.p[3] = GemmP{net->H3t, NH, net->D4t, NOUT, NOUT, net->part + 3 * PS};
    return gemm(w, 4, s);
}

static int forward_rows(dv_mlp* net, const bf16* X, int64_t rows, int64_t rows_valid, float* out, cudaStream_t s) {
    ChainP g = chain_of(net, X, rows, rows_valid);
    g.out = out;
    return chain<false>(g, (int)(rows / 128), s);
}

int predict(dv_mlp* net, const StageInputs& in, const double* ytr, double* pred, cudaStream_t s) {
    const int64_t rows = (in.nc + 127) / 128 * 128;
    if (rows > net->inf_rows) {
        set_error("dv_mlp: inference buffers smaller than the model (call dv_mlp_reserve)");
        return DV_ERR_ARG;
    }
    DV_LAUNCH(dv::K_MLP, s, k_features<<<g1(in.nc, 128), 128, 0, s>>>(in, net->norm, 0, 1, in.nc, net->Xi, rows, 0));
    DV_CUDA(cudaGetLastError());
    DV_TRY(forward_rows(net, net->Xi, rows, in.nc, net->Oi, s));
    DV_LAUNCH(dv::K_MLP, s, k_apply<<<g1(in.nc), 256, 0, s>>>(in, net->norm, net->Oi, ytr, pred));
    return launch_ok("k_apply");
}

int record_features(dv_mlp* net, const StageInputs& in, int64_t first, int64_t stride, int64_t cnt, cudaStream_t s) {
    if (net->count + cnt > net->cap) return DV_OK;
    DV_LAUNCH(dv::K_MLP, s, k_features<<<g1(cnt, 128), 128, 0, s>>>(in, net->norm, first, stride, cnt, net->Xs, net->cap,
                                                                      net->count));
    return launch_ok("k_features");
}

int record_targets(dv_mlp* net, const StageInputs& in, const double* zstar, const double* zext, int64_t first,
                   int64_t stride, int64_t cnt, cudaStream_t s) {
    if (net->count + cnt > net->cap) return DV_OK;
    DV_LAUNCH(dv::K_MLP, s, k_targets<<<g1(cnt), 256, 0, s>>>(in, zstar, zext, first, stride, cnt, net->Ts, net->count));
    DV_CUDA(cudaGetLastError());
    net->count += cnt;
    return DV_OK;
}

}  // namespace mlp

int selftest_mbar_timeout(int polls, int* err, cudaStream_t s) {
    mlp::k_selftest_mbar<<<1, 32, 0, s>>>(polls, err);
    DV_CUDA(cudaGetLastError());
    return DV_OK;
}
}  // namespace dv

using namespace dv;
using namespace dv::mlp;

namespace {
template <class T>
int dalloc(T** p, int64_t n) {
    if (cudaMalloc((void**)p, sizeof(T) * (size_t)std::max<int64_t>(n, 1)) != cudaSuccess)
        return cuda_fail(cudaGetLastError(), "cudaMalloc(mlp)");
    return cudaMemset(*p, 0, sizeof(T) * (size_t)std::max<int64_t>(n, 1)) == cudaSuccess ? DV_OK
                                                                                       : cuda_fail(cudaGetLastError(), "cudaMemset(mlp)");
}
void bf16_round_host(const float* x, int64_t n, std::vector<uint16_t>& out) {
    out.resize(n);
    for (int64_t i = 0; i < n; ++i) {
        uint32_t u;
        memcpy(&u, &x[i], 4);
        const uint32_t r = u + 0x7FFFu + ((u >> 16) & 1u);   // round to nearest even (finite inputs)
        out[i] = (uint16_t)(r >> 16);
    }
}
}  // namespace

extern "C" {

int dv_mlp_create(int64_t sample_capacity, uint64_t seed, dv_mlp** out) {
    std::lock_guard<std::recursive_mutex> lk_(dv::capture_mutex());
    if (!out || sample_capacity < 0) { set_error("dv_mlp_create: bad argument"); return DV_ERR_ARG; }
    dv_mlp* n = new dv_mlp();
    n->cap = (sample_capacity + NB - 1) / NB * NB;
    int rc = DV_OK;
    const int64_t TB = NB / 128;
    auto A = [&](auto** p, int64_t cnt) { if (rc == DV_OK) rc = dalloc(p, cnt); };
    A(&n->P, NPARAM); A(&n->G, NPARAM); A(&n->Mo, NPARAM); A(&n->Vo, NPARAM);
    A(&n->W1, (int64_t)NH * NIN); A(&n->W2, (int64_t)NH * NH); A(&n->W3, (int64_t)NH * NH); A(&n->W4, (int64_t)NOUT * NH);
    A(&n->W2t, (int64_t)NH * NH); A(&n->W3t, (int64_t)NH * NH); A(&n->W4t, (int64_t)NOUT * NH);
    A(&n->norm, NNORM);
    A(&n->Xs, std::max<int64_t>(n->cap, NB) * NIN); A(&n->Ts, std::max<int64_t>(n->cap, NB) * 8);
    A(&n->Xb, (int64_t)NB * NIN); A(&n->Xbt, (int64_t)NB * NIN); A(&n->Tb, (int64_t)NB * 8);
    for (bf16** p : {&n->H1t, &n->H2t, &n->H3t, &n->D3t, &n->D2t, &n->D1t})
        A(p, (int64_t)NB * NH);
    A(&n->D4t, (int64_t)NB * NOUT);
    A(&n->part, 4LL * NSPLIT * 128 * 128); A(&n->bpart, 4LL * TB * 128); A(&n->lossp, LOSS_KEEP * TB);
    A(&n->d_err, 1);
    if (rc == DV_OK && cudaMallocHost((void**)&n->h_loss, sizeof(float) * LOSS_KEEP * TB) != cudaSuccess)
        rc = cuda_fail(cudaGetLastError(), "cudaMallocHost(mlp)");
    if (rc != DV_OK) { dv_mlp_destroy(n); return rc; }
    // initial parameters: uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) hidden weights, zero biases, zero output
    // layer (the untrained network predicts no correction: the plain extrapolation)
    std::vector<float> P(NPARAM, 0.0f);
    uint64_t st = seed * 0x9e3779b97f4a7c15ull + 1;
    auto uni = [&]() {
        st ^= st << 13; st ^= st >> 7; st ^= st << 17;
        return (double)(st >> 11) * (1.0 / 9007199254740992.0);
    };
    auto fill = [&](int64_t off, int64_t cnt, double fan) {
        const double a = 1.0 / std::sqrt(fan);
        for (int64_t i = 0; i < cnt; ++i) P[off + i] = (float)((2.0 * uni() - 1.0) * a);
    };
    fill(OFF_W1, (int64_t)NH * NIN, NFEAT);
    fill(OFF_W2, (int64_t)NH * NH, NH);
    fill(OFF_W3, (int64_t)NH * NH, NH);
    double nrm[NNORM] = {0.02, 0.5, 40.0, 1.0, 5.0, 1e7, 2e-3, 5e-2, 4.0, 0.1, 0.5, 1e6, 10.0,
                         1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 8.0};
    rc = dv_mlp_set_params(n, P.data(), NPARAM, nrm, NNORM);
    if (rc != DV_OK) { dv_mlp_destroy(n); return rc; }
    *out = n;
    return DV_OK;
}

int dv_mlp_destroy(dv_mlp* n) {
    std::lock_guard<std::recursive_mutex> lk_(dv::capture_mutex());
    if (!n) return DV_OK;
    void* ptrs[] = {n->P, n->G, n->Mo, n->Vo, n->W1, n->W2, n->W3, n->W4, n->W2t, n->W3t, n->W4t, n->norm, n->Xs, n->Ts,
                    n->Xb, n->Xbt, n->H1t, n->H2t, n->H3t, n->D4t, n->D3t, n->D2t, n->D1t, n->Tb, n->part, n->bpart,
                    n->lossp, n->Xi, n->Oi, n->d_err};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (n->h_loss) cudaFreeHost(n->h_loss);
    delete n;
    return DV_OK;
}

int dv_mlp_reserve(dv_mlp* n, int64_t ncell) {
    if (!n || ncell <= 0) { set_error("dv_mlp_reserve: bad argument"); return DV_ERR_ARG; }
    const int64_t rows = (ncell + 127) / 128 * 128;
    if (rows <= n->inf_rows) return DV_OK;
    for (void* p : {(void*)n->Xi, (void*)n->Oi})
        if (p) cudaFree(p);
    n->Xi = nullptr;
    n->Oi = nullptr;
    n->inf_rows = 0;
    int rc = dalloc(&n->Xi, rows * NIN);
    if (rc == DV_OK) rc = dalloc(&n->Oi, rows * NOUT);
    if (rc == DV_OK) n->inf_rows = rows;
    return rc;
}

int dv_mlp_set_params(dv_mlp* n, const float* params, int64_t nparams, const double* norm, int32_t nnorm) {
    if (!n || !params || nparams != NPARAM || (norm && nnorm != NNORM)) {
        set_error("dv_mlp_set_params: expected DV_MLP_NPARAM parameters and DV_MLP_NNORM constants");
        return DV_ERR_ARG;
    }
    DV_CUDA(cudaMemcpy(n->P, params, sizeof(float) * NPARAM, cudaMemcpyHostToDevice));
    DV_CUDA(cudaMemset(n->Mo, 0, sizeof(float) * NPARAM));
    DV_CUDA(cudaMemset(n->Vo, 0, sizeof(float) * NPARAM));
    n->adam_t = 0;
    if (norm) {
        memcpy(n->norm_h, norm, sizeof(double) * NNORM);
        DV_CUDA(cudaMemcpy(n->norm, norm, sizeof(double) * NNORM, cudaMemcpyHostToDevice));
    }
    DV_TRY(pack(n, 0));
    DV_CUDA(cudaDeviceSynchronize());
    return DV_OK;
}

int dv_mlp_get_params(const dv_mlp* n, float* params, double* norm) {
    if (!n || !params) { set_error("dv_mlp_get_params: null argument"); return DV_ERR_ARG; }
    DV_CUDA(cudaMemcpy(params, n->P, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost));
    if (norm) memcpy(norm, n->norm_h, sizeof(double) * NNORM);
    return DV_OK;
}

int64_t dv_mlp_sample_count(const dv_mlp* n) { return n ? n->count : -1; }

int dv_mlp_get_samples(const dv_mlp* n, int64_t first, int64_t count, float* X, float* T) {
    if (!n || first < 0 || count < 0 || first + count > n->count || (!X && !T)) {
        set_error("dv_mlp_get_samples: bad argument");
        return DV_ERR_ARG;
    }
    if (count == 0) return DV_OK;
    if (X) {        // the store is in panels of 8 features: copy each panel's rows, then transpose
        std::vector<uint16_t> pan((size_t)count * 8);
        for (int p = 0; p < NIN / 8; ++p) {
            DV_CUDA(cudaMemcpy(pan.data(), n->Xs + pidx(first, p * 8, n->cap), sizeof(uint16_t) * pan.size(),
                               cudaMemcpyDeviceToHost));
            for (int64_t r = 0; r < count; ++r)
                for (int q = 0; q < 8; ++q) {
                    const uint32_t bits = (uint32_t)pan[(size_t)r * 8 + q] << 16;
                    float v;
                    memcpy(&v, &bits, sizeof v);
                    X[(size_t)r * NIN + p * 8 + q] = v;
                }
        }
    }
    if (T) DV_CUDA(cudaMemcpy(T, n->Ts + first * 8, sizeof(float) * (size_t)count * 8, cudaMemcpyDeviceToHost));
    return DV_OK;
}

int dv_mlp_clear_samples(dv_mlp* n) {
    if (!n) { set_error("null argument"); return DV_ERR_ARG; }
    n->count = 0;
    return DV_OK;
}

// Forward pass of rows of host features (row-major fp32, rounded to bf16) -> outputs [rows][NOUT].
int dv_mlp_forward_host(dv_mlp* n, const float* X, int64_t rows, float* out) {
    if (!n || !X || !out || rows <= 0) { set_error("dv_mlp_forward_host: bad argument"); return DV_ERR_ARG; }
    const int64_t R = (rows + 127) / 128 * 128;
    DV_TRY(dv_mlp_reserve(n, R));
    std::vector<uint16_t> xb;
    bf16_round_host(X, rows * NIN, xb);
    std::vector<uint16_t> panel((size_t)R * NIN, 0);
    for (int64_t r = 0; r < rows; ++r)
        for (int k = 0; k < NIN; ++k) panel[pidx(r, k, R)] = xb[r * NIN + k];
    DV_CUDA(cudaMemcpy(n->Xi, panel.data(), panel.size() * 2, cudaMemcpyHostToDevice));
    DV_TRY(forward_rows(n, n->Xi, R, rows, n->Oi, 0));
    DV_CUDA(cudaMemcpy(out, n->Oi, sizeof(float) * rows * NOUT, cudaMemcpyDeviceToHost));
    int e = 0;
    DV_CUDA(cudaMemcpy(&e, n->d_err, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) { set_error("dv_mlp: a tensor-core product's completion wait timed out"); return DV_ERR_CUDA; }
    return DV_OK;
}

// One tensor-core product D [M][N] = A [M][K] B[N][K]^T of host fp32 matrices rounded to BF16 (M a
// multiple of 128, N a multiple of 16 up to 128, K a multiple of 16), FP32 result: the check of the
// product kernel itself.  Allocates its device buffers.
int dv_mlp_gemm_host(int32_t M, int32_t N, int32_t K, const float* A, const float* B, float* D) {
    if (M <= 0 || M % 128 || N < 16 || N > 128 || N % 16 || K <= 0 || K % 16 || !A || !B || !D) {
        set_error("dv_mlp_gemm_host: M multiple of 128, N in 16..128 multiple of 16, K multiple of 16");
        return DV_ERR_ARG;
    }
    std::vector<uint16_t> ab, bb;
    bf16_round_host(A, (int64_t)M * K, ab);
    bf16_round_host(B, (int64_t)N * K, bb);
    std::vector<uint16_t> ap((size_t)M * K), bp((size_t)N * K);
    for (int64_t r = 0; r < M; ++r)
        for (int k = 0; k < K; ++k) ap[pidx(r, k, M)] = ab[r * K + k];
    for (int64_t r = 0; r < N; ++r)
        for (int k = 0; k < K; ++k) bp[pidx(r, k, N)] = bb[r * K + k];
    bf16 *dA = nullptr, *dB = nullptr;
    float* dD = nullptr;
    int* derr = nullptr;
    int rc = DV_OK;
    if (cudaMalloc((void**)&dA, ap.size() * 2) != cudaSuccess || cudaMalloc((void**)&dB, bp.size() * 2) != cudaSuccess ||
        cudaMalloc((void**)&dD, sizeof(float) * (size_t)M * N) != cudaSuccess || cudaMalloc((void**)&derr, sizeof(int)) != cudaSuccess)
        rc = cuda_fail(cudaGetLastError(), "cudaMalloc(gemm check)");
    if (rc == DV_OK) {
        cudaMemcpy(dA, ap.data(), ap.size() * 2, cudaMemcpyHostToDevice);
        cudaMemcpy(dB, bp.data(), bp.size() * 2, cudaMemcpyHostToDevice);
        cudaMemset(derr, 0, sizeof(int));
        GemmBatch g;
        memset(&g, 0, sizeof g);
        g.p[0] = GemmP{dA, M, dB, N, N, dD};
        g.per = M / 128; g.kpanels = K / 8; g.err = derr;
        rc = gemm(g, 1, 0);
        if (rc == DV_OK && cudaDeviceSynchronize() != cudaSuccess) rc = cuda_fail(cudaGetLastError(), "k_gemm");
        int e = 0;
        if (rc == DV_OK) cudaMemcpy(&e, derr, sizeof(int), cudaMemcpyDeviceToHost);
        if (rc == DV_OK && e) { set_error("dv_mlp: a tensor-core product's completion wait timed out"); rc = DV_ERR_CUDA; }
        if (rc == DV_OK) cudaMemcpy(D, dD, sizeof(float) * (size_t)M * N, cudaMemcpyDeviceToHost);
    }
    for (void* q : {(void*)dA, (void*)dB, (void*)dD, (void*)derr})
        if (q) cudaFree(q);
    return rc;
}

// Gradient of the batch loss mean((O - T)^2) over the used outputs for host features X [rows][NIN] and
// targets T [rows][8] (already scaled; rows <= DV_MLP_BATCH), into grad [DV_MLP_NPARAM]; *loss = the mean.
int dv_mlp_gradient_host(dv_mlp* n, const float* X, const float* T, int64_t rows, float* grad, double* loss) {
    if (!n || !X || !T || !grad || rows <= 0 || rows > NB) { set_error("dv_mlp_gradient_host: bad argument"); return DV_ERR_ARG; }
    std::vector<uint16_t> xb;
    bf16_round_host(X, rows * NIN, xb);
    std::vector<uint16_t> rm((size_t)NB * NIN, 0), fm((size_t)NB * NIN, 0);
    std::vector<float> tb((size_t)NB * 8, 0.0f);
    for (int64_t r = 0; r < rows; ++r) {
        for (int k = 0; k < NIN; ++k) {
            rm[pidx(r, k, NB)] = xb[r * NIN + k];
            fm[pidx(k, r, NIN)] = xb[r * NIN + k];
        }
        for (int k = 0; k < 8; ++k) tb[r * 8 + k] = T[r * 8 + k];
    }
    DV_CUDA(cudaMemcpy(n->Xb, rm.data(), rm.size() * 2, cudaMemcpyHostToDevice));
    DV_CUDA(cudaMemcpy(n->Xbt, fm.data(), fm.size() * 2, cudaMemcpyHostToDevice));
    DV_CUDA(cudaMemcpy(n->Tb, tb.data(), tb.size() * 4, cudaMemcpyHostToDevice));
    DV_TRY(grad_batch(n, rows, 0, -1, n->lossp, 0));
    DV_LAUNCH(dv::K_MLP, 0, k_collect_grad<<<g1(NPARAM), 256, 0, 0>>>(n->part, n->bpart, n->G));
    DV_TRY(launch_ok("k_collect_grad"));
    DV_CUDA(cudaMemcpy(grad, n->G, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost));
    std::vector<float> lp(NB / 128);
    DV_CUDA(cudaMemcpy(lp.data(), n->lossp, sizeof(float) * lp.size(), cudaMemcpyDeviceToHost));
    double s = 0.0;
    for (float x : lp) s += x;
    if (loss) *loss = s / ((double)rows * NOUT_USED);
    int e = 0;
    DV_CUDA(cudaMemcpy(&e, n->d_err, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) { set_error("dv_mlp: a tensor-core product's completion wait timed out"); return DV_ERR_CUDA; }
    return DV_OK;
}

// Adam on the recorded samples: `steps` batches of DV_MLP_BATCH samples drawn (with replacement, by a
// hash of seed, step and row) from the recorded set; the output scales are set first from the recorded
// targets (RMS per variable) unless keep_scales.  loss_hist (host, `steps` entries) receives each
// batch's mean loss when non-NULL.
int dv_mlp_train(dv_mlp* n, int32_t steps, float lr, uint64_t seed, int32_t keep_scales, float* loss_hist, void* stream) {
    if (!n || steps < 0) { set_error("dv_mlp_train: bad argument"); return DV_ERR_ARG; }
    if (n->count < NB) { set_error("dv_mlp_train: fewer recorded samples than one batch"); return DV_ERR_ARG; }
    cudaStream_t s = (cudaStream_t)stream;
    if (!keep_scales) {
        std::vector<float> T((size_t)n->count * 8);
        DV_CUDA(cudaMemcpyAsync(T.data(), n->Ts, sizeof(float) * T.size(), cudaMemcpyDeviceToHost, s));
        DV_CUDA(cudaStreamSynchronize(s));
        for (int v = 0; v < NOUT_USED; ++v) {
            double ss = 0.0;
            for (int64_t r = 0; r < n->count; ++r) ss += (double)T[r * 8 + v] * T[r * 8 + v];
            n->norm_h[13 + v] = std::max(std::sqrt(ss / (double)n->count), 1e-6);
        }
        DV_CUDA(cudaMemcpyAsync(n->norm, n->norm_h, sizeof(double) * NNORM, cudaMemcpyHostToDevice, s));
    }
    const int TB = NB / 128;
    for (int it = 0; it < steps; ++it) {
        const int slot = it % LOSS_KEEP;
        DV_TRY(grad_batch(n, NB, (int64_t)(seed & 0x7fffffffffffll), n->adam_t, n->lossp + slot * TB, s));
        n->adam_t += 1;
        const float b1 = 0.9f, b2 = 0.999f;
        const float c1 = 1.0f - std::pow(b1, (float)n->adam_t), c2 = 1.0f - std::pow(b2, (float)n->adam_t);
        DV_LAUNCH(dv::K_MLP, s, k_update<<<g1(NPARAM), 256, 0, s>>>(n->part, n->bpart, n->P, n->Mo, n->Vo, lr, b1, b2, 1e-8f, c1,
                                                                   c2, packed(n)));
        DV_CUDA(cudaGetLastError());
        if (loss_hist && (slot == LOSS_KEEP - 1 || it == steps - 1)) {      // the partial sums of up to LOSS_KEEP steps at once
            DV_CUDA(cudaMemcpyAsync(n->h_loss, n->lossp, sizeof(float) * (slot + 1) * TB, cudaMemcpyDeviceToHost, s));
            DV_CUDA(cudaStreamSynchronize(s));
            for (int q = 0; q <= slot; ++q) {
                double t = 0.0;
                for (int b = 0; b < TB; ++b) t += n->h_loss[q * TB + b];
                loss_hist[it - slot + q] = (float)(t / ((double)NB * NOUT_USED));
            }
        }
    }
    DV_CUDA(cudaStreamSynchronize(s));
    int e = 0;
    DV_CUDA(cudaMemcpy(&e, n->d_err, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) { set_error("dv_mlp: a tensor-core product's completion wait timed out"); return DV_ERR_CUDA; }
    return DV_OK;
}

}  // extern "C"
