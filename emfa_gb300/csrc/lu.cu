// Dense LU factorisation of the impedance matrix, for solves that factor once
// and then solve and refine (the batched EFIE problems, whose restarted
// Krylov solves need hundreds of iterations).  The reference has no dense
// direct solver on this path: EMSolver/EFIE.cpp:89 keeps a commented-out
// Eigen LU, and its EFIE/CFIE solves are GMRES/BiCGStab only.
//
// Factorisation, FP32 complex, blocked right-looking, block LU_NB = 64, row
// exchanges within each diagonal block (the rows of block k only trade places
// among themselves).  One step per diagonal block:
//   k_lu_diag     one CTA: pivoted LU of the diagonal block, then explicit
//                 inverses of its unit-lower and upper factors
//   k_lu_panels   U12 = L11^-1 P A12 and L21 = A21 U11^-1 with those
//                 inverses (P the block's row exchange, applied by reading
//                 A12 through the permutation), and their split-FP16
//                 operand planes, scaled per column / row by powers of two
//   k_lu_update_tc  A22 -= L21 U12 on the tensor cores (tcgen05, K = 128
//                 real per block), tiles of 256 or 64 rows x 64 complex
//                 columns of A22 moved through shared memory by TMA
// While two or more blocks follow, blocks go in pairs: the first block
// updates only the second block's columns and rows, and one pass with both
// blocks' panels (packed together by the second's k_lu_panels, K = 128
// complex) updates the rest, so A22 is read and written once per two blocks.
// The chain that every block waits for (panels, the next block's 64 columns,
// its diagonal block) runs on a high-priority stream as dependent launches,
// the update of the other columns beside it on the caller's.  The row
// exchanges reach the columns left of each block in one pass at the end
// (k_lu_rowperm_left).
// Up to a few thousand unknowns a factorisation is that chain's latency: at
// n = 1470, per block, diagonal 38 us (63 with one warp's panel steps),
// panels 8 to 9 (24 with 64-wide chunks and loads waited for one by one),
// columns 3.8 and 5.3 (11 and 16), and no gap of more than 1.5 us (a separate
// packing launch was 9.5 a pair and each crossing of streams 3 to 4).  EFIE
// jobs of 8 incidences: n = 480, 1.26 -> 0.88 ms; 1470, 3.50 -> 2.25; 3630,
// 8.85 -> 5.39; 5070, 13.1 -> 8.2.
// Rows of the factor are padded to an even number of complex elements
// (16-byte TMA strides).
// Solve for many right-hand sides (RHS-major, (r, u) at r n + u): gather by
// the row permutation, then one launch for the forward (L) and one for the
// backward (U) sweep (k_lu_wave): a CTA per row block, in wavefront order,
// applies the block's explicit inverse once the blocks before it are solved.
//
// A pivot that is exactly zero is replaced by 1e-30 and recorded in the
// factor's info word, so the caller can fall back to an iterative solve.
#include "emfa_internal.cuh"
#include "gemm.cuh"
#include "lu.cuh"
#include "tcgen05.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

namespace emfa {

namespace {

constexpr int NB = LU_NB;
constexpr int LDS = NB + 1;  // padded shared-memory row

__device__ __forceinline__ float2 cm(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ float2 cfma(float2 a, float2 b, float2 c)  // c + a b
{
    return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
}
__device__ __forceinline__ float2 cinv(float2 a)
{
    const float d = a.x * a.x + a.y * a.y;
    return make_float2(a.x / d, -a.y / d);
}

// Pivoted LU of the diagonal block [k0, k0 + nb)^2 and the inverses of its
// factors.  perm[k0 + i] = the original row now at k0 + i (rows of earlier
// blocks never move into this one, so original = k0 + local index).
//
// Factorisation by 16-column panels.  Rows never move: a pivot row only
// leaves the active set, and its step number is its position in the factor
// (ord, pos).  Per panel:
//   1. the 16 column steps, a chain of latencies: eight warps hold two
//      columns each (lane l: rows l and l + 32).  The warp of a step's column
//      finds the pivot (largest |.|^2 among the active rows, the lowest row
//      on ties: two warp reductions), fetches its row by shuffles, scales the
//      column and updates its own second column at once; after both steps it
//      publishes the multipliers in shared memory, one barrier, and the other
//      warps follow.  660 cycles a step; 1230 with one warp that held all 16
//      columns, 820 with a column a warp and a barrier every step, 690 with
//      four columns a warp.
//   2. all warps: the panel's pivot rows on the columns to its right
//      (unit-lower triangular solve, four lanes per column, each row's
//      entries read ahead of the sums before it: 3.8k -> 1.9k cycles), then
//      the rank-16 update of the active rows there (a thread keeps its
//      column's 16 pivot entries in registers)
// Inverses: the 8 x 8 diagonal blocks of L and U by substitution (a thread
// per column), then three merge levels of the 2 x 2 block inverse,
//   [L11 0; L21 L22]^-1 = [X11 0; -X22 L21 X11  X22],
//   [U11 U12; 0 U22]^-1 = [Y11 -Y11 U12 Y22; 0 Y22],
// each two rounds of small products over all block pairs at once.
// The block's products with their roundings written out (which product of a
// pair is the fused one), so that the factor's bits do not hang on how a
// compiler contracts the code around them.
__device__ __forceinline__ float norm2(float2 a) { return fmaf(a.x, a.x, __fmul_rn(a.y, a.y)); }
__device__ __forceinline__ float2 cmul_rn(float2 a, float2 b)
{
    return make_float2(fmaf(a.x, b.x, -__fmul_rn(a.y, b.y)), fmaf(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float2 csub_rn(float2 x, float2 l, float2 u)  // x - l u
{
    return make_float2(__fsub_rn(x.x, fmaf(l.x, u.x, -__fmul_rn(l.y, u.y))),
                       __fsub_rn(x.y, fmaf(l.y, u.x, __fmul_rn(l.x, u.y))));
}
// 1 / a for a warp's common a: even lanes divide for the real part and odd
// ones for the imaginary, one division deep instead of two
__device__ __forceinline__ float2 cinv_warp(float2 a)
{
    const float d = fmaf(a.y, a.y, __fmul_rn(a.x, a.x));
    const float q = (threadIdx.x & 1 ? -a.y : a.x) / d;
    return make_float2(__shfl_sync(0xffffffffu, q, 0), __shfl_sync(0xffffffffu, q, 1));
}

constexpr int DIAG_THREADS = 512;
constexpr int PW = 16;  // panel width
constexpr int CPW = 2;

// One merge level of the blocked inverses: for every pair of b-blocks on the
// diagonal, T = L21 X11 and T = Y11 U12, then X21 = -X22 T and Y12 = -T Y22.
// Bound by shared-memory reads: a thread takes a tile of RT x CT entries (of
// T, then of X21 or Y12), RT + CT reads for RT CT products (12.2k -> 7.4k
// cycles for b = 32, 4.2k -> 3.1k for 16, 1.8k -> 1.0k for 8, against two
// reads a product).
template <int b>
__device__ __forceinline__ void diag_merge(const float2* __restrict__ D, float2* __restrict__ WL,
                                           float2* __restrict__ WU, float2* __restrict__ TM)
{
    constexpr int pairs = (NB / 2) / b, per = pairs * b * b, NI = (2 * per + DIAG_THREADS - 1) / DIAG_THREADS;
    constexpr int RT = NI >= 4 ? 2 : 1, CT = NI >= 2 ? 2 : 1, RS = b / RT, CS = b / CT;
    static_assert(RT * CT == NI && 2 * pairs * RS * CS == DIAG_THREADS, "one tile a thread");
    const int half = threadIdx.x / (DIAG_THREADS / 2), q = threadIdx.x % (DIAG_THREADS / 2);  // half: L or U
    const int pr = q / (RS * CS), r = (q % (RS * CS)) / CS, c = q % CS, i0 = pr * 2 * b;
    float2* T = TM + half * per + pr * b * b;
    const auto product = [&](const float2* x, int ldx, const float2* y, int ldy, float2 (&s)[RT][CT]) {
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int j = 0; j < CT; ++j) s[i][j] = make_float2(0.f, 0.f);
#pragma unroll 8
        for (int k = 0; k < b; ++k) {
            float2 xv[RT], yv[CT];
#pragma unroll
            for (int i = 0; i < RT; ++i) xv[i] = x[(r + i * RS) * ldx + k];
#pragma unroll
            for (int j = 0; j < CT; ++j) yv[j] = y[k * ldy + c + j * CS];
#pragma unroll
            for (int i = 0; i < RT; ++i)
#pragma unroll
                for (int j = 0; j < CT; ++j) s[i][j] = cfma(xv[i], yv[j], s[i][j]);
        }
    };
    const int d11 = i0 * LDS + i0, d21 = (i0 + b) * LDS + i0, d12 = i0 * LDS + i0 + b, d22 = (i0 + b) * LDS + i0 + b;
    float2 s[RT][CT];
    if (half == 0)
        product(D + d21, LDS, WL + d11, LDS, s);
    else
        product(WU + d11, LDS, D + d12, LDS, s);
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < CT; ++j) T[(r + i * RS) * b + c + j * CS] = s[i][j];
    __syncthreads();
    if (half == 0)
        product(WL + d22, LDS, T, b, s);
    else
        product(T, b, WU + d22, LDS, s);
    float2* O = half == 0 ? WL + d21 : WU + d12;
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < CT; ++j) O[(r + i * RS) * LDS + c + j * CS] = make_float2(-s[i][j].x, -s[i][j].y);
    __syncthreads();
}

__global__ void __launch_bounds__(DIAG_THREADS) k_lu_diag(float2* __restrict__ A, int n, int lda, int k0, int nb,
                                                          int* __restrict__ perm, float2* __restrict__ linv,
                                                          float2* __restrict__ uinv, int* __restrict__ info)
{
    extern __shared__ float2 s_lu[];
    float2* D = s_lu;               // [NB][LDS] the factors, in factor order
    float2* WL = D + NB * LDS;      // [NB][LDS] the block by original row while it is factored, then L^-1
    float2* WU = WL + NB * LDS;     // [NB][LDS] U^-1
    float2* TM = WU + NB * LDS;     // [2048] products of a merge level
    __shared__ float2 lbuf[2][CPW][NB];  // the multipliers of a group of columns
    __shared__ int pos[NB];         // factor position of each row (NB + row while active)
    __shared__ int ord[NB];         // row at each factor position
    __shared__ float2 invd[NB];
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    float2* W = WL;
    griddep_wait();  // launched as a dependent of the update of its columns
#pragma unroll
    for (int t = 0; t < NB * NB / DIAG_THREADS; ++t) {
        const int q = tid + t * DIAG_THREADS, i = q / NB, j = q % NB;
        W[i * LDS + j] = (i < nb && j < nb) ? A[(size_t)(k0 + i) * lda + k0 + j] : make_float2(0.f, 0.f);
    }
    if (tid < NB) pos[tid] = NB + tid;
    __syncthreads();
    unsigned act = (l < nb ? 1u : 0u) | (l + 32 < nb ? 2u : 0u);  // rows l, l + 32 still active
    for (int c0 = 0; c0 < nb; c0 += PW) {
        const int pe = min(PW, nb - c0);  // the panel's pivots
        if (w < PW / CPW) {
            float2 x[2][CPW];  // rows l, l + 32 of the warp's columns
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int c = 0; c < CPW; ++c) x[r][c] = W[(l + 32 * r) * LDS + c0 + w * CPW + c];
#pragma unroll 1
            for (int g = 0; g * CPW < pe; ++g) {
                float2(*lcol)[NB] = lbuf[g & 1];
                if (w == g) {
#pragma unroll
                    for (int q = 0; q < CPW; ++q) {
                        const int j = c0 + g * CPW + q;
                        if (j >= nb) break;  // uniform
                        // the largest |.|^2 among the active rows, then the lowest row that has it
                        const unsigned k0b = act & 1 ? __float_as_uint(norm2(x[0][q])) : 0u;
                        const unsigned k1b = act & 2 ? __float_as_uint(norm2(x[1][q])) : 0u;
                        const unsigned best = __reduce_max_sync(0xffffffffu, max(k0b, k1b));
                        const unsigned row = (act & 1) && k0b == best   ? l
                                             : (act & 2) && k1b == best ? l + 32
                                                                        : 2 * NB;
                        const int p = (int)__reduce_min_sync(0xffffffffu, row);
                        const int pl = p & 31, pr = p >> 5;
                        float2 u[CPW];  // the pivot row
#pragma unroll
                        for (int c = q; c < CPW; ++c) {
                            const float2 v = pr ? x[1][c] : x[0][c];
                            u[c].x = __shfl_sync(0xffffffffu, v.x, pl);
                            u[c].y = __shfl_sync(0xffffffffu, v.y, pl);
                        }
                        if (u[q].x == 0.f && u[q].y == 0.f) {
                            if (l == 0) atomicCAS(info, 0, k0 + j + 1);
                            u[q] = make_float2(1e-30f, 0.f);
                            if (l == pl) {
                                if (pr)
                                    x[1][q] = u[q];
                                else
                                    x[0][q] = u[q];
                            }
                        }
                        if (l == pl) act &= ~(1u << pr);
                        const float2 ipv = cinv_warp(u[q]);
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const bool on = act >> r & 1;
                            const float2 lm = cmul_rn(x[r][q], ipv);
                            x[r][q].x = on ? lm.x : x[r][q].x;
                            x[r][q].y = on ? lm.y : x[r][q].y;
#pragma unroll
                            for (int c = q + 1; c < CPW; ++c) {
                                const float2 y = csub_rn(x[r][c], lm, u[c]);
                                x[r][c].x = on ? y.x : x[r][c].x;
                                x[r][c].y = on ? y.y : x[r][c].y;
                            }
                            lcol[q][l + 32 * r] = x[r][q];
                        }
                        if (l == 0) {
                            ord[j] = p;
                            pos[p] = j;
                        }
                    }
                }
                asm volatile("bar.sync 1, %0;" ::"r"(32 * (PW / CPW)) : "memory");
                if (w != g) {
#pragma unroll
                    for (int q = 0; q < CPW; ++q) {
                        const int j = c0 + g * CPW + q;
                        if (j >= nb) break;  // uniform
                        const int p = ord[j], pl = p & 31, pr = p >> 5;
                        if (l == pl) act &= ~(1u << pr);
                        if (w > g) {
                            float2 lm[2];
#pragma unroll
                            for (int r = 0; r < 2; ++r) lm[r] = lcol[q][l + 32 * r];
#pragma unroll
                            for (int c = 0; c < CPW; ++c) {
                                float2 u = pr ? x[1][c] : x[0][c];
                                u.x = __shfl_sync(0xffffffffu, u.x, pl);
                                u.y = __shfl_sync(0xffffffffu, u.y, pl);
#pragma unroll
                                for (int r = 0; r < 2; ++r) {
                                    const float2 y = csub_rn(x[r][c], lm[r], u);
                                    const bool on = act >> r & 1;
                                    x[r][c].x = on ? y.x : x[r][c].x;
                                    x[r][c].y = on ? y.y : x[r][c].y;
                                }
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int c = 0; c < CPW; ++c) W[(l + 32 * r) * LDS + c0 + w * CPW + c] = x[r][c];
        }
        __syncthreads();
        const int c1 = c0 + PW;  // columns right of the panel
        if (c1 < nb) {
            // the panel's pivot rows on the columns right of it: forward
            // substitution with the panel's unit-lower part, four lanes per
            // column (lane sub keeps the solved entries k = sub mod 4)
            if (w < (4 * (nb - c1) + 31) / 32) {  // whole warps
                const int sub = tid & 3, c = c1 + (tid >> 2), cc = min(c, NB - 1);
                float2 u[PW / 4], lk[PW / 4], a;
#pragma unroll
                for (int t = 0; t < PW / 4; ++t) u[t] = make_float2(0.f, 0.f);
                float2* row = W + ord[c0] * LDS;
                a = row[cc];
#pragma unroll
                for (int i = 0; i < PW; ++i) {
                    // the next pivot row's entries are read ahead of this row's sums
                    float2* next = W + ord[c0 + min(i + 1, PW - 1)] * LDS;
                    float2 ln[PW / 4], an = make_float2(0.f, 0.f);
                    if (i + 1 < PW) {
                        an = next[cc];
#pragma unroll
                        for (int t = 0; t < PW / 4; ++t)
                            if (4 * t < i + 1) ln[t] = next[c0 + sub + 4 * t];
                    }
                    float2 part = make_float2(0.f, 0.f);
#pragma unroll
                    for (int t = 0; t < PW / 4; ++t)
                        if (4 * t < i) {
                            const float2 y = cfma(lk[t], u[t], part);
                            part.x = sub + 4 * t < i ? y.x : part.x;
                            part.y = sub + 4 * t < i ? y.y : part.y;
                        }
                    part.x += __shfl_xor_sync(0xffffffffu, part.x, 1);
                    part.y += __shfl_xor_sync(0xffffffffu, part.y, 1);
                    part.x += __shfl_xor_sync(0xffffffffu, part.x, 2);
                    part.y += __shfl_xor_sync(0xffffffffu, part.y, 2);
                    const float2 v = make_float2(a.x - part.x, a.y - part.y);
                    if ((i & 3) == sub) u[i >> 2] = v;
                    if (sub == 0 && c < nb) row[c] = v;
                    row = next;
                    a = an;
#pragma unroll
                    for (int t = 0; t < PW / 4; ++t)
                        if (4 * t < i + 1) lk[t] = ln[t];
                }
            }
            __syncthreads();
            const int nc = nb - c1, lg = nc > 32 ? 6 : nc > 16 ? 5 : 4;  // 2^lg >= nc columns
            const int c = c1 + (tid & ((1 << lg) - 1));
            if (c < nb) {
                float2 uk[PW];
#pragma unroll
                for (int k = 0; k < PW; ++k) uk[k] = W[ord[c0 + k] * LDS + c];
                for (int r = tid >> lg; r < nb; r += DIAG_THREADS >> lg) {
                    if (pos[r] < NB) continue;
                    float2 s = W[r * LDS + c];
#pragma unroll
                    for (int k = 0; k < PW; ++k) s = csub_rn(s, W[r * LDS + c0 + k], uk[k]);
                    W[r * LDS + c] = s;
                }
            }
            __syncthreads();
        }
    }
    // the factors in factor order: shared memory (rows and columns past nb
    // are zero) and A
#pragma unroll
    for (int t = 0; t < NB * NB / DIAG_THREADS; ++t) {
        const int q = tid + t * DIAG_THREADS, r = q / NB, c = q % NB;
        const int i = r < nb ? pos[r] : r;
        const float2 v = W[r * LDS + c];
        D[i * LDS + c] = v;
        if (r < nb && c < nb) A[(size_t)(k0 + i) * lda + k0 + c] = v;
    }
    if (tid < nb) perm[k0 + tid] = k0 + ord[tid];
    __syncthreads();
    for (int q = tid; q < NB * LDS; q += blockDim.x) {
        WL[q] = make_float2(0.f, 0.f);
        WU[q] = make_float2(0.f, 0.f);
    }
    __syncthreads();
    if (tid < NB) invd[tid] = tid < nb ? cinv(D[tid * LDS + tid]) : make_float2(1.f, 0.f);
    if (tid >= nb && tid < NB) D[tid * LDS + tid] = make_float2(1.f, 0.f);  // identity past the block
    __syncthreads();
    // 8 x 8 diagonal blocks: threads 0..63 columns of L^-1, 64..127 of U^-1
    if (tid < 2 * NB) {
        const int t = tid & 63, b0 = t & ~7, c = t & 7;
        float2 x[8];
        if (tid < NB) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float2 s = make_float2(0.f, 0.f);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (k >= c && k < i) s = cfma(D[(b0 + i) * LDS + b0 + k], x[k], s);
                x[i] = i < c ? make_float2(0.f, 0.f) : i == c ? make_float2(1.f, 0.f) : make_float2(-s.x, -s.y);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) WL[(b0 + i) * LDS + b0 + c] = x[i];
        } else {
#pragma unroll
            for (int i = 7; i >= 0; --i) {
                float2 s = make_float2(0.f, 0.f);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (k > i && k <= c) s = cfma(D[(b0 + i) * LDS + b0 + k], x[k], s);
                x[i] = i > c ? make_float2(0.f, 0.f)
                             : cm(make_float2((i == c ? 1.f : 0.f) - s.x, -s.y), invd[b0 + i]);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) WU[(b0 + i) * LDS + b0 + c] = x[i];
        }
    }
    __syncthreads();
    diag_merge<8>(D, WL, WU, TM);
    diag_merge<16>(D, WL, WU, TM);
    griddep_launch();  // the panels' CTAs take their places during the last level
    diag_merge<32>(D, WL, WU, TM);
    const size_t kb = (size_t)(k0 / NB) * NB * NB;
#pragma unroll
    for (int t = 0; t < NB * NB / DIAG_THREADS; ++t) {
        const int q = tid + t * DIAG_THREADS, i = q / NB, j = q % NB;
        const bool in = i < nb && j < nb;
        linv[kb + q] = in ? WL[i * LDS + j] : make_float2(0.f, 0.f);
        uinv[kb + q] = in ? WU[i * LDS + j] : make_float2(0.f, 0.f);
    }
    __syncthreads();
}

// The row exchanges of every diagonal block applied to the columns left of
// the block (the factor's L part), once the factorisation is done: the
// exchanges stay within a block and those columns are final by then.  CTA
// per (32 columns, block).
__global__ void __launch_bounds__(256) k_lu_rowperm_left(float2* __restrict__ A, int n, int lda,
                                                         const int* __restrict__ perm)
{
    __shared__ float2 T[NB][33];
    __shared__ int moved;
    const int k0 = blockIdx.y * NB, nb = min(NB, n - k0), c0 = blockIdx.x * 32;
    if (c0 >= k0) return;  // uniform over the CTA
    if (threadIdx.x == 0) moved = 0;
    __syncthreads();
    if (threadIdx.x < nb && perm[k0 + threadIdx.x] != k0 + (int)threadIdx.x) moved = 1;
    __syncthreads();
    if (!moved) return;
    for (int q = threadIdx.x; q < nb * 32; q += blockDim.x) {
        const int r = q / 32, c = c0 + q % 32;
        if (c < k0) T[r][q % 32] = A[(size_t)perm[k0 + r] * lda + c];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < nb * 32; q += blockDim.x) {
        const int r = q / 32, c = c0 + q % 32;
        if (c < k0) A[(size_t)(k0 + r) * lda + c] = T[r][q % 32];
    }
}

// ---------------------------------------------------------------------------
// Trailing update on the tensor cores: A22 -= L21 U12 as one real GEMM with
// split-FP16 operands (tcgen05.mma kind::f16, FP32 accumulation in tensor
// memory).  The accumulator is laid out transposed, D[real column][row], so
// that the epilogue's 32 lanes read and write 32 consecutive floats of a row
// of A22 (coalesced):
//   U operand row 2j   = t_j (Re u_kj, -Im u_kj)_k     (K = 2 nb = 128 halves)
//   U operand row 2j+1 = t_j (Im u_kj,  Re u_kj)_k
//   L operand row i    = s_i (Re l_ik,  Im l_ik)_k
//   D[2j + e][i] = t_j s_i (Re, Im)_e (L21 U12)_ij
// with t_j, s_i powers of two per column of U12 and per row of L21 (largest
// |Re|, |Im| scaled into [2^14, 2^15)), each operand split into hi = fp16(x)
// and lo = fp16(x - hi), and D = Uh Lh + Uh Ll + Ul Lh (the lo-lo term is
// below 2^-21 of the product).
// ---------------------------------------------------------------------------
namespace lutc {
constexpr int TM = 128;                                  // real columns of A22 per tile (MMA M): 64 complex
constexpr int KH = 4 * NB;                               // halves per operand row: two blocks' panels
constexpr int U_BYTES = TM * 128;                        // one 64-half K slice of one U plane
constexpr int C_BYTES = 64 * 128 * 4;                    // 64 rows x 64 complex of A22
constexpr int THREADS = 320;                             // producer, MMA, 8 epilogue warps

// TN: rows of A22 per tile (MMA N)
template <int TN>
struct Tile {
    static constexpr bool WIDE = TN == 256;               // two CTAs an SM, else one
    static constexpr int L_BYTES = TN * 128;              // one K slice of one L plane
    static constexpr int STAGE = 2 * U_BYTES + 2 * L_BYTES;  // both planes of both operands: 96 KB, 48 KB
    static constexpr int NST = WIDE ? 1 : 4;              // K slices staged: of the narrow tile all four
    static constexpr int NC = TN / 64;                    // 64-row chunks of A22
    static constexpr int SLOTS = WIDE ? 3 : 1;            // chunks staged: three fill the wide tile's stage
    static constexpr int C_OFF = WIDE ? 0 : NST * STAGE;
    static constexpr int BAR_OFF = WIDE ? STAGE : NST * STAGE + C_BYTES;
    static constexpr int SMEM = BAR_OFF + 1024 /*align*/ + 256 /*barriers*/;
};
}  // namespace lutc

__device__ __forceinline__ float2 col_max_scale(float m)
{
    int e = 0;
    frexpf(m, &e);  // m = f 2^e, f in [0.5, 1); m = 0 gives e = 0
    return make_float2(ldexpf(1.f, 15 - e), ldexpf(1.f, e - 15));
}

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }

// hi/lo FP16 pairs of (a, b)
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo)
{
    const __half ha = __float2half_rn(a), hb = __float2half_rn(b);
    hi = h2_bits(__halves2half2(ha, hb));
    lo = h2_bits(__halves2half2(__float2half_rn(a - __half2float(ha)), __float2half_rn(b - __half2float(hb))));
}

// Panels of step k0, written to A and packed as the trailing update's
// split-FP16 operand planes (rows indexed from k1 = k0 + nb; plane p of the U
// operand starts at row p 2n, of the L operand at row p n):
//   blockIdx.y = 0: U12 = L11^-1 P A12 on the CW-column chunk blockIdx.x,
//                   P the diagonal block's row exchange (row perm[k0 + i] of
//                   A12 is read for row i)
//   blockIdx.y = 1: L21 = A21 U11^-1 on the CW-row chunk blockIdx.x
// The chunk's product is kept in shared memory, scaled per column of U12 /
// row of L21, and written as 16-byte pieces of contiguous operand rows.
constexpr int CW = 32;          // columns or rows of a chunk
constexpr int LDC = CW + 1;     // row of U12's chunk in shared memory
constexpr int CHUNK = NB * LDC > CW * LDS ? NB * LDC : CW * LDS;

__global__ void __launch_bounds__(256) k_lu_panels(float2* __restrict__ A, int n, int lda, int k0, int nb,
                                                   const int* __restrict__ perm, const float2* __restrict__ linv,
                                                   const float2* __restrict__ uinv, __half* __restrict__ Uop,
                                                   __half* __restrict__ Lop, float* __restrict__ inv_t,
                                                   float* __restrict__ inv_s, int pack)
{
    constexpr int NT = CW / 16;       // product entries of a thread along the chunk (4 along the block)
    extern __shared__ float2 s_lu[];
    float2* X = s_lu;           // [NB][LDS] the inverse
    float2* Y = X + NB * LDS;   // the chunk, then the product: [NB][LDC] (U12) or [CW][LDS] (L21)
    float2* P = Y + CHUNK;      // pack 2: the chunk of the block before, laid out like Y
    __shared__ float sc[CW];    // scale of each product column (U12) or row (L21)
    const int mode = blockIdx.y;
    const int k1 = k0 + nb, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    griddep_launch();
    griddep_wait();  // the diagonal block
    const int e0 = k1 + blockIdx.x * CW;  // first column (U12) or row (L21) of the chunk
    const int ne = min(CW, n - e0);
    const float2* iv = (mode == 0 ? linv : uinv) + (size_t)(k0 / NB) * NB * NB;
    {
        // every load in flight before the first is stored
        constexpr int TX = NB * NB / 256, TY = NB * CW / 256;
        float2 x[TX], y[TY], z[TY];
        int row[TY];  // U12: the row the block's exchange puts at i
#pragma unroll
        for (int t = 0; t < TY; ++t) {
            const int i = (tid + t * 256) / CW;
            row[t] = mode == 0 && i < nb ? perm[k0 + i] : 0;
        }
#pragma unroll
        for (int t = 0; t < TX; ++t) x[t] = iv[tid + t * 256];
#pragma unroll
        for (int t = 0; t < TY; ++t) {
            const int q = tid + t * 256;
            const int i = mode == 0 ? q / CW : q / NB, j = mode == 0 ? q % CW : q % NB;
            const float2 zero = make_float2(0.f, 0.f);
            if (mode == 0) {
                y[t] = i < nb && j < ne ? A[(size_t)row[t] * lda + e0 + j] : zero;
                z[t] = pack == 2 && j < ne ? A[(size_t)(k0 - NB + i) * lda + e0 + j] : zero;
            } else {
                y[t] = i < ne && j < nb ? A[(size_t)(e0 + i) * lda + k0 + j] : zero;
                z[t] = pack == 2 && i < ne ? A[(size_t)(e0 + i) * lda + k0 - NB + j] : zero;
            }
        }
#pragma unroll
        for (int t = 0; t < TX; ++t) {
            const int q = tid + t * 256;
            X[(q / NB) * LDS + q % NB] = x[t];
        }
#pragma unroll
        for (int t = 0; t < TY; ++t) {
            const int q = tid + t * 256, o = mode == 0 ? (q / CW) * LDC + q % CW : (q / NB) * LDS + q % NB;
            Y[o] = y[t];
            if (pack == 2) P[o] = z[t];
        }
    }
    __syncthreads();
    const int tx = tid & 15, ty = tid >> 4;
    // C = L R: [NB][CW] = X Y (U12), [CW][NB] = Y X (L21)
    const auto product = [&](auto na_, auto nb_, const float2* L, int ldl, const float2* R, int ldr, const auto& out) {
        constexpr int NA = decltype(na_)::value, NBB = decltype(nb_)::value;
        float2 acc[NA][NBB];
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
            for (int b = 0; b < NBB; ++b) acc[a][b] = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int k = 0; k < NB; ++k) {
            float2 l[NA], r[NBB];
#pragma unroll
            for (int a = 0; a < NA; ++a) l[a] = L[(ty + 16 * a) * ldl + k];
#pragma unroll
            for (int b = 0; b < NBB; ++b) r[b] = R[k * ldr + tx + 16 * b];
#pragma unroll
            for (int a = 0; a < NA; ++a)
#pragma unroll
                for (int b = 0; b < NBB; ++b) acc[a][b] = cfma(l[a], r[b], acc[a][b]);
        }
        __syncthreads();  // Y is overwritten by the product
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
            for (int b = 0; b < NBB; ++b) out(ty + 16 * a, tx + 16 * b, acc[a][b]);
    };
    // entries past the chunk or the block are zero products
    if (mode == 0)
        product(std::integral_constant<int, 4>(), std::integral_constant<int, NT>(), X, LDS, Y, LDC, [&](int i, int j, float2 v) {
            Y[i * LDC + j] = v;
            if (i < nb && j < ne) A[(size_t)(k0 + i) * lda + e0 + j] = v;
        });
    else
        product(std::integral_constant<int, NT>(), std::integral_constant<int, 4>(), Y, LDS, X, LDS, [&](int i, int j, float2 v) {
            Y[i * LDS + j] = v;
            if (i < ne && j < nb) A[(size_t)(e0 + i) * lda + k0 + j] = v;
        });
    __syncthreads();
    // scales: per column of U12 (mode 0) or row of L21 (mode 1), CW / 8 per
    // warp, over both blocks of a pair
#pragma unroll
    for (int c = warp * (CW / 8); c < (warp + 1) * (CW / 8); ++c) {
        float mx = 0.f;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (u >= 2 && pack != 2) break;  // uniform
            const float2* T = u < 2 ? Y : P;
            const int k = lane + 32 * (u & 1);
            const float2 a = mode == 0 ? T[k * LDC + c] : T[c * LDS + k];
            mx = fmaxf(mx, fmaxf(fabsf(a.x), fabsf(a.y)));
        }
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) {
            const float2 s2 = col_max_scale(mx);
            sc[c] = s2.x;
            if (c < ne) (mode == 0 ? inv_t : inv_s)[e0 - k1 + c] = s2.y;
        }
    }
    __syncthreads();
    // the operand rows in 16-byte pieces (4 k values): block p's piece ch is
    // piece 16 p + ch of the row; a pair's first block is P
#pragma unroll 1
    for (int p = 0; p < pack; ++p) {
        const float2* T = p + 1 < pack ? P : Y;
        if (mode == 0) {
            // item (column c, part e, piece ch)
#pragma unroll
            for (int t = 0; t < CW * 2 * 16 / 256; ++t) {
                const int q = tid + t * 256, c = q >> 5, e = (q >> 4) & 1, ch = q & 15;
                if (c >= ne) continue;
                const float t2 = sc[c];
                uint4 h, lo;
                uint32_t* hp = &h.x;
                uint32_t* lp = &lo.x;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float2 v = T[(4 * ch + u) * LDC + c];
                    if (e == 0)
                        split2(t2 * v.x, -(t2 * v.y), hp[u], lp[u]);
                    else
                        split2(t2 * v.y, t2 * v.x, hp[u], lp[u]);
                }
                const size_t r = (size_t)(2 * (e0 - k1 + c) + e);
                reinterpret_cast<uint4*>(Uop + r * lutc::KH)[16 * p + ch] = h;
                reinterpret_cast<uint4*>(Uop + ((size_t)2 * n + r) * lutc::KH)[16 * p + ch] = lo;
            }
        } else {
            // item (row i, piece ch)
#pragma unroll
            for (int t = 0; t < CW * 16 / 256; ++t) {
                const int q = tid + t * 256, i = q >> 4, ch = q & 15;
                if (i >= ne) continue;
                const float s = sc[i];
                uint4 h, lo;
                uint32_t* hp = &h.x;
                uint32_t* lp = &lo.x;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float2 v = T[i * LDS + 4 * ch + u];
                    split2(s * v.x, s * v.y, hp[u], lp[u]);
                }
                const size_t r = (size_t)(e0 - k1 + i);
                reinterpret_cast<uint4*>(Lop + r * lutc::KH)[16 * p + ch] = h;
                reinterpret_cast<uint4*>(Lop + ((size_t)n + r) * lutc::KH)[16 * p + ch] = lo;
            }
        }
    }
}

// A22 -= L21 U12 on the tile of 64 complex columns (blockIdx.x + ct0) and
// TN rows (blockIdx.y < bend) of [k1, n)^2; blockIdx.y >= bend goes on along
// the first row of tiles (columns blockIdx.y - bend + 1).  nslices K slices of 64 halves: 2 for
// one block's panels (K = 64 complex), 4 for two blocks'.
//   warp 0      TMA producer: per K slice Uh, Ul (128 rows) and Lh, Ll (TN
//               rows), 128-byte swizzle
//   warp 1      allocates TN tensor-memory columns and issues
//               tcgen05.mma M = 128, N = TN, K = 16: 12 per slice
//   warps 2..9  epilogue, per 64-row chunk of the tile of A22 (TMA loads, 32
//               KB): each warp takes a quadrant of the tensor-memory lanes
//               (32 real columns) and 32 rows and subtracts the scaled
//               accumulator in shared memory; one thread stores the chunk
//               back with TMA.  Rows and columns past the matrix are
//               zero-filled on load and clipped on store.
// TN = 256, two CTAs an SM, for the bulk of the trailing matrix, bound by
// the traffic of A22: one stage; once the MMAs are done it holds three
// chunks, and the fourth takes the first slot when that slot's store has
// read it.  TN = 64, one CTA an SM, where the tiles are too few to fill the
// SMs and the next diagonal block waits for them: every slice and the chunk
// are in flight from the start, and four times the CTAs share the rows (a
// block's next 64 columns at n = 1470: 10.8 -> 3.8 us for two slices, 16 -> 5.3
// for four).
// Every wait is bounded; on timeout the kernel records a code in *err, skips
// the stores that would follow, drains its copies and MMAs and frees tensor
// memory.
template <int TN>
__global__ void __launch_bounds__(lutc::THREADS, TN == 256 ? 2 : 1)
    k_lu_update_tc(const __grid_constant__ CUtensorMap tmU, const __grid_constant__ CUtensorMap tmL,
                   const __grid_constant__ CUtensorMap tmC, int n, int k1, int ct0, int bend, int nslices,
                   const float* __restrict__ inv_t, const float* __restrict__ inv_s, int* __restrict__ err)
{
    using namespace tc;
    using S = lutc::Tile<TN>;
    constexpr int NST = S::NST;
    extern __shared__ uint8_t smem_raw[];
    __shared__ float rs[TN];  // 1 / s_i of the tile's rows
    __shared__ int eok;
    __shared__ volatile int stopped;  // a wait of this CTA ran out
    uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sC = base + S::C_OFF;
    uint64_t* full = (uint64_t*)(base + S::BAR_OFF);  // [NST]
    uint64_t* empty = full + NST;                     // [NST]
    uint64_t* accum = empty + NST;
    uint64_t* cfull = accum + 1;  // [SLOTS] chunk slots of A22
    uint32_t* tmem_slot = (uint32_t*)(cfull + S::SLOTS);

    griddep_launch();  // the diagonal block's CTA may take its place beside the last of these
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m = n - k1;
    const int by = blockIdx.y;
    const int cc0 = (by < bend ? blockIdx.x + ct0 : by - bend + 1) * 64, r0 = by < bend ? by * TN : 0;

    if (threadIdx.x == 0) {
        stopped = 0;
        for (int s = 0; s < NST; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        mbar_init(accum, 1);
        for (int c = 0; c < S::SLOTS; ++c) mbar_init(cfull + c, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    griddep_wait();  // the panels (barriers and tensor memory above do not need them)
    const int xC = 2 * (k1 + cc0), yC = k1 + r0;  // tile origin in the float view of A

    if (warp == 0) {
        if (lane == 0) {
            int issued = 0;
            for (int s = 0; s < nslices; ++s) {
                uint8_t* st = base + (s % NST) * S::STAGE;
                if (s >= NST && !mbar_wait(empty + s % NST, (s / NST - 1) & 1, err, 11)) break;
                mbar_expect_tx(full + s % NST, S::STAGE);
                tma_load_2d(st, &tmU, full + s % NST, 64 * s, 2 * cc0);
                tma_load_2d(st + lutc::U_BYTES, &tmU, full + s % NST, 64 * s, 2 * n + 2 * cc0);
                tma_load_2d(st + 2 * lutc::U_BYTES, &tmL, full + s % NST, 64 * s, r0);
                tma_load_2d(st + 2 * lutc::U_BYTES + S::L_BYTES, &tmL, full + s % NST, 64 * s, n + r0);
                issued = s + 1;
            }
            if (!S::WIDE) {
                mbar_expect_tx(cfull, lutc::C_BYTES);
                tma_load_2d(sC, &tmC, cfull, xC, yC);
            }
            // the issued copies must have landed before the CTA exits
            for (int s = issued > NST ? issued - NST : 0; s < issued; ++s)
                mbar_wait(full + s % NST, (s / NST) & 1, err, 12);
            if (!S::WIDE) mbar_wait(cfull, 0, err, 12);
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = idesc_f16(lutc::TM, TN);
        const uint64_t d0 = sw128_desc(smem_u32(base));
        for (int s = 0; s < nslices; ++s) {
            if (!warp_wait(full + s % NST, (s / NST) & 1, err, 13)) {
                stopped = 1;
                __threadfence_block();
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t uh = d0 + (uint64_t)((s % NST) * (S::STAGE >> 4)), ul = uh + (lutc::U_BYTES >> 4);
            const uint64_t lh = ul + (lutc::U_BYTES >> 4), ll = lh + (S::L_BYTES >> 4);
            mma_f16_block(tmem, uh, lh, idesc, s > 0 ? 1u : 0u);
            mma_f16_block(tmem, uh, ll, idesc, 1u);
            mma_f16_block(tmem, ul, lh, idesc, 1u);
            if (s + NST < nslices) commit_elect(empty + s % NST);
        }
        // every MMA issued must be complete before the epilogue and before
        // tensor memory is released
        commit_elect(accum);
        warp_wait(accum, 0, err, 14);
    } else {
        const int q = warp & 3, hf = (warp - 2) >> 2;
        const bool leader = threadIdx.x == 64;
        const int l = 32 * q + lane;  // lane of tensor memory: real column of the tile
        const int jc = cc0 + (l >> 1);  // complex column, from k1
        const float itj = jc < m ? inv_t[jc] : 0.f;
        for (int i = threadIdx.x - 64; i < TN; i += 256) rs[i] = r0 + i < m ? inv_s[r0 + i] : 0.f;
        if (leader) {
            // the wide tile's operand buffer is free once the MMAs are done
            int ok = (int)mbar_wait(accum, 0, err, 15);
            if (ok) ok = stopped == 0;
            if (S::WIDE && ok)
                for (int c = 0; c < S::SLOTS; ++c) {
                    mbar_expect_tx(cfull + c, lutc::C_BYTES);
                    tma_load_2d(sC + c * lutc::C_BYTES, &tmC, cfull + c, xC, yC + 64 * c);
                }
            eok = ok;
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (eok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int c = 0; c < S::NC; ++c) {
                const int slot = c % S::SLOTS;
                float* cs = (float*)(sC + slot * lutc::C_BYTES);  // [64][128] floats
                int got = 0;
                if (lane == 0) {
                    got = stopped == 0 && mbar_wait(cfull + slot, c / S::SLOTS, err, 16);
                    if (!got) stopped = 1;
                }
                got = __shfl_sync(0xffffffffu, got, 0);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int rr = 32 * hf + 16 * h;  // first row of the group, in the chunk
                    float acc[16];
                    tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(64 * c + rr), acc);
                    if (got) {
#pragma unroll
                        for (int r = 0; r < 16; ++r) {
                            float* p = cs + (rr + r) * 128 + l;
                            *p = *p - acc[r] * (itj * rs[64 * c + rr + r]);
                        }
                    }
                }
                fence_proxy_async();
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (leader && stopped == 0) {
                    tma_store_2d(&tmC, cs, xC, yC + 64 * c);
                    bulk_store_commit();
                    if (c + S::SLOTS < S::NC) {
                        bulk_store_wait_read();  // the slot takes a later chunk
                        mbar_expect_tx(cfull + slot, lutc::C_BYTES);
                        tma_load_2d(cs, &tmC, cfull + slot, xC, yC + 64 * (c + S::SLOTS));
                    }
                }
            }
            if (leader) bulk_store_wait();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TN) : "memory");
    }
}

// W[r][i] = B[r][perm[i]]
__global__ void k_lu_gather(const float2* __restrict__ B, const int* __restrict__ perm, int n, int nrhs,
                            float2* __restrict__ W)
{
    const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (size_t)n * nrhs) return;
    const int r = (int)(id / n), i = (int)(id % n);
    W[id] = B[(size_t)r * n + perm[i]];
}

constexpr int RC = 8;  // right-hand sides per CTA of a triangular solve

// Both triangular solves as one launch each, in wavefront order.  A CTA
// takes a ticket when it starts: ticket t is row block t of the forward (L)
// sweep, block nblk - 1 - t of the backward (U) sweep, so a CTA only waits for
// blocks whose CTAs started before it.  Row block k:
//   acc = W[block k] - sum over the blocks j before k (forward: j < k;
//         backward: j > k) of A[block k][block j] x_j
//   x_k = inv_k acc, stored in Out, then the block's flag is raised
// Each x_j is read once its flag is up (bounded wait: on timeout, or once
// any wait has given up, the kernel records an error and stops waiting); the
// 64 x 64 blocks of A stream through a cp.async double buffer, the inverse
// last.  A chain of blocks bounds it: 4.0 -> 2.7 us a block (eight right-hand
// sides, 228 -> 155 us a sweep on the batch's mean) since the inverse no longer
// loads on the chain and the error word is polled with every 64th read of a flag
// only.  RC right-hand sides per CTA (blockIdx.y).  Thread: row i = tid / 4, right-hand sides
// 2 (tid % 4) and the next.
constexpr int WLD = NB + 2;  // tile row stride in float2: 16-byte aligned, 8 rows on distinct banks

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int src_bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// tile rows [r0, r0 + 64) x columns [c0, c0 + 64) of A into T (rows past n
// or columns past n read as zeros)
__device__ __forceinline__ void tile_async(float2* T, const float2* __restrict__ A, int n, int lda, int r0, int c0)
{
    for (int q = threadIdx.x; q < NB * (NB / 2); q += blockDim.x) {
        const int i = q / (NB / 2), c = 2 * (q % (NB / 2));  // 16-byte piece: two complex
        const int r = r0 + i, cc = c0 + c;
        const int nv = (r < n) ? max(0, min(2, n - cc)) : 0;  // valid complex in the piece
        // clamped source stays 16-byte aligned: lda and the column are even
        const float2* src = A + (size_t)min(r, n - 1) * lda + min(cc, (n - 1) & ~1);
        cp_async16(T + i * WLD + c, src, 8 * nv);
    }
}

template <int DIR>
__global__ void __launch_bounds__(256) k_lu_wave(const float2* __restrict__ A, int n, int lda, int nblk,
                                                 const float2* __restrict__ inv, int nrhs,
                                                 const float2* __restrict__ W, float2* __restrict__ Out,
                                                 int* __restrict__ ticket, int* __restrict__ flag,
                                                 int* __restrict__ err, long long limit)
{
    extern __shared__ float2 s_w[];
    float2* T0 = s_w;                 // [NB][WLD] tile buffers
    float2* T1 = T0 + NB * WLD;
    __shared__ float2 xs[NB][RC];     // x_j of the tile, then acc
    __shared__ int s_t, s_ok;
    const int tid = threadIdx.x, i = tid >> 2, r = 2 * (tid & 3);
    if (tid == 0) s_t = atomicAdd(ticket + blockIdx.y, 1);
    __syncthreads();
    const int t = s_t;
    const int k = DIR == 0 ? t : nblk - 1 - t;
    const int k0 = k * NB, nbk = min(NB, n - k0);
    const int rb = blockIdx.y * RC, nr = min(RC, nrhs - rb);
    int* fl = flag + (size_t)blockIdx.y * nblk;
    float2 acc[2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
        acc[h] = (i < nbk && r + h < nr) ? W[(size_t)(rb + r + h) * n + k0 + i] : make_float2(0.f, 0.f);
    // the blocks this row block depends on, in the order they are solved
    const int nd = DIR == 0 ? k : nblk - 1 - k;
    auto dep = [&](int s) { return DIR == 0 ? s : nblk - 1 - s; };
    // the block's inverse is the tile after the last one: in shared memory by
    // the time the chain reaches it
    const float2* iv = inv + (size_t)k * NB * NB;
    auto fetch = [&](float2* T, int s) {
        if (s < nd)
            tile_async(T, A, n, lda, k0, dep(s) * NB);
        else
            for (int q = tid; q < NB * NB / 2; q += blockDim.x)
                cp_async16(T + (q / (NB / 2)) * WLD + 2 * (q % (NB / 2)), iv + 2 * q, 16);
        cp_async_commit();
    };
    fetch(T0, 0);
    bool ok = true;
    for (int s = 0; s < nd; ++s) {
        float2* T = (s & 1) ? T1 : T0;
        fetch((s & 1) ? T0 : T1, s + 1);
        const int j = dep(s), j0 = j * NB, nbj = min(NB, n - j0);
        if (tid == 0) {
            int got = ok;
            if (got) {
                const long long t0 = clock64();
                for (int spin = 1; *(volatile int*)(fl + j) == 0; ++spin) {
                    // now and then: a second read would double the time to see the flag
                    if ((spin & 63) == 0 && (*(volatile int*)err || clock64() - t0 > limit)) {
                        atomicCAS(err, 0, 21);
                        got = 0;
                        break;
                    }
                }
            }
            __threadfence();
            s_ok = got;
        }
        __syncthreads();
        ok = s_ok;
        if (ok)
            for (int q = tid; q < NB * RC; q += blockDim.x) {
                const int c = q / RC, rr = q % RC;
                xs[c][rr] = (c < nbj && rr < nr) ? __ldcg(Out + (size_t)(rb + rr) * n + j0 + c) : make_float2(0.f, 0.f);
            }
        cp_async_wait<1>();
        __syncthreads();
        if (ok) {
            // the block's 64-term product on its own, then subtracted (the
            // rounding of a sweep that updates W block by block)
            float2 p[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll 8
            for (int c = 0; c < NB; ++c) {
                const float2 l = T[i * WLD + c];
#pragma unroll
                for (int h = 0; h < 2; ++h) p[h] = cfma(l, xs[c][r + h], p[h]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) acc[h] = make_float2(acc[h].x - p[h].x, acc[h].y - p[h].y);
        }
        __syncthreads();
    }
    cp_async_wait<0>();
    // x_k = inv_k acc
#pragma unroll
    for (int h = 0; h < 2; ++h) xs[i][r + h] = acc[h];
    const float2* Ti = (nd & 1) ? T1 : T0;
    __syncthreads();
    float2 x[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll 8
    for (int c = 0; c < NB; ++c) {
        const float2 m = Ti[i * WLD + c];
#pragma unroll
        for (int h = 0; h < 2; ++h) x[h] = cfma(m, xs[c][r + h], x[h]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if (i < nbk && r + h < nr) Out[(size_t)(rb + r + h) * n + k0 + i] = x[h];
    __threadfence();
    __syncthreads();
    if (tid == 0) atomicExch(fl + k, 1);
}

}  // namespace

// trailing-update operands: U planes [2][2n][128] and L planes [2][n][128]
// halves, then 1/t_j and 1/s_i (n floats each)
static size_t ops_bytes(int n) { return (size_t)6 * n * lutc::KH * sizeof(__half) + 2 * sizeof(float) * (size_t)n; }

size_t lu_bytes(int n)
{
    const size_t nblk = (size_t)(n + NB - 1) / NB;
    return sizeof(float2) * (size_t)(n + (n & 1)) * n + sizeof(int) * (size_t)n + 2 * sizeof(float2) * nblk * NB * NB + 256 * 4 +
           ops_bytes(n);
}

// FP16 operand map: rows of 128 halves (256 bytes), box 64 halves x box_rows,
// 128-byte swizzle, zero fill past the last row
static emfa_status_t ops_map(Ctx* c, CUtensorMap* m, const void* ptr, uint64_t rows, uint32_t box_rows)
{
    auto fn = tensor_map_encoder();
    if (!fn) {
        set_error(c, "cuTensorMapEncodeTiled unavailable");
        return EMFA_ERR_CUDA;
    }
    cuuint64_t dims[2] = {(cuuint64_t)lutc::KH, rows};
    cuuint64_t strides[1] = {(cuuint64_t)lutc::KH * sizeof(__half)};
    cuuint32_t box[2] = {64, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error(c, "lu_factor: cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
        return EMFA_ERR_CUDA;
    }
    return EMFA_OK;
}

// A as a float matrix of `rows` rows x 2n columns, rows lda complex apart;
// box 128 floats (64 complex) x 64 rows, no swizzle; loads past the matrix
// (or past `rows`) read zeros and stores there are clipped
static emfa_status_t tile_map(Ctx* c, CUtensorMap* m, const void* A, int n, int lda, int rows)
{
    auto fn = tensor_map_encoder();
    if (!fn) {
        set_error(c, "cuTensorMapEncodeTiled unavailable");
        return EMFA_ERR_CUDA;
    }
    cuuint64_t dims[2] = {2 * (cuuint64_t)n, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)lda * sizeof(float2)};
    cuuint32_t box[2] = {128, 64};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(A), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error(c, "lu_factor: cuTensorMapEncodeTiled (A) failed (" + std::to_string((int)r) + ")");
        return EMFA_ERR_CUDA;
    }
    return EMFA_OK;
}

// three padded 64 x 64 blocks and the merge products (2048): about 116 KB,
// so the CTA fits on an SM beside one CTA of the trailing update
static size_t panels_smem() { return sizeof(float2) * (NB * LDS + 2 * CHUNK); }
static size_t diag_smem() { return sizeof(float2) * (3 * NB * LDS + 2048); }

static emfa_status_t lu_set_smem(Ctx* c)
{
    EMFA_TRY(ensure_smem(c, k_lu_diag, diag_smem()));
    EMFA_TRY(ensure_smem(c, k_lu_panels, panels_smem()));
    EMFA_TRY(ensure_smem(c, k_lu_wave<0>, sizeof(float2) * 2 * NB * WLD));
    EMFA_TRY(ensure_smem(c, k_lu_wave<1>, sizeof(float2) * 2 * NB * WLD));
    EMFA_TRY(ensure_smem(c, k_lu_update_tc<64>, lutc::Tile<64>::SMEM));
    return ensure_smem(c, k_lu_update_tc<256>, lutc::Tile<256>::SMEM);
}

emfa_status_t lu_factor(Ctx* c, const void* Z, int n, LuFactor& F, cudaStream_t st)
{
    if (n <= 0) {
        set_error(c, "lu_factor: n must be positive");
        return EMFA_ERR_INVALID;
    }
    EMFA_TRY(lu_set_smem(c));
    F.n = n;
    F.lda = n + (n & 1);  // rows 16-byte aligned: the update moves tiles of A with TMA
    F.nblk = (n + NB - 1) / NB;
    const int lda = F.lda;
    EMFA_TRY(F.a.alloc(c, sizeof(float2) * (size_t)lda * n));
    EMFA_TRY(F.perm.alloc(c, sizeof(int) * (size_t)n));
    EMFA_TRY(F.linv.alloc(c, sizeof(float2) * (size_t)F.nblk * NB * NB));
    EMFA_TRY(F.uinv.alloc(c, sizeof(float2) * (size_t)F.nblk * NB * NB));
    EMFA_TRY(F.info.alloc(c, 256));
    EMFA_TRY(F.ops.alloc(c, ops_bytes(n)));
    float2* A = dptr<float2>(F.a);
    __half* Uop = dptr<__half>(F.ops);
    __half* Lop = Uop + (size_t)4 * n * lutc::KH;
    float* inv_t = (float*)(Lop + (size_t)2 * n * lutc::KH);
    float* inv_s = inv_t + n;
    int* info = dptr<int>(F.info);
    CUtensorMap tmU, tmL, tmL64, tmC;
    EMFA_TRY(ops_map(c, &tmU, Uop, (uint64_t)4 * n, lutc::TM));
    EMFA_TRY(ops_map(c, &tmL, Lop, (uint64_t)2 * n, 256));
    EMFA_TRY(ops_map(c, &tmL64, Lop, (uint64_t)2 * n, 64));
    EMFA_TRY(tile_map(c, &tmC, A, n, lda, n));
    EMFA_CUDA(c, cudaMemcpy2DAsync(A, sizeof(float2) * (size_t)lda, Z, sizeof(float2) * (size_t)n,
                                   sizeof(float2) * (size_t)n, (size_t)n, cudaMemcpyDeviceToDevice, st));
    EMFA_CUDA(c, cudaMemsetAsync(info, 0, 3 * sizeof(int), st));
    // lookahead: the chain of panels, the next block's columns and its
    // diagonal block runs on a high-priority stream, and the rest of each
    // trailing update on st beside it.  Within the chain the update of the
    // block's columns and the diagonal block are dependent launches, so that
    // the diagonal block's one CTA holds its place on an SM before the rest
    // of the update fills them (released on every return)
    struct Aux {
        cudaStream_t s = nullptr;
        cudaEvent_t panel = nullptr, rest = nullptr;
        bool open = false;  // work on s that the caller's stream does not wait for yet
        ~Aux()
        {
            // an error return: the caller frees what that work reads and writes
            if (open) cudaStreamSynchronize(s);
            if (panel) cudaEventDestroy(panel);
            if (rest) cudaEventDestroy(rest);
            if (s) cudaStreamDestroy(s);
        }
    } aux;
    if (F.nblk > 2) {
        int lo = 0, hi = 0;
        EMFA_CUDA(c, cudaDeviceGetStreamPriorityRange(&lo, &hi));
        EMFA_CUDA(c, cudaStreamCreateWithPriority(&aux.s, cudaStreamNonBlocking, hi));
        EMFA_CUDA(c, cudaEventCreateWithFlags(&aux.panel, cudaEventDisableTiming));
        EMFA_CUDA(c, cudaEventCreateWithFlags(&aux.rest, cudaEventDisableTiming));
    }
    cudaStream_t hs = aux.s ? aux.s : st;
    const auto wait_for = [&](cudaStream_t waiter, cudaEvent_t e, cudaStream_t s) -> emfa_status_t {
        EMFA_CUDA(c, cudaEventRecord(e, s));
        EMFA_CUDA(c, cudaStreamWaitEvent(waiter, e, 0));
        return EMFA_OK;
    };
    auto diag = [&](int kb) -> emfa_status_t {
        const int k0 = kb * NB, nb = std::min(NB, n - k0);
        EMFA_CUDA(c, launch_dependent(k_lu_diag, dim3(1), dim3(DIAG_THREADS), diag_smem(), hs, A, n, lda, k0, nb,
                                      dptr<int>(F.perm), dptr<float2>(F.linv), dptr<float2>(F.uinv), info));
        c->kernel_launches += 1;
        return EMFA_OK;
    };
    // A22 -= L21 U12 on column tiles [ct0, ct0 + nct) (64 complex columns
    // each) of [k1, n)^2, and on the first 64 rows of the next `along` tiles.
    // 64-row tiles where one wave of them fits the SMs beside the diagonal
    // block's (or with `along`, whose tiles are single rows of 64)
    const int sms = c->sm_count > 0 ? c->sm_count : 148;
    auto update = [&](int k1, int ct0, int nct, int along, int nslices, cudaStream_t s) -> emfa_status_t {
        const int rows = n - k1;
        const bool low = along > 0 || (long)nct * ((rows + 63) / 64) < sms;
        const int rt = (rows + (low ? 63 : 255)) / (low ? 64 : 256);
        const float *it = inv_t, *is = inv_s;
        const auto launch = [&](auto kernel, int smem) {
            const dim3 grd((unsigned)nct, (unsigned)(rt + along));
            const CUtensorMap& tl = low ? tmL64 : tmL;
            if (s == hs)
                return launch_dependent(kernel, grd, dim3(lutc::THREADS), (size_t)smem, s, tmU, tl, tmC, n, k1, ct0, rt,
                                        nslices, it, is, info + 1);
            kernel<<<grd, lutc::THREADS, smem, s>>>(tmU, tl, tmC, n, k1, ct0, rt, nslices, it, is, info + 1);
            return cudaGetLastError();
        };
        EMFA_CUDA(c, low ? launch(k_lu_update_tc<64>, lutc::Tile<64>::SMEM)
                         : launch(k_lu_update_tc<256>, lutc::Tile<256>::SMEM));
        c->kernel_launches += 1;
        return EMFA_OK;
    };
    auto panels = [&](int k0, int nb, int pack, bool dependent) -> emfa_status_t {
        const dim3 grd((unsigned)((n - k0 - nb + CW - 1) / CW), 2);
        const float2 *li = dptr<float2>(F.linv), *ui = dptr<float2>(F.uinv);
        const int* pm = dptr<int>(F.perm);
        if (dependent)
            EMFA_CUDA(c, launch_dependent(k_lu_panels, grd, dim3(256), panels_smem(), hs, A, n, lda, k0, nb, pm, li, ui,
                                          Uop, Lop, inv_t, inv_s, pack));
        else
            k_lu_panels<<<grd, 256, panels_smem(), hs>>>(A, n, lda, k0, nb, pm, li, ui, Uop, Lop, inv_t, inv_s, pack);
        c->kernel_launches += 1;
        return EMFA_OK;
    };
    if (aux.s) EMFA_TRY(wait_for(hs, aux.panel, st));
    aux.open = aux.s != nullptr;
    EMFA_TRY(diag(0));
    int kb = 0;
    while (kb < F.nblk) {
        const int k0 = kb * NB, nb = std::min(NB, n - k0), rest = n - k0 - nb;
        if (rest <= 0) break;
        const int k1 = k0 + nb, ch = (rest + NB - 1) / NB;
        EMFA_TRY(panels(k0, nb, 1, false));
        if (aux.s && F.nblk - kb - 1 >= 2) {
            // blocks kb and kb + 1 as a pair: block kb's update of the next
            // block's columns and rows only, then one K = 128 update of the
            // rest with both blocks' panels (A22 is read and written once
            // for the two)
            const int k2 = k1 + NB, ch2 = (n - k2 + NB - 1) / NB;
            EMFA_TRY(update(k1, 0, 1, ch - 1, 2, hs));
            EMFA_TRY(diag(kb + 1));
            EMFA_TRY(panels(k1, NB, 2, true));
            if (ch2 > 1) EMFA_TRY(wait_for(st, aux.panel, hs));
            EMFA_TRY(update(k2, 0, 1, 0, 4, hs));  // columns of block kb + 2
            EMFA_TRY(diag(kb + 2));
            if (ch2 > 1) {
                EMFA_TRY(update(k2, 1, ch2 - 1, 0, 4, st));
                EMFA_TRY(wait_for(hs, aux.rest, st));
            }
            kb += 2;
            continue;
        }
        if (aux.s && ch > 1) {
            EMFA_TRY(wait_for(st, aux.panel, hs));
            EMFA_TRY(update(k1, 0, 1, 0, 2, hs));
            EMFA_TRY(diag(kb + 1));
            EMFA_TRY(update(k1, 1, ch - 1, 0, 2, st));
            EMFA_TRY(wait_for(hs, aux.rest, st));
        } else {
            EMFA_TRY(update(k1, 0, ch, 0, 2, hs));
            EMFA_TRY(diag(kb + 1));
        }
        kb += 1;
    }
    if (aux.s) EMFA_TRY(wait_for(st, aux.panel, hs));
    aux.open = false;
    if (F.nblk > 1) {
        k_lu_rowperm_left<<<dim3((unsigned)(F.nblk - 1) * (NB / 32), (unsigned)F.nblk), 256, 0, st>>>(
            A, n, lda, dptr<int>(F.perm));
        c->kernel_launches += 1;
    }
    EMFA_CUDA(c, cudaGetLastError());
    return EMFA_OK;
}

emfa_status_t lu_check_solves(Ctx* c, const LuFactor& F, cudaStream_t st)
{
    int h = 0;
    EMFA_CUDA(c, cudaMemcpyAsync(&h, dptr<int>(F.info) + 2, sizeof(int), cudaMemcpyDeviceToHost, st));
    EMFA_CUDA(c, cudaStreamSynchronize(st));
    if (h) {
        set_error(c, "lu_apply: a wait of the triangular solves timed out (code " + std::to_string(h) + ")");
        return EMFA_ERR_TIMEOUT;
    }
    return EMFA_OK;
}

emfa_status_t lu_zero_pivot(Ctx* c, const LuFactor& F, int* first, cudaStream_t st)
{
    int h[2] = {0, 0};
    EMFA_CUDA(c, cudaMemcpyAsync(h, F.info.ptr, sizeof(h), cudaMemcpyDeviceToHost, st));
    EMFA_CUDA(c, cudaStreamSynchronize(st));
    *first = h[0];
    if (h[1]) {
        set_error(c, "lu_factor: a wait of the tensor-core trailing update timed out (stage " + std::to_string(h[1]) +
                         ")");
        return EMFA_ERR_TIMEOUT;
    }
    return EMFA_OK;
}

emfa_status_t lu_apply(Ctx* c, const LuFactor& F, const float2* B, int nrhs, float2* X, float2* work,
                       cudaStream_t st)
{
    const int n = F.n;
    const size_t tot = (size_t)n * nrhs;
    float2* W = work;           // permuted right-hand sides
    float2* Y = work + tot;     // L^-1 P b
    const float2* A = dptr<float2>(F.a);
    const int gy = (nrhs + RC - 1) / RC;
    // tickets and flags of both sweeps: 2 (gy + gy nblk) ints
    void* wp = nullptr;
    const size_t words = 2 * ((size_t)gy + (size_t)gy * F.nblk);
    EMFA_TRY(ctx_workspace(c, WS_LU_WAVE, sizeof(int) * words, &wp));
    int* tk = (int*)wp;
    int* fl = tk + 2 * gy;
    EMFA_CUDA(c, cudaMemsetAsync(tk, 0, sizeof(int) * words, st));
    k_lu_gather<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(B, dptr<int>(F.perm), n, nrhs, W);
    const size_t sm = sizeof(float2) * 2 * NB * WLD;
    const long long limit = 2000000000LL;  // about 1 s
    k_lu_wave<0><<<dim3((unsigned)F.nblk, (unsigned)gy), 256, sm, st>>>(A, n, F.lda, F.nblk, dptr<float2>(F.linv),
                                                                        nrhs, W, Y, tk, fl, dptr<int>(F.info) + 2,
                                                                        limit);
    k_lu_wave<1><<<dim3((unsigned)F.nblk, (unsigned)gy), 256, sm, st>>>(
        A, n, F.lda, F.nblk, dptr<float2>(F.uinv), nrhs, Y, X, tk + gy, fl + (size_t)gy * F.nblk,
        dptr<int>(F.info) + 2, limit);
    c->kernel_launches += 3;
    EMFA_CUDA(c, cudaGetLastError());
    return EMFA_OK;
}

}  // namespace emfa
