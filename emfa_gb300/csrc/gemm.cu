// Multi-right-hand-side dense complex product on CUDA cores:
//   Y[r][f] = sum_k Z[f][k] X[r][k]      (Z row-major N x N, X / Y RHS-major)
// the dense products of iml::BICGSTAB / iml::GMRES (EMIterative/iml.cpp:22,186)
// for many right-hand sides at once.
//
// 64 (f) x 64 (r) CTA tile, 16-wide K slices staged through shared memory,
// 4 x 4 complex outputs per thread; up to 16 right-hand sides, and in FP64
// always, a warp-per-row GEMV instead.  ACC selects the accumulation:
//   float / double : plain accumulation in that type
//   CHUNKED        : FP32 products and sums over 64-wide K chunks, chunk sums
//                    accumulated in FP64 (the refinement residual of the
//                    mixed-precision solver: ~FP32-product accuracy without
//                    FP64 FMA throughput)
#include "emfa_internal.cuh"
#include "emfa_math.cuh"
#include "gemm.cuh"

#include <algorithm>
#include <climits>

namespace emfa {

template <typename T, bool CHUNKED>
__global__ void __launch_bounds__(256) k_cgemm(const Cx<T>* __restrict__ Z, size_t ldz, const Cx<T>* __restrict__ X,
                                               int n, int nrhs, Cx<T>* __restrict__ Y,
                                               const Cx<T>* __restrict__ Bsub, Cx<double>* __restrict__ Yd)
{
    constexpr int BM = 64, BN = 64, BK = 16;
    __shared__ Cx<T> As[BK][BM + 1];
    __shared__ Cx<T> Bs[BK][BN + 1];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int f0 = blockIdx.x * BM, r0 = blockIdx.y * BN;
    Cx<T> acc[4][4];
    double accd[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            acc[i][j] = cx(T(0), T(0));
            accd[i][j][0] = accd[i][j][1] = 0.0;
        }
    // loader mapping: 256 threads load 64 rows x 16 k: row = tid / 4, k = (tid % 4) * 4 .. +3
    const int lrow = threadIdx.x >> 2, lk = (threadIdx.x & 3) * 4;
    int kt = 0;
    for (int k0 = 0; k0 < n; k0 += BK, ++kt) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            int k = k0 + lk + q;
            int f = f0 + lrow, r = r0 + lrow;
            As[lk + q][lrow] = (f < n && k < n) ? Z[(size_t)f * ldz + k] : cx(T(0), T(0));
            Bs[lk + q][lrow] = (r < nrhs && k < n) ? X[(size_t)r * n + k] : cx(T(0), T(0));
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            Cx<T> a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][tx + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][ty + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j].re = fma(a[i].re, b[j].re, acc[i][j].re);
                    acc[i][j].re = fma(-a[i].im, b[j].im, acc[i][j].re);
                    acc[i][j].im = fma(a[i].re, b[j].im, acc[i][j].im);
                    acc[i][j].im = fma(a[i].im, b[j].re, acc[i][j].im);
                }
        }
        __syncthreads();
        if (CHUNKED && ((kt & 3) == 3 || k0 + BK >= n)) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    accd[i][j][0] += (double)acc[i][j].re;
                    accd[i][j][1] += (double)acc[i][j].im;
                    acc[i][j] = cx(T(0), T(0));
                }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        int r = r0 + ty + 16 * j;
        if (r >= nrhs) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int f = f0 + tx + 16 * i;
            if (f >= n) continue;
            size_t o = (size_t)r * n + f;
            if (CHUNKED) {
                // Yd = Bsub - Z X  (residual) when Bsub given, else Z X
                double re = accd[i][j][0], im = accd[i][j][1];
                if (Bsub) {
                    re = (double)Bsub[o].re - re;
                    im = (double)Bsub[o].im - im;
                }
                Yd[o] = cx(re, im);
            } else {
                Y[o] = acc[i][j];
            }
        }
    }
}

// Few right-hand sides (the 64-wide tile above would leave most of its RHS
// columns empty): a warp per RPW rows of Z, lanes striding k, RB right-hand
// sides accumulated in registers, then reduced by shuffles.  Each warp reads
// its rows once (coalesced 512-byte segments for complex128) and the RHS
// entries from L1/L2.  FP64 is bound by the FMA rate.  FP32 is bound by the
// latency of its loads, so U steps of k are loaded before any is used and
// the rows of a warp are few where the warps would be (rpw_f32).  A sum's
// terms and their order depend on none of RB, RPW and U.
template <typename T, int RB, int RPW>
__global__ void __launch_bounds__(256) k_cgemv(const Cx<T>* __restrict__ Z, size_t ldz, const Cx<T>* __restrict__ X,
                                               int n, int nrhs, Cx<T>* __restrict__ Y)
{
    constexpr int U = sizeof(T) == 8 ? 1 : RPW * RB >= 16 ? 2 : 4;
    const int warp = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int f0 = warp * RPW;
    if (f0 >= n) return;
    // block blockIdx.y of RB right-hand sides; the last may be short: its
    // missing columns repeat the last one and are not stored
    X += (size_t)blockIdx.y * RB * n;
    Y += (size_t)blockIdx.y * RB * n;
    nrhs = min(RB, nrhs - (int)blockIdx.y * RB);
    T ar[RPW][RB], ai[RPW][RB];
#pragma unroll
    for (int i = 0; i < RPW; ++i)
#pragma unroll
        for (int r = 0; r < RB; ++r) ar[i][r] = ai[i][r] = T(0);
    const auto step = [&](const Cx<T> (&z)[RPW], int r, Cx<T> x) {
#pragma unroll
        for (int i = 0; i < RPW; ++i) {
            ar[i][r] = fma(z[i].re, x.re, ar[i][r]);
            ar[i][r] = fma(-z[i].im, x.im, ar[i][r]);
            ai[i][r] = fma(z[i].re, x.im, ai[i][r]);
            ai[i][r] = fma(z[i].im, x.re, ai[i][r]);
        }
    };
    int k = lane;
    if constexpr (U > 1) {
        const Cx<T>* zr[RPW];
#pragma unroll
        for (int i = 0; i < RPW; ++i) zr[i] = Z + (size_t)min(f0 + i, n - 1) * ldz;
        const Cx<T>* xr[RB];
#pragma unroll
        for (int r = 0; r < RB; ++r) xr[r] = X + (size_t)min(r, nrhs - 1) * n;
        for (; k + 32 * (U - 1) < n; k += 32 * U) {
            Cx<T> z[U][RPW], x[U][RB];
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int i = 0; i < RPW; ++i) z[u][i] = zr[i][k + 32 * u];
#pragma unroll
                for (int r = 0; r < RB; ++r) x[u][r] = xr[r][k + 32 * u];
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int r = 0; r < RB; ++r) step(z[u], r, x[u][r]);
        }
    }
    for (; k < n; k += 32) {
        Cx<T> z[RPW];
#pragma unroll
        for (int i = 0; i < RPW; ++i) z[i] = f0 + i < n ? Z[(size_t)(f0 + i) * ldz + k] : cx(T(0), T(0));
#pragma unroll
        for (int r = 0; r < RB; ++r)
            if (r < nrhs) step(z, r, X[(size_t)r * n + k]);
    }
#pragma unroll
    for (int i = 0; i < RPW; ++i)
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            if (r >= nrhs) break;
            T re = ar[i][r], im = ai[i][r];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                re += __shfl_xor_sync(0xffffffffu, re, o);
                im += __shfl_xor_sync(0xffffffffu, im, o);
            }
            if (lane == 0 && f0 + i < n) Y[(size_t)r * n + f0 + i] = cx(re, im);
        }
}

template <typename T, int RPW>
static void launch_gemv(const Cx<T>* z, size_t ldz, const Cx<T>* x, int n, int nrhs, Cx<T>* y, cudaStream_t st)
{
    // blocks of up to 8 right-hand sides of even size (grid y)
    const int blocks = (nrhs + 7) / 8, rb = (nrhs + blocks - 1) / blocks;
    const dim3 grd(((n + RPW - 1) / RPW + 7) / 8, blocks);
    switch (rb) {
    case 1: k_cgemv<T, 1, RPW><<<grd, 256, 0, st>>>(z, ldz, x, n, nrhs, y); break;
    case 2: k_cgemv<T, 2, RPW><<<grd, 256, 0, st>>>(z, ldz, x, n, nrhs, y); break;
    case 3: k_cgemv<T, 3, RPW><<<grd, 256, 0, st>>>(z, ldz, x, n, nrhs, y); break;
    case 4: k_cgemv<T, 4, RPW><<<grd, 256, 0, st>>>(z, ldz, x, n, nrhs, y); break;
    case 5: k_cgemv<T, 5, RPW><<<grd, 256, 0, st>>>(z, ldz, x, n, nrhs, y); break;
    case 6: k_cgemv<T, 6, RPW><<<grd, 256, 0, st>>>(z, ldz, x, n, nrhs, y); break;
    case 7: k_cgemv<T, 7, RPW><<<grd, 256, 0, st>>>(z, ldz, x, n, nrhs, y); break;
    default: k_cgemv<T, 8, RPW><<<grd, 256, 0, st>>>(z, ldz, x, n, nrhs, y); break;
    }
}

// Rows of a warp, FP32.  More rows read the right-hand sides fewer times
// (they come from L1 and L2 once n x rb no longer fits L1), fewer rows make
// more warps.  us at 1 | 2 | 4 rows: n = 480 x 8, 37 | 41 | 41; 2000 x 5,
// 54 | 53 | 64; 2000 x 8, 57 | 73 | 60; 2000 x 12, 64 | 61 | 55; 3000 x 3,
// 54 | 49 | 55; 3000 x 8, 78 | 97 | 72; 5067 x 1, 69 | 97 | 171; 5067 x 5,
// 251 | 147 | 189; 5067 x 9, 338 | 233 | 307; 5067 x 16, 470 | 456 | 246.
// Four rows a warp, one step of k at a time and blocks of 1, 2, 4 or 8 took
// 60, 100, 138, 166, 194, 74 for 3 and 191, 217, 372, 751 and 1100.
static int rpw_f32(int n, int rb)
{
    if (rb <= 2 || (long)n * rb < 9000) return 1;
    return rb <= 5 ? 2 : 4;
}

template <typename T>
static emfa_status_t cgemv_blocks(Ctx* c, const void* Z, size_t ldz, const void* X, int n, int nrhs, void* Y,
                                  cudaStream_t st)
{
    const Cx<T>*z = (const Cx<T>*)Z, *x = (const Cx<T>*)X;
    Cx<T>* y = (Cx<T>*)Y;
    if constexpr (sizeof(T) == 8) {
        launch_gemv<T, 1>(z, ldz, x, n, nrhs, y, st);
    } else {
        const int blocks = (nrhs + 7) / 8, rpw = rpw_f32(n, (nrhs + blocks - 1) / blocks);
        if (rpw == 1)
            launch_gemv<T, 1>(z, ldz, x, n, nrhs, y, st);
        else if (rpw == 2)
            launch_gemv<T, 2>(z, ldz, x, n, nrhs, y, st);
        else
            launch_gemv<T, 4>(z, ldz, x, n, nrhs, y, st);
    }
    c->kernel_launches += 1;
    EMFA_CUDA(c, cudaGetLastError());
    return EMFA_OK;
}

// ---------------------------------------------------------------------------
// FP32 product of a block of right-hand sides on the CUDA cores: a cluster of
// CTAs per tile of 16 FT rows of Z and 8 RT right-hand sides, each CTA a part
// of k.  Bound by the FP32 FMAs: a thread keeps FT x RT sums, so FT + RT
// 8-byte reads of shared memory feed 4 FT RT FMAs.  Both operands are rows
// along k, copied 16 k at a time (cp.async, CT_STAGES deep) into rows of 17
// elements: the 16 rows that half a warp reads lie in distinct banks.  The
// cluster's partial sums meet in distributed shared memory, added in rank
// order: the parts fill the SMs where n / (16 FT) tiles do not, shorten the
// sums (and with them their error), and need no scratch.  Up to 40
// right-hand sides a thread also closes its sums every 64 k: the error at
// n = 5067, 6.5e-7 -> 2.2e-7.
// us on GB300 | GEMV (up to 32) or digit planes: 480 x 37, 38 | 57; 1033 x 37,
// 52 | 68; 2000 x 17, 56 | 67, x 37, 68 | 102, x 80, 96 | 125; 3000 x 37,
// 102 | 156; 5067 x 16, 123 | 252, x 37, 205 | 350 (FMA rate: 103, 111 with
// the padding to 40), x 80, 403 | 483.  The 64 x 64 tiles below took 97, 170,
// 299, 308, 465, 801 and 814 for the ones of 17 and 37.
// ---------------------------------------------------------------------------
constexpr int CT_THREADS = 128, CT_BK = 16, CT_LD = CT_BK + 1, CT_STAGES = 3, CT_SPLITS = 8, CT_FLUSH = 4;

constexpr int ct_resident(int rt) { return rt <= 5 ? 4 : 3; }  // CTAs an SM

__device__ __forceinline__ void cp_async8_zfill(void* smem, const void* gmem, bool in)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
                 "l"(gmem), "r"(in ? 8 : 0)
                 : "memory");
}

// MASKED: Z has `rows` rows; only the results that mask ([nrhs][rows] bytes) marks
// are stored, and a tile without any does nothing; *again 0: there are none at all
template <int FT, int RT, bool MASKED>
__global__ void __launch_bounds__(CT_THREADS, ct_resident(RT)) k_ctile(const float2* __restrict__ Z, size_t ldz,
                                                      const float2* __restrict__ X, int n, int nrhs, int kper,
                                                      float2* __restrict__ Y, int rows, const unsigned char* __restrict__ mask,
                                                      const int* __restrict__ again)
{
    constexpr int BM = 16 * FT, BN = 8 * RT, STAGE = (BM + BN) * CT_LD;
    extern __shared__ float2 s_ct[];  // [stage][BM + BN][CT_LD], then the partial sums [BN][BM]
    const int tid = threadIdx.x, tf = tid & 15, tr = tid >> 4;
    const int f0 = blockIdx.y * BM, r0 = blockIdx.z * BN, m = MASKED ? rows : n;
    if constexpr (MASKED) {  // the same answer in every CTA of the cluster
        if (*again == 0) return;
        bool any = false;
        for (int q = tid; q < BM * BN; q += CT_THREADS) {
            const int f = f0 + q % BM, r = r0 + q / BM;
            any |= f < m && r < nrhs && mask[(size_t)r * m + f];
        }
        if (!__syncthreads_or(any)) return;
    }
    const int rank = blockIdx.x, csize = gridDim.x;
    const int k0 = rank * kper, k1 = min(n, k0 + kper), steps = k1 > k0 ? (k1 - k0 + CT_BK - 1) / CT_BK : 0;
    const auto load = [&](int t) {
        float2* st = s_ct + (t % CT_STAGES) * STAGE;
        const int k = k0 + t * CT_BK + tf;
#pragma unroll
        for (int i = 0; i < BM / 8; ++i) {
            const int f = tr + 8 * i;
            const bool in = k < k1 && f0 + f < m;
            cp_async8_zfill(st + f * CT_LD + tf, Z + (in ? (size_t)(f0 + f) * ldz + k : 0), in);
        }
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            const int r = tr + 8 * i;
            const bool in = k < k1 && r0 + r < nrhs;
            cp_async8_zfill(st + (BM + r) * CT_LD + tf, X + (in ? (size_t)(r0 + r) * n + k : 0), in);
        }
    };
    constexpr bool TWO = FT * RT <= 20;  // sums of CT_FLUSH steps, and their sum
    float2 acc[FT][RT], tot[TWO ? FT : 1][TWO ? RT : 1];
#pragma unroll
    for (int i = 0; i < FT; ++i)
#pragma unroll
        for (int j = 0; j < RT; ++j) {
            acc[i][j] = make_float2(0.f, 0.f);
            if constexpr (TWO) tot[i][j] = make_float2(0.f, 0.f);
        }
#pragma unroll
    for (int t = 0; t < CT_STAGES - 1; ++t) {
        if (t < steps) load(t);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int t = 0; t < steps; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(CT_STAGES - 2) : "memory");
        __syncthreads();  // stage t has landed for every thread, and stage t - 1 has been read
        if (t + CT_STAGES - 1 < steps) load(t + CT_STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float2* A = s_ct + (t % CT_STAGES) * STAGE + tf * CT_LD;
        const float2* B = s_ct + (t % CT_STAGES) * STAGE + (BM + tr) * CT_LD;
#pragma unroll 4
        for (int kk = 0; kk < CT_BK; ++kk) {
            float2 a[FT], b[RT];
#pragma unroll
            for (int i = 0; i < FT; ++i) a[i] = A[16 * i * CT_LD + kk];
#pragma unroll
            for (int j = 0; j < RT; ++j) b[j] = B[8 * j * CT_LD + kk];
#pragma unroll
            for (int i = 0; i < FT; ++i)
#pragma unroll
                for (int j = 0; j < RT; ++j) {
                    acc[i][j].x = fmaf(a[i].x, b[j].x, acc[i][j].x);
                    acc[i][j].y = fmaf(a[i].x, b[j].y, acc[i][j].y);
                    acc[i][j].x = fmaf(-a[i].y, b[j].y, acc[i][j].x);
                    acc[i][j].y = fmaf(a[i].y, b[j].x, acc[i][j].y);
                }
        }
        if constexpr (TWO)
            if (t % CT_FLUSH == CT_FLUSH - 1 || t == steps - 1) {
#pragma unroll
                for (int i = 0; i < FT; ++i)
#pragma unroll
                    for (int j = 0; j < RT; ++j) {
                        tot[i][j].x += acc[i][j].x;
                        tot[i][j].y += acc[i][j].y;
                        acc[i][j] = make_float2(0.f, 0.f);
                    }
            }
    }
    if constexpr (TWO) {
#pragma unroll
        for (int i = 0; i < FT; ++i)
#pragma unroll
            for (int j = 0; j < RT; ++j) acc[i][j] = tot[i][j];
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (csize == 1) {
#pragma unroll
        for (int j = 0; j < RT; ++j)
#pragma unroll
            for (int i = 0; i < FT; ++i) {
                const int f = f0 + tf + 16 * i, r = r0 + tr + 8 * j;
                if (f < m && r < nrhs && (!MASKED || mask[(size_t)r * m + f])) Y[(size_t)r * n + f] = acc[i][j];
            }
        return;
    }
    __syncthreads();  // the last stages have been read
#pragma unroll
    for (int j = 0; j < RT; ++j)
#pragma unroll
        for (int i = 0; i < FT; ++i) s_ct[(tr + 8 * j) * BM + tf + 16 * i] = acc[i][j];
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
    // rank's share of the tile, from every part in rank order
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(s_ct);
    for (int q = rank * CT_THREADS + tid; q < BM * BN; q += csize * CT_THREADS) {
        const int f = f0 + q % BM, r = r0 + q / BM;
        if (f >= m || r >= nrhs || (MASKED && !mask[(size_t)r * m + f])) continue;
        float2 v[CT_SPLITS], t = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < CT_SPLITS; ++c)
            if (c < csize) {
                uint32_t ra;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(base + 8u * q), "r"(c));
                asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v[c].x), "=f"(v[c].y) : "r"(ra) : "memory");
            }
#pragma unroll
        for (int c = 0; c < CT_SPLITS; ++c)
            if (c < csize) {
                t.x += v[c].x;
                t.y += v[c].y;
            }
        Y[(size_t)r * n + f] = t;
    }
    // no CTA leaves while another may still read its sums
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int FT, int RT, bool MASKED = false>
static emfa_status_t launch_ctile(Ctx* c, const void* Z, size_t ldz, const void* X, int n, int nrhs, void* Y,
                                  cudaStream_t st, int rows = 0, const unsigned char* mask = nullptr, const int* again = nullptr)
{
    constexpr int BM = 16 * FT, BN = 8 * RT;
    constexpr size_t stages = sizeof(float2) * CT_STAGES * (BM + BN) * CT_LD, sums = sizeof(float2) * BM * BN;
    constexpr size_t smem = stages > sums ? stages : sums;
    EMFA_TRY(ensure_smem(c, k_ctile<FT, RT, MASKED>, smem));
    const int ft = ((MASKED ? rows : n) + BM - 1) / BM, rt = (nrhs + BN - 1) / BN;
    const int sms = c->sm_count > 0 ? c->sm_count : 148;
    // parts of k: the fewest steps of the busiest SM, whose CTAs share its
    // FMAs (below two and a half a SM they wait for their loads instead),
    // with about four steps a CTA of filling and adding, in one wave
    int splits = 1;
    long best = LONG_MAX;
    for (int q = 1; q <= CT_SPLITS; ++q) {
        const long per_sm = ((long)ft * rt * q + sms - 1) / sms, steps = (n + q * CT_BK - 1) / (q * CT_BK) + 4;
        if (q > 1 && per_sm > ct_resident(RT)) break;
        const long cost = steps * std::max(2 * per_sm, 5L);
        if (cost < best) {
            best = cost;
            splits = q;
        }
    }
    const int kper = ((n + splits - 1) / splits + CT_BK - 1) / CT_BK * CT_BK;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)splits, (unsigned)ft, (unsigned)rt);
    cfg.blockDim = dim3(CT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)splits;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    EMFA_CUDA(c, cudaLaunchKernelEx(&cfg, k_ctile<FT, RT, MASKED>, (const float2*)Z, ldz, (const float2*)X, n, nrhs, kper,
                                    (float2*)Y, rows, mask, again));
    c->kernel_launches += 1;
    return EMFA_OK;
}

static emfa_status_t cgemm_f32_tiles(Ctx* c, const void* Z, size_t ldz, const void* X, int n, int nrhs, void* Y,
                                     cudaStream_t st)
{
    // even tiles of up to 80 right-hand sides, eight a step
    const int blocks = (nrhs + 79) / 80, rt = ((nrhs + blocks - 1) / blocks + 7) / 8;
    switch (rt) {
    case 1:
    case 2: return launch_ctile<4, 2>(c, Z, ldz, X, n, nrhs, Y, st);
    case 3: return launch_ctile<4, 3>(c, Z, ldz, X, n, nrhs, Y, st);
    case 4: return launch_ctile<4, 4>(c, Z, ldz, X, n, nrhs, Y, st);
    case 5: return launch_ctile<4, 5>(c, Z, ldz, X, n, nrhs, Y, st);
    case 6: return launch_ctile<4, 6>(c, Z, ldz, X, n, nrhs, Y, st);
    case 7: return launch_ctile<4, 7>(c, Z, ldz, X, n, nrhs, Y, st);
    case 8: return launch_ctile<4, 8>(c, Z, ldz, X, n, nrhs, Y, st);
    case 9: return launch_ctile<4, 9>(c, Z, ldz, X, n, nrhs, Y, st);
    default: return launch_ctile<4, 10>(c, Z, ldz, X, n, nrhs, Y, st);
    }
}

emfa_status_t cgemm_f32_masked(Ctx* c, const void* Z, size_t ldz, int rows, const void* X, int n, int nrhs, void* Y,
                               const unsigned char* mask, const int* again, cudaStream_t st)
{
    return launch_ctile<4, 10, true>(c, Z, ldz, X, n, nrhs, Y, st, rows, mask, again);
}

// One FP32 product, the kernel chosen (us, GEMV | tiles): the GEMV up to 4
// right-hand sides (5067 x 3, 102 | 121), below n = 4000 up to 8 (3000 x 8, 74 | 68, x 5,
// 65 | 68; 5067 x 5, 151 | 121) and below 2500 up to 16 (2000 x 12, 57 | 62;
// 3000 x 12, 88 | 68; 5067 x 16, 252 | 123).
emfa_status_t cgemm_f32_block(Ctx* c, const void* Z, size_t ldz, const void* X, int n, int nrhs, void* Y,
                              cudaStream_t st)
{
    if (nrhs <= 4 || (nrhs <= 8 && n < 4000) || (nrhs <= 16 && n < 2500)) return cgemv_blocks<float>(c, Z, ldz, X, n, nrhs, Y, st);
    return cgemm_f32_tiles(c, Z, ldz, X, n, nrhs, Y, st);
}

emfa_status_t cgemm_f32(Ctx* c, const void* Z, size_t ldz, const void* X, int n, int nrhs, void* Y, cudaStream_t st)
{
    if (nrhs <= 16) return cgemv_blocks<float>(c, Z, ldz, X, n, nrhs, Y, st);
    dim3 grd((n + 63) / 64, (nrhs + 63) / 64);
    k_cgemm<float, false><<<grd, 256, 0, st>>>((const Cx<float>*)Z, ldz, (const Cx<float>*)X, n, nrhs, (Cx<float>*)Y,
                                               nullptr, nullptr);
    c->kernel_launches += 1;
    EMFA_CUDA(c, cudaGetLastError());
    return EMFA_OK;
}

// FP64: the GEMV for any number of right-hand sides.  Both are bound by the
// FP64 pipe, but the 64 x 64 tiles, for which this was once chosen above 16
// right-hand sides, leave most SMs idle at these sizes (n = 1080 has 17 tiles
// of rows): n = 1080 x 91, 4456 us with the tiles, 859 us; 2430 x 181, 9.9 ms
// against 7.3 ms; 5070 x 360, 81 ms against 61 ms.
emfa_status_t cgemm_f64(Ctx* c, const void* Z, size_t ldz, const void* X, int n, int nrhs, void* Y, cudaStream_t st)
{
    return cgemv_blocks<double>(c, Z, ldz, X, n, nrhs, Y, st);
}

emfa_status_t cgemm_f32_chunked(Ctx* c, const void* Z, size_t ldz, const void* X, int n, int nrhs, const void* Bsub,
                                void* Yd, cudaStream_t st)
{
    dim3 grd((n + 63) / 64, (nrhs + 63) / 64);
    {
        TimedLaunch tl(c, KT_RESIDUAL, st, 8.0 * n * (double)n * nrhs);
        k_cgemm<float, true><<<grd, 256, 0, st>>>((const Cx<float>*)Z, ldz, (const Cx<float>*)X, n, nrhs, nullptr,
                                                  (const Cx<float>*)Bsub, (Cx<double>*)Yd);
    }
    c->kernel_launches += 1;
    EMFA_CUDA(c, cudaGetLastError());
    return EMFA_OK;
}

}  // namespace emfa
