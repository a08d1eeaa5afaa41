// Y = Z X in FP64 or FP32 accuracy on the 5th-generation tensor cores.
//
// GB300's FP64 pipe runs at 1/64 of the FP32 one, so the CUDA-core FP64 product
// (gemm.cu) is bound by it from a few right-hand sides on.  Here both operands
// are cut into eight signed 8-bit digits,
//     z = 2^(e-63) sum_s d_s 2^(8 (7 - s)),   |d_s| <= 128,
// with one power of two per row of Z and per right-hand side (the fixed-point
// form of an FP64 significand: an entry keeps all 53 bits down to 2^-10 of its
// row's scale), and the digits' products run as FP16 MMAs (integers up to 128
// are exact in FP16, their products in FP32).  Digit pairs (i, j) of one level
// i + j share an accumulator; levels 0..7 are kept (36 of the 64 pairs).  128
// columns of at most eight pairs add up to at most 2^24, so every FP32
// accumulator holds an exact integer, and the sums across those groups are
// exact in 64-bit integers: the result is one rounding of the sum, whatever the
// order, so K can be split over CTAs freely.
//
// Accuracy.  In units of the two scales, a real product is off by at most
// 7 x 2^14 x 2^48 / 2^126 for level 8, 2^-69 for the rest below it, and 2 x 2^-64
// for the cut of its factors: 2^-60.8, 2n times that a component of the sum.  A
// floating-point sum's error goes with S = sum |z||x| instead, and S may be far
// below the scales (columns of Z scaled against x, a large entry that meets a
// zero).  So S itself is formed, per component, by one more FP16 product of the
// operands' magnitudes (10 bits each, every nonzero counted; th::k_hgemm, 1/36
// of the digit products), and k_combine keeps a digit result only where
//     S >= FLOOR (37/512 in FP64, 161/512 in FP32):
// there 2n 2^-60.8 <= (2 ceil(n / 32) + 5) 2^-52 S, the first-order bound of the
// CUDA-core product's own sum (gemm.cu), for every n; FP32, by the same count,
// 2n 2^-29.7 <= (2 ceil(n / 32) + 5) 2^-23 S.  The other results, and those of a
// row or right-hand side with an infinity or NaN, are summed in their own type:
// in FP64 by k_combine's CTA (a term a thread), in FP32 by gemm.cu's tiles.
// Impedance-like operands have S of 0.04 to 2: of 100 CFIE Krylov products a few
// hundredths of a percent of the results are summed again.  Measured against
// extended precision at n = 2430, impedance-like with a dominant diagonal: 9e-17
// of the result, the CUDA-core sums 3e-15.
//
// Kernel k_slice<BN>: one 128 x BN tile and one range of K per CTA, 18 warps:
//   warp 0      TMA producer, K in blocks of 64 columns (128-byte rows): the
//               eight B planes of a block in one 3-D copy into one of two
//               buffers, the A planes one by one through a ring
//   warp 1      tensor memory, MMAs (M = 128, N = BN, K = 16): per block, plane
//               i of A with planes 0..7-i of B, the k-steps outside, so that
//               consecutive MMAs add to different levels (each level has its
//               own BN columns).  After two blocks level i is complete once
//               plane i of A is done, and is committed for the drain
//   warps 2..17 drain: a level's columns to integers (FP32 arithmetic only:
//               conversions share the slow pipe), added to a 64-bit sum per
//               output; warps 2..9 levels 0-3, warps 10..17 levels 4-7
// The MMAs are bound by shared-memory operand reads (4 KB + BN 32 B a MMA at
// 128 B/cycle).  A first form staged 32 columns of all planes at a time, in
// 64-byte rows: the copies (1536 rows a stage, four cycles each) set its pace,
// 416 us at n = 2430 x 181 right-hand sides with the tensor pipe 32 % active,
// whatever the drain did.  A single thread issuing MMAs with descriptors from
// its own registers bounded the second (382 us, 86 cycles a MMA); now 298 us,
// 48 %.
// On GB300, a product of n unknowns and R right-hand sides, its split of Z and
// the magnitudes' product (10 us and 18 us) included, against 64 x 64 CUDA-core
// tiles and against the GEMV that sums again where every result needs it:
// 1080 x 91: 4456, 860 -> 120 us;  2430 x 181: 9928, 7300 -> 450 us.  All results
// of columns scaled against x by 10^4: 1.66 and 11.5 ms.
// FP32 (complex64) operands take four digits, 31 bits below the scale, of which
// the ten pairs of levels 0..3 are kept (a real product is off by at most 3 x 2^14
// x 2^16 / 2^62 for level 4, 2^-39 below it, 2 x 2^-32 for the cut: 2^-29.7 of the
// scales): one rounding to FP32 of a sum that is exact to that, against an FP32
// sum's rounding at every term.
#include "emfa_internal.cuh"
#include "emfa_math.cuh"
#include "gemm_slice.cuh"
#include "tcgen05.cuh"

#include <algorithm>
#include <climits>

namespace emfa {

namespace sl {

constexpr int BM = 128;
constexpr int BK = 64;       // halves of K per block: 128-byte rows
constexpr int GROUP = 2;     // blocks per drain: 128 columns
constexpr int RING = 4;      // A planes in flight
constexpr int THREADS = 32 * (2 + 16);
constexpr int SLICE_NONFINITE = INT_MAX;

// per element type: digits, bits of a scaled value, the top word's exponent
// field, and the least S of a digit result (see above)
template <typename T> struct Cut;
template <> struct Cut<double> {
    static constexpr int NS = 8, BITS = 63, MANT = 20, FIELD_MAX = 0x7ff, EXP_ONE = 1022;
    static constexpr float FLOOR = 37.f / 512.f;
    using Word = unsigned long long;
};
template <> struct Cut<float> {
    static constexpr int NS = 4, BITS = 31, MANT = 23, FIELD_MAX = 0xff, EXP_ONE = 126;
    static constexpr float FLOOR = 161.f / 512.f;
    using Word = unsigned;
};
// magnitudes are FP16 values of 2^15 times the entry over its scale
constexpr float MAG_UNIT = 1.f / 32768.f;

// NS digits; the drain's 16 warps: lane quadrant, column part, four levels each
template <int NS, int BN>
struct Smem {
    static constexpr int SETS = NS / 4;        // of four levels
    static constexpr int PARTS = 4 / SETS;     // of the columns
    static constexpr int EPI = 4 * PARTS;      // warps that drain a level
    static constexpr int A_BYTES = BM * BK * 2;  // one plane
    static constexpr int B_SLICE = BN * BK * 2;
    static constexpr int B_BYTES = NS * B_SLICE;
    static constexpr int TMEM_COLS = NS * BN < 32 ? 32 : NS * BN;
    static constexpr int TOTAL = RING * A_BYTES + 2 * B_BYTES + 1024 /*align*/ + 512 /*barriers*/;
};

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(tc::smem_u32(dst)), "l"((uint64_t)map), "r"(tc::smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

// CW consecutive columns (32 lanes x 32 bit) of tensor memory in one round trip
template <int CW>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float* v)
{
    static_assert(CW == 8 || CW == 16, "");
    if constexpr (CW == 16) {
        tc::tmem_ld16(taddr, v);
    } else {
        uint32_t r[8];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
                     :
                     : "memory");
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
    }
}

// an integer |v| <= 2^24 held in FP32, plus INT_BIAS, as int: v = 4096 h + l
// with both halves read off the mantissa of a sum with 1.5 * 2^23 (whose bits
// are INT_BIAS; 4096 times them vanish modulo 2^32)
constexpr int INT_BIAS = 0x4B400000;
__device__ __forceinline__ int biased_int(float v)
{
    const float big = 12582912.0f;
    const float h = fmaf(v, 1.0f / 4096.0f, big);
    const float l = fmaf(h - big, -4096.0f, v) + big;
    return (int)(((unsigned)__float_as_int(h) << 12) + (unsigned)__float_as_int(l));
}

// acc += x w, one multiply-add, w = 256^i from a kernel argument (w8): a power
// of two known to the compiler becomes four shifts and additions on the ALU pipe, and the drain (30 cycles a
// value of that pipe) then set the kernel's pace
__device__ __forceinline__ void mad_wide(unsigned long long& acc, int x, int w)
{
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(acc) : "r"(x), "r"(w));
}

template <int NS, int BN>
__global__ void __launch_bounds__(THREADS, 1)
    k_slice(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int M, int C,
            int kblocks, int per_split, int4 w8, long long* __restrict__ part, int* __restrict__ err)
{
    using S = Smem<NS, BN>;
    using namespace tc;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sA = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);  // [RING]
    uint8_t* sB = sA + RING * S::A_BYTES;                                       // [2][plane]
    uint64_t* a_full = (uint64_t*)(sB + 2 * S::B_BYTES);
    uint64_t* a_empty = a_full + RING;
    uint64_t* b_full = a_empty + RING;
    uint64_t* b_empty = b_full + 2;
    uint64_t* acc_full = b_empty + 2;
    uint64_t* acc_empty = acc_full + NS;
    uint64_t* done = acc_empty + NS;
    uint32_t* tmem_slot = (uint32_t*)(done + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int f0 = blockIdx.y * BM, c0 = blockIdx.x * BN;
    const int k0 = blockIdx.z * per_split, nk = min(per_split, kblocks - k0);  // blocks; nk >= 1

    if (threadIdx.x == 0) {
        for (int i = 0; i < RING; ++i) {
            mbar_init(a_full + i, 1);
            mbar_init(a_empty + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(b_full + i, 1);
            mbar_init(b_empty + i, 1);
        }
        for (int l = 0; l < NS; ++l) {
            mbar_init(acc_full + l, 1);
            mbar_init(acc_empty + l, S::EPI);
        }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(S::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int na = 0, nb = 0;  // A planes and B blocks issued
            bool ok = true;
            auto load_b = [&](int kb) {
                const int s = kb & 1;
                if (kb >= 2 && !mbar_wait(b_empty + s, ((kb >> 1) - 1) & 1, err, 21)) return false;
                mbar_expect_tx(b_full + s, S::B_BYTES);
                tma_load_3d(sB + s * S::B_BYTES, &tmB, b_full + s, (k0 + kb) * BK, c0, 0);
                nb = kb + 1;
                return true;
            };
            ok = load_b(0);
            for (int kb = 0; kb < nk && ok; ++kb)
                for (int i = 0; i < NS && ok; ++i) {
                    const int s = na % RING;
                    if (na >= RING && !mbar_wait(a_empty + s, ((na / RING) - 1) & 1, err, 22)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(a_full + s, S::A_BYTES);
                    tma_load_3d(sA + s * S::A_BYTES, &tmA, a_full + s, (k0 + kb) * BK, f0, i);
                    ++na;
                    if (i == 1 && kb + 1 < nk) ok = load_b(kb + 1);  // its buffer was free a block ago
                }
            // every copy issued must have landed before the CTA exits
            for (int i = na - RING > 0 ? na - RING : 0; i < na; ++i) mbar_wait(a_full + (i % RING), (i / RING) & 1, err, 23);
            for (int i = nb - 2 > 0 ? nb - 2 : 0; i < nb; ++i) mbar_wait(b_full + (i & 1), (i >> 1) & 1, err, 23);
        }
    } else if (warp == 1) {
        // the whole warp walks the loop and one elected lane issues: the
        // descriptors then are warp-uniform values, in uniform registers
        constexpr uint32_t idesc = idesc_f16(BM, BN);
        const uint32_t dhi = (uint32_t)(sw128_desc(0) >> 32);
        const uint32_t a_lo = (uint32_t)sw128_desc(smem_u32(sA)), b_lo = (uint32_t)sw128_desc(smem_u32(sB));
        bool ok = true;
        for (int kb = 0; kb < nk && ok; ++kb) {
            const int g = kb / GROUP;
            const bool first = kb % GROUP == 0, last = kb % GROUP == GROUP - 1 || kb == nk - 1;
            ok = warp_wait(b_full + (kb & 1), (kb >> 1) & 1, err, 24);
            if (first && g > 0)
                for (int l = 0; l < NS && ok; ++l) ok = warp_wait(acc_empty + l, (g - 1) & 1, err, 26);
            if (!ok) break;
            const uint32_t lb = b_lo + (kb & 1) * (S::B_BYTES >> 4);
            const uint32_t add0 = first ? 0u : 1u;
#pragma unroll
            for (int i = 0; i < NS; ++i) {
                const int s = (kb * NS + i) % RING;
                if (!warp_wait(a_full + s, ((kb * NS + i) / RING) & 1, err, 25)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t la = a_lo + s * (S::A_BYTES >> 4);
#pragma unroll
                for (int j = 0; j < NS - i; ++j)
                    mma_f16_block(tmem + (uint32_t)((i + j) * BN), ((uint64_t)dhi << 32) | la,
                                  ((uint64_t)dhi << 32) | (lb + j * (S::B_SLICE >> 4)), idesc, i == 0 ? add0 : 1u);
                commit_elect(a_empty + s);
                if (last) commit_elect(acc_full + i);
            }
            commit_elect(b_empty + (kb & 1));
        }
        commit_elect(done);
        warp_wait(done, 0, err, 27);
    } else {
        // drain warps: lane quadrant warp % 4, part of the columns, four levels
        constexpr int CW = BN / S::PARTS, LW = CW < 16 ? CW : 16;
        const int q = warp & 3, part_c = ((warp - 2) >> 2) % S::PARTS, set = ((warp - 2) >> 2) / S::PARTS;
        const uint32_t tw = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(part_c * CW);
        unsigned long long sum[CW];
        const int weight[4] = {w8.x, w8.y, w8.z, w8.w};
#pragma unroll
        for (int i = 0; i < CW; ++i) sum[i] = 0;
        const int groups = (nk + GROUP - 1) / GROUP;
        bool ok = true;
        for (int g = 0; g < groups && ok; ++g) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int l = 4 * set + j;
                int w = lane == 0 ? (int)mbar_wait(acc_full + l, g & 1, err, 28) : 0;
                w = __shfl_sync(0xffffffffu, w, 0);
                if (!w) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int c = 0; c < CW; c += LW) {
                    float v[LW];
                    tmem_ld<LW>(tw + (uint32_t)(l * BN + c), v);
                    if (c + LW == CW) {  // all read: the level may be written again
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(acc_empty + l);
                    }
#pragma unroll
                    for (int i = 0; i < LW; ++i) mad_wide(sum[c + i], biased_int(v[i]), weight[3 - j]);
                }
            }
        }
        // the bias of every drain and level; modulo 2^64, so the sums may have wrapped
        const unsigned long long bias = (unsigned long long)groups * INT_BIAS * 0x01010101ull;
        const int f = f0 + 32 * q + lane;
        if (ok && f < M) {
            long long* o = part + ((size_t)blockIdx.z * S::SETS + set) * C * M;
#pragma unroll
            for (int i = 0; i < CW; ++i) {
                const int col = c0 + part_c * CW + i;
                if (col < C) o[(size_t)col * M + f] = (long long)(sum[i] - bias);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::TMEM_COLS) : "memory");
    }
}

// ---------------------------------------------------------------------------
// operand preparation, integers only
// ---------------------------------------------------------------------------
// exponent and leading mantissa bits of |x|: an integer that orders magnitudes
__device__ __forceinline__ int top_word(double x) { return __double2hiint(x) & 0x7fffffff; }
__device__ __forceinline__ int top_word(float x) { return __float_as_int(x) & 0x7fffffff; }

// scale of a row from its largest top word: the exponent field eb, at least 1,
// with |x| < 127/128 2^(eb - EXP_ONE), so that the leading digit stays below 128
template <typename T>
__device__ __forceinline__ int scale_field(int top)
{
    return max(1, (top + (1 << (Cut<T>::MANT - 6))) >> Cut<T>::MANT);
}

// biased digits of x at scale eb: byte s of the result is d_(NS-1-s) + 128
__device__ __forceinline__ unsigned long long digits(double x, int eb)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int ef = (int)((b >> 52) & 0x7ff);
    unsigned long long m = b & 0xFFFFFFFFFFFFFull;
    if (ef) m |= 1ull << 52;
    const int s = (ef ? ef : 1) - eb + 10;  // 9 or 10 for the largest
    long long v;
    if (s >= 0)
        v = (long long)(m << s);
    else
        v = s < -54 ? 0 : (long long)((m + (1ull << (-s - 1))) >> -s);
    if ((long long)b < 0) v = -v;
    return ((unsigned long long)v + 0x0080808080808080ull) ^ (0x80ull << 56);
}
__device__ __forceinline__ unsigned digits(float x, int eb)
{
    const unsigned b = (unsigned)__float_as_int(x);
    const int ef = (int)((b >> 23) & 0xff);
    unsigned m = b & 0x7fffffu;
    if (ef) m |= 1u << 23;
    const int s = (ef ? ef : 1) - eb + 7;  // 6 or 7 for the largest
    int v;
    if (s >= 0)
        v = (int)(m << s);
    else
        v = s < -25 ? 0 : (int)((m + (1u << (-s - 1))) >> -s);
    if ((int)b < 0) v = -v;
    return ((unsigned)v + 0x00808080u) ^ 0x80000000u;
}

// |x| 2^15 / 2^(eb - EXP_ONE) as an FP16 value: 10 mantissa bits, cut off; below
// FP16's range the smallest value, so that only a zero is zero
template <typename T>
__device__ __forceinline__ unsigned magnitude(T x, int eb)
{
    int ef, m;  // exponent field and 10 mantissa bits
    bool zero;
    if constexpr (sizeof(T) == 8) {
        const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
        zero = b == 0;
        ef = (int)(b >> 52);
        m = (int)(b >> 42) & 0x3ff;
        if (ef == 0 && !zero) {  // subnormal
            const int z = __clzll((long long)b) - 11;
            ef = 1 - z;
            m = (int)((b << z) >> 42) & 0x3ff;
        }
    } else {
        const unsigned b = (unsigned)__float_as_int(x) & 0x7fffffffu;
        zero = b == 0;
        ef = (int)(b >> 23);
        m = (int)(b >> 13) & 0x3ff;
        if (ef == 0 && !zero) {
            const int z = __clz((int)b) - 8;
            ef = 1 - z;
            m = (int)((b << z) >> 13) & 0x3ff;
        }
    }
    const int e = ef - eb + 29;
    const int low = e < -9 ? 1 : max(1, (m | 0x400) >> (1 - min(e, 1)));
    return zero ? 0u : (unsigned)(e >= 1 ? (e << 10) | m : low);
}

// digit s of a complex pair as two FP16 integers: the byte under the exponent
// of 1024 is 1024 + d + 128
template <typename Word>
__device__ __forceinline__ unsigned pair_digit(Word a, Word b, int s)
{
    const int byte = (int)sizeof(Word) - 1 - s;
    const unsigned wa = (unsigned)(byte & 4 ? (unsigned long long)a >> 32 : a),
                   wb = (unsigned)(byte & 4 ? (unsigned long long)b >> 32 : b);
    const unsigned x = (__byte_perm(wa, wb, (byte & 3) | ((4 + (byte & 3)) << 8)) & 0x00ff00ffu) | 0x64006400u;
    const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&x), __half2half2(__float2half_rn(1152.f)));
    return *reinterpret_cast<const unsigned*>(&r);
}

__device__ __forceinline__ int block_max_int(int m, int* red)
{
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) red[w] = m;
    __syncthreads();
    if (w == 0) {
        m = l < (int)(blockDim.x >> 5) ? red[l] : 0;
        for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (l == 0) red[0] = m;
    }
    __syncthreads();
    return red[0];
}

// CTA per row of Z: its scale, then its digits and, in the plane after them, its
// magnitudes (the row is read twice, the second time from L2)
template <typename T>
__global__ void __launch_bounds__(256) k_slice_rows(const Cx<T>* __restrict__ Z, size_t ldz, int n, size_t ldk,
                                                    __half* __restrict__ D, int* __restrict__ ex)
{
    using Word = typename Cut<T>::Word;
    __shared__ int red[32];
    const int i = blockIdx.x;
    const Cx<T>* z = Z + (size_t)i * ldz;
    int m = 0;
#pragma unroll 4
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const Cx<T> v = z[k];
        m = max(m, max(top_word(v.re), top_word(v.im)));
    }
    m = block_max_int(m, red);
    const bool bad = m >> Cut<T>::MANT == Cut<T>::FIELD_MAX;
    const int eb = scale_field<T>(m);
    if (threadIdx.x == 0) ex[i] = bad ? SLICE_NONFINITE : eb;
    const size_t plane = (size_t)gridDim.x * ldk / 2;
    unsigned* o = reinterpret_cast<unsigned*>(D) + (size_t)i * (ldk / 2);
    constexpr Word zero = (Word)0x8080808080808080ull;
    // two elements a thread, one 8-byte store a plane (the rows of D are padded
    // to 16 bytes: an odd row's last store ends in the padding)
    for (int k = 2 * threadIdx.x; k < n; k += 2 * blockDim.x) {
        const Cx<T> v = z[k], u = k + 1 < n ? z[k + 1] : cx(T(0), T(0));
        const Word a = bad ? zero : digits(v.re, eb), b = bad ? zero : digits(v.im, eb);
        const Word c = bad ? zero : digits(u.re, eb), d = bad ? zero : digits(u.im, eb);
#pragma unroll
        for (int s = 0; s < Cut<T>::NS; ++s)
            *reinterpret_cast<uint2*>(o + s * plane + k) = make_uint2(pair_digit(a, b, s), pair_digit(c, d, s));
        *reinterpret_cast<uint2*>(o + Cut<T>::NS * plane + k) =
            bad ? make_uint2(0u, 0u)
                : make_uint2(magnitude(v.re, eb) | magnitude(v.im, eb) << 16,
                             magnitude(u.re, eb) | magnitude(u.im, eb) << 16);
    }
}

// CTA per right-hand side: B rows 2r = (Re, -Im) and 2r + 1 = (Im, Re), of the
// magnitudes (|Re|, |Im|) and (|Im|, |Re|).  unit[r]: the magnitudes' unit;
// *again: no result to be summed again so far.
template <typename T>
__global__ void __launch_bounds__(256) k_slice_rhs(const Cx<T>* __restrict__ X, int n, int nrhs, size_t ldk,
                                                   __half* __restrict__ D, int* __restrict__ ex,
                                                   float* __restrict__ unit, int* __restrict__ again)
{
    using Word = typename Cut<T>::Word;
    __shared__ int red[32];
    const int r = blockIdx.x;
    const Cx<T>* x = X + (size_t)r * n;
    int m = 0;
#pragma unroll 4
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const Cx<T> v = x[k];
        m = max(m, max(top_word(v.re), top_word(v.im)));
    }
    m = block_max_int(m, red);
    const bool bad = m >> Cut<T>::MANT == Cut<T>::FIELD_MAX;
    const int eb = scale_field<T>(m);
    if (threadIdx.x == 0) {
        ex[r] = bad ? SLICE_NONFINITE : eb;
        unit[r] = MAG_UNIT;
        if (r == 0) *again = 0;
    }
    const size_t plane = (size_t)2 * nrhs * ldk / 2;
    unsigned* o0 = reinterpret_cast<unsigned*>(D) + (size_t)(2 * r) * (ldk / 2);
    unsigned* o1 = o0 + ldk / 2;
    constexpr Word zero = (Word)0x8080808080808080ull;
#pragma unroll 2
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const Cx<T> v = x[k];
        const Word a = bad ? zero : digits(v.re, eb), b = bad ? zero : digits(v.im, eb),
                   nb = bad ? zero : digits(-v.im, eb);
#pragma unroll
        for (int s = 0; s < Cut<T>::NS; ++s) {
            o0[s * plane + k] = pair_digit(a, nb, s);
            o1[s * plane + k] = pair_digit(b, a, s);
        }
        const unsigned re = bad ? 0u : magnitude(v.re, eb), im = bad ? 0u : magnitude(v.im, eb);
        o0[Cut<T>::NS * plane + k] = re | im << 16;
        o1[Cut<T>::NS * plane + k] = im | re << 16;
    }
}

// (hi 2^32 + lo) 2^ex, rounded to nearest even once (twice below the normal range)
__device__ __forceinline__ double to_double(long long hi, long long lo, int ex)
{
    // 128-bit two's complement t1:t0
    unsigned long long t0 = ((unsigned long long)hi << 32), t1 = (unsigned long long)(hi >> 32);
    const unsigned long long s0 = t0 + (unsigned long long)lo;
    t1 += (unsigned long long)(lo >> 63) + (s0 < t0 ? 1ull : 0ull);
    t0 = s0;
    const bool neg = (long long)t1 < 0;
    if (neg) {
        t0 = ~t0 + 1ull;
        t1 = ~t1 + (t0 == 0 ? 1ull : 0ull);
    }
    if (!(t0 | t1)) return 0.0;
    // top 64 significant bits, the rest as a sticky bit
    int lz;
    unsigned long long m;
    if (t1) {
        lz = __clzll((long long)t1);
        m = lz ? (t1 << lz) | (t0 >> (64 - lz)) : t1;
        if (lz ? (t0 << lz) : t0) m |= 1ull;
    } else {
        lz = 64 + __clzll((long long)t0);
        m = t0 << (lz - 64);
    }
    unsigned long long q = m >> 11;
    const unsigned rest = (unsigned)m & 0x7ffu;
    q += (rest > 0x400u || (rest == 0x400u && (q & 1ull))) ? 1ull : 0ull;  // [2^52, 2^53]
    const int e = 127 - lz - 52 + ex;  // value = q 2^e
    double v;
    if (e + 1075 >= 1 && e + 1075 <= 2045)
        v = __longlong_as_double((long long)(((unsigned long long)(e + 1074) << 52) + q));
    else
        v = scalbn((double)q, e);
    return neg ? -v : v;
}

// report (optional): a page-locked host word that gets *err.
// Y (rows n apart a right-hand side) from the partial sums of all splits where the digits are as good as a sum in
// T (S at least FLOOR, or zero: no product at all); a pipeline that gave up (err)
// leaves NaN.  The rest is summed in T: FP64 by the CTA, one result after the
// other, a term a thread (a few results cost a few us, all of them about the
// GEMV's time); FP32 results are marked in `mask` for gemm.cu's tiles.
template <typename T>
__global__ void __launch_bounds__(256) k_combine(const long long* __restrict__ part, int splits, int rows, int n, int nrhs,
                                                 const int* __restrict__ exz, const int* __restrict__ exx,
                                                 const float2* __restrict__ S, const Cx<T>* __restrict__ Z, size_t ldz,
                                                 const Cx<T>* __restrict__ X, const int* __restrict__ err,
                                                 Cx<T>* __restrict__ Y, unsigned char* __restrict__ mask,
                                                 int* __restrict__ again, int* __restrict__ report)
{
    if (report && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && *err) *(volatile int*)report = *err;
    const int f = blockIdx.x * blockDim.x + threadIdx.x, r = blockIdx.y;
    const bool live = f < rows;
    bool sum = false;
    Cx<T> y = cx(T(0), T(0));
    if (live) {
        const int ez = exz[f], ex = exx[r];
        const float2 s = S[(size_t)r * rows + f];
        if (*err) {
            y.re = y.im = (T)__longlong_as_double(0x7ff8000000000000ll);
        } else if (ez == SLICE_NONFINITE || ex == SLICE_NONFINITE || (s.x > 0.f && s.x < Cut<T>::FLOOR) ||
                   (s.y > 0.f && s.y < Cut<T>::FLOOR)) {
            sum = true;
        } else {
            const size_t plane = (size_t)2 * nrhs * rows;
            const long long* p0 = part + (size_t)(2 * r) * rows + f;
            // z = V 2^(e - BITS), e = field - EXP_ONE; the lowest kept level, NS - 1, weighs 2^(8 (NS - 1)) in V V
            const int e = ez + ex - 2 * (Cut<T>::EXP_ONE + Cut<T>::BITS) + 8 * (Cut<T>::NS - 1);
            long long s0 = 0, s1 = 0;  // levels 0-3
            if constexpr (Cut<T>::NS == 8) {
                long long l0 = 0, l1 = 0;
                for (int q = 0; q < splits; ++q, p0 += 2 * plane) {
                    s0 += p0[0];
                    s1 += p0[rows];
                    l0 += p0[plane];
                    l1 += p0[plane + rows];
                }
                y = cx((T)to_double(s0, l0, e), (T)to_double(s1, l1, e));
            } else {
                for (int q = 0; q < splits; ++q, p0 += plane) {
                    s0 += p0[0];
                    s1 += p0[rows];
                }
                y = cx((T)to_double(s0 >> 32, s0 & 0xffffffffll, e), (T)to_double(s1 >> 32, s1 & 0xffffffffll, e));
            }
        }
    }
    if constexpr (Cut<T>::NS == 8) {
        __shared__ unsigned todo[8];
        __shared__ Cx<T> red[2][8];
        const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
        const unsigned b = __ballot_sync(0xffffffffu, sum);
        if (l == 0) todo[w] = b;
        if (__syncthreads_or(sum)) {  // uniform
            const Cx<T>* x = X + (size_t)r * n;
            int turn = 0;
            for (int q = 0; q < 8; ++q)
                for (unsigned left = todo[q]; left; left &= left - 1, turn ^= 1) {
                    const int t = 32 * q + __ffs((int)left) - 1;
                    const Cx<T>* z = Z + (size_t)(blockIdx.x * blockDim.x + t) * ldz;
                    T re = 0, im = 0;
#pragma unroll 4
                    for (int k = threadIdx.x; k < n; k += 256) {
                        const Cx<T> a = z[k], v = x[k];
                        re = fma(a.re, v.re, re);
                        re = fma(-a.im, v.im, re);
                        im = fma(a.re, v.im, im);
                        im = fma(a.im, v.re, im);
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        re += __shfl_xor_sync(0xffffffffu, re, o);
                        im += __shfl_xor_sync(0xffffffffu, im, o);
                    }
                    if (l == 0) red[turn][w] = cx(re, im);
                    __syncthreads();  // the next result's sums go to the other half
                    if ((int)threadIdx.x == t) {
                        y = red[turn][0];
#pragma unroll
                        for (int i = 1; i < 8; ++i) {
                            y.re += red[turn][i].re;
                            y.im += red[turn][i].im;
                        }
                    }
                }
        }
        if (live) Y[(size_t)r * n + f] = y;
    } else if (live) {
        mask[(size_t)r * rows + f] = sum;
        if (sum)
            *again = 1;
        else
            Y[(size_t)r * n + f] = y;
    }
}

}  // namespace sl

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static size_t slice_ld(int n) { return ((size_t)2 * n + 7) & ~(size_t)7; }  // 16-byte rows

// ns digits and the magnitudes
static size_t slice_plane_bytes(int ns, int n, int rows)
{
    return Carver::round(sizeof(__half) * (ns + 1) * (size_t)rows * slice_ld(n)) + Carver::round(sizeof(int) * (size_t)rows);
}

// A context keeps at most this much of planes between calls: a single product
// splits Z by blocks of rows that fit (the digits of the right-hand sides, formed
// anew for each block, are about 1 % of a block's time at n = 6000 x 181), and a
// solve, whose products all read the planes, gives larger ones back at its end.
constexpr size_t PLANES_KEPT = (size_t)1 << 30;
static int rows_kept(int ns, int n)
{
    const size_t row = sizeof(__half) * (ns + 1) * slice_ld(n);
    return (int)std::min<size_t>((size_t)n, std::max<size_t>(PLANES_KEPT / row / sl::BM, 1) * sl::BM);
}

static emfa_status_t slice_map(Ctx* c, CUtensorMap* m, const void* ptr, uint64_t inner, uint64_t rows, size_t ld,
                               uint64_t planes, uint32_t box_rows, uint32_t box_planes)
{
    auto fn = tensor_map_encoder();
    if (!fn) {
        set_error(c, "cuTensorMapEncodeTiled unavailable");
        return EMFA_ERR_CUDA;
    }
    cuuint64_t dims[3] = {inner, rows, planes};
    cuuint64_t strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)ld * 2 * rows};
    cuuint32_t box[3] = {(cuuint32_t)sl::BK, box_rows, box_planes};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error(c, "cuTensorMapEncodeTiled (digit planes) failed (" + std::to_string((int)r) + ")");
        return EMFA_ERR_CUDA;
    }
    return EMFA_OK;
}

// error words of the products: ints 8 (a solve's) and 9 (single products') of
// the context's GEMM error slot
static emfa_status_t slice_err(Ctx* c, int word, int** err)
{
    void* ep = nullptr;
    EMFA_TRY(ctx_workspace(c, WS_GEMM_ERR, 64, &ep));
    *err = (int*)ep + word;
    return EMFA_OK;
}

emfa_status_t slice_word(Ctx* c, int** err, cudaStream_t st)
{
    EMFA_TRY(slice_err(c, 9, err));
    if (!c->slice_word_clear) EMFA_CUDA(c, cudaMemsetAsync(*err, 0, sizeof(int), st));
    c->slice_word_clear = true;
    return EMFA_OK;
}

static emfa_status_t timed_out(Ctx* c, int stage)
{
    set_error(c, "digit-plane tensor-core product: a pipeline wait timed out (stage " + std::to_string(stage) + ")");
    return EMFA_ERR_TIMEOUT;
}

emfa_status_t slice_report(Ctx* c)
{
    std::lock_guard<std::mutex> lk(c->slice_mu);
    volatile int* told = c->pinned + Ctx::PINNED - 1;
    const int stage = *told;
    if (!stage) return EMFA_OK;
    *told = 0;
    c->slice_word_clear = false;
    return timed_out(c, stage);
}

// The planes take twice the matrix's memory, in workspaces of the context that
// calls on its own stream share: a context with an HBM budget, a caller's
// stream (its calls may overlap others of the context, and may be captured) and
// planes above 16 GB keep the CUDA-core product, which needs no memory.
static bool slice_allowed(Ctx* c, int ns, int n, cudaStream_t st)
{
    if (n < 128 || c->budget || c->stream_ordered || st != c->stream || slice_plane_bytes(ns - 1, n, n) > ((size_t)16 << 30))
        return false;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone;
}

bool slice_worthwhile(Ctx* c, int n, int nrhs, bool built, cudaStream_t st)
{
    if (!slice_allowed(c, sl::Cut<double>::NS, n, st)) return false;
    // Measured (us, a call with its one split of Z | the CUDA-core GEMV): n = 256, 24 right-hand sides 63 | 51,
    // 40: 65 | 68; 480, 12: 67 | 53, 16: 69 | 71; 750, 8: 71 | 91; 1080, 6: 86 | 83, 8: 86 | 118; 2430, 4: 184 | 192;
    // 5070, 4: 540 | 842.  The split of Z, which a solve makes once, is 8 us of it at n = 480, 15 at 1080, 60 at 2430.
    if (built) return nrhs >= (n >= 2000 ? 3 : n >= 1000 ? 6 : n >= 600 ? 8 : n >= 480 ? 12 : 32);
    return nrhs >= (n >= 2000 ? 4 : n >= 600 ? 8 : n >= 480 ? 16 : 32);
}

// One FP32 product with its split of Z, where it beats the CUDA cores' tiles
// (us, this | tiles: n = 1033 x 360, 139 | 98; 1500 x 360, 177 | 191; 2000 x 280, 252 | 241,
// x 360, 263 | 346; 3000 x 160, 294 | 296, x 240, 359 | 386, x 360, 443 | 689; 5067 x 96, 574 | 529,
// x 128, 604 | 677, x 360, 1187 | 1621): above 100 right-hand sides and 600000 results.  With every
// result summed again (columns scaled against x) 5067 x 360 takes 2921; 64 x 64 tiles, 2350.  Errors on
// normal entries, n = 480 to 5067: this 3e-8, the tiles 2.1e-7 to 8.1e-7, the GEMV 1.2e-7 to 3.3e-7, 64 x 64 tiles
// 5.5e-7 to 1.8e-6.
static bool slice_worthwhile_f32(Ctx* c, int n, int nrhs, cudaStream_t st)
{
    return nrhs > 100 && (long)n * nrhs > 600000 && slice_allowed(c, sl::Cut<float>::NS, n, st);
}

template <typename T>
static emfa_status_t prepare_t(Ctx* c, int slot, const void* Z, size_t ldz, int n, int rows, SlicePlanes* out,
                               cudaStream_t st)
{
    constexpr int NS = sl::Cut<T>::NS;
    const size_t ldk = slice_ld(n);
    void* wp = nullptr;
    EMFA_TRY(ctx_workspace(c, slot, slice_plane_bytes(NS, n, rows) + 512, &wp));
    Carver cv{(char*)wp};
    __half* d = cv.take<__half>((NS + 1) * (size_t)rows * ldk);
    int* ex = cv.take<int>(rows);
    sl::k_slice_rows<T><<<rows, 256, 0, st>>>((const Cx<T>*)Z, ldz, n, ldk, d, ex);
    c->kernel_launches += 1;
    EMFA_CUDA(c, cudaGetLastError());
    *out = SlicePlanes{d, ex, Z, ldz, n, rows, ldk};
    return EMFA_OK;
}

emfa_status_t slice_prepare(Ctx* c, int slot, const void* Z, size_t ldz, int n, SlicePlanes* out, cudaStream_t st)
{
    int* err = nullptr;
    EMFA_TRY(slice_err(c, 8, &err));
    EMFA_CUDA(c, cudaMemsetAsync(err, 0, sizeof(int), st));
    return prepare_t<double>(c, slot, Z, ldz, n, n, out, st);
}

// Column tile (narrow for few right-hand sides; the wide one fills tensor
// memory with a level's sums each), and over how many CTAs a tile's K is split:
// the split with the fewest K blocks in the longest chain of CTAs an SM runs, a
// CTA's fixed cost (pipeline fill, last drain, partial sums written and read
// again) counted as two and a half blocks.
template <typename T> struct Tile;
template <> struct Tile<double> { static constexpr int NARROW = 16, WIDE = 64; };
template <> struct Tile<float> { static constexpr int NARROW = 32, WIDE = 128; };

template <typename T>
static void slice_shape(Ctx* c, int n, int rows, int nrhs, int* bn, int* splits, int* per_split)
{
    const int sms = c->sm_count > 0 ? c->sm_count : 148;
    *bn = 2 * nrhs <= Tile<T>::NARROW ? Tile<T>::NARROW : Tile<T>::WIDE;
    const int blocks = (2 * n + sl::BK - 1) / sl::BK, groups = (blocks + sl::GROUP - 1) / sl::GROUP;
    const long tiles = (long)((rows + sl::BM - 1) / sl::BM) * ((2 * nrhs + *bn - 1) / *bn);
    long best = -1;
    for (int s = 1; s <= std::min(groups, 16); ++s) {
        const int g = (groups + s - 1) / s, used = (groups + g - 1) / g;
        const long waves = (tiles * used + sms - 1) / sms;
        const long cost = waves * (2 * g * sl::GROUP + 5);
        if (best < 0 || cost < best) {
            best = cost;
            *splits = used;
            *per_split = g * sl::GROUP;
        }
    }
}

template <int NS, int BN>
static emfa_status_t launch_slice(Ctx* c, const CUtensorMap& ta, const CUtensorMap& tb, int n, int rows, int nrhs, int splits,
                                  int per_split, long long* part, int* err, cudaStream_t st)
{
    using S = sl::Smem<NS, BN>;
    EMFA_TRY(ensure_smem(c, sl::k_slice<NS, BN>, S::TOTAL));
    const dim3 grd((2 * nrhs + BN - 1) / BN, (rows + sl::BM - 1) / sl::BM, splits);
    sl::k_slice<NS, BN><<<grd, sl::THREADS, S::TOTAL, st>>>(ta, tb, rows, 2 * nrhs, (2 * n + sl::BK - 1) / sl::BK,
                                                            per_split, make_int4(1, 1 << 8, 1 << 16, 1 << 24), part,
                                                            err);
    c->kernel_launches += 1;
    EMFA_CUDA(c, cudaGetLastError());
    return EMFA_OK;
}

template <typename T>
static emfa_status_t apply_t(Ctx* c, int slot, const SlicePlanes& p, const void* X, int nrhs, void* Y, int* err,
                             int* report, cudaStream_t st)
{
    constexpr int NS = sl::Cut<T>::NS, SETS = NS / 4, NARROW = Tile<T>::NARROW, WIDE = Tile<T>::WIDE;
    const int n = p.n, rows = p.rows;
    // blocks of right-hand sides bound the scratch: 512, fewer above n = 7000
    // (256 MB of digits)
    const int RB = (int)std::min<size_t>(512, std::max<size_t>(1, ((size_t)256 << 20) / (sizeof(__half) * (NS + 1) * 2 * 64 * p.ldk)) * 64);
    const int rmax = std::min(nrhs, RB);
    int bn, splits, per_split;
    slice_shape<T>(c, n, rows, rmax, &bn, &splits, &per_split);
    const size_t brow = (size_t)2 * rmax * p.ldk;
    int smax = splits;
    if (nrhs % RB) {
        int b2, s2, p2;
        slice_shape<T>(c, n, rows, nrhs % RB, &b2, &s2, &p2);
        // scratch of the last block: fewer columns, perhaps more splits
        smax = std::max(splits, (int)(((long)s2 * (nrhs % RB) + rmax - 1) / rmax));
    }
    const size_t res = (size_t)rmax * rows, parts = (size_t)smax * 2 * SETS * res;
    void* wp = nullptr;
    EMFA_TRY(ctx_workspace(c, slot,
                           Carver::round(sizeof(__half) * (NS + 1) * brow) + 2 * Carver::round(sizeof(int) * (size_t)rmax) +
                               Carver::round(sizeof(long long) * parts) + Carver::round(sizeof(float2) * res) +
                               Carver::round(res) + 2048,
                           &wp));
    Carver cv{(char*)wp};
    __half* b = cv.take<__half>((NS + 1) * brow);
    int* ex = cv.take<int>(rmax);
    float* unit = cv.take<float>(rmax);
    long long* part = cv.take<long long>(parts);
    float2* sums = cv.take<float2>(res);
    unsigned char* mask = cv.take<unsigned char>(res);
    int* again = cv.take<int>(1);
    CUtensorMap ta, tb;
    EMFA_TRY(slice_map(c, &ta, p.d, 2 * (uint64_t)n, (uint64_t)rows, p.ldk, NS, sl::BM, 1));
    for (int r0 = 0; r0 < nrhs; r0 += RB) {
        const int nr = std::min(RB, nrhs - r0);
        const Cx<T>* x = (const Cx<T>*)X + (size_t)r0 * n;
        slice_shape<T>(c, n, rows, nr, &bn, &splits, &per_split);
        EMFA_TRY(slice_map(c, &tb, b, 2 * (uint64_t)n, 2 * (uint64_t)nr, p.ldk, NS, (uint32_t)bn, NS));
        Cx<T>* y = (Cx<T>*)Y + (size_t)r0 * n;
        sl::k_slice_rhs<T><<<nr, 256, 0, st>>>(x, n, nr, p.ldk, b, ex, unit, again);
        c->kernel_launches += 1;
        EMFA_CUDA(c, cudaGetLastError());
        EMFA_TRY((bn == NARROW ? launch_slice<NS, NARROW> : launch_slice<NS, WIDE>)(c, ta, tb, n, rows, nr, splits,
                                                                                  per_split, part, err, st));
        EMFA_TRY(hgemm_planes(c, p.d + NS * (size_t)rows * p.ldk, b + NS * (size_t)2 * nr * p.ldk, rows, n, nr, p.ldk, unit,
                              sums, err, st));
        sl::k_combine<T><<<dim3((rows + 255) / 256, nr), 256, 0, st>>>(part, splits, rows, n, nr, p.ex, ex, sums,
                                                                       (const Cx<T>*)p.Z, p.ldz, x, err, y, mask, again,
                                                                       report);
        c->kernel_launches += 1;
        EMFA_CUDA(c, cudaGetLastError());
        if (NS == 4) EMFA_TRY(cgemm_f32_masked(c, p.Z, p.ldz, rows, x, n, nr, y, mask, again, st));
    }
    return EMFA_OK;
}

emfa_status_t slice_apply(Ctx* c, int slot, const SlicePlanes& p, const void* X, int nrhs, void* Y, cudaStream_t st)
{
    int* err = nullptr;
    EMFA_TRY(slice_err(c, 8, &err));
    return apply_t<double>(c, slot, p, X, nrhs, Y, err, nullptr, st);
}

emfa_status_t slice_check(Ctx* c, cudaStream_t st)
{
    int* err = nullptr;
    EMFA_TRY(slice_err(c, 8, &err));
    int h = 0;
    EMFA_CUDA(c, cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st));
    EMFA_CUDA(c, cudaStreamSynchronize(st));
    return h ? timed_out(c, h) : EMFA_OK;
}

void slice_release(Ctx* c)
{
    for (int slot : {WS_SLICE_Z, WS_SLICE_B})
        if (c->ws[slot].bytes > PLANES_KEPT) c->ws[slot].release();
}

template <typename T>
static emfa_status_t matvec_t(Ctx* c, const void* Z, size_t ldz, const void* X, int n, int nrhs, void* Y,
                              cudaStream_t st, bool* done)
{
    // the whole sequence of launches at once: another thread's product on this
    // context's stream uses the same workspaces before or after it
    std::lock_guard<std::mutex> lk(c->slice_mu);
    int* err = nullptr;
    EMFA_TRY(slice_word(c, &err, st));
    const int step = rows_kept(sl::Cut<T>::NS, n);
    emfa_status_t s = EMFA_OK;
    for (int f0 = 0; f0 < n && s == EMFA_OK; f0 += step) {
        SlicePlanes p;
        s = prepare_t<T>(c, WS_SLICE_MV, (const Cx<T>*)Z + (size_t)f0 * ldz, ldz, n, std::min(step, n - f0), &p, st);
        if (s == EMFA_OK)
            s = apply_t<T>(c, WS_SLICE_MV_B, p, X, nrhs, (Cx<T>*)Y + f0, err, c->pinned + Ctx::PINNED - 1, st);
    }
    if (s == EMFA_ERR_OOM) {
        cudaGetLastError();  // no room: the caller's CUDA-core product
        return EMFA_OK;
    }
    EMFA_TRY(s);
    *done = true;
    return EMFA_OK;
}

emfa_status_t slice_matvec(Ctx* c, int prec, const void* Z, size_t ldz, const void* X, int n, int nrhs, void* Y,
                           cudaStream_t st, bool* done)
{
    *done = false;
    if (prec == EMFA_F64)
        return slice_worthwhile(c, n, nrhs, false, st) ? matvec_t<double>(c, Z, ldz, X, n, nrhs, Y, st, done) : EMFA_OK;
    return slice_worthwhile_f32(c, n, nrhs, st) ? matvec_t<float>(c, Z, ldz, X, n, nrhs, Y, st, done) : EMFA_OK;
}

}  // namespace emfa
