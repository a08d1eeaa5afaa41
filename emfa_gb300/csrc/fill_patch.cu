// Impedance fill by patches of RWGs, for the fills whose cost is the kernel
// values G = exp(-jkR)/R of triangle point pairs: the FP64 fills (EFIE and
// CFIE, 3 x 3 points) and the configuration's 7 x 7-point EFIE fill (FP32 and
// FP64).
//
// An entry takes four triangle pairs and every triangle pair serves up to nine
// entries, so a thread per entry evaluates each kernel value nine times.  Here
// the RWGs are grouped into compact patches of 24 (k-d bisection of the edge
// midpoints, about 23 triangles a patch, whatever order the mesh lists them
// in), and a CTA takes a patch pair (bf <= bs):
//   1. a thread per triangle pair evaluates the point pairs once and reduces
//      them to the values of the pair's (field corner, source corner)
//      combinations, into shared memory;
//   2. a thread per entry adds its four values, and the self terms from the
//      FP64 table, and stores the entry and, off the diagonal of patches, its
//      mirror image: the regular part of an EFIE entry is the same both ways,
//      of a CFIE entry the EFIE part is, and the MFIE part of either direction
//      is formed from the same kernel values.
//
// EFIE, step 1: with v_i, w_j the triangles' corners, lambda the barycentric
// coordinates of the points and S_ij = sum_pq w_p w_q lambda_i(p) lambda_j(q)
// G_pq, the pair's value for the free vertices v_a and w_b is
//   1/4 sum_ij S_ij (v_i - v_a).(w_j - w_b) - 1/k^2 sum_ij S_ij,
// four terms (i != a, j != b) of nine edge-vector products: no cancellation,
// the edge vectors are differences of corners, and about 10 operations a
// combination instead of 6 a point pair.
//
// Bound: the FP64 pipe (16 cycles a warp instruction and SM) for the FP64
// fills, FP32 issue for the FP32 one.  On GB300, against a thread per entry:
//   EFIE FP64, N = 2427:        22.4 -> 2.8 ms a fill (the kernel 22.3 -> 2.6)
//   CFIE FP64, N = 1080:        5.75 -> 1.71 ms the kernel (N = 2430: 28.4 -> 8.2 ms a fill)
//   EFIE 7 x 7 FP32, N = 1920:  1.81 -> 0.20 ms (2.9 -> 0.41 a fill, with the table)
#include "emfa_internal.cuh"
#include "emfa_math.cuh"
#include "fill_entry.cuh"
#include "fill_patch.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

namespace emfa {

namespace {

constexpr int PB = 24;           // RWGs a patch: 48 (triangle, corner) slots; the CFIE values of a patch
                                 // pair take 74 KB, so two CTAs fit an SM
constexpr int PS = 2 * PB;       // slots, and triangles, a patch has at most
constexpr int SC_N = 512;        // sin/cos table entries over one turn

// ---------------------------------------------------------------------------
// kernel value G = exp(-jkR)/R from the squared distance
// ---------------------------------------------------------------------------
// FP64: every operation on the FP64 pipe counts (it is 64 times slower than
// the FP32 one), so the seeds come from the FP32 and integer pipes:
// - 1/sqrt from the FP32 reciprocal square root of the mantissa (exponent
//   handled in integers), one Halley step (relative error 2^-23 -> 2^-66),
//   then one Newton correction of R;
// - sin and cos of pi x, x = n/256 + t: exact rounding of 256 x by the 1.5
//   2^52 trick, sin/cos(pi n/256) from a table, and the Taylor series of
//   sin/cos(pi t), |pi t| <= pi/512, to t^5 and t^4 (the first omitted terms
//   are 1e-17 and 7e-17), combined by the addition theorem.
// 24 FP64 instructions against about 55 for sqrt, 1/R and sincospi.  Valid
// for kR/pi below 2^42; beyond, kR itself has no correct digit.
__device__ __forceinline__ void green(double d2, double kpi, const double2* __restrict__ sc, double& gr, double& gi,
                                      double& r, double& rinv)
{
    const int hi = __double2hiint(d2), lo = __double2loint(d2);
    const int ex = hi >> 20;  // the sign bit is clear
    if ((unsigned)(ex - 1) < 0x7feu - 1u) {
        const int h = (ex - 1023) >> 1, par = (ex - 1023) & 1;
        const float m = __int_as_float(((127 + par) << 23) | ((hi & 0xfffff) << 3) | (int)((unsigned)lo >> 29));
        const int fb = __float_as_int(rsqrtf(m));  // 1/sqrt of [1, 4): (1/2, 1]
        double y = __hiloint2double((((fb >> 23) - 127 + 1023 - h) << 20) | ((fb & 0x7fffff) >> 3), fb << 29);
        const double e = fma(-(d2 * y), y, 1.0);
        y = fma(y * e, fma(0.375, e, 0.5), y);
        const double hy = __hiloint2double(__double2hiint(y) - (1 << 20), __double2loint(y));  // y / 2
        r = d2 * y;
        r = fma(fma(-r, r, d2), hy, r);
        rinv = y;
    } else {  // zero, subnormal, infinite or NaN
        r = sqrt(d2);
        rinv = 1.0 / r;
    }
    const double x = r * kpi;
    const double big = 6755399441055744.0;  // 1.5 * 2^52
    const double t = fma(x, 256.0, big);
    const double2 a = sc[__double2loint(t) & (SC_N - 1)];
    const double u = fma(t - big, -1.0 / 256.0, x) * 3.14159265358979323846;
    const double u2 = u * u;
    const double sd = u * fma(u2, fma(u2, 1.0 / 120.0, -1.0 / 6.0), 1.0);
    const double cd = u2 * fma(u2, 1.0 / 24.0, -0.5);  // cos - 1
    // rounding the sum a + (a cd -+ b sd) once keeps the table's accuracy
    const double s = a.x + fma(a.x, cd, a.y * sd);
    const double c = a.y + fma(a.y, cd, -(a.x * sd));
    gr = c * rinv;
    gi = -s * rinv;
}

// FP32: 1/sqrt from the hardware approximation, one correction each of R and
// 1/R (within about half an ulp of the IEEE square root and reciprocal, which
// cost twice the instructions: the four values of a far RWG pair nearly
// cancel, so G keeps every bit it can)
__device__ __forceinline__ void green(float d2, float kpi, const double2*, float& gr, float& gi, float& r,
                                      float& rinv)
{
    float y = rsqrtf(d2);
    r = d2 * y;
    r = fmaf(fmaf(-r, r, d2), 0.5f * y, r);
    rinv = fmaf(y, fmaf(-r, y, 1.0f), y);
    float s, c;
    sincos_pi_taylor(r * kpi, &s, &c);
    gr = c * rinv;
    gi = -s * rinv;
}

template <typename T> __device__ __forceinline__ T fma_t(T a, T b, T c);
template <> __device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
template <> __device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }

// weight x barycentric coordinates of the 7-point rule (gauss7), in T: a
// product or a conversion in FP64 would cost the FP32 fill more than the rest
// of its row
constexpr double BARY7[7][4] = {
    {0.333333333333333, 0.333333333333333, 1.0 - 0.333333333333333 - 0.333333333333333, 2 * 0.112500000000000},
    {0.797426985353087, 0.101286507323456, 1.0 - 0.797426985353087 - 0.101286507323456, 2 * 0.062969590272413},
    {0.101286507323456, 0.797426985353087, 1.0 - 0.101286507323456 - 0.797426985353087, 2 * 0.062969590272413},
    {0.101286507323456, 0.101286507323456, 1.0 - 0.101286507323456 - 0.101286507323456, 2 * 0.062969590272413},
    {0.470142064105115, 0.470142064105115, 1.0 - 0.470142064105115 - 0.470142064105115, 2 * 0.066197076394253},
    {0.470142064105115, 0.059715871789770, 1.0 - 0.470142064105115 - 0.059715871789770, 2 * 0.066197076394253},
    {0.059715871789770, 0.470142064105115, 1.0 - 0.059715871789770 - 0.470142064105115, 2 * 0.066197076394253}};

template <typename T>
struct Rule7 {
    T w[7][3];
};
template <typename T>
constexpr Rule7<T> rule7()
{
    Rule7<T> r{};
    for (int q = 0; q < 7; ++q)
        for (int j = 0; j < 3; ++j) r.w[q][j] = (T)(BARY7[q][3] * BARY7[q][j]);
    return r;
}
__device__ constexpr Rule7<float> R7F = rule7<float>();
__device__ constexpr Rule7<double> R7D = rule7<double>();
template <typename T>
__device__ __forceinline__ constexpr T w7(int q, int j)
{
    if constexpr (std::is_same<T, float>::value)
        return R7F.w[q][j];
    else
        return R7D.w[q][j];
}

// ---------------------------------------------------------------------------
// what the kernels share
// ---------------------------------------------------------------------------
struct Sphere {
    double x, y, z, w;  // centre, radius
};

struct PatchArgs {
    const int* rwg;               // [nb][PB] RWG ids, ascending, -1 beyond the patch's count
    const int* nt;                // [nb] triangles
    const int* tri;               // [nb][PS] triangle ids
    const unsigned char* slot;    // [nb][PS][4] slot of (triangle, corner), 255: none of the patch's
    const unsigned char* side;    // [nb][PS] slot of side a of RWG i, at 2 i + a
    const Sphere* sphere;        // [nb] centre and radius around the patch's RWG centres
    const double2* sc;            // [SC_N] sin, cos of 2 pi i / SC_N
    int nb;
};

// patch pair (bf, bs), bf <= bs, of a linear index; row bf holds nb - bf pairs
__device__ __forceinline__ void patch_pair(long long li, int nb, int* bf_out, int* bs_out)
{
    const float t = 2.0f * nb + 1.0f;
    int bf = (int)((t - sqrtf(fmaxf(t * t - 8.0f * (float)li, 0.0f))) * 0.5f);
    auto row0 = [&](int b) { return (long long)b * nb - (long long)b * (b - 1) / 2; };
    bf = min(max(bf, 0), nb - 1);
    while (bf > 0 && row0(bf) > li) --bf;
    while (bf + 1 < nb && row0(bf + 1) <= li) ++bf;
    *bf_out = bf;
    *bs_out = bf + (int)(li - row0(bf));
}

// The CTA's patch pair, found by one thread (the far test is FP64): x, y, and
// in z whether all RWG centres of one patch are farther than thr from all of
// the other's (thr < 0: not asked).
__device__ __forceinline__ int3 patch_pair_cta(const PatchArgs& pa, double thr, int3* shared)
{
    if (threadIdx.x == 0) {
        int3 r = make_int3(0, 0, 0);
        patch_pair(blockIdx.x, pa.nb, &r.x, &r.y);
        if (thr >= 0) {
            const Sphere a = pa.sphere[r.x], b = pa.sphere[r.y];
            const double dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
            r.z = sqrt(dx * dx + dy * dy + dz * dz) - (a.w + b.w) > thr * (1.0 + 1e-5);
        }
        *shared = r;
    }
    __syncthreads();
    return *shared;
}

template <typename T>
__device__ __forceinline__ bool rwg_far(const RwgPack<T>& F, const RwgPack<T>& S, const FillConst<T>& c)
{
    V3<T> fc = divr(v3(F.cen[0][0], F.cen[0][1], F.cen[0][2]) + v3(F.cen[1][0], F.cen[1][1], F.cen[1][2]), T(2));
    V3<T> sc = divr(v3(S.cen[0][0], S.cen[0][1], S.cen[0][2]) + v3(S.cen[1][0], S.cen[1][1], S.cen[1][2]), T(2));
    return norm(fc - sc) > c.thr_edm;
}

template <typename T, int NP> struct Staged {  // one patch's triangles in shared memory
    T pts[PS * 3 * NP];  // NP points a triangle, 3 NP apart (an odd stride: no bank conflicts)
    T v[PS * 9];     // corners
    int id[PS];
    unsigned char slot[PS * 4];
    unsigned char act[PS * 4];  // the active corners, then 255
};

template <typename T, int NP>
__device__ __forceinline__ void stage_patch(Staged<T, NP>& s, const PatchArgs& pa, int b, const T* __restrict__ pts,
                                            const T* __restrict__ verts, const int* __restrict__ tris)
{
    const int nt = pa.nt[b];
    const int* ids = pa.tri + (size_t)b * PS;
    for (int i = threadIdx.x; i < nt * 3 * NP; i += blockDim.x)
        s.pts[i] = pts[(size_t)ids[i / (3 * NP)] * (3 * NP) + i % (3 * NP)];
    for (int i = threadIdx.x; i < nt * 9; i += blockDim.x)
        s.v[i] = verts[3 * (size_t)tris[3 * (size_t)ids[i / 9] + (i % 9) / 3] + i % 3];
    for (int i = threadIdx.x; i < nt; i += blockDim.x) s.id[i] = ids[i];
    for (int i = threadIdx.x; i < nt * 4; i += blockDim.x) s.slot[i] = pa.slot[(size_t)b * PS * 4 + i];
    for (int i = threadIdx.x; i < nt; i += blockDim.x) {
        int k = 0;
        for (int a = 0; a < 3; ++a)
            if (pa.slot[((size_t)b * PS + i) * 4 + a] != 255) s.act[4 * i + k++] = (unsigned char)a;
        for (; k < 4; ++k) s.act[4 * i + k] = 255;
    }
}

// ---------------------------------------------------------------------------
// EFIE: 3 x 3 points (self pairs from the table) or 7 x 7 points (self and
// edge-adjacent pairs from the table; a triangle lists three neighbours, so on a
// mesh with more at an edge a pair may be in one direction's table only)
// ---------------------------------------------------------------------------
template <typename T, int NP>
__global__ void __launch_bounds__(256) k_fill_patch_efie(const RwgPack<T>* __restrict__ rw, FillConst<T> c,
                                                         const double2* __restrict__ tab,
                                                         const int* __restrict__ nbr, const T* __restrict__ pts,
                                                         const T* __restrict__ verts, const int* __restrict__ tris,
                                                         PatchArgs pa, Cx<T>* __restrict__ Z, size_t ldz)
{
    extern __shared__ double2 s_raw[];
    Cx<T>* val = reinterpret_cast<Cx<T>*>(s_raw);  // [PS][PS]
    __shared__ double2 sc[std::is_same<T, double>::value ? SC_N : 1];
    __shared__ Staged<T, NP> sf, ss;
    __shared__ int3 s_pair;
    const int3 pair = patch_pair_cta(pa, c.edm_mode != 2 ? (double)c.thr_edm : -1.0, &s_pair);
    const int bf = pair.x, bs = pair.y;
    const bool far = pair.z != 0;
    if (!far) {  // uniform over the CTA
        const int ntf = pa.nt[bf], nts = pa.nt[bs];
        stage_patch<T, NP>(sf, pa, bf, pts, verts, tris);
        stage_patch<T, NP>(ss, pa, bs, pts, verts, tris);
        if (std::is_same<T, double>::value)
            for (int i = threadIdx.x; i < SC_N; i += blockDim.x) sc[i] = pa.sc[i];
        __syncthreads();
        for (int pr = threadIdx.x; pr < ntf * nts; pr += blockDim.x) {
            const int tf = pr / nts, ts = pr - tf * nts;
            const int idf = sf.id[tf], ids = ss.id[ts];
            bool table = idf == ids;  // both ways: no regular value is read
            if (NP == 7 && !table) table = table_slot(nbr, idf, ids) >= 0 && table_slot(nbr, ids, idf) >= 0;
            T sr[3][3], si[3][3];  // S_ij
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) sr[i][j] = si[i][j] = T(0);
            if (!table) {
                T Q[NP][3];
#pragma unroll
                for (int q = 0; q < NP; ++q)
#pragma unroll
                    for (int x = 0; x < 3; ++x) Q[q][x] = ss.pts[ts * 3 * NP + 3 * q + x];
#pragma unroll(NP == 3 ? 3 : 1)
                for (int p = 0; p < NP; ++p) {
                    const T px = sf.pts[tf * 3 * NP + 3 * p], py = sf.pts[tf * 3 * NP + 3 * p + 1],
                            pz = sf.pts[tf * 3 * NP + 3 * p + 2];
                    T hr[3] = {T(0), T(0), T(0)}, hi[3] = {T(0), T(0), T(0)};
#pragma unroll
                    for (int q = 0; q < NP; ++q) {
                        const T dx = px - Q[q][0], dy = py - Q[q][1], dz = pz - Q[q][2];
                        T gr, gi, r, rinv;
                        green(dx * dx + dy * dy + dz * dz, c.kpi, sc, gr, gi, r, rinv);
                        if (NP == 3) {
                            hr[q] = gr;
                            hi[q] = gi;
                        } else {
#pragma unroll
                            for (int j = 0; j < 3; ++j) {
                                const T w = w7<T>(q, j);
                                hr[j] = fma_t(w, gr, hr[j]);
                                hi[j] = fma_t(w, gi, hi[j]);
                            }
                        }
                    }
                    if (NP == 3) {
                        // lambda_j(q) = 1/6, and 1/2 more for j = q; the p sum follows below
                        const T tr = (hr[0] + hr[1] + hr[2]) * T(1.0 / 6.0), ti = (hi[0] + hi[1] + hi[2]) * T(1.0 / 6.0);
#pragma unroll
                        for (int j = 0; j < 3; ++j) {
                            sr[p < 3 ? p : 0][j] = fma_t(T(0.5), hr[j], tr);
                            si[p < 3 ? p : 0][j] = fma_t(T(0.5), hi[j], ti);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            const T w = w7<T>(p, i);
#pragma unroll
                            for (int j = 0; j < 3; ++j) {
                                sr[i][j] = fma_t(w, hr[j], sr[i][j]);
                                si[i][j] = fma_t(w, hi[j], si[i][j]);
                            }
                        }
                    }
                }
                if (NP == 3) {
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        const T tr = (sr[0][j] + sr[1][j] + sr[2][j]) * T(1.0 / 6.0),
                                ti = (si[0][j] + si[1][j] + si[2][j]) * T(1.0 / 6.0);
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            sr[i][j] = fma_t(T(0.5), sr[i][j], tr);
                            si[i][j] = fma_t(T(0.5), si[i][j], ti);
                        }
                    }
                }
            }
            T er = T(0), ei = T(0);  // sum of all S_ij, times 1/k^2
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                er += sr[i][0] + sr[i][1] + sr[i][2];
                ei += si[i][0] + si[i][1] + si[i][2];
            }
            er *= c.inv_k2;
            ei *= c.inv_k2;
            // edge vectors E_i = v_(i+1) - v_i; D_ij = E_i . F_j / 4
            T D[3][3];
            {
                const T* a = sf.v + 9 * tf;
                const T* b = ss.v + 9 * ts;
                T F[3][3];
#pragma unroll
                for (int j = 0; j < 3; ++j)
#pragma unroll
                    for (int x = 0; x < 3; ++x) F[j][x] = T(0.25) * (b[3 * ((j + 1) % 3) + x] - b[3 * j + x]);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    T E[3];
#pragma unroll
                    for (int x = 0; x < 3; ++x) E[x] = a[3 * ((i + 1) % 3) + x] - a[3 * i + x];
#pragma unroll
                    for (int j = 0; j < 3; ++j) D[i][j] = E[0] * F[j][0] + E[1] * F[j][1] + E[2] * F[j][2];
                }
            }
            // corner a: v_(a+1) - v_a = E_a and v_(a+2) - v_a = -E_(a+2)
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const int la = sf.slot[4 * tf + a];
                const int a1 = (a + 1) % 3, a2 = (a + 2) % 3;
                if (la == 255) continue;
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const int lb = ss.slot[4 * ts + b];
                    const int b1 = (b + 1) % 3, b2 = (b + 2) % 3;
                    if (lb == 255) continue;
                    T zr = fma_t(sr[a1][b1], D[a][b], -er), zi = fma_t(si[a1][b1], D[a][b], -ei);
                    zr = fma_t(-sr[a1][b2], D[a][b2], zr);
                    zi = fma_t(-si[a1][b2], D[a][b2], zi);
                    zr = fma_t(-sr[a2][b1], D[a2][b], zr);
                    zi = fma_t(-si[a2][b1], D[a2][b], zi);
                    zr = fma_t(sr[a2][b2], D[a2][b2], zr);
                    zi = fma_t(si[a2][b2], D[a2][b2], zi);
                    val[la * PS + lb] = cx(zr, zi);
                }
            }
        }
        __syncthreads();
    }
    const unsigned char* sidef = pa.side + (size_t)bf * PS;
    const unsigned char* sides = pa.side + (size_t)bs * PS;
    const T w2 = NP == 3 ? c.ce : T(1);  // the 3-point weights; the 7-point ones are in S
    for (int e = threadIdx.x; e < PB * PB; e += blockDim.x) {
        const int lf = e / PB, ls = e - lf * PB;
        const int f = pa.rwg[(size_t)bf * PB + lf], s = pa.rwg[(size_t)bs * PB + ls];
        if (f < 0 || s < 0) continue;
        const RwgPack<T>& F = rw[f];
        const RwgPack<T>& S = rw[s];
        Cx<T> out = cx(T(0), T(0)), out_t = out;
        if (far || (c.edm_mode != 2 && rwg_far(F, S, c))) {
            if (c.edm_mode == 1) {
                out = edm_value(F, S, c);
                out_t = edm_value(S, F, c);
            }
        } else {
            T zr = T(0), zi = T(0), yr = T(0), yi = T(0);  // regular part of (f, s) and of (s, f)
            // table terms, of (f, s) and of (s, f), summed in FP64 and rounded once to T
            // (few entries have any: the sums start, and are rounded, where one does)
            double tr = 0, ti = 0, ur = 0, ui = 0;
            bool any = false;
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                const int la = sidef[2 * lf + a] * PS, tf = F.tri[a];
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    Cx<T> v = val[la + sides[2 * ls + b]];
                    if (a != b) v = cx(-v.re, -v.im);
                    const int ts = S.tri[b];
                    const double sgn = a == b ? 1.0 : -1.0;
                    if (NP == 3) {
                        zr += v.re;
                        zi += v.im;
                        if (tf != ts) continue;
                        const double2* p = tab + 3 * (9 * (size_t)tf + 3 * F.e[a] + S.e[b]);
                        const double2* q = tab + 3 * (9 * (size_t)ts + 3 * S.e[b] + F.e[a]);
                        const int var = a == 0 && b == 0 ? 0 : 1;
                        any = true;
                        tr += sgn * p[var].x + p[2].x;
                        ti += sgn * p[var].y + p[2].y;
                        ur += sgn * q[var].x + q[2].x;
                        ui += sgn * q[var].y + q[2].y;
                    } else {
                        const int sl = table_slot(nbr, tf, ts), st = table_slot(nbr, ts, tf);
                        if (sl >= 0) {
                            const double2 p = tab[36 * (size_t)tf + 9 * sl + 3 * F.e[a] + S.e[b]];
                            any = true;
                            tr += sgn * p.x;
                            ti += sgn * p.y;
                        } else {
                            zr += v.re;
                            zi += v.im;
                        }
                        if (st >= 0) {
                            const double2 q = tab[36 * (size_t)ts + 9 * st + 3 * S.e[b] + F.e[a]];
                            any = true;
                            ur += sgn * q.x;
                            ui += sgn * q.y;
                        } else {
                            yr += v.re;
                            yi += v.im;
                        }
                    }
                }
            }
            if (NP == 3) {
                yr = zr;
                yi = zi;
            }
            const T kz = (T)c.coef_efie * (F.len * S.len);
            Cx<T> t = cx(T(0), T(0)), u = t;
            if (any) {
                t = cx((T)tr, (T)ti);
                u = cx((T)ur, (T)ui);
            }
            out = cx(-kz * (w2 * zi + t.im), kz * (w2 * zr + t.re));
            out_t = cx(-kz * (w2 * yi + u.im), kz * (w2 * yr + u.re));
        }
        Z[(size_t)f * ldz + s] = out;
        if (bf != bs) Z[(size_t)s * ldz + f] = out_t;
    }
}

// ---------------------------------------------------------------------------
// CFIE, FP64, 3 x 3 points.  A (field corner, source corner) combination sums,
// with d = P - Q, rf = P - v_a, rs = Q - w_b and H = (1 + jkR) G / R^2,
//   EFIE  (rf.rs/4 - 1/k^2) G                       both ways
//   MFIE  [(rf.d)(nf.rs) - (rf.rs)(nf.d)] H         for Z(f, s)
//         [(rf.rs)(ns.d) - (rs.d)(ns.rf)] H         for Z(s, f)
// over the nine G and H held in registers.  nf.d depends on q alone and ns.d
// on p alone (the field points lie in one plane, the source points in another),
// so for a field corner and a source point q the p sums are
//   A = sum H (rf.d),  B = sum H rf,  C = sum G rf,  D = sum H ((ns.d) rf - (ns.rf) d)
// and each source corner adds rs.(jC - (nf.d) B) + (nf.rs) A and rs.(jC + D)
// (the combination constants folded into G and H).  A thread takes a triangle
// pair and walks the field triangle's active corners: the patch lists its
// triangles by their number of active corners, so a warp's lanes, which run
// over the source triangles, walk the same number.  (A thread per combination
// with every product formed per point pair, or lanes with different corners,
// ran 2750 FP64 instructions a triangle pair; this form about 1600.)
// ---------------------------------------------------------------------------
constexpr int CFIE_THREADS = 256;
__global__ void __launch_bounds__(CFIE_THREADS, 2) k_fill_patch_cfie(const RwgPack<double>* __restrict__ rw, FillConst<double> c,
                                                         const double2* __restrict__ tab,
                                                         const double* __restrict__ pts,
                                                         const double* __restrict__ nrm,
                                                         const double* __restrict__ verts,
                                                         const int* __restrict__ tris, PatchArgs pa,
                                                         Cx<double>* __restrict__ Z, size_t ldz)
{
    extern __shared__ double2 s_raw[];
    double2* val = s_raw;               // [PS][PS], Z(f, s)
    double2* val_t = s_raw + PS * PS;   // [PS][PS], Z(s, f)
    __shared__ double2 sc[SC_N];
    __shared__ Staged<double, 3> sf, ss;
    __shared__ int3 s_pair;
    const int3 pair = patch_pair_cta(pa, -1.0, &s_pair);
    const int bf = pair.x, bs = pair.y;
    const int ntf = pa.nt[bf], nts = pa.nt[bs];
    stage_patch<double, 3>(sf, pa, bf, pts, verts, tris);
    stage_patch<double, 3>(ss, pa, bs, pts, verts, tris);
    for (int i = threadIdx.x; i < SC_N; i += blockDim.x) sc[i] = pa.sc[i];
    __syncthreads();
    for (int pr = threadIdx.x; pr < ntf * nts; pr += blockDim.x) {
        const int tf = pr / nts, ts = pr - tf * nts;
        const int idf = sf.id[tf], ids = ss.id[ts];
        double gr[9], gi[9], hr[9], hi[9];  // ce/4 G, cm H
        const double* Pp = sf.pts + 9 * tf;
        const double* Qp = ss.pts + 9 * ts;
        double tr = 0.0, ti = 0.0;  // sum of G
        if (idf != ids) {
            const double ce4 = 0.25 * c.ce;
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const double dx = Pp[3 * p] - Qp[3 * q], dy = Pp[3 * p + 1] - Qp[3 * q + 1],
                                 dz = Pp[3 * p + 2] - Qp[3 * q + 2];
                    double r, rinv, g_r, g_i;
                    green(dx * dx + dy * dy + dz * dz, c.kpi, sc, g_r, g_i, r, rinv);
                    const double kr = r * c.k, r2 = c.cm * (rinv * rinv);
                    hr[3 * p + q] = (g_r - kr * g_i) * r2;
                    hi[3 * p + q] = (g_i + kr * g_r) * r2;
                    tr += gr[3 * p + q] = ce4 * g_r;
                    ti += gi[3 * p + q] = ce4 * g_i;
                }
        } else {
#pragma unroll
            for (int i = 0; i < 9; ++i) gr[i] = gi[i] = hr[i] = hi[i] = 0.0;
        }
        // j times -4/k^2 of the sum of ce/4 G
        tr *= -4.0 * c.inv_k2;
        ti *= -4.0 * c.inv_k2;
        const double nfx = nrm[3 * (size_t)idf], nfy = nrm[3 * (size_t)idf + 1], nfz = nrm[3 * (size_t)idf + 2];
        const double nsx = nrm[3 * (size_t)ids], nsy = nrm[3 * (size_t)ids + 1], nsz = nrm[3 * (size_t)ids + 2];
        double nsd[3];
#pragma unroll
        for (int p = 0; p < 3; ++p)
            nsd[p] = nsx * (Pp[3 * p] - Qp[0]) + nsy * (Pp[3 * p + 1] - Qp[1]) + nsz * (Pp[3 * p + 2] - Qp[2]);
#pragma unroll 1
        for (int ia = 0; ia < 3; ++ia) {
            const int a = sf.act[4 * tf + ia];
            if (a == 255) break;
            double rf[3][3], nsrf[3];
            const double* va = sf.v + 9 * tf + 3 * a;
#pragma unroll
            for (int p = 0; p < 3; ++p) {
#pragma unroll
                for (int x = 0; x < 3; ++x) rf[p][x] = Pp[3 * p + x] - va[x];
                nsrf[p] = nsx * rf[p][0] + nsy * rf[p][1] + nsz * rf[p][2];
            }
            double vr[3], vi[3], wr[3], wi[3];  // Z(f, s) and Z(s, f) by source corner
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                vr[b] = wr[b] = -ti;
                vi[b] = wi[b] = tr;
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const double qx = Qp[3 * q], qy = Qp[3 * q + 1], qz = Qp[3 * q + 2];
                double Ar = 0, Ai = 0, B[6] = {0, 0, 0, 0, 0, 0}, C[6] = {0, 0, 0, 0, 0, 0}, D[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    const double h_r = hr[3 * p + q], h_i = hi[3 * p + q], g_r = gr[3 * p + q], g_i = gi[3 * p + q];
                    const double d[3] = {Pp[3 * p] - qx, Pp[3 * p + 1] - qy, Pp[3 * p + 2] - qz};
                    const double rfd = rf[p][0] * d[0] + rf[p][1] * d[1] + rf[p][2] * d[2];
                    Ar = fma(h_r, rfd, Ar);
                    Ai = fma(h_i, rfd, Ai);
#pragma unroll
                    for (int x = 0; x < 3; ++x) {
                        const double u = fma(nsd[p], rf[p][x], -(nsrf[p] * d[x]));
                        B[x] = fma(h_r, rf[p][x], B[x]);
                        B[3 + x] = fma(h_i, rf[p][x], B[3 + x]);
                        C[x] = fma(g_r, rf[p][x], C[x]);
                        C[3 + x] = fma(g_i, rf[p][x], C[3 + x]);
                        D[x] = fma(h_r, u, D[x]);
                        D[3 + x] = fma(h_i, u, D[3 + x]);
                    }
                }
                const double nfd = nfx * (Pp[0] - qx) + nfy * (Pp[1] - qy) + nfz * (Pp[2] - qz);
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    B[x] = fma(-nfd, B[x], -C[3 + x]);
                    B[3 + x] = fma(-nfd, B[3 + x], C[x]);
                    D[x] -= C[3 + x];
                    D[3 + x] += C[x];
                }
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const double* wb = ss.v + 9 * ts + 3 * b;
                    const double rx = qx - wb[0], ry = qy - wb[1], rz = qz - wb[2];
                    const double nfrs = nfx * rx + nfy * ry + nfz * rz;
                    vr[b] = fma(nfrs, Ar, vr[b] + (rx * B[0] + ry * B[1] + rz * B[2]));
                    vi[b] = fma(nfrs, Ai, vi[b] + (rx * B[3] + ry * B[4] + rz * B[5]));
                    wr[b] += rx * D[0] + ry * D[1] + rz * D[2];
                    wi[b] += rx * D[3] + ry * D[4] + rz * D[5];
                }
            }
            const int la = sf.slot[4 * tf + a];
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const int lb = ss.slot[4 * ts + b];
                if (lb == 255) continue;
                val[la * PS + lb] = make_double2(vr[b], vi[b]);
                val_t[la * PS + lb] = make_double2(wr[b], wi[b]);
            }
        }
    }
    __syncthreads();
    const unsigned char* sidef = pa.side + (size_t)bf * PS;
    const unsigned char* sides = pa.side + (size_t)bs * PS;
    for (int e = threadIdx.x; e < PB * PB; e += blockDim.x) {
        const int lf = e / PB, ls = e - lf * PB;
        const int f = pa.rwg[(size_t)bf * PB + lf], s = pa.rwg[(size_t)bs * PB + ls];
        if (f < 0 || s < 0) continue;
        const RwgPack<double>& F = rw[f];
        const RwgPack<double>& S = rw[s];
        double zr = 0, zi = 0, tr = 0, ti = 0;
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const int la = sidef[2 * lf + a] * PS;
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                double2 v = val[la + sides[2 * ls + b]], t = val_t[la + sides[2 * ls + b]];
                if (F.tri[a] == S.tri[b]) {
                    v = tab[9 * (size_t)F.tri[a] + 3 * F.e[a] + S.e[b]];
                    t = tab[9 * (size_t)S.tri[b] + 3 * S.e[b] + F.e[a]];
                }
                zr += a == b ? v.x : -v.x;
                zi += a == b ? v.y : -v.y;
                tr += a == b ? t.x : -t.x;
                ti += a == b ? t.y : -t.y;
            }
        }
        const double l = F.len * S.len;
        Z[(size_t)f * ldz + s] = cx(zr * l, zi * l);
        if (bf != bs) Z[(size_t)s * ldz + f] = cx(tr * l, ti * l);
    }
}

__global__ void k_sincos_table(double2* __restrict__ sc)
{
    const int i = threadIdx.x;
    double s, c;
    sincospi((double)i / (SC_N / 2), &s, &c);
    sc[i] = make_double2(s, c);
}

// doubles in an order that integers keep (so that no coordinate, NaN included, breaks the sort)
uint64_t order_key(double x)
{
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return (u >> 63) ? ~u : u | (1ull << 63);
}

// leaves of PB consecutive entries of `id` that are close together: bisection
// along the longest extent of the edge midpoints
void bisect(std::vector<int>& id, const std::vector<double>& mid, int lo, int hi)
{
    const int blocks = (hi - lo + PB - 1) / PB;
    if (blocks <= 1) {
        std::sort(id.begin() + lo, id.begin() + hi);
        return;
    }
    int axis = 0;
    double best = -1.0;
    for (int x = 0; x < 3; ++x) {
        double mn = mid[3 * (size_t)id[lo] + x], mx = mn;
        for (int i = lo; i < hi; ++i) {
            mn = std::min(mn, mid[3 * (size_t)id[i] + x]);
            mx = std::max(mx, mid[3 * (size_t)id[i] + x]);
        }
        if (mx - mn > best) {
            best = mx - mn;
            axis = x;
        }
    }
    const int cut = lo + (blocks / 2) * PB;
    std::nth_element(id.begin() + lo, id.begin() + cut, id.begin() + hi, [&](int a, int b) {
        const uint64_t ka = order_key(mid[3 * (size_t)a + axis]), kb = order_key(mid[3 * (size_t)b + axis]);
        return ka != kb ? ka < kb : a < b;
    });
    bisect(id, mid, lo, cut);
    bisect(id, mid, cut, hi);
}

}  // namespace

// Per-geometry plan of the patch fill (host, once).  g->patch_ok is false for
// an RWG table whose free vertices are not corners of their triangles: its
// fills keep a thread per entry.
static emfa_status_t patch_plan(Ctx* c, Geom* g, cudaStream_t st)
{
    if (g->patch_ready) return EMFA_OK;
    const int n = g->n, nb = (n + PB - 1) / PB;
    std::vector<int> id(n), corner(2 * (size_t)n);
    std::vector<double> mid(3 * (size_t)n), cen(3 * (size_t)n);
    g->patch_ok = true;
    for (int u = 0; u < n; ++u) {
        const int* r = &g->rwg[6 * (size_t)u];
        id[u] = u;
        for (int x = 0; x < 3; ++x) {
            mid[3 * (size_t)u + x] = 0.5 * (g->verts[3 * (size_t)r[0] + x] + g->verts[3 * (size_t)r[1] + x]);
            double s = 0.0;  // the RWG's centre: mean of its triangles' centroids
            for (int a = 0; a < 2; ++a)
                for (int j = 0; j < 3; ++j) s += g->verts[3 * (size_t)g->tris[3 * (size_t)r[4 + a] + j] + x];
            cen[3 * (size_t)u + x] = s / 6.0;
        }
        for (int a = 0; a < 2; ++a) {
            int e = -1;
            for (int j = 0; j < 3; ++j)
                if (g->tris[3 * (size_t)r[4 + a] + j] == r[2 + a]) e = j;  // the last match, as k_pack_rwg
            if (e < 0) g->patch_ok = false;
            corner[2 * (size_t)u + a] = e;
        }
    }
    if (!g->patch_ok) {
        g->patch_ready = true;
        return EMFA_OK;
    }
    bisect(id, mid, 0, n);
    std::vector<int> rwg((size_t)nb * PB, -1), nt(nb, 0), tri((size_t)nb * PS, 0);
    std::vector<unsigned char> slot((size_t)nb * PS * 4, 255), side((size_t)nb * PS, 0);
    std::vector<Sphere> sph(nb);
    std::vector<int> seen(g->nt, -1);  // patch that listed the triangle last
    std::vector<int> at(g->nt, 0);
    std::vector<int> sides_of(g->nt, 0);
    for (int b = 0; b < nb; ++b) {
        const int lo = b * PB, cnt = std::min(PB, n - lo);
        int slots = 0;
        double m[3] = {0, 0, 0}, rad = 0.0;
        // the patch's triangles, those with the most of its RWG sides first
        int* list = &tri[(size_t)b * PS];
        for (int i = 0; i < cnt; ++i)
            for (int a = 0; a < 2; ++a) {
                const int t = g->rwg[6 * (size_t)id[lo + i] + 4 + a];
                if (seen[t] != b) {
                    seen[t] = b;
                    sides_of[t] = 0;
                    list[nt[b]++] = t;
                }
                sides_of[t] += 1;
            }
        std::stable_sort(list, list + nt[b], [&](int x, int y) { return sides_of[x] > sides_of[y]; });
        for (int i = 0; i < nt[b]; ++i) at[list[i]] = i;
        for (int i = 0; i < cnt; ++i) {
            const int u = id[lo + i];
            rwg[(size_t)b * PB + i] = u;
            for (int x = 0; x < 3; ++x) m[x] += cen[3 * (size_t)u + x] / cnt;
            for (int a = 0; a < 2; ++a) {
                const int t = g->rwg[6 * (size_t)u + 4 + a];
                unsigned char& sl = slot[((size_t)b * PS + at[t]) * 4 + corner[2 * (size_t)u + a]];
                if (sl == 255) sl = (unsigned char)slots++;
                side[(size_t)b * PS + 2 * i + a] = sl;
            }
        }
        for (int i = 0; i < cnt; ++i) {
            const double* p = &cen[3 * (size_t)id[lo + i]];
            const double d = std::sqrt((p[0] - m[0]) * (p[0] - m[0]) + (p[1] - m[1]) * (p[1] - m[1]) +
                                       (p[2] - m[2]) * (p[2] - m[2]));
            rad = std::max(rad, d);
        }
        sph[b] = Sphere{m[0], m[1], m[2], rad};
    }
    struct Part {
        DevView* view;
        const void* src;
        size_t bytes;
    } parts[] = {{&g->patch_rwg, rwg.data(), sizeof(int) * rwg.size()},
                 {&g->patch_nt, nt.data(), sizeof(int) * nt.size()},
                 {&g->patch_tri, tri.data(), sizeof(int) * tri.size()},
                 {&g->patch_slot, slot.data(), slot.size()},
                 {&g->patch_side, side.data(), side.size()},
                 {&g->patch_sphere, sph.data(), sizeof(Sphere) * sph.size()}};
    size_t total = sizeof(double2) * SC_N;
    for (const Part& p : parts) total += (p.bytes + 255) & ~(size_t)255;
    std::vector<char> host(total, 0);  // one copy
    EMFA_TRY(g->patch_block.alloc(c, total));
    size_t off = sizeof(double2) * SC_N;
    g->patch_sc = DevView{g->patch_block.ptr, off};
    for (const Part& p : parts) {
        std::memcpy(host.data() + off, p.src, p.bytes);
        *p.view = DevView{(char*)g->patch_block.ptr + off, p.bytes};
        off += (p.bytes + 255) & ~(size_t)255;
    }
    EMFA_CUDA(c, cudaMemcpyAsync(g->patch_block.ptr, host.data(), total, cudaMemcpyHostToDevice, st));
    k_sincos_table<<<1, SC_N, 0, st>>>(dptr<double2>(g->patch_sc));
    c->kernel_launches += 1;
    EMFA_CUDA(c, cudaGetLastError());
    EMFA_CUDA(c, cudaStreamSynchronize(st));  // host staging goes out of scope; other streams may use the plan
    g->patch_nb = nb;
    g->patch_ready = true;
    return EMFA_OK;
}

template <typename T>
emfa_status_t launch_fill_patch(Ctx* c, Geom* g, const GeomDev<T>& d, const emfa_fill_params_t* p,
                                const FillConst<T>& fc, const double2* tab, void* Z, size_t ldz, cudaStream_t st,
                                bool* done)
{
    const emfa_status_t plan = patch_plan(c, g, st);
    *done = plan == EMFA_OK && g->patch_ok;
    if (plan == EMFA_ERR_OOM) cudaGetLastError();  // no room for the plan: a thread per entry needs none
    else EMFA_TRY(plan);
    if (!*done) return EMFA_OK;
    const int nb = g->patch_nb;
    const PatchArgs pa{dptr<int>(g->patch_rwg),           dptr<int>(g->patch_nt),     dptr<int>(g->patch_tri),
                       dptr<unsigned char>(g->patch_slot), dptr<unsigned char>(g->patch_side),
                       dptr<Sphere>(g->patch_sphere),     dptr<double2>(g->patch_sc), nb};
    const unsigned grd = (unsigned)((long long)nb * (nb + 1) / 2);
    const size_t sm = sizeof(Cx<T>) * PS * PS;
    const bool cfg = p->discretisation == EMFA_DISC_CONFIG;
    TimedLaunch tl(c, KT_FILL_Z, st, (double)g->n * g->n);
    if (cfg) {
        EMFA_TRY(ensure_smem(c, k_fill_patch_efie<T, 7>, sm));
        k_fill_patch_efie<T, 7><<<grd, 256, sm, st>>>(dptr<RwgPack<T>>(d.rwg), fc, tab, dptr<int>(g->nbr),
                                                      dptr<T>(d.tri_q7), dptr<T>(d.verts), dptr<int>(d.tris), pa,
                                                      reinterpret_cast<Cx<T>*>(Z), ldz);
    } else if constexpr (std::is_same<T, double>::value) {
        if (p->kind == EMFA_CFIE) {
            EMFA_TRY(ensure_smem(c, k_fill_patch_cfie, 2 * sm));
            k_fill_patch_cfie<<<grd, CFIE_THREADS, 2 * sm, st>>>(dptr<RwgPack<double>>(d.rwg), fc, tab, dptr<double>(d.tri_q3),
                                                        dptr<double>(d.tri_n), dptr<double>(d.verts),
                                                        dptr<int>(d.tris), pa, reinterpret_cast<Cx<double>*>(Z), ldz);
        } else {
            EMFA_TRY(ensure_smem(c, k_fill_patch_efie<double, 3>, sm));
            k_fill_patch_efie<double, 3><<<grd, 256, sm, st>>>(
                dptr<RwgPack<double>>(d.rwg), fc, tab, nullptr, dptr<double>(d.tri_q3), dptr<double>(d.verts),
                dptr<int>(d.tris), pa, reinterpret_cast<Cx<double>*>(Z), ldz);
        }
    } else {
        *done = false;  // the FP32 3 x 3-point fills have their own tiles
        return EMFA_OK;
    }
    c->kernel_launches += 1;
    EMFA_CUDA(c, cudaGetLastError());
    return EMFA_OK;
}

template emfa_status_t launch_fill_patch<float>(Ctx*, Geom*, const GeomDev<float>&, const emfa_fill_params_t*,
                                                const FillConst<float>&, const double2*, void*, size_t, cudaStream_t,
                                                bool*);
template emfa_status_t launch_fill_patch<double>(Ctx*, Geom*, const GeomDev<double>&, const emfa_fill_params_t*,
                                                 const FillConst<double>&, const double2*, void*, size_t,
                                                 cudaStream_t, bool*);

}  // namespace emfa
