// Multilevel fast multipole CFIE operator (EMSolver/MLFMA.cpp).
//
// Host (float arithmetic, the reference's own rules, so box order, multipole
// counts, sample points and stencils are the reference's):
//   bounding cube and level count   MLFMA_Boundary::init (MLFMA_Boundary.cpp:15-35)
//   octree, box order of unknowns   buildBox / buildFirstLevel / buildCurLevel (MLFMA.cpp:688-805)
//   near / far lists                setBoxParameter (MLFMA.cpp:807-866)
//   multipoles, Gauss-Legendre      getMultipoleNumber / levelRootsAndWeights (MLFMA.cpp:877-915)
//   3x3 Lagrange stencils           calculateInterpolationMtr / lagrangeIPWeights (MLFMA.cpp:917-1002)
// Device (FP32 patterns; level patterns in 3 Cartesian components as in the
// reference, the transverse radiation / receive patterns in 2, theta and phi
// of each sample's own basis):
//   k_trans_table  translation operators (parallelLevelTrans, MLFMA.cpp:1191-1222) in FP64, once
//                  per distinct box offset (at most 7^3 per level) instead of per box pair
//   k_radrec       radiation / receive patterns (MLFMA.cpp:1244-1292,1393-1422)
//   k_near_fill    near-field CFIE blocks per (field box, near box) (MLFMA.cpp:1004-1131)
//   per mat-vec (MLFMA.cpp:454-686), up to 8 right-hand sides per pass, level patterns planar:
//     k_agg_finest    finest-level aggregation
//     k_upward        interpolation + shift, child -> parent: the 3 x 3 Lagrange stencil as two
//                     1-D passes (theta into shared memory, then phi)
//     k_translate     translation of every level at once, by sibling groups: each source pattern read
//                     once for the up to eight boxes of a parent
//     k_downward      anterpolation from the parent (transposed stencil as two 1-D passes), by chunks
//                     of phi rows, added to the translated pattern
//     k_finish        the finest level: anterpolation, disaggregation and near-field product (or
//                     k_downward and k_disagg_near, for boxes too large for shared memory)
#include "emfa_internal.cuh"
#include "emfa_math.cuh"
#include "fill_entry.cuh"
#include "gemm.cuh"

#include <algorithm>
#include <cmath>
#include <complex>

namespace emfa {

struct C3f {
    float2 x, y, z;
};
// a transverse pattern in the (theta, phi) basis of its sample direction
struct C2f {
    float2 t, p;
};

__device__ __forceinline__ float2 cmulf(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ float2 caddf(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 cscalef(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
__device__ __forceinline__ C3f c3zero() { return C3f{make_float2(0, 0), make_float2(0, 0), make_float2(0, 0)}; }
__device__ __forceinline__ void c3fma(C3f& acc, float2 s, const C3f& v)
{
    acc.x = caddf(acc.x, cmulf(s, v.x));
    acc.y = caddf(acc.y, cmulf(s, v.y));
    acc.z = caddf(acc.z, cmulf(s, v.z));
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace mh {

const float PI = 3.14159265358979323846f;

struct Box {
    float c[3];
    int parent = -1;
    int oct = 0;      // child index (x*2+y)*2+z within the parent
    int ix[3] = {0, 0, 0};          // place on the level's grid
    int offset = 0, count = 0;      // its unknowns in box order
    int child0 = 0, nchild = 0;     // its children on the next level
};

// a level's boxes and their near lists (CSR)
struct Level {
    std::vector<Box> b;
    std::vector<int> nptr{0}, near;
};

// Legendre value / derivative recurrence of GaussLegendre::Evaluation, for
// GL roots side by side (one recurrence is a chain of divisions)
constexpr int GL = 8;
static void gl_eval(const float* x, int n, float* v, float* d)
{
    float vsub1[GL], vsub2[GL];
    for (int r = 0; r < GL; ++r) {
        vsub1[r] = x[r];
        vsub2[r] = 1;
        v[r] = 1;
        d[r] = 0;
    }
    for (int i = 2; i <= n; ++i)
        for (int r = 0; r < GL; ++r) {
            v[r] = ((2 * i - 1) * x[r] * vsub1[r] - (i - 1) * vsub2[r]) / i;
            if (i == n) d[r] = i * (1 / (x[r] * x[r] - 1)) * (x[r] * v[r] - vsub1[r]);
            vsub2[r] = vsub1[r];
            vsub1[r] = v[r];
        }
}

// GaussLegendre::set (EMComponent/Quadrature.cpp:93-112): Newton from the
// Chebyshev-like guess, float arithmetic, roots ascending
static void gauss_legendre(int n, std::vector<float>& r, std::vector<float>& w)
{
    r.assign(n, 0);
    w.assign(n, 0);
    for (int i0 = 0; i0 < n; i0 += GL) {
        float x[GL], v[GL], d[GL], xn[GL], vn[GL], dn[GL];
        bool live[GL];
        for (int q = 0; q < GL; ++q) {
            const int i = std::min(i0 + q, n - 1);
            x[q] = (float)std::cos((double)(PI * (i + 0.75f) / (n + 0.5f)));
            live[q] = true;
        }
        gl_eval(x, n, v, d);
        int guard = 0;
        for (bool any = true; any;) {
            for (int q = 0; q < GL; ++q) xn[q] = x[q] - v[q] / d[q];
            gl_eval(xn, n, vn, dn);
            const bool stop = ++guard >= 1000;
            any = false;
            for (int q = 0; q < GL; ++q)
                if (live[q]) {  // a root that has converged keeps its last step
                    live[q] = std::fabs((double)(v[q] / d[q])) > 2e-7f && !stop;
                    any |= live[q];
                    x[q] = xn[q];
                    v[q] = vn[q];
                    d[q] = dn[q];
                }
        }
        for (int q = 0; q < GL && i0 + q < n; ++q) {
            r[n - 1 - i0 - q] = x[q];
            w[n - 1 - i0 - q] = 2 / ((1 - x[q] * x[q]) * d[q] * d[q]);
        }
    }
}

// lagrangeIPWeights (MLFMA.cpp:962-1002): 3-point stencils of the samples
// `cur` (parent level) in the samples `nxt` (child level), clamped at the ends
static void lagrange(const std::vector<float>& nxt, const std::vector<float>& cur, std::vector<int>& loc,
                     std::vector<float>& el)
{
    size_t cols = cur.size();
    loc.assign(3 * cols, 0);
    el.assign(3 * cols, 0);
    size_t nlast = nxt.size() - 1;
    size_t nid = 2;
    float low = nxt[1], high = nxt[nlast - 1];
    for (size_t cid = 0; cid < cols; ++cid) {
        const float xx = cur[cid];
        size_t p1, p2, p3;
        if (xx < low) {
            p1 = 0; p2 = 1; p3 = 2;
        } else if (xx > high) {
            p1 = nlast - 2; p2 = nlast - 1; p3 = nlast;
        } else {
            nid += nxt[nid] < xx ? 1 : 0;
            size_t off = (nxt[nid] - xx < xx - nxt[nid - 1]) ? 1 : 0;
            p1 = nid + off - 2; p2 = nid + off - 1; p3 = nid + off;
        }
        loc[3 * cid] = (int)p1; loc[3 * cid + 1] = (int)p2; loc[3 * cid + 2] = (int)p3;
        const float x0 = nxt[p1], x1 = nxt[p2], x2 = nxt[p3];
        el[3 * cid] = (xx - x1) * (xx - x2) / ((x0 - x1) * (x0 - x2));
        el[3 * cid + 1] = (xx - x0) * (xx - x2) / ((x1 - x0) * (x1 - x2));
        el[3 * cid + 2] = (xx - x0) * (xx - x1) / ((x2 - x0) * (x2 - x1));
    }
}

static float fnorm3(const float* a, const float* b)
{
    float x = a[0] - b[0], y = a[1] - b[1], z = a[2] - b[2];
    return std::sqrt(x * x + y * y + z * z);
}

}  // namespace mh

// per-level device data
struct MLevel {
    int nbox = 0, L = 0, K = 0;
    float len = 0;
    DevView parent, oct;                 // parent index and octant per box (int)
    DevView child_ptr, child_idx;        // CSR children (int)
    // translation by sibling groups: the children of one box of the level
    // above, at most four a group (TransGroup), and their source boxes, the
    // children of the boxes near the parent
    DevView grp, grp_src;
    int ngrp = 0;
    DevView trans;                       // float2 [343][K]
    DevView up, down;                    // planar float2 [right-hand side][nbox][3][K]
    // interpolation to this level from the level below, separable: 3-point
    // Lagrange stencils in theta (per theta index of this level: child theta,
    // weight) and in phi (per phi index: child phi row, weight)
    DevView ip_tl, ip_te, ip_pl, ip_pe;
    // anterpolation from the level above, as two transposed 1-D Lagrange
    // stencils: theta (CSR over this level's theta index: parent theta, weight)
    // and phi (CSR over this level's phi index: parent phi, weight)
    DevView th_ptr, th_src, th_w, ph_ptr, ph_src, ph_w;
    size_t down_smem = 0;               // shared bytes per CTA (theta-pass rows, and the shifted rows where
    bool down_staged = true;            //   they fit beside them)
    DevView down_win;                    // int2 per chunk: parent phi rows its phi stencils read
    DevView up_phase;                    // float2 [8][K]: exp(-j k k.(parent - child)) for the level below
    int up_rows = 0;                    // interpolation from the level below: phi rows per CTA,
    size_t up_child_bytes = 0;          //   shared bytes of one child's theta pass,
    int up_batch = 0;                   //   children per shared-memory pass,
    DevView up_win;                      //   int2 per chunk: the child phi rows it reads
};

}  // namespace emfa

struct emfa_mlfma {
    emfa::Ctx* ctx = nullptr;
    emfa::Geom* geom = nullptr;
    emfa_mlfma_params_t p{};
    int levels = 0;   // finest level number L (levels 2..L carry patterns)
    int n = 0;
    float k = 0;
    std::vector<int> perm;         // box order -> RWG index
    std::vector<int> level_boxes;  // boxes per level 0..L
    std::vector<int> poles;        // multipoles per level 2..L
    std::vector<emfa::MLevel> lv;  // index level - 2
    int rcap = 1;                  // right-hand sides the level patterns hold (one apply chunk)
    emfa::DevBuf fine_tables, level_tables;  // the lists and tables below and of every level
    emfa::DevBuf trans_tables, patterns;     // translation operators, up and down patterns of every level
    emfa::DevView perm_d, box_of;  // int [n]
    emfa::DevBuf rad, rec;         // C2f [n][Kf]: theta, phi components in each sample's basis
    emfa::DevView tp;               // float [6][Kf]: theta_hat, phi_hat of the finest samples
    emfa::DevView coeff;            // float [Kf]
    emfa::DevView box_off, box_cnt; // finest boxes: first unknown, count
    emfa::DevView near_ptr, near_box, near_col, row_cols;  // CSR near lists, column base per slot, C_b per box
    emfa::DevView row_base;         // size_t per finest box: first value of the box's rows
    emfa::DevBuf near_val;         // float2 [nnz]
    emfa::DevView near_cbase;      // per finest box: first entry of
    emfa::DevBuf near_cidx;        //   the column unknowns of its near rows
    size_t nnz = 0;
    emfa::DevView trans_work;       // TransWork per CTA of the translation
    int trans_ctas = 0;
    bool wide = false;             // a level's pattern elements need more than 32 bits (k_translate)
    int max_cols = 0;              // near columns of a box, most
    emfa::DevBuf tmp_in, tmp_out;  // complex64 scratch for residuals
    // SAI preconditioner P (CSR over box-order rows), built when p.precond
    bool precond = false;
    size_t sai_nnz = 0;
    std::vector<int> sai_rptr, sai_rows, sai_cptr, sai_cols, sai_own;  // host copies of the lists
    emfa::DevBuf csr_ptr, csr_col, csr_val;  // int [n+1], int [nnz], float2 [nnz]
    emfa::DevBuf pre_tmp, pre_b;             // complex64 scratch: Z x, P b
};

namespace emfa {

// ---------------------------------------------------------------------------
// device kernels
// ---------------------------------------------------------------------------
// radiation / receive patterns of every unknown (box order) at every finest
// sample.  Both are transverse (k . rad = 0: rad is projected off k; the
// receive pattern is alpha conj(rad) plus k x (...)), so they are stored as
// their theta and phi components in the sample's own basis (tp: theta_hat,
// phi_hat per sample), 16 bytes a sample instead of the 24 of x, y, z.
__global__ void k_radrec(const RwgPack<float>* __restrict__ rw, const int* __restrict__ perm,
                         const int* __restrict__ box_of, const float* __restrict__ centers,
                         const float* __restrict__ kdir, const float* __restrict__ tp, int n, int K, float k,
                         float alpha, C2f* __restrict__ rad, C2f* __restrict__ rec)
{
    size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (size_t)n * K) return;
    const int u = (int)(id / K), kk = (int)(id % K);
    const RwgPack<float>& R = rw[perm[u]];
    const float* c = centers + 3 * box_of[u];
    const V3<float> kh = v3(kdir[3 * kk], kdir[3 * kk + 1], kdir[3 * kk + 2]);
    const V3<float> cen = v3(c[0], c[1], c[2]);
    const float w3 = 1.0f / 3.0f;
    float2 ra[3] = {{0, 0}, {0, 0}, {0, 0}}, rh[3] = {{0, 0}, {0, 0}, {0, 0}};
    for (int s = 0; s < 2; ++s) {
        const float sg = s == 0 ? 1.0f : -1.0f;
        const V3<float> fv = v3(R.v[s][0], R.v[s][1], R.v[s][2]);
        const V3<float> nn = v3(R.n[s][0], R.n[s][1], R.n[s][2]);
        for (int q = 0; q < 3; ++q) {
            const V3<float> g = v3(R.q3[s][q][0], R.q3[s][q][1], R.q3[s][q][2]);
            const V3<float> rho = (g - fv) * (sg * w3);
            const V3<float> nr = cross(nn, rho);
            float sn, cs;
            sincos_pi(k * dot(kh, g - cen) / mh::PI, &sn, &cs);
            // rad: rho e^{+j phase}; half receive: (n x rho) e^{-j phase}
            ra[0] = caddf(ra[0], make_float2(rho.x * cs, rho.x * sn));
            ra[1] = caddf(ra[1], make_float2(rho.y * cs, rho.y * sn));
            ra[2] = caddf(ra[2], make_float2(rho.z * cs, rho.z * sn));
            rh[0] = caddf(rh[0], make_float2(nr.x * cs, -nr.x * sn));
            rh[1] = caddf(rh[1], make_float2(nr.y * cs, -nr.y * sn));
            rh[2] = caddf(rh[2], make_float2(nr.z * cs, -nr.z * sn));
        }
    }
    // rad - (k . rad) k
    float2 kd = make_float2(kh.x * ra[0].x + kh.y * ra[1].x + kh.z * ra[2].x, kh.x * ra[0].y + kh.y * ra[1].y + kh.z * ra[2].y);
    ra[0] = make_float2(ra[0].x - kd.x * kh.x, ra[0].y - kd.y * kh.x);
    ra[1] = make_float2(ra[1].x - kd.x * kh.y, ra[1].y - kd.y * kh.y);
    ra[2] = make_float2(ra[2].x - kd.x * kh.z, ra[2].y - kd.y * kh.z);
    // k x half-receive
    float2 hx = make_float2(kh.y * rh[2].x - kh.z * rh[1].x, kh.y * rh[2].y - kh.z * rh[1].y);
    float2 hy = make_float2(kh.z * rh[0].x - kh.x * rh[2].x, kh.z * rh[0].y - kh.x * rh[2].y);
    float2 hz = make_float2(kh.x * rh[1].x - kh.y * rh[0].x, kh.x * rh[1].y - kh.y * rh[0].y);
    const float h = R.len / 2;
    const float b = 1.0f - alpha;
    const float e[6] = {tp[kk],         tp[K + kk],     tp[2 * K + kk],
                        tp[3 * K + kk], tp[4 * K + kk], tp[5 * K + kk]};  // theta_hat, phi_hat
    C3f o, q;
    o.x = cscalef(ra[0], h);
    o.y = cscalef(ra[1], h);
    o.z = cscalef(ra[2], h);
    q.x = make_float2(h * (alpha * ra[0].x + b * hx.x), h * (-alpha * ra[0].y + b * hx.y));
    q.y = make_float2(h * (alpha * ra[1].x + b * hy.x), h * (-alpha * ra[1].y + b * hy.y));
    q.z = make_float2(h * (alpha * ra[2].x + b * hz.x), h * (-alpha * ra[2].y + b * hz.y));
    auto proj = [](const C3f& v, const float* u) {
        return make_float2(u[0] * v.x.x + u[1] * v.y.x + u[2] * v.z.x, u[0] * v.x.y + u[1] * v.y.y + u[2] * v.z.y);
    };
    rad[id] = C2f{proj(o, e), proj(o, e + 3)};
    rec[id] = C2f{proj(q, e), proj(q, e + 3)};
}

// near-field blocks, row-major per field box over the concatenated near-box
// columns: a warp per field unknown, lanes over the columns (near_cidx), so that
// the row is stored coalesced and the lanes share the work whatever the boxes'
// sizes.  Bound by FP32 issue.  With a thread per (unknown, near box), idle
// beyond a box's own near boxes and as slow as the largest one of its warp,
// 43,320 unknowns took 1.59 ms; now 0.76.
__global__ void __launch_bounds__(128) k_near_fill(const RwgPack<float>* __restrict__ rw, const int* __restrict__ perm,
                                                   const int* __restrict__ box_of, const int* __restrict__ box_off,
                                                   const int* __restrict__ row_cols,
                                                   const size_t* __restrict__ row_base,
                                                   const int* __restrict__ near_cbase,
                                                   const int* __restrict__ near_cidx, int n, FillConst<float> fc,
                                                   const double2* __restrict__ sing, float2* __restrict__ val)
{
    const int u = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (u >= n) return;
    const int b = box_of[u], rc = row_cols[b];
    const int* ci = near_cidx + near_cbase[b];
    const RwgPack<float>& F = rw[perm[u]];
    float2* out = val + row_base[b] + (size_t)(u - box_off[b]) * rc;
    for (int j = lane; j < rc; j += 32) {
        const Cx<float> z = z_entry<float, true>(F, rw[perm[ci[j]]], fc, sing);
        out[j] = make_float2(z.re, z.im);
    }
}

// Level patterns (up and down) are planar: box b's component c occupies
// float2 [(3 b + c) K, (3 b + c + 1) K), so a warp reads 32 consecutive
// samples of one plane at once.

// finest aggregation: CTA per finest box, threads over samples; each
// radiation pattern is read once for up to RB right-hand sides (nr of them:
// x[r][u] at r n + u, patterns of RHS r at out + r ostride)
// (the box's theta and phi sums, then expanded to x, y, z once per sample)
template <int RB>
__global__ void k_agg_finest(const float2* __restrict__ x, int n, int nr, const C2f* __restrict__ rad,
                             const float* __restrict__ tp, const int* __restrict__ box_off,
                             const int* __restrict__ box_cnt, int K, float2* __restrict__ out, size_t ostride)
{
    const int b = blockIdx.x;
    const int o = box_off[b], cnt = box_cnt[b];
    x += (size_t)blockIdx.y * n;  // RB = 1: a right-hand side a grid row
    out += blockIdx.y * ostride;
    for (int kk = threadIdx.x; kk < K; kk += blockDim.x) {
        float2 at[RB], ap[RB];
#pragma unroll
        for (int r = 0; r < RB; ++r) at[r] = ap[r] = make_float2(0, 0);
        for (int u = 0; u < cnt; ++u) {
            const C2f rv = rad[(size_t)(o + u) * K + kk];
#pragma unroll
            for (int r = 0; r < RB; ++r)
                if (RB == 1 || r < nr) {
                    const float2 xv = x[(size_t)r * n + o + u];
                    at[r] = caddf(at[r], cmulf(xv, rv.t));
                    ap[r] = caddf(ap[r], cmulf(xv, rv.p));
                }
        }
        const float e[6] = {tp[kk], tp[K + kk], tp[2 * K + kk], tp[3 * K + kk], tp[4 * K + kk], tp[5 * K + kk]};
#pragma unroll
        for (int r = 0; r < RB; ++r)
            if (RB == 1 || r < nr) {
                float2* ob = out + r * ostride + (size_t)3 * b * K + kk;
                ob[0] = caddf(cscalef(at[r], e[0]), cscalef(ap[r], e[3]));
                ob[K] = caddf(cscalef(at[r], e[1]), cscalef(ap[r], e[4]));
                ob[2 * K] = caddf(cscalef(at[r], e[2]), cscalef(ap[r], e[5]));
            }
    }
}

// interpolation + phase shift: CTA per (parent box, chunk of parent phi rows
// [pp0, pp0 + R)); thread per parent sample (pp, t), k = pp Lp + t.  The
// Lagrange stencil is separable: per child (in batches that fit shared memory)
//   1. theta pass: u[row][t] = sum_it tel(t, it) child(row, tloc(t, it)) for
//      the child phi rows [win.x, win.y) the chunk reads, into shared memory;
//   2. phi pass: parent(pp, t) += phase_oct(pp, t) sum_ip pel(pp, ip) u[ploc(pp, ip)][t].
__global__ void k_upward(const float2* __restrict__ child, int Lc, const int* __restrict__ child_ptr,
                         const int* __restrict__ child_idx, const int* __restrict__ child_oct,
                         const int* __restrict__ tl, const float* __restrict__ te, const int* __restrict__ pl,
                         const float* __restrict__ pe, const int2* __restrict__ win, int batch,
                         const float2* __restrict__ phase, int Lp, int R, float2* __restrict__ out, size_t cstride,
                         size_t ostride)
{
    extern __shared__ float2 s_u[];  // [child in batch][3][rows of the window][Lp]
    child += blockIdx.z * cstride;  // right-hand side blockIdx.z
    out += blockIdx.z * ostride;
    const int b = blockIdx.x;
    const int Kc = 2 * Lc * Lc, K = 2 * Lp * Lp;
    const int pp0 = blockIdx.y * R;
    const int nr = min(R, 2 * Lp - pp0);
    const int2 w2 = win[blockIdx.y];
    const int usz = (w2.y - w2.x) * Lp;  // one plane of one child
    const int it = threadIdx.x;
    const bool act = it < nr * Lp;
    const int pp = pp0 + (act ? it / Lp : 0), t = act ? it % Lp : 0;
    const int kp = pp * Lp + t;
    int prow[3];
    float pw[3];
#pragma unroll
    for (int ip = 0; ip < 3; ++ip) {
        prow[ip] = (pl[3 * pp + ip] - w2.x) * Lp + t;
        pw[ip] = pe[3 * pp + ip];
    }
    const int c0 = child_ptr[b], nch = child_ptr[b + 1] - c0;
    C3f acc = c3zero();
    for (int cb = 0; cb < nch; cb += batch) {
        const int nb = min(batch, nch - cb);
        __syncthreads();  // the previous batch has been read
        for (int cc = 0; cc < nb; ++cc) {
            const float2* src = child + (size_t)3 * child_idx[c0 + cb + cc] * Kc;
            float2* dst = s_u + (size_t)cc * 3 * usz;
            for (int i = threadIdx.x; i < usz; i += blockDim.x) {
                const int r = i / Lp, tt = i - r * Lp;
                const int base = (w2.x + r) * Lc;
                float2 vx = make_float2(0, 0), vy = vx, vz = vx;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const int kc = base + tl[3 * tt + q];
                    const float w = te[3 * tt + q];
                    vx = caddf(vx, cscalef(src[kc], w));
                    vy = caddf(vy, cscalef(src[Kc + kc], w));
                    vz = caddf(vz, cscalef(src[2 * Kc + kc], w));
                }
                dst[i] = vx;
                dst[usz + i] = vy;
                dst[2 * usz + i] = vz;
            }
        }
        __syncthreads();
        if (act)
            for (int cc = 0; cc < nb; ++cc) {
                const float2* u = s_u + (size_t)cc * 3 * usz;
                C3f v = c3zero();
#pragma unroll
                for (int ip = 0; ip < 3; ++ip) {
                    v.x = caddf(v.x, cscalef(u[prow[ip]], pw[ip]));
                    v.y = caddf(v.y, cscalef(u[usz + prow[ip]], pw[ip]));
                    v.z = caddf(v.z, cscalef(u[2 * usz + prow[ip]], pw[ip]));
                }
                c3fma(acc, phase[child_oct[child_idx[c0 + cb + cc]] * K + kp], v);
            }
    }
    if (act) {
        float2* ob = out + (size_t)3 * b * K + kp;
        ob[0] = acc.x;
        ob[K] = acc.y;
        ob[2 * K] = acc.z;
    }
}

// Translation, all levels in one launch: down(b) = sum over far boxes f of
// T[offset(b, f)] up(f), sample by sample.  The far boxes of the siblings under
// one parent are nearly the same: all are children of the boxes near the
// parent, and the operator depends on the offset alone.  A warp takes up to
// four siblings and 32 samples (a lane each) and reads each source pattern once
// for all of them, the siblings' sums in registers; near offsets have T = 0 in
// the table, so the siblings need no lists of their own.  The table of the
// CTA's 32 samples (343 offsets, 88 KB) is staged in shared memory, and a
// child's octant shifts its offset by a constant.  Four patterns are in flight
// at a time (lists are padded to fours with an offset that is near for every
// octant); warps take groups from a counter.
// Per (source, sibling): one 8-byte shared load and 12 FMA, against an 8-byte
// table and a 24-byte pattern load through L1 when a thread took one box's far
// list (5-wavelength sphere, 122,880 unknowns: 518 us for the five levels with
// the anterpolation, the L1 data path 80 % busy).  Now 248 us, and 109 for the
// anterpolation above the finest level; still bound by L1 wavefronts (81 %), half
// of them the siblings' table values.  Eight siblings a
// warp, or two patterns in flight, were no faster (spills; latency).
constexpr int TRANS_LEVELS = 24;  // octree levels a launch takes
// sixteen warps, two CTAs an SM by the table: a product in us with 12 | 14 | 16 |
// 18 warps (64 registers up to 16): 122880 x 1, 778 | 782 | 766 | 808; 43320 x 8,
// 1635 | 1633 | 1600 | 1619
constexpr int TRANS_WARPS = 16, TRANS_K = 32, TRANS_OFF = 343, TRANS_NC = 4, TRANS_BATCH = 4;
constexpr size_t TRANS_SMEM = sizeof(float2) * TRANS_OFF * TRANS_K;
struct TransGroup {
    int s0, s1, nc, pad;      // sources [s0, s1), multiples of TRANS_BATCH; siblings
    int2 child[TRANS_NC];     // box, its octant's shift in table rows x 32
};
struct TransWork {  // one CTA: a level's groups [g0, g1), samples [k0, k0 + 32)
    int level, k0, g0, g1;
};
struct TransLevel {
    const float2* up;
    float2* down;
    const float2* trans;
    const int4* src;          // per two sources: first element of the pattern (WIDE: first plane), row x 32 of its offset
    const TransGroup* grp;
    int K;
    size_t stride;            // complex64 from one right-hand side to the next
};
struct TransLevels {
    TransLevel l[TRANS_LEVELS];
};

// WIDE: a level has patterns of more than 2^32 values, whose elements the 32 bits
// of a source entry do not count (a few percent slower)
template <int NC, bool WIDE>
__device__ __forceinline__ void translate_group(const TransGroup& G, const int4* __restrict__ src,
                                                const float2* __restrict__ tab, const float2* __restrict__ u, int K,
                                                int k, bool store, float2* __restrict__ down)
{
    C3f acc[NC];
    const float2* t0[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        acc[c] = c3zero();
        t0[c] = tab + G.child[c].y;
    }
    const float2 *u1 = u + K, *u2 = u1 + K;
    const int s1 = G.s1;
#pragma unroll 1
    for (int s = G.s0; s < s1; s += TRANS_BATCH) {
        unsigned at[TRANS_BATCH];
        int row[TRANS_BATCH];
#pragma unroll
        for (int j = 0; j < TRANS_BATCH; j += 2) {
            const int4 e = src[(s + j) >> 1];
            at[j] = (unsigned)e.x;
            row[j] = e.y;
            at[j + 1] = (unsigned)e.z;
            row[j + 1] = e.w;
        }
        C3f v[TRANS_BATCH];
#pragma unroll
        for (int j = 0; j < TRANS_BATCH; ++j) {
            const size_t o = WIDE ? (size_t)at[j] * (unsigned)K : at[j];
            v[j] = C3f{u[o], u1[o], u2[o]};
        }
#pragma unroll
        for (int j = 0; j < TRANS_BATCH; ++j) {
            const C3f w = v[j];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float2 t = t0[c][row[j]];
                acc[c].x.x = fmaf(t.x, w.x.x, fmaf(-t.y, w.x.y, acc[c].x.x));
                acc[c].x.y = fmaf(t.x, w.x.y, fmaf(t.y, w.x.x, acc[c].x.y));
                acc[c].y.x = fmaf(t.x, w.y.x, fmaf(-t.y, w.y.y, acc[c].y.x));
                acc[c].y.y = fmaf(t.x, w.y.y, fmaf(t.y, w.y.x, acc[c].y.y));
                acc[c].z.x = fmaf(t.x, w.z.x, fmaf(-t.y, w.z.y, acc[c].z.x));
                acc[c].z.y = fmaf(t.x, w.z.y, fmaf(t.y, w.z.x, acc[c].z.y));
            }
        }
    }
    if (store) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            float2* o = down + (size_t)3 * G.child[c].x * K + k;
            o[0] = acc[c].x;
            o[K] = acc[c].y;
            o[2 * K] = acc[c].z;
        }
    }
}

template <bool WIDE>
__global__ void __launch_bounds__(32 * TRANS_WARPS, 2) k_translate(const __grid_constant__ TransLevels lv,
                                                                   const TransWork* __restrict__ work, int nr)
{
    extern __shared__ float2 s_tab[];  // [offset][32 samples]
    __shared__ int s_next;
    const TransWork w = work[blockIdx.x];
    const TransLevel& L = lv.l[w.level];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = min(w.k0 + lane, L.K - 1);  // the last chunk's spare lanes repeat the last sample
    if (threadIdx.x == 0) s_next = 0;
    for (int o = warp; o < TRANS_OFF; o += TRANS_WARPS) s_tab[o * TRANS_K + lane] = L.trans[(size_t)o * L.K + k];
    __syncthreads();
    const int n = (w.g1 - w.g0) * nr;
    const bool store = w.k0 + lane < L.K;
    const float2* tab = s_tab + lane;
    for (;;) {
        int i = lane == 0 ? atomicAdd(&s_next, 1) : 0;
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= n) break;
        const int r = nr == 1 ? 0 : i % nr;
        const TransGroup& G = L.grp[w.g0 + (nr == 1 ? i : i / nr)];
        const float2* u = L.up + r * L.stride + k;
        float2* down = L.down + r * L.stride;
        switch (G.nc) {
        case 1: translate_group<1, WIDE>(G, L.src, tab, u, L.K, k, store, down); break;
        case 2: translate_group<2, WIDE>(G, L.src, tab, u, L.K, k, store, down); break;
        case 3: translate_group<3, WIDE>(G, L.src, tab, u, L.K, k, store, down); break;
        default: translate_group<4, WIDE>(G, L.src, tab, u, L.K, k, store, down); break;
        }
    }
}

// Anterpolation from a parent pattern, theta pass: for the parent phi rows
// [w2.x, w2.y) and every theta column tc of the child
//   h[comp][pp - w2.x][tc] = sum over the transposed theta stencil of
//                            w * conj(phase(pp, t)) * parent(pp, t)
// into shared memory.  STAGED: the parent's samples are shifted first (each
// serves about three columns), into s_q, then summed; else each column shifts
// the samples that it reads, to the same bits, for rows too long for both.
template <bool STAGED>
__device__ __forceinline__ void anterp_theta(const float2* __restrict__ src, const float2* __restrict__ ph, int2 w2,
                                             int L, int Lp, const int* __restrict__ th_ptr,
                                             const int* __restrict__ th_src, const float* __restrict__ th_w,
                                             float2* s_q, float2* s_h)
{
    const int Kp = 2 * Lp * Lp, base = w2.x * Lp, qsz = (w2.y - w2.x) * Lp, hsz = (w2.y - w2.x) * L;
    if constexpr (STAGED) {
        for (int i = threadIdx.x; i < qsz; i += blockDim.x) {
            const float2 p = ph[base + i], c = make_float2(p.x, -p.y);  // exp(+j k k.(parent - child))
            s_q[i] = cmulf(c, src[base + i]);
            s_q[qsz + i] = cmulf(c, src[Kp + base + i]);
            s_q[2 * qsz + i] = cmulf(c, src[2 * Kp + base + i]);
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < hsz; i += blockDim.x) {
        const int r = i / L, tc = i - r * L;
        float2 sx = make_float2(0, 0), sy = sx, sz = sx;
        if constexpr (STAGED) {
            const float2* q = s_q + r * Lp;
            for (int a = th_ptr[tc]; a < th_ptr[tc + 1]; ++a) {
                const int t = th_src[a];
                const float w = th_w[a];
                sx = caddf(sx, cscalef(q[t], w));
                sy = caddf(sy, cscalef(q[qsz + t], w));
                sz = caddf(sz, cscalef(q[2 * qsz + t], w));
            }
        } else {
            for (int a = th_ptr[tc]; a < th_ptr[tc + 1]; ++a) {
                const int k = base + r * Lp + th_src[a];
                const float w = th_w[a];
                const float2 p = ph[k], c = make_float2(p.x, -p.y);
                sx = caddf(sx, cscalef(cmulf(c, src[k]), w));
                sy = caddf(sy, cscalef(cmulf(c, src[Kp + k]), w));
                sz = caddf(sz, cscalef(cmulf(c, src[2 * Kp + k]), w));
            }
        }
        s_h[i] = sx;
        s_h[hsz + i] = sy;
        s_h[2 * hsz + i] = sz;
    }
    __syncthreads();
}

// phi pass: the transposed phi stencil of child sample k = pc L + tc over h
__device__ __forceinline__ void anterp_phi(int pc, int tc, int w0, int L, int hsz, const int* __restrict__ ph_ptr,
                                           const int* __restrict__ ph_src, const float* __restrict__ ph_w,
                                           const float2* s_h, float2& sx, float2& sy, float2& sz)
{
    for (int a = ph_ptr[pc]; a < ph_ptr[pc + 1]; ++a) {
        const int r = (ph_src[a] - w0) * L + tc;
        const float w = ph_w[a];
        sx = caddf(sx, cscalef(s_h[r], w));
        sy = caddf(sy, cscalef(s_h[hsz + r], w));
        sz = caddf(sz, cscalef(s_h[2 * hsz + r], w));
    }
}

// a level's anterpolation, added to its translated pattern: CTA per (box, chunk
// of phi rows [pc0, pc0 + R)), i.e. the contiguous samples [pc0 L, (pc0 + R) L)
// of the box (samples k = pc L + tc, phi-major)
template <bool STAGED>
__global__ void k_downward(int L, int R, const float2* __restrict__ pdown, int Lp, const int2* __restrict__ win,
                           const int* __restrict__ parent, const int* __restrict__ oct,
                           const float2* __restrict__ pphase, const int* __restrict__ th_ptr,
                           const int* __restrict__ th_src, const float* __restrict__ th_w,
                           const int* __restrict__ ph_ptr, const int* __restrict__ ph_src,
                           const float* __restrict__ ph_w, float2* __restrict__ out, size_t ustride, size_t pstride)
{
    extern __shared__ float2 s_h[];  // [3][rows of the window][L], then, STAGED, the shifted rows [3][rows][Lp]
    // right-hand side blockIdx.z: strides in complex64 (this level, parent level)
    out += blockIdx.z * ustride;
    pdown += blockIdx.z * pstride;
    const int b = blockIdx.x;
    const int K = 2 * L * L;
    const int pc0 = blockIdx.y * R;
    const int ns = min(R, 2 * L - pc0) * L;
    const int2 w2 = win[blockIdx.y];
    const int hsz = (w2.y - w2.x) * L;
    const int Kp = 2 * Lp * Lp;
    anterp_theta<STAGED>(pdown + (size_t)3 * parent[b] * Kp, pphase + (size_t)oct[b] * Kp, w2, L, Lp, th_ptr, th_src, th_w,
                 s_h + 3 * hsz, s_h);
    for (int i = threadIdx.x; i < ns; i += blockDim.x) {
        const int k = pc0 * L + i;
        const int pc = k / L, tc = k - pc * L;
        float2* ob = out + (size_t)3 * b * K + k;
        float2 sx = ob[0], sy = ob[K], sz = ob[2 * K];
        anterp_phi(pc, tc, w2.x, L, hsz, ph_ptr, ph_src, ph_w, s_h, sx, sy, sz);
        ob[0] = sx;
        ob[K] = sy;
        ob[2 * K] = sz;
    }
}

// The finest level's anterpolation, the disaggregation and the near field in
// one pass, CTA per finest box, up to RB right-hand sides (nr of them):
//   1. per right-hand side, the box's down pattern: translated part plus
//      anterpolation, projected on theta_hat and phi_hat of each sample, times
//      its quadrature coefficient, into shared memory; the x of the box's near
//      columns beside it;
//   2. a warp per unknown: receive pattern times down pattern, then the near row.
// As two kernels (the anterpolation writing x, y, z patterns that each unknown
// read and projected again, and gathered its near x itself) this took 252 us on
// 122,880 unknowns, latency-bound; now 181.
struct FinishArgs {
    const float2* x;
    int n, nr;
    const C2f* rec;
    const float* tp;
    const float2* down;
    size_t dstride;
    const float* coeff;
    int L, Lp;
    const float2* pdown;  // parent level's patterns; null: the finest level is the top one
    size_t pstride;
    const int *parent, *oct;
    const float2* pphase;
    const int *th_ptr, *th_src;
    const float* th_w;
    const int *ph_ptr, *ph_src;
    const float* ph_w;
    const int *box_off, *box_cnt, *row_cols;
    const size_t* row_base;
    const int *near_cbase, *near_cidx;
    const float2* val;
    int parts;  // 0 near + far, 1 near, 2 far
    float2* y;
};
// Eight warps: the phases between the CTA's barriers have a few hundred
// outputs each and a box a handful of unknowns.  A product in us with 4 | 8 |
// 12 warps: 122880 x 1, 792 | 780 | 840; 10830 x 4, 282 | 260 | 271; 43320 x 8,
// 1884 | 1630 | 1700.
constexpr int FINISH_WARPS = 8;

template <int RB>
__global__ void __launch_bounds__(32 * FINISH_WARPS) k_finish(const __grid_constant__ FinishArgs A)
{
    extern __shared__ float2 s_h[];  // [3][2 Lp][L], [3][2 Lp][Lp], down [RB][2][K], x [RB][near columns]
    const int b = blockIdx.x, L = A.L, K = 2 * L * L, Lp = A.Lp, n = A.n;
    const int r0 = blockIdx.y, nr = RB == 1 ? 1 : A.nr;  // RB = 1: a right-hand side a grid row
    const float2* x = A.x + (size_t)r0 * n;
    float2* y = A.y + (size_t)r0 * n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int hsz = A.pdown ? 2 * Lp * L : 0, qsz = A.pdown ? 2 * Lp * Lp : 0;
    float2* s_q = s_h + 3 * hsz;
    float2* s_d = s_q + 3 * qsz;
    float2* s_x = s_d + (size_t)RB * 2 * K;
    const int o = A.box_off[b], cnt = A.box_cnt[b], rc = A.parts == 2 ? 0 : A.row_cols[b];
    const int* ci = A.near_cidx + A.near_cbase[b];
    for (int j = threadIdx.x; j < rc; j += blockDim.x) {
        const int cj = ci[j];
#pragma unroll
        for (int r = 0; r < RB; ++r)
            if (RB == 1 || r < nr) s_x[r * rc + j] = x[(size_t)r * n + cj];
    }
    if (A.parts != 1)
        for (int r = 0; r < nr; ++r) {
            if (A.pdown)
                anterp_theta<true>(A.pdown + (r0 + r) * A.pstride + (size_t)3 * A.parent[b] * qsz, A.pphase + (size_t)A.oct[b] * qsz,
                             make_int2(0, 2 * Lp), L, Lp, A.th_ptr, A.th_src, A.th_w, s_q, s_h);
            const float2* d = A.down + (r0 + r) * A.dstride + (size_t)3 * b * K;
            for (int k = threadIdx.x; k < K; k += blockDim.x) {
                float2 sx = d[k], sy = d[K + k], sz = d[2 * K + k];
                if (A.pdown) {
                    const int pc = k / L;
                    anterp_phi(pc, k - pc * L, 0, L, hsz, A.ph_ptr, A.ph_src, A.ph_w, s_h, sx, sy, sz);
                }
                const float e[6] = {A.tp[k],         A.tp[K + k],     A.tp[2 * K + k],
                                    A.tp[3 * K + k], A.tp[4 * K + k], A.tp[5 * K + k]};
                const float cf = A.coeff[k];
                s_d[(2 * r) * K + k] = cscalef(caddf(caddf(cscalef(sx, e[0]), cscalef(sy, e[1])), cscalef(sz, e[2])), cf);
                s_d[(2 * r + 1) * K + k] = cscalef(caddf(caddf(cscalef(sx, e[3]), cscalef(sy, e[4])), cscalef(sz, e[5])), cf);
            }
        }
    __syncthreads();
    const int kf = A.parts == 1 ? 0 : K;
    for (int u = warp; u < cnt; u += FINISH_WARPS) {
        float2 acc[RB];
#pragma unroll
        for (int r = 0; r < RB; ++r) acc[r] = make_float2(0, 0);
        const C2f* rr = A.rec + (size_t)(o + u) * K;
#pragma unroll 4
        for (int k = lane; k < kf; k += 32) {
            const C2f rv = rr[k];
#pragma unroll
            for (int r = 0; r < RB; ++r)
                if (RB == 1 || r < nr)
                    acc[r] = caddf(acc[r], caddf(cmulf(rv.t, s_d[(2 * r) * K + k]), cmulf(rv.p, s_d[(2 * r + 1) * K + k])));
        }
        const float2* vrow = A.val + A.row_base[b] + (size_t)u * A.row_cols[b];
#pragma unroll 4
        for (int j = lane; j < rc; j += 32) {
            const float2 v = vrow[j];
#pragma unroll
            for (int r = 0; r < RB; ++r)
                if (RB == 1 || r < nr) acc[r] = caddf(acc[r], cmulf(v, s_x[r * rc + j]));
        }
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            if (RB > 1 && r >= nr) break;
#pragma unroll
            for (int q = 16; q > 0; q >>= 1) {
                acc[r].x += __shfl_xor_sync(0xffffffffu, acc[r].x, q);
                acc[r].y += __shfl_xor_sync(0xffffffffu, acc[r].y, q);
            }
            if (lane == 0) y[(size_t)r * n + o + u] = acc[r];
        }
    }
}

// disaggregation + near field: warp per unknown (box order), for up to RB
// right-hand sides (nr of them; x, y at r n, down patterns at r dstride): the
// receive pattern and the near row are read once.  The near row of unknown u
// is contiguous in val (row_cols[b] values); its column unknowns are listed
// once per box in near_cidx.
template <int RB>
__global__ void k_disagg_near(const float2* __restrict__ x, int nr, const C2f* __restrict__ rec,
                              const float* __restrict__ tp, const float2* __restrict__ down, size_t dstride,
                              const float* __restrict__ coeff, int K,
                              const int* __restrict__ box_of, const int* __restrict__ box_off,
                              const int* __restrict__ row_cols, const size_t* __restrict__ row_base,
                              const int* __restrict__ near_cbase, const int* __restrict__ near_cidx,
                              const float2* __restrict__ val, int n, int skip_near, float2* __restrict__ y)
{
    const int warp = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (warp >= n) return;
    x += (size_t)blockIdx.y * n;  // RB = 1: a right-hand side a grid row
    y += (size_t)blockIdx.y * n;
    down += blockIdx.y * dstride;
    const int u = warp, b = box_of[u];
    float2 acc[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) acc[r] = make_float2(0, 0);
    const C2f* rr = rec + (size_t)u * K;
    const float2* dd = down + (size_t)3 * b * K;
#pragma unroll 4
    for (int kk = lane; kk < K; kk += 32) {
        const C2f rv = rr[kk];
        const float cf = coeff[kk];
        const float e[6] = {tp[kk], tp[K + kk], tp[2 * K + kk], tp[3 * K + kk], tp[4 * K + kk], tp[5 * K + kk]};
#pragma unroll
        for (int r = 0; r < RB; ++r)
            if (RB == 1 || r < nr) {
                const float2* d = dd + r * dstride;
                const float2 dx = d[kk], dy = d[K + kk], dz = d[2 * K + kk];
                // theta and phi components of the down pattern at this sample
                const float2 dt = caddf(caddf(cscalef(dx, e[0]), cscalef(dy, e[1])), cscalef(dz, e[2]));
                const float2 dp = caddf(caddf(cscalef(dx, e[3]), cscalef(dy, e[4])), cscalef(dz, e[5]));
                const float2 t = caddf(cmulf(rv.t, dt), cmulf(rv.p, dp));
                acc[r] = caddf(acc[r], cscalef(t, cf));
            }
    }
    if (!skip_near) {
        const int rc = row_cols[b];
        const float2* vrow = val + row_base[b] + (size_t)(u - box_off[b]) * rc;
        const int* ci = near_cidx + near_cbase[b];
#pragma unroll 4
        for (int j = lane; j < rc; j += 32) {
            const float2 v = vrow[j];
            const int cj = ci[j];
#pragma unroll
            for (int r = 0; r < RB; ++r)
                if (RB == 1 || r < nr) acc[r] = caddf(acc[r], cmulf(v, x[(size_t)r * n + cj]));
        }
    }
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        if (RB > 1 && r >= nr) break;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            acc[r].x += __shfl_xor_sync(0xffffffffu, acc[r].x, o);
            acc[r].y += __shfl_xor_sync(0xffffffffu, acc[r].y, o);
        }
        if (lane == 0) y[(size_t)r * n + u] = acc[r];
    }
}

__global__ void k_gather_c64(const float2* __restrict__ src, const int* __restrict__ idx, int n, int nrhs,
                             float2* __restrict__ dst)
{
    size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (size_t)n * nrhs) return;
    size_t r = id / n, u = id % n;
    dst[id] = src[r * n + idx[u]];
}

__global__ void k_scatter_c128(const double2* __restrict__ src, const int* __restrict__ idx, int n, int nrhs,
                               double2* __restrict__ dst)
{
    size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (size_t)n * nrhs) return;
    size_t r = id / n, u = id % n;
    dst[r * n + idx[u]] = src[id];
}

__global__ void k_resid_c64(const float2* __restrict__ B, const float2* __restrict__ Y, double2* __restrict__ R, size_t tot)
{
    size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id < tot) R[id] = make_double2((double)B[id].x - (double)Y[id].x, (double)B[id].y - (double)Y[id].y);
}

__global__ void k_f64_to_f32(const double2* __restrict__ X, float2* __restrict__ Y, size_t tot)
{
    size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id < tot) Y[id] = make_float2((float)X[id].x, (float)X[id].y);
}

// ---------------------------------------------------------------------------
// SAI preconditioner (MLFMA::parallelPreconditioner, EMSolver/MLFMA.cpp:1346-1391)
// ---------------------------------------------------------------------------
// near-field entry Z(uf, us) in box order, zero when the boxes are not near
__device__ __forceinline__ float2 near_entry(int uf, int us, const int* __restrict__ box_of,
                                             const int* __restrict__ box_off, const int* __restrict__ near_ptr,
                                             const int* __restrict__ near_box, const int* __restrict__ near_col,
                                             const int* __restrict__ row_cols, const size_t* __restrict__ row_base,
                                             const float2* __restrict__ val)
{
    const int bf = box_of[uf], bs = box_of[us];
    for (int sl = near_ptr[bf]; sl < near_ptr[bf + 1]; ++sl)
        if (near_box[sl] == bs)
            return val[row_base[bf] + (size_t)(uf - box_off[bf]) * row_cols[bf] + near_col[sl] + (us - box_off[bs])];
    return make_float2(0.f, 0.f);
}

__device__ __forceinline__ float2 cconjmul(float2 a, float2 b)  // conj(a) b
{
    return make_float2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}

__device__ __forceinline__ float2 warp_sum2(float2 v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    return v;
}

// One CTA (4 warps) per finest box: A = Z_near(rows, cols) (m x n, column
// major in shared memory), complex Householder QR, then for each unknown u
// of the box the least-squares column P(cols, u) = R^-1 Q^H e_(own + u),
// written to its CSR slot.  FP32, as the reference's value_t.
__global__ void __launch_bounds__(128) k_sai(const int* __restrict__ rptr, const int* __restrict__ rows,
                                             const int* __restrict__ cptr, const int* __restrict__ cols,
                                             const int* __restrict__ own, const int* __restrict__ box_cnt,
                                             const size_t* __restrict__ ebase, const int* __restrict__ dest,
                                             const int* __restrict__ box_of, const int* __restrict__ box_off,
                                             const int* __restrict__ near_ptr, const int* __restrict__ near_box,
                                             const int* __restrict__ near_col, const int* __restrict__ row_cols,
                                             const size_t* __restrict__ row_base, const float2* __restrict__ val,
                                             int max_rows, int max_cols, float2* __restrict__ csr_val)
{
    extern __shared__ float2 sm[];
    const int b = blockIdx.x;
    const int m = rptr[b + 1] - rptr[b], n = cptr[b + 1] - cptr[b], nb = box_cnt[b], o = own[b];
    const int* R = rows + rptr[b];
    const int* C = cols + cptr[b];
    float2* A = sm;                                        // [n][m]
    float2* rd = A + (size_t)max_rows * max_cols;          // R diagonal [n]
    float* tau = reinterpret_cast<float*>(rd + max_cols);  // [n]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float2* bv = reinterpret_cast<float2*>(tau + max_cols + (max_cols & 1)) + (size_t)warp * (max_rows + max_cols);
    float2* yv = bv + max_rows;
    for (int idx = threadIdx.x; idx < m * n; idx += blockDim.x) {
        const int f = idx % m, s = idx / m;
        A[idx] = near_entry(R[f], C[s], box_of, box_off, near_ptr, near_box, near_col, row_cols, row_base, val);
    }
    __syncthreads();
    for (int j = 0; j < n; ++j) {
        float2* aj = A + (size_t)j * m;
        if (warp == 0) {
            float xs = 0.f;
            for (int i = j + lane; i < m; i += 32) xs += aj[i].x * aj[i].x + aj[i].y * aj[i].y;
#pragma unroll
            for (int q = 16; q > 0; q >>= 1) xs += __shfl_xor_sync(0xffffffffu, xs, q);
            if (lane == 0) {
                // H_j x = al e_j with al = -e^(i arg x0) |x|: no cancellation in v0
                const float xn = sqrtf(xs);
                const float2 x0 = aj[j];
                const float ax = sqrtf(x0.x * x0.x + x0.y * x0.y);
                const float2 al = ax > 0.f ? make_float2(-x0.x / ax * xn, -x0.y / ax * xn) : make_float2(-xn, 0.f);
                const float2 v0 = make_float2(x0.x - al.x, x0.y - al.y);
                const float vn = xs - ax * ax + v0.x * v0.x + v0.y * v0.y;
                aj[j] = v0;
                rd[j] = al;
                tau[j] = vn > 0.f ? 2.f / vn : 0.f;
            }
        }
        __syncthreads();
        const float t = tau[j];
        for (int k = j + 1 + warp; k < n; k += 4) {
            float2* ak = A + (size_t)k * m;
            float2 s = make_float2(0.f, 0.f);
            for (int i = j + lane; i < m; i += 32) {
                const float2 p = cconjmul(aj[i], ak[i]);
                s.x += p.x;
                s.y += p.y;
            }
            s = warp_sum2(s);
            for (int i = j + lane; i < m; i += 32) {
                const float2 v = aj[i];
                ak[i].x -= t * (s.x * v.x - s.y * v.y);
                ak[i].y -= t * (s.x * v.y + s.y * v.x);
            }
        }
        __syncthreads();
    }
    for (int u = warp; u < nb; u += 4) {
        for (int i = lane; i < m; i += 32) bv[i] = make_float2(i == o + u ? 1.f : 0.f, 0.f);
        __syncwarp();
        for (int j = 0; j < n; ++j) {  // b <- H_j b: Q^H e
            const float2* aj = A + (size_t)j * m;
            float2 s = make_float2(0.f, 0.f);
            for (int i = j + lane; i < m; i += 32) {
                const float2 p = cconjmul(aj[i], bv[i]);
                s.x += p.x;
                s.y += p.y;
            }
            s = warp_sum2(s);
            const float t = tau[j];
            for (int i = j + lane; i < m; i += 32) {
                const float2 v = aj[i];
                bv[i].x -= t * (s.x * v.x - s.y * v.y);
                bv[i].y -= t * (s.x * v.y + s.y * v.x);
            }
            __syncwarp();
        }
        for (int i = n - 1; i >= 0; --i) {  // R y = b (R above the diagonal in A, diagonal in rd)
            float2 s = make_float2(0.f, 0.f);
            for (int k = i + 1 + lane; k < n; k += 32) {
                const float2 r = A[(size_t)k * m + i], y = yv[k];
                s.x += r.x * y.x - r.y * y.y;
                s.y += r.x * y.y + r.y * y.x;
            }
            s = warp_sum2(s);
            if (lane == 0) {
                const float2 d = rd[i];
                const float dd = d.x * d.x + d.y * d.y;
                const float2 num = make_float2(bv[i].x - s.x, bv[i].y - s.y);
                yv[i] = dd > 0.f ? make_float2((num.x * d.x + num.y * d.y) / dd, (num.y * d.x - num.x * d.y) / dd)
                                 : make_float2(0.f, 0.f);
            }
            __syncwarp();
        }
        for (int c = lane; c < n; c += 32) csr_val[dest[ebase[b] + (size_t)u * n + c]] = yv[c];
        __syncwarp();
    }
}

// translation operator of every far-box offset at every sample (FP64, the
// series of parallelLevelTrans, MLFMA.cpp:1191-1222): thread per (offset,
// sample); cf holds each offset's (2q+1)(-j)^q h_q, rec the Legendre
// recurrence's (2q-1)/q and (q-1)/q.  Bound by the FP64 pipe: five instructions
// a term (with the division by q and the products in the loop, the levels of
// 43,320 unknowns took 1.12 ms; now 0.34).
__global__ void k_trans_table(const double2* __restrict__ cf, const double2* __restrict__ rec,
                              const int* __restrict__ minl, int lmax, const float* __restrict__ kd, int K, double len,
                              float2* __restrict__ tr)
{
    const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (size_t)343 * K) return;
    const int off = (int)(id / K), kk = (int)(id % K);
    const int ml = minl[off];
    if (ml < 0) {  // near offsets: no translation
        tr[id] = make_float2(0.f, 0.f);
        return;
    }
    const int dx = off / 49 - 3, dy = (off / 7) % 7 - 3, dz = off % 7 - 3;
    const double D0 = dx * len, D1 = dy * len, D2 = dz * len;
    const double Dn = sqrt(D0 * D0 + D1 * D1 + D2 * D2);
    const double ct = ((double)kd[3 * kk] * D0 + (double)kd[3 * kk + 1] * D1 + (double)kd[3 * kk + 2] * D2) / Dn;
    const double2* c = cf + (size_t)off * (lmax + 1);
    double vr = c[0].x, vi = c[0].y, p0 = 1.0, p1 = ct;
    if (ml >= 1) {
        vr = fma(ct, c[1].x, vr);
        vi = fma(ct, c[1].y, vi);
    }
    for (int q = 2; q <= ml; ++q) {
        const double2 ab = rec[q], cq = c[q];
        const double P = fma(ab.x, ct * p1, -(ab.y * p0));
        p0 = p1;
        p1 = P;
        vr = fma(P, cq.x, vr);
        vi = fma(P, cq.y, vi);
    }
    tr[id] = make_float2((float)vr, (float)vi);
}

// y = P x, P in CSR (row per thread)
__global__ void k_sai_apply(const int* __restrict__ ptr, const int* __restrict__ col, const float2* __restrict__ val,
                            const float2* __restrict__ x, int n, float2* __restrict__ y)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float2 acc = make_float2(0.f, 0.f);
    for (int k = ptr[i]; k < ptr[i + 1]; ++k) acc = caddf(acc, cmulf(val[k], x[col[k]]));
    y[i] = acc;
}

// ---------------------------------------------------------------------------
// host build
// ---------------------------------------------------------------------------
// phi rows per CTA of the downward pass: an even count giving chunks of about
// 256 samples (sample pairs never straddle a chunk)
static int down_rows(int L)
{
    const int nchunk = (2 * L * L + 255) / 256;
    const int r = (2 * L + nchunk - 1) / nchunk;
    return r + (r & 1);
}

template <typename T>
static emfa_status_t upload(Ctx* c, DevBuf& b, const std::vector<T>& v, cudaStream_t st)
{
    EMFA_TRY(b.alloc(c, sizeof(T) * std::max<size_t>(v.size(), 1)));
    if (!v.empty()) EMFA_CUDA(c, cudaMemcpyAsync(b.ptr, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, st));
    return EMFA_OK;
}

// Host plan: everything the reference computes before its operators, in its
// float arithmetic (tree, box order, near/far lists, multipoles, samples).
struct Plan {
    int L = 0;
    float k = 0;
    std::vector<float> blen;
    std::vector<mh::Level> lev;
    std::vector<int> poles;
    std::vector<std::vector<float>> gt, gp, gw, kd;
    std::vector<std::vector<float>> wt1, wp1;  // 1-D Gauss weights in theta and phi (gw = wp1 x wt1)
    std::vector<int> perm, box_of, off, cnt;  // perm: box order -> RWG index
    std::vector<float> cen;
    std::vector<float> cp;  // RWG centres (v1 + v2) / 2, RWG order
};

static bool build_plan(const std::vector<double>& verts, int nv, const std::vector<int>& rwg, int n,
                       const emfa_mlfma_params_t& prm, Plan& P, std::string& err)
{
    const float freq = (float)prm.freq;
    const float cc = 299792458.0f;
    const float k = ((2.0f * mh::PI) * freq) / cc;  // PI2 * f / cc
    P.k = k;
    const float lambda = cc / freq;
    // float vertices, as the reference holds them
    std::vector<float> vf(verts.size());
    for (size_t i = 0; i < vf.size(); ++i) vf[i] = (float)verts[i];
    // MLFMA_Boundary::init
    float mn[3] = {3.4e38f, 3.4e38f, 3.4e38f}, mx[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
    for (int i = 0; i < nv; ++i)
        for (int d = 0; d < 3; ++d) {
            mn[d] = std::min(mn[d], vf[3 * i + d]);
            mx[d] = std::max(mx[d], vf[3 * i + d]);
        }
    float cen[3], half;
    for (int d = 0; d < 3; ++d) cen[d] = (mn[d] + mx[d]) * 0.5f;
    float maxlen = std::max(std::max(mx[0] - mn[0], mx[1] - mn[1]), mx[2] - mn[2]) + 0.1f * lambda;
    half = maxlen / 2;
    float bmin[3], bmax[3];
    for (int d = 0; d < 3; ++d) {
        bmin[d] = cen[d] - half;
        bmax[d] = cen[d] + half;
    }
    const float delta = (float)prm.box_threshold * lambda;
    int L = 0;
    for (float ml = maxlen; ml > delta; ++L) ml /= 2;
    if (L < 2) {
        err = "level number of MLFMA is too small (MLFMA box threshold is too large)";
        return false;
    }
    P.L = L;
    const float big = bmax[0] - bmin[0];
    float root[3];
    for (int d = 0; d < 3; ++d) root[d] = (bmin[d] + bmax[d]) * 0.5f;
    // RWG centres: (v1 + v2) / 2
    std::vector<float>& cp = P.cp;
    cp.assign(3 * (size_t)n, 0.f);
    for (int u = 0; u < n; ++u)
        for (int d = 0; d < 3; ++d) cp[3 * u + d] = (vf[3 * rwg[6 * u] + d] + vf[3 * rwg[6 * u + 1] + d]) * 0.5f;
    // octree (buildBox): the unknowns of every box are a range of one order,
    // which each level refines by a stable counting sort within the boxes
    auto& lev = P.lev;
    auto& blen = P.blen;
    lev.assign(L + 1, mh::Level());
    blen.assign(L + 1, 0.f);
    mh::Box rb;
    std::copy(root, root + 3, rb.c);
    rb.count = n;
    lev[0].b.push_back(rb);
    std::vector<int>& order = P.perm;
    std::vector<int> next(n);
    std::vector<unsigned char> oct(n);
    order.resize(n);
    for (int u = 0; u < n; ++u) order[u] = u;
    float cur = big / 2;
    blen[1] = cur;
    for (int l = 1; l <= L; ++l) {
        if (l > 1) {
            cur /= 2;
            blen[l] = cur;
        }
        auto& up = lev[l - 1].b;
        auto& down = lev[l].b;
        down.reserve(std::min<size_t>((size_t)n, 8 * up.size()));
        for (size_t pi = 0; pi < up.size(); ++pi) {
            mh::Box& pb = up[pi];
            const int q0 = pb.offset, q1 = pb.offset + pb.count;
            int pos[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            for (int q = q0; q < q1; ++q) {
                const float* x = &cp[3 * (size_t)order[q]];
                const int xf = x[0] < pb.c[0] ? 0 : 1, yf = x[1] < pb.c[1] ? 0 : 1, zf = x[2] < pb.c[2] ? 0 : 1;
                oct[q] = (unsigned char)((xf * 2 + yf) * 2 + zf);
                ++pos[oct[q]];
            }
            pb.child0 = (int)down.size();
            int at = q0;
            for (int idx = 0; idx < 8; ++idx) {
                const int cnt = pos[idx], x = idx >> 2, y = (idx >> 1) & 1, z = idx & 1;
                pos[idx] = at;
                if (!cnt) continue;
                mh::Box ch;
                ch.c[0] = pb.c[0] + (x - 0.5f) * cur;
                ch.c[1] = pb.c[1] + (y - 0.5f) * cur;
                ch.c[2] = pb.c[2] + (z - 0.5f) * cur;
                ch.parent = (int)pi;
                ch.oct = idx;
                ch.ix[0] = 2 * pb.ix[0] + x;
                ch.ix[1] = 2 * pb.ix[1] + y;
                ch.ix[2] = 2 * pb.ix[2] + z;
                ch.offset = at;
                ch.count = cnt;
                at += cnt;
                down.push_back(ch);
            }
            pb.nchild = (int)down.size() - pb.child0;
            for (int q = q0; q < q1; ++q) next[pos[oct[q]]++] = order[q];
        }
        order.swap(next);
    }
    // setBoxParameter: level 1 all near; level >= 2 near if the centres are
    // less than 1.75 boxes apart, that is at most one box in each direction
    // (sqrt(3) < 1.75 < 2)
    for (size_t f = 0; f < lev[1].b.size(); ++f) {
        for (size_t s2 = 0; s2 < lev[1].b.size(); ++s2) lev[1].near.push_back((int)s2);
        lev[1].nptr.push_back((int)lev[1].near.size());
    }
    for (int l = 2; l <= L; ++l) {
        const mh::Level& pl = lev[l - 1];
        mh::Level& cl = lev[l];
        cl.near.reserve(27 * cl.b.size());
        for (const auto& b : cl.b) {
            for (int s2 = pl.nptr[b.parent]; s2 < pl.nptr[b.parent + 1]; ++s2) {
                const mh::Box& pn = pl.b[pl.near[s2]];
                for (int cidx = pn.child0; cidx < pn.child0 + pn.nchild; ++cidx) {
                    const int* x = cl.b[cidx].ix;
                    if ((unsigned)(x[0] - b.ix[0] + 1) < 3u && (unsigned)(x[1] - b.ix[1] + 1) < 3u &&
                        (unsigned)(x[2] - b.ix[2] + 1) < 3u)
                        cl.near.push_back(cidx);
                }
            }
            cl.nptr.push_back((int)cl.near.size());
        }
    }
    // box order of the unknowns
    const auto& fin = lev[L].b;
    P.box_of.resize(n);
    for (size_t b = 0; b < fin.size(); ++b) {
        P.off.push_back(fin[b].offset);
        P.cnt.push_back(fin[b].count);
        std::fill_n(P.box_of.begin() + fin[b].offset, fin[b].count, (int)b);
        P.cen.insert(P.cen.end(), fin[b].c, fin[b].c + 3);
    }
    // multipoles, samples, weights, directions
    const int nl = L - 1;
    P.poles.assign(nl, 0);
    auto& gt = P.gt;
    auto& gp = P.gp;
    auto& gw = P.gw;
    auto& kd = P.kd;
    gt.assign(nl, {});
    P.wt1.assign(nl, {});
    P.wp1.assign(nl, {});
    gp.assign(nl, {});
    gw.assign(nl, {});
    kd.assign(nl, {});
    for (int l = 2; l <= L; ++l) {
        int i = l - 2;
        float kdl = 1.732051f * k * blen[l];
        // the reference's rule, or the excess-bandwidth rule of the
        // configuration (d0 = 3 digits: d0^(2/3) = 9^(1/3))
        int Pm = prm.truncation == 1 ? (int)(kdl + 1.8f * cbrtf(9.0f) * cbrtf(kdl)) : (int)(kdl + 6 * cbrtf(kdl));
        P.poles[i] = Pm;
        std::vector<float> rt, wt, rp, wp;
        mh::gauss_legendre(Pm, rt, wt);
        mh::gauss_legendre(2 * Pm, rp, wp);
        gt[i] = rt;
        gp[i] = rp;
        P.wt1[i] = wt;
        P.wp1[i] = wp;
        gw[i].resize(2 * (size_t)Pm * Pm);
        kd[i].resize(3 * 2 * (size_t)Pm * Pm);
        size_t q = 0;
        for (int pp = 0; pp < 2 * Pm; ++pp)
            for (int t = 0; t < Pm; ++t, ++q) gw[i][q] = wp[pp] * wt[t];
        const float PIh = 0.5f * mh::PI;
        for (int pp = 0; pp < 2 * Pm; ++pp) {
            float phi = mh::PI * (rp[pp] + 1);
            float ps = (float)std::sin((double)phi), pc = (float)std::cos((double)phi);
            for (int t = 0; t < Pm; ++t) {
                float th = PIh * (rt[t] + 1);
                float ts = (float)std::sin((double)th), tc = (float)std::cos((double)th);
                size_t kk = (size_t)pp * Pm + t;
                kd[i][3 * kk] = ts * pc;
                kd[i][3 * kk + 1] = ts * ps;
                kd[i][3 * kk + 2] = tc;
            }
        }
    }
    return true;
}

// SAI lists (MLFMA::setBoxParameter and parallelPreconditioner, EMSolver/MLFMA.cpp:719-741,1346-1370):
// per finest box, the near unknowns whose centre lies within row / col
// threshold x finest box length of the box centre, in near-box order; then
// the batched QR on the device and P in CSR over box-order rows
static emfa_status_t sai_build(emfa_mlfma* M, const Plan& P, cudaStream_t st)
{
    Ctx* c = M->ctx;
    if (!(M->p.row_threshold >= 0.87) || !(M->p.col_threshold >= 0.87)) {
        set_error(c, "MLFMA preconditioner: row_threshold and col_threshold must be >= 0.87 (a box's own "
                     "unknowns lie within sqrt(3)/2 box lengths of its centre)");
        return EMFA_ERR_INVALID;
    }
    const mh::Level& fl = P.lev[P.L];
    const auto& fin = fl.b;
    const float bl = P.blen[P.L];
    const float thr_r = (float)M->p.row_threshold * bl, thr_c = (float)M->p.col_threshold * bl;
    const int nbox = (int)fin.size(), n = M->n;
    auto& rptr = M->sai_rptr;
    auto& rows = M->sai_rows;
    auto& cptr = M->sai_cptr;
    auto& cols = M->sai_cols;
    auto& own = M->sai_own;
    rptr.assign(1, 0);
    cptr.assign(1, 0);
    rows.clear();
    cols.clear();
    own.clear();
    std::vector<size_t> ebase;
    size_t nnz = 0;
    int max_rows = 1, max_cols = 1;
    for (int b = 0; b < nbox; ++b) {
        int o = -1;
        for (int sl = fl.nptr[b]; sl < fl.nptr[b + 1]; ++sl) {
            const int nb = fl.near[sl];
            if (nb == b) o = (int)(rows.size() - rptr.back());
            for (int i = 0; i < fin[nb].count; ++i) {
                const int idx = fin[nb].offset + i;
                const float dist = mh::fnorm3(&P.cp[3 * (size_t)P.perm[idx]], fin[b].c);
                if (dist <= thr_r) rows.push_back(idx);
                if (dist <= thr_c) cols.push_back(idx);
            }
        }
        rptr.push_back((int)rows.size());
        cptr.push_back((int)cols.size());
        own.push_back(o);
        const int m = rptr[b + 1] - rptr[b], nc = cptr[b + 1] - cptr[b];
        max_rows = std::max(max_rows, m);
        max_cols = std::max(max_cols, nc);
        ebase.push_back(nnz);
        nnz += (size_t)nc * fin[b].count;
    }
    // CSR of P over rows = cols[c], columns = the box's own unknowns, the
    // entries of a row in the order the boxes produce them
    std::vector<int> cnt(n + 1, 0), dest(std::max<size_t>(nnz, 1)), ccol(std::max<size_t>(nnz, 1));
    for (int b = 0; b < nbox; ++b)
        for (int u = 0; u < fin[b].count; ++u)
            for (int k = cptr[b]; k < cptr[b + 1]; ++k) cnt[cols[k] + 1] += 1;
    for (int i = 0; i < n; ++i) cnt[i + 1] += cnt[i];
    std::vector<int> fillp(cnt.begin(), cnt.end() - 1);
    for (int b = 0; b < nbox; ++b)
        for (int u = 0; u < fin[b].count; ++u)
            for (int k = cptr[b]; k < cptr[b + 1]; ++k) {
                const size_t e = ebase[b] + u * (size_t)(cptr[b + 1] - cptr[b]) + (k - cptr[b]);
                const int pos = fillp[cols[k]]++;
                dest[e] = pos;
                ccol[pos] = fin[b].offset + u;
            }
    const size_t smem = sizeof(float2) * ((size_t)max_rows * max_cols + max_cols) +
                        sizeof(float) * (max_cols + (max_cols & 1)) + sizeof(float2) * 4 * (size_t)(max_rows + max_cols);
    if (smem > 220 * 1024) {
        set_error(c, "MLFMA preconditioner: a near block of " + std::to_string(max_rows) + " x " +
                         std::to_string(max_cols) + " does not fit in shared memory (use smaller boxes)");
        return EMFA_ERR_UNSUPPORTED;
    }
    M->sai_nnz = nnz;
    DevBuf d_rptr, d_rows, d_cptr, d_cols, d_own, d_ebase, d_dest;
    EMFA_TRY(upload(c, d_rptr, rptr, st));
    EMFA_TRY(upload(c, d_rows, rows, st));
    EMFA_TRY(upload(c, d_cptr, cptr, st));
    EMFA_TRY(upload(c, d_cols, cols, st));
    EMFA_TRY(upload(c, d_own, own, st));
    EMFA_TRY(upload(c, d_ebase, ebase, st));
    EMFA_TRY(upload(c, d_dest, dest, st));
    EMFA_TRY(upload(c, M->csr_ptr, cnt, st));
    EMFA_TRY(upload(c, M->csr_col, ccol, st));
    EMFA_TRY(M->csr_val.alloc(c, sizeof(float2) * std::max<size_t>(nnz, 1)));
    EMFA_TRY(M->pre_tmp.alloc(c, sizeof(float2) * (size_t)n));
    EMFA_TRY(ensure_smem(c, k_sai, smem));
    k_sai<<<nbox, 128, smem, st>>>(dptr<int>(d_rptr), dptr<int>(d_rows), dptr<int>(d_cptr), dptr<int>(d_cols),
                                   dptr<int>(d_own), dptr<int>(M->box_cnt), dptr<size_t>(d_ebase), dptr<int>(d_dest),
                                   dptr<int>(M->box_of), dptr<int>(M->box_off), dptr<int>(M->near_ptr),
                                   dptr<int>(M->near_box), dptr<int>(M->near_col), dptr<int>(M->row_cols),
                                   dptr<size_t>(M->row_base), dptr<float2>(M->near_val), max_rows, max_cols,
                                   dptr<float2>(M->csr_val));
    c->kernel_launches += 1;
    EMFA_CUDA(c, cudaGetLastError());
    EMFA_CUDA(c, cudaStreamSynchronize(st));  // the list buffers and host vectors are released on return
    M->precond = true;
    return EMFA_OK;
}

// Host tables gathered for one device buffer and one copy; the views point
// into it after upload().  The host copy must outlive the copy's stream order.
struct Stage {
    std::vector<char> host;
    std::vector<std::pair<DevView*, size_t>> at;
    template <typename T>
    void put(DevView& v, const T* a, size_t n)
    {
        const size_t o = (host.size() + 255) & ~(size_t)255;
        host.resize(o + sizeof(T) * std::max<size_t>(n, 1));
        if (n) std::copy(a, a + n, reinterpret_cast<T*>(host.data() + o));
        v.bytes = sizeof(T) * n;
        at.push_back({&v, o});
    }
    template <typename T>
    void put(DevView& v, const std::vector<T>& a)
    {
        put(v, a.data(), a.size());
    }
    emfa_status_t upload(Ctx* c, DevBuf& b, cudaStream_t st)
    {
        EMFA_TRY(b.alloc(c, std::max<size_t>(host.size(), 1)));
        EMFA_CUDA(c, cudaMemcpyAsync(b.ptr, host.data(), host.size(), cudaMemcpyHostToDevice, st));
        for (auto& x : at) x.first->ptr = (char*)b.ptr + x.second;
        return EMFA_OK;
    }
};

// column unknowns of each finest box's near rows, in value order: a warp per box
__global__ void k_near_cidx(int nbox, const int* __restrict__ near_ptr, const int* __restrict__ near_box,
                            const int* __restrict__ near_col, const int* __restrict__ box_off,
                            const int* __restrict__ box_cnt, const int* __restrict__ cbase, int* __restrict__ cidx)
{
    const int b = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (b >= nbox) return;
    for (int sl = near_ptr[b]; sl < near_ptr[b + 1]; ++sl) {
        const int nb = near_box[sl], off = box_off[nb], cnt = box_cnt[nb];
        int* o = cidx + cbase[b] + near_col[sl];
        for (int q = lane; q < cnt; q += 32) o[q] = off + q;
    }
}

// The level patterns of nr right-hand sides, one buffer
static emfa_status_t alloc_patterns(emfa_mlfma* M, int nr)
{
    size_t tot = 0;
    for (auto& ml : M->lv) tot += 2 * Carver::round(sizeof(float2) * 3 * (size_t)ml.nbox * ml.K * nr);
    M->rcap = 0;
    EMFA_TRY(M->patterns.alloc(M->ctx, tot));
    char* p = (char*)M->patterns.ptr;
    for (auto& ml : M->lv) {
        const size_t per = sizeof(float2) * 3 * (size_t)ml.nbox * ml.K * nr;
        for (DevView* v : {&ml.up, &ml.down}) {
            v->ptr = p;
            v->bytes = per;
            p += Carver::round(per);
        }
    }
    M->rcap = nr;
    return EMFA_OK;
}

// Set-up.  The device has about 1.3 ms of work at 43 k unknowns (singular
// table, patterns, near field, translation series), the host about 3 ms
// (tree and lists, series, stencils), and 120 allocations and as many copies
// had cost 3 ms more with the first product and the release.  So the
// singular table runs beside the tree, patterns and near field beside the
// level tables, and the tables travel as two buffers: 10.6 -> 4.2 ms, with a
// first product of four right-hand sides and the release 13.7 -> 6.5.
static emfa_status_t mlfma_build(emfa_mlfma* M, cudaStream_t st)
{
    Ctx* c = M->ctx;
    Geom* g = M->geom;
    const int n = g->n;
    M->n = n;
    emfa_fill_params_t fp{EMFA_CFIE, EMFA_F32, M->p.freq, M->p.alpha, 0, 0, 0};
    Stage fine, tables, series;  // series: read by k_trans_table only
    struct Landed {  // no return leaves a copy from the stages in flight
        cudaStream_t s;
        ~Landed() { cudaStreamSynchronize(s); }
    } landed{st};
    DevBuf tab;
    EMFA_TRY(geom_prepare_f32(g, st));
    EMFA_TRY(tab.alloc(c, sizeof(double2) * (size_t)g->nt * 9));
    EMFA_TRY(build_singular_table(c, g, &fp, dptr<double2>(tab), st));
    Plan P;
    std::string err;
    if (!build_plan(g->verts, g->nv, g->rwg, n, M->p, P, err)) {
        set_error(c, err);
        return EMFA_ERR_INVALID;
    }
    const int L = P.L;
    const float k = P.k;
    M->k = k;
    M->levels = L;
    auto& lev = P.lev;
    auto& gt = P.gt;
    auto& gp = P.gp;
    auto& gw = P.gw;
    auto& kd = P.kd;
    const auto& fin = lev[L].b;
    M->level_boxes.clear();
    for (int l = 0; l <= L; ++l) M->level_boxes.push_back((int)lev[l].b.size());
    M->perm = P.perm;
    M->poles = P.poles;
    const int nl = L - 1;
    if (nl > TRANS_LEVELS) {
        set_error(c, "mlfma: more than " + std::to_string(TRANS_LEVELS + 1) + " octree levels (box threshold too small)");
        return EMFA_ERR_UNSUPPORTED;
    }
    M->lv.clear();
    M->lv.resize(nl);
    for (int l = 2; l <= L; ++l) {
        const int i = l - 2;
        MLevel& ml = M->lv[i];
        ml.nbox = (int)lev[l].b.size();
        ml.L = P.poles[i];
        ml.K = 2 * ml.L * ml.L;
        ml.len = P.blen[l];
        if ((size_t)3 * ml.nbox * ml.K > 0xffffffffull) M->wide = true;
    }
    // the interpolation and anterpolation passes may use more than the default 48 KB of shared memory
    EMFA_TRY(ensure_smem(c, k_upward, 96 * 1024));
    EMFA_TRY(ensure_smem(c, k_downward<true>, 200 * 1024));
    EMFA_TRY(ensure_smem(c, k_downward<false>, 200 * 1024));
    EMFA_TRY(ensure_smem(c, k_translate<false>, TRANS_SMEM));
    EMFA_TRY(ensure_smem(c, k_translate<true>, TRANS_SMEM));
    // finest-level lists and tables
    MLevel& fl = M->lv[nl - 1];
    const int Kf = fl.K;
    DevView cen_d, kdir_d;
    {
        std::vector<float> coeff(Kf);
        const float PIh = 0.5f * mh::PI;
        size_t q = 0;
        for (int pp = 0; pp < 2 * fl.L; ++pp)
            for (int t = 0; t < fl.L; ++t, ++q)
                coeff[q] = (float)(gw[nl - 1][q] * std::sin((double)(PIh * (gt[nl - 1][t] + 1))));
        const float z0 = 120.0f * mh::PI;
        const float cn = k * k * z0 / 32;
        for (auto& v : coeff) v = cn * v;
        fine.put(M->coeff, coeff);
    }
    fine.put(M->perm_d, M->perm);
    fine.put(M->box_of, P.box_of);
    fine.put(M->box_off, P.off);
    fine.put(M->box_cnt, P.cnt);
    fine.put(cen_d, P.cen);
    fine.put(kdir_d, kd[nl - 1]);
    // theta_hat, phi_hat of every finest sample direction (FP64 from the
    // sample's float direction, stored in float): phi_hat = z x k / |z x k|,
    // theta_hat = phi_hat x k (the Gauss-Legendre theta nodes avoid the poles)
    {
        std::vector<float> tp((size_t)6 * Kf);
        const auto& kv = kd[nl - 1];
        for (int kk = 0; kk < Kf; ++kk) {
            const double kx = kv[3 * kk], ky = kv[3 * kk + 1], kz = kv[3 * kk + 2];
            const double rho = std::sqrt(kx * kx + ky * ky);
            const double px = -ky / rho, py = kx / rho;
            const double tx = py * kz, ty = -px * kz, tz = px * ky - py * kx;
            const double tv[6] = {tx, ty, tz, px, py, 0.0};
            for (int j = 0; j < 6; ++j) tp[(size_t)j * Kf + kk] = (float)tv[j];
        }
        fine.put(M->tp, tp);
    }
    // near field: column bases, row bases
    const int nfin = (int)fin.size();
    std::vector<int> ncol, rcols, cbase{0};
    std::vector<size_t> rbase;
    size_t nnz = 0;
    ncol.reserve(lev[L].near.size());
    for (int b = 0; b < nfin; ++b) {
        int cols = 0;
        for (int sl = lev[L].nptr[b]; sl < lev[L].nptr[b + 1]; ++sl) {
            ncol.push_back(cols);
            cols += fin[lev[L].near[sl]].count;
        }
        rcols.push_back(cols);
        cbase.push_back(cbase.back() + cols);
        M->max_cols = std::max(M->max_cols, cols);
        rbase.push_back(nnz);
        nnz += (size_t)cols * fin[b].count;
    }
    M->nnz = nnz;
    fine.put(M->near_ptr, lev[L].nptr);
    fine.put(M->near_box, lev[L].near);
    fine.put(M->near_col, ncol);
    fine.put(M->row_cols, rcols);
    fine.put(M->row_base, rbase);
    fine.put(M->near_cbase, cbase);
    EMFA_TRY(fine.upload(c, M->fine_tables, st));
    EMFA_TRY(M->near_cidx.alloc(c, sizeof(int) * (size_t)std::max(cbase.back(), 1)));
    EMFA_TRY(M->near_val.alloc(c, sizeof(float2) * std::max<size_t>(nnz, 1)));
    EMFA_TRY(M->rad.alloc(c, sizeof(C2f) * (size_t)n * Kf));
    EMFA_TRY(M->rec.alloc(c, sizeof(C2f) * (size_t)n * Kf));
    {
        k_near_cidx<<<(unsigned)((nfin + 3) / 4), 128, 0, st>>>(
            nfin, dptr<int>(M->near_ptr), dptr<int>(M->near_box), dptr<int>(M->near_col), dptr<int>(M->box_off),
            dptr<int>(M->box_cnt), dptr<int>(M->near_cbase), dptr<int>(M->near_cidx));
        FillConst<float> fc = make_fill_const<float>(&fp);
        k_near_fill<<<(unsigned)(((size_t)n * 32 + 127) / 128), 128, 0, st>>>(
            dptr<RwgPack<float>>(g->g32.rwg), dptr<int>(M->perm_d), dptr<int>(M->box_of), dptr<int>(M->box_off),
            dptr<int>(M->row_cols), dptr<size_t>(M->row_base), dptr<int>(M->near_cbase), dptr<int>(M->near_cidx), n,
            fc, dptr<double2>(tab), dptr<float2>(M->near_val));
        const size_t tot = (size_t)n * Kf;
        k_radrec<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(dptr<RwgPack<float>>(g->g32.rwg), dptr<int>(M->perm_d),
                                                               dptr<int>(M->box_of), dptr<float>(cen_d),
                                                               dptr<float>(kdir_d), dptr<float>(M->tp), n, Kf, k,
                                                               (float)M->p.alpha, dptr<C2f>(M->rad),
                                                               dptr<C2f>(M->rec));
        c->kernel_launches += 3;
        EMFA_CUDA(c, cudaGetLastError());
    }
    // under a budget the singular table goes before the level tables come (and
    // the host waits here for the near field, which it otherwise overlaps)
    if (c->budget) tab.release();
    // per-level tables
    struct Series {
        DevView hl, rec, minl, kd;
    };
    std::vector<Series> sv(nl);
    for (int l = 2; l <= L; ++l) {
        const int i = l - 2;
        MLevel& ml = M->lv[i];
        const int K = ml.K;
        const auto& bx = lev[l].b;
        const auto& up = lev[l - 1];
        std::vector<int> par, oc, cptr{0}, cidx;
        for (auto& b : bx) {
            par.push_back(b.parent);
            oc.push_back(b.oct);
        }
        // sibling groups: the far boxes of a box are the children of the boxes
        // near its parent that are not near itself (setBoxParameter), in that order
        std::vector<TransGroup> grp;
        std::vector<int2> gsrc;
        for (int self = 0; self < (int)up.b.size(); ++self) {
            const mh::Box& pb = up.b[self];
            const int s0 = (int)gsrc.size();
            for (int sl = up.nptr[self]; sl < up.nptr[self + 1]; ++sl) {
                const int pn = up.near[sl];
                if (pn == self) continue;  // the siblings are near one another
                const mh::Box& nbx = up.b[pn];
                for (int f = nbx.child0; f < nbx.child0 + nbx.nchild; ++f) {
                    // from the source box to the parent's first octant, in boxes
                    int off = 0;
                    for (int d = 0; d < 3; ++d) off = 7 * off + (2 * pb.ix[d] - bx[f].ix[d]) + 3;
                    gsrc.push_back(make_int2(M->wide ? 3 * f : (int)(unsigned)((size_t)3 * f * K), off * TRANS_K));
                }
            }
            // the offset (0, 0, 0) is near for every octant: T = 0
            while (gsrc.size() % TRANS_BATCH) gsrc.push_back(make_int2(gsrc.back().x, 171 * TRANS_K));  // gsrc.size() > s0 here
            const int nc = pb.nchild, parts = (nc + TRANS_NC - 1) / TRANS_NC;
            for (int q = 0; q < parts; ++q) {
                TransGroup tg{};
                tg.s0 = s0;
                tg.s1 = (int)gsrc.size();
                for (int j = nc * q / parts; j < nc * (q + 1) / parts; ++j) {
                    const int o = bx[pb.child0 + j].oct;
                    tg.child[tg.nc++] = make_int2(pb.child0 + j, (49 * (o >> 2) + 7 * ((o >> 1) & 1) + (o & 1)) * TRANS_K);
                }
                grp.push_back(tg);
            }
        }
        ml.ngrp = (int)grp.size();
        if (l < L)
            for (auto& b : bx) {
                for (int ch = b.child0; ch < b.child0 + b.nchild; ++ch) cidx.push_back(ch);
                cptr.push_back((int)cidx.size());
            }
        tables.put(ml.parent, par);
        tables.put(ml.oct, oc);
        tables.put(ml.grp_src, gsrc);
        tables.put(ml.grp, grp);
        tables.put(ml.child_ptr, cptr);
        tables.put(ml.child_idx, cidx);
        // translation operators per offset: sum_l (2l+1)(-j)^l h_l^(2)(kD) P_l(k.D/|D|),
        // l <= min(poles, floor(kD)) (MLFMA.cpp:1203-1219), in FP64: the Hankel
        // recurrence per distance here, the Legendre sums per sample on the device
        {
            const int lmax = ml.L;
            std::vector<double2> hlv((size_t)343 * (lmax + 1), make_double2(0, 0));
            std::vector<int> minl(343, -1);
            std::vector<std::pair<double, int>> dist;  // distances so far and an offset of each
            for (int dx = -3; dx <= 3; ++dx)
                for (int dy = -3; dy <= 3; ++dy)
                    for (int dz = -3; dz <= 3; ++dz) {
                        if (std::abs(dx) <= 1 && std::abs(dy) <= 1 && std::abs(dz) <= 1) continue;
                        const int off = ((dx + 3) * 7 + (dy + 3)) * 7 + (dz + 3);
                        double D[3] = {dx * (double)ml.len, dy * (double)ml.len, dz * (double)ml.len};
                        double Dn = std::sqrt(D[0] * D[0] + D[1] * D[1] + D[2] * D[2]);
                        double x = (double)k * Dn;
                        int minL = (int)std::min((float)ml.L, (float)(k * (float)Dn));
                        minL = std::min(minL, lmax);
                        minl[off] = minL;
                        double2* out = &hlv[(size_t)off * (lmax + 1)];
                        // offsets of one distance share the series
                        size_t same = 0;
                        while (same < dist.size() && dist[same].first != Dn) ++same;
                        if (same < dist.size()) {
                            std::copy_n(&hlv[(size_t)dist[same].second * (lmax + 1)], minL + 1, out);
                            continue;
                        }
                        dist.push_back({Dn, off});
                        std::vector<std::complex<double>> hl(minL + 1);
                        hl[0] = std::complex<double>(std::sin(x), std::cos(x)) / x;
                        if (minL >= 1)
                            hl[1] = std::complex<double>(std::sin(x) / x - std::cos(x), std::cos(x) / x + std::sin(x)) / x;
                        for (int q = 2; q <= minL; ++q) hl[q] = ((2.0 * q - 1) / x) * hl[q - 1] - hl[q - 2];
                        for (int q = 0; q <= minL; ++q) {
                            // (2q+1) (-j)^q h_q
                            const double w = 2.0 * q + 1, hr = w * hl[q].real(), hi = w * hl[q].imag();
                            out[q] = (q & 3) == 0   ? make_double2(hr, hi)
                                     : (q & 3) == 1 ? make_double2(hi, -hr)
                                     : (q & 3) == 2 ? make_double2(-hr, -hi)
                                                    : make_double2(-hi, hr);
                        }
                    }
            std::vector<double2> recv(lmax + 1, make_double2(0, 0));
            for (int q = 1; q <= lmax; ++q) recv[q] = make_double2((2.0 * q - 1) / q, (q - 1.0) / q);
            series.put(sv[i].hl, hlv);
            series.put(sv[i].rec, recv);
            series.put(sv[i].minl, minl);
            series.put(sv[i].kd, kd[i]);
        }
    }
    // translation work: up to 48 groups a CTA (three a warp and right-hand side,
    // so that the table's staging is a few percent; 122880 x 1, us with 24 | 36 | 48 |
    // 72: 762 | 751 | 739 | 742), fewer where that leaves SMs idle
    {
        std::vector<TransWork> tw;
        size_t tasks = 0;
        for (const MLevel& ml : M->lv) tasks += (size_t)ml.ngrp * ((ml.K + TRANS_K - 1) / TRANS_K);
        const size_t sms = c->sm_count > 0 ? c->sm_count : 148;
        const int per = (int)std::min<size_t>(48, std::max<size_t>(6, tasks / (8 * sms)));
        for (int i = nl - 1; i >= 0; --i) {
            const MLevel& ml = M->lv[i];
            const int parts = std::max(1, (ml.ngrp + per / 2) / per);
            for (int k0 = 0; k0 < ml.K; k0 += TRANS_K)
                for (int p = 0; p < parts; ++p)
                    tw.push_back(TransWork{i, k0, (int)((long long)ml.ngrp * p / parts),
                                           (int)((long long)ml.ngrp * (p + 1) / parts)});
        }
        M->trans_ctas = (int)tw.size();
        tables.put(M->trans_work, tw);
    }
    // interpolation level i+1 (child, fewer samples) -> level i (parent), i = 0..nl-2
    for (int i = 0; i + 1 < nl; ++i) {
        MLevel& pm = M->lv[i];
        MLevel& cm = M->lv[i + 1];
        std::vector<int> tloc, ploc;
        std::vector<float> tel, pel;
        mh::lagrange(gt[i + 1], gt[i], tloc, tel);
        mh::lagrange(gp[i + 1], gp[i], ploc, pel);
        const int Kp = pm.K, Lc = cm.L;
        tables.put(pm.ip_tl, tloc);
        tables.put(pm.ip_te, tel);
        tables.put(pm.ip_pl, ploc);
        tables.put(pm.ip_pe, pel);
        {
            // phi-row chunks of about 256 parent samples, a thread each (two rows
            // above 181 samples a row, one above 512), and the child rows each reads
            if (pm.L > 1024) {
                set_error(c, "mlfma: more than 1024 multipoles (level too large)");
                return EMFA_ERR_UNSUPPORTED;
            }
            pm.up_rows = pm.L > 512 ? 1 : down_rows(pm.L);
            const int nchunk = (2 * pm.L + pm.up_rows - 1) / pm.up_rows;
            std::vector<int2> win(nchunk);
            int most = 0;
            for (int ch = 0; ch < nchunk; ++ch) {
                int lo = 2 * Lc, hi = 0;
                for (int pp = ch * pm.up_rows; pp < std::min(2 * pm.L, (ch + 1) * pm.up_rows); ++pp)
                    for (int ip = 0; ip < 3; ++ip) {
                        lo = std::min(lo, ploc[3 * pp + ip]);
                        hi = std::max(hi, ploc[3 * pp + ip] + 1);
                    }
                win[ch] = make_int2(lo, hi);
                most = std::max(most, hi - lo);
            }
            pm.up_child_bytes = sizeof(float2) * 3 * (size_t)most * pm.L;
            pm.up_batch = (int)std::min<size_t>(8, (96 * 1024) / pm.up_child_bytes);
            if (pm.up_batch < 1) {
                set_error(c, "mlfma: interpolation rows exceed shared memory (level too large)");
                return EMFA_ERR_UNSUPPORTED;
            }
            tables.put(pm.up_win, win);
        }
        // phases for the children of level i: exp(-j k kp . (parent - child)), per octant
        std::vector<float2> ph((size_t)8 * Kp);
        for (int o = 0; o < 8; ++o) {
            int x = o >> 2, y = (o >> 1) & 1, z = o & 1;
            float rv[3] = {-(x - 0.5f) * cm.len, -(y - 0.5f) * cm.len, -(z - 0.5f) * cm.len};
            for (int kk = 0; kk < Kp; ++kk) {
                double a = (double)k * ((double)kd[i][3 * kk] * rv[0] + (double)kd[i][3 * kk + 1] * rv[1] +
                                         (double)kd[i][3 * kk + 2] * rv[2]);
                ph[(size_t)o * Kp + kk] = make_float2((float)std::cos(a), (float)-std::sin(a));
            }
        }
        tables.put(pm.up_phase, ph);
        // anterpolation into level i+1: the transposed theta and phi Lagrange
        // stencils, each weight scaled by w_parent / w_child of its own axis
        // (the 2-D weights are products: gw = wp x wt)
        {
            const int Lp = pm.L;
            auto transpose = [](const std::vector<int>& loc, const std::vector<float>& el, int np, int nc,
                                const std::vector<float>& wpar, const std::vector<float>& wch, std::vector<int>& ptr,
                                std::vector<int>& src, std::vector<float>& wt) {
                std::vector<std::vector<std::pair<int, float>>> lst(nc);
                for (int x = 0; x < np; ++x)
                    for (int q = 0; q < 3; ++q) {
                        const int y = loc[3 * x + q];
                        lst[y].push_back({x, el[3 * x + q] * wpar[x] / wch[y]});
                    }
                ptr.assign(1, 0);
                src.clear();
                wt.clear();
                for (int y = 0; y < nc; ++y) {
                    for (auto& e : lst[y]) {
                        src.push_back(e.first);
                        wt.push_back(e.second);
                    }
                    ptr.push_back((int)src.size());
                }
            };
            std::vector<int> tptr, tsrc, pptr, psrc;
            std::vector<float> tw, pw;
            transpose(tloc, tel, Lp, Lc, P.wt1[i], P.wt1[i + 1], tptr, tsrc, tw);
            transpose(ploc, pel, 2 * Lp, 2 * Lc, P.wp1[i], P.wp1[i + 1], pptr, psrc, pw);
            tables.put(cm.th_ptr, tptr);
            tables.put(cm.th_src, tsrc);
            tables.put(cm.th_w, tw);
            tables.put(cm.ph_ptr, pptr);
            tables.put(cm.ph_src, psrc);
            tables.put(cm.ph_w, pw);
            // phi-row chunks of about 256 samples, and the parent rows each reads
            const int rows = down_rows(Lc);
            const int nchunk = (2 * Lc + rows - 1) / rows;
            std::vector<int2> dw(nchunk);
            int most = 0;
            for (int ch = 0; ch < nchunk; ++ch) {
                int lo = 2 * Lp, hi = 0;
                for (int pc = ch * rows; pc < std::min(2 * Lc, (ch + 1) * rows); ++pc)
                    for (int a = pptr[pc]; a < pptr[pc + 1]; ++a) {
                        lo = std::min(lo, psrc[a]);
                        hi = std::max(hi, psrc[a] + 1);
                    }
                if (hi <= lo) lo = hi = 0;
                dw[ch] = make_int2(lo, hi);
                most = std::max(most, hi - lo);
            }
            // both sets of rows up to an extent of about 180 wavelengths
            cm.down_smem = sizeof(float2) * 3 * (size_t)most * (Lc + Lp);
            cm.down_staged = cm.down_smem <= 200 * 1024;
            if (!cm.down_staged) cm.down_smem = sizeof(float2) * 3 * (size_t)most * Lc;
            if (cm.down_smem > 200 * 1024) {
                set_error(c, "mlfma: anterpolation rows exceed shared memory (level too large)");
                return EMFA_ERR_UNSUPPORTED;
            }
            tables.put(cm.down_win, dw);
        }
    }
    EMFA_TRY(tables.upload(c, M->level_tables, st));
    DevBuf series_d;
    EMFA_TRY(series.upload(c, series_d, st));
    size_t tt = 0;
    for (auto& ml : M->lv) tt += Carver::round(sizeof(float2) * (size_t)343 * ml.K);
    EMFA_TRY(M->trans_tables.alloc(c, tt));
    EMFA_TRY(alloc_patterns(M, 1));
    tt = 0;
    for (int i = 0; i < nl; ++i) {
        MLevel& ml = M->lv[i];
        const size_t tot = (size_t)343 * ml.K;
        ml.trans.ptr = (char*)M->trans_tables.ptr + tt;
        ml.trans.bytes = sizeof(float2) * tot;
        tt += Carver::round(ml.trans.bytes);
        k_trans_table<<<(unsigned)((tot + 127) / 128), 128, 0, st>>>(dptr<double2>(sv[i].hl), dptr<double2>(sv[i].rec),
                                                                     dptr<int>(sv[i].minl), ml.L,
                                                                     dptr<float>(sv[i].kd), ml.K, (double)ml.len,
                                                                     dptr<float2>(ml.trans));
        c->kernel_launches += 1;
    }
    EMFA_CUDA(c, cudaGetLastError());
    if (M->p.precond) EMFA_TRY(sai_build(M, P, st));
    EMFA_CUDA(c, cudaGetLastError());
    EMFA_CUDA(c, cudaStreamSynchronize(st));  // the host tables and the temporary buffers are released on return
    return EMFA_OK;
}

// right-hand sides per pass of the operator's kernels
constexpr int RHS_CHUNK = 8;

// level patterns for nr right-hand sides (scratch: grown, never copied)
static emfa_status_t reserve_rhs(emfa_mlfma* M, int nr) { return nr <= M->rcap ? EMFA_OK : alloc_patterns(M, nr); }

// shared bytes of k_finish<RB>
static size_t finish_smem(emfa_mlfma* M, int rb)
{
    const int nl = M->levels - 1;
    const MLevel& fl = M->lv[nl - 1];
    const size_t Lp = nl > 1 ? M->lv[nl - 2].L : 0;
    return sizeof(float2) * (6 * Lp * (fl.L + Lp) + (size_t)rb * (2 * fl.K + M->max_cols));
}
// k_finish where at least two of its CTAs fit an SM; larger finest boxes (many
// samples or near columns) keep the anterpolation and the warp-per-unknown
// disaggregation as two kernels
constexpr size_t FINISH_SMEM_MAX = 100 * 1024;
template <int RB>
static emfa_status_t launch_finish(emfa_mlfma* M, const float2* x, int nr, float2* y, int parts, cudaStream_t st)
{
    const int nl = M->levels - 1;
    MLevel& fl = M->lv[nl - 1];
    MLevel& pm = M->lv[nl > 1 ? nl - 2 : 0];
    const bool par = nl > 1;
    const FinishArgs a{x, M->n, nr, dptr<C2f>(M->rec), dptr<float>(M->tp), dptr<float2>(fl.down),
                       (size_t)3 * fl.nbox * fl.K, dptr<float>(M->coeff), fl.L, par ? pm.L : 0,
                       par ? dptr<float2>(pm.down) : nullptr, (size_t)3 * pm.nbox * pm.K, dptr<int>(fl.parent),
                       dptr<int>(fl.oct), dptr<float2>(pm.up_phase), dptr<int>(fl.th_ptr), dptr<int>(fl.th_src),
                       dptr<float>(fl.th_w), dptr<int>(fl.ph_ptr), dptr<int>(fl.ph_src), dptr<float>(fl.ph_w),
                       dptr<int>(M->box_off), dptr<int>(M->box_cnt), dptr<int>(M->row_cols), dptr<size_t>(M->row_base),
                       dptr<int>(M->near_cbase), dptr<int>(M->near_cidx), dptr<float2>(M->near_val), parts, y};
    const size_t sm = finish_smem(M, RB);
    EMFA_TRY(ensure_smem(M->ctx, k_finish<RB>, sm));
    k_finish<RB><<<dim3(fl.nbox, RB == 1 ? nr : 1), 32 * FINISH_WARPS, sm, st>>>(a);
    return EMFA_OK;
}

template <int RB>
static void launch_agg_disagg(emfa_mlfma* M, bool agg, const float2* x, int nr, float2* y, int parts, cudaStream_t st)
{
    const int nl = M->levels - 1;
    MLevel& fl = M->lv[nl - 1];
    const int Kf = fl.K, n = M->n;
    const size_t lstride = (size_t)3 * fl.nbox * Kf;
    if (agg)  // 256 threads cover the samples of a box in one turn (27000 x 2, 412 -> 405 us a product)
        k_agg_finest<RB><<<dim3(fl.nbox, RB == 1 ? nr : 1), 256, 0, st>>>(x, n, nr, dptr<C2f>(M->rad), dptr<float>(M->tp),
                                                  dptr<int>(M->box_off), dptr<int>(M->box_cnt), Kf,
                                                  dptr<float2>(fl.up), lstride);
    else
        k_disagg_near<RB><<<dim3((unsigned)(((size_t)n * 32 + 255) / 256), RB == 1 ? nr : 1), 256, 0, st>>>(
            x, nr, dptr<C2f>(M->rec), dptr<float>(M->tp), dptr<float2>(fl.down), lstride, dptr<float>(M->coeff),
            parts == 1 ? 0 : Kf,
            dptr<int>(M->box_of), dptr<int>(M->box_off), dptr<int>(M->row_cols), dptr<size_t>(M->row_base),
            dptr<int>(M->near_cbase), dptr<int>(M->near_cidx), dptr<float2>(M->near_val), n, parts == 2 ? 1 : 0, y);
}

// Right-hand sides a CTA of the finest level's kernels takes (1, 2, 4 or 8):
// all of them, so that the radiation and receive patterns are read from HBM
// once, unless they stay in L2 anyway; then one each, on its own grid row, which
// fills the SMs at these sizes (10,830 unknowns, 4 right-hand sides:
// k_finish 115 -> 74 us, a product 328 -> 274 us).
static int finest_rhs(emfa_mlfma* M, int nr)
{
    const size_t pat = sizeof(C2f) * (size_t)M->n * M->lv[M->levels - 2].K;
    if (nr <= 1 || pat <= ((size_t)64 << 20)) return 1;
    return nr <= 2 ? 2 : nr <= 4 ? 4 : 8;
}

static void agg_disagg(emfa_mlfma* M, bool agg, const float2* x, int nr, int rb, float2* y, int parts, cudaStream_t st)
{
    if (rb == 1)
        launch_agg_disagg<1>(M, agg, x, nr, y, parts, st);
    else if (rb == 2)
        launch_agg_disagg<2>(M, agg, x, nr, y, parts, st);
    else if (rb == 4)
        launch_agg_disagg<4>(M, agg, x, nr, y, parts, st);
    else
        launch_agg_disagg<8>(M, agg, x, nr, y, parts, st);
}

// y = Z x for nr <= RHS_CHUNK vectors (RHS-major, box order, complex64);
// parts: 0 near + far, 1 near, 2 far
static emfa_status_t mlfma_apply(emfa_mlfma* M, const float2* x, float2* y, int nr, cudaStream_t st, int parts = 0)
{
    Ctx* c = M->ctx;
    EMFA_TRY(reserve_rhs(M, nr));
    const int nl = M->levels - 1;
    const int rb = finest_rhs(M, nr);
    agg_disagg(M, true, x, nr, rb, y, parts, st);
    for (int i = nl - 2; i >= 0; --i) {
        MLevel& pm = M->lv[i];
        MLevel& cm = M->lv[i + 1];
        const int R = pm.up_rows;
        const int bs = 32 * ((R * pm.L + 31) / 32);
        const dim3 grid((unsigned)pm.nbox, (unsigned)((2 * pm.L + R - 1) / R), (unsigned)nr);
        k_upward<<<grid, bs, pm.up_child_bytes * pm.up_batch, st>>>(
            dptr<float2>(cm.up), cm.L, dptr<int>(pm.child_ptr), dptr<int>(pm.child_idx), dptr<int>(cm.oct),
            dptr<int>(pm.ip_tl), dptr<float>(pm.ip_te), dptr<int>(pm.ip_pl), dptr<float>(pm.ip_pe),
            dptr<int2>(pm.up_win), pm.up_batch, dptr<float2>(pm.up_phase), pm.L, R, dptr<float2>(pm.up),
            (size_t)3 * cm.nbox * cm.K, (size_t)3 * pm.nbox * pm.K);
    }
    EMFA_CUDA(c, cudaGetLastError());
    TransLevels lv;
    for (int i = 0; i < nl; ++i) {
        MLevel& ml = M->lv[i];
        lv.l[i] = TransLevel{dptr<float2>(ml.up),     dptr<float2>(ml.down),      dptr<float2>(ml.trans),
                             dptr<int4>(ml.grp_src), dptr<TransGroup>(ml.grp), ml.K, (size_t)3 * ml.nbox * ml.K};
    }
    (M->wide ? k_translate<true> : k_translate<false>)<<<M->trans_ctas, 32 * TRANS_WARPS, TRANS_SMEM, st>>>(lv, dptr<TransWork>(M->trans_work), nr);
    const bool fused = finish_smem(M, rb) <= FINISH_SMEM_MAX;
    for (int i = 1; i < (fused ? nl - 1 : nl); ++i) {
        MLevel& ml = M->lv[i];
        MLevel& pm = M->lv[i - 1];
        const int R = down_rows(ml.L);
        const int bs = std::min(256, 32 * ((R * ml.L + 31) / 32));
        const dim3 grid((unsigned)ml.nbox, (unsigned)((2 * ml.L + R - 1) / R), (unsigned)nr);
        (ml.down_staged ? k_downward<true> : k_downward<false>)<<<grid, bs, ml.down_smem, st>>>(
            ml.L, R, dptr<float2>(pm.down), pm.L, dptr<int2>(ml.down_win), dptr<int>(ml.parent), dptr<int>(ml.oct),
            dptr<float2>(pm.up_phase), dptr<int>(ml.th_ptr), dptr<int>(ml.th_src), dptr<float>(ml.th_w),
            dptr<int>(ml.ph_ptr), dptr<int>(ml.ph_src), dptr<float>(ml.ph_w), dptr<float2>(ml.down),
            (size_t)3 * ml.nbox * ml.K, (size_t)3 * pm.nbox * pm.K);
    }
    if (!fused)
        agg_disagg(M, false, x, nr, rb, y, parts, st);
    else if (rb == 1)
        EMFA_TRY(launch_finish<1>(M, x, nr, y, parts, st));
    else if (rb == 2)
        EMFA_TRY(launch_finish<2>(M, x, nr, y, parts, st));
    else if (rb == 4)
        EMFA_TRY(launch_finish<4>(M, x, nr, y, parts, st));
    else
        EMFA_TRY(launch_finish<8>(M, x, nr, y, parts, st));
    c->kernel_launches += (fused ? 0 : 1) + 2 * nl;
    EMFA_CUDA(c, cudaGetLastError());
    return EMFA_OK;
}

// MLFMA as a Krylov operator (iteration vectors complex64, box order)
// y = P x for n_rhs vectors
static emfa_status_t sai_apply(emfa_mlfma* M, const float2* x, float2* y, int nrhs, cudaStream_t st)
{
    for (int r = 0; r < nrhs; ++r)
        k_sai_apply<<<(M->n + 255) / 256, 256, 0, st>>>(dptr<int>(M->csr_ptr), dptr<int>(M->csr_col),
                                                          dptr<float2>(M->csr_val), x + (size_t)r * M->n, M->n,
                                                          y + (size_t)r * M->n);
    M->ctx->kernel_launches += nrhs;
    EMFA_CUDA(M->ctx, cudaGetLastError());
    return EMFA_OK;
}

struct MlfmaOp : LinOp {
    emfa_mlfma* M = nullptr;
    bool pre = false;  // left-preconditioned operator P Z
    emfa_status_t apply(Ctx*, const void* X, void* Y, int nrhs, cudaStream_t st) override
    {
        if (pre) {
            // P (Z x): one right-hand side at a time through the preconditioner's scratch
            for (int r = 0; r < nrhs; ++r) {
                EMFA_TRY(mlfma_apply(M, (const float2*)X + (size_t)r * n, dptr<float2>(M->pre_tmp), 1, st));
                EMFA_TRY(sai_apply(M, dptr<float2>(M->pre_tmp), (float2*)Y + (size_t)r * n, 1, st));
            }
            return EMFA_OK;
        }
        for (int r0 = 0; r0 < nrhs; r0 += RHS_CHUNK)
            EMFA_TRY(mlfma_apply(M, (const float2*)X + (size_t)r0 * n, (float2*)Y + (size_t)r0 * n,
                                 std::min(RHS_CHUNK, nrhs - r0), st));
        return EMFA_OK;
    }
    emfa_status_t residual(Ctx* c, const double2* X, const void* B, double2* R, int nrhs, float2* xt,
                           cudaStream_t st) override
    {
        const size_t tot = (size_t)n * nrhs;
        EMFA_TRY(M->tmp_out.bytes >= sizeof(float2) * tot ? EMFA_OK : M->tmp_out.alloc(c, sizeof(float2) * tot));
        k_f64_to_f32<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(X, xt, tot);
        EMFA_TRY(apply(c, xt, M->tmp_out.ptr, nrhs, st));
        k_resid_c64<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>((const float2*)B, dptr<float2>(M->tmp_out), R, tot);
        c->kernel_launches += 2;
        return EMFA_OK;
    }
};

}  // namespace emfa

using namespace emfa;

extern "C" {

emfa_status_t emfa_mlfma_create(emfa_ctx_t* ctx, emfa_geom_t* geom, const emfa_mlfma_params_t* p, emfa_mlfma_t** out)
{
    if (!ctx || !geom || !p || !out || !(p->freq > 0) || !(p->box_threshold > 0) ||
        (p->truncation != 0 && p->truncation != 1)) {
        set_error(ctx, "emfa_mlfma_create: bad arguments");
        return EMFA_ERR_INVALID;
    }
    EMFA_CUDA(ctx, cudaSetDevice(ctx->device));
    emfa_mlfma_t* M = new emfa_mlfma_t();
    M->ctx = ctx;
    M->geom = geom;
    M->p = *p;
    emfa_status_t s = mlfma_build(M, ctx->stream);
    if (s != EMFA_OK) {
        delete M;
        return s;
    }
    // the operator holds its geometry (and through it the context) until it
    // is destroyed, whatever order the caller closes them in
    geom_retain(geom);
    *out = M;
    return EMFA_OK;
}

emfa_status_t emfa_mlfma_plan(const double* verts_host, int n_vert, const int* rwg_host, int n_rwg,
                              const emfa_mlfma_params_t* p, int* levels, int* level_boxes, int level_cap, int* poles,
                              int* perm)
{
    if (!verts_host || !rwg_host || !p || n_vert <= 0 || n_rwg <= 0 || !levels) return EMFA_ERR_INVALID;
    if (p->truncation != 0 && p->truncation != 1) {
        set_global_error("emfa_mlfma_plan: truncation must be 0 or 1");
        return EMFA_ERR_INVALID;
    }
    std::vector<double> v(verts_host, verts_host + 3 * (size_t)n_vert);
    std::vector<int> r(rwg_host, rwg_host + 6 * (size_t)n_rwg);
    Plan P;
    std::string err;
    if (!build_plan(v, n_vert, r, n_rwg, *p, P, err)) {
        set_global_error("emfa_mlfma_plan: " + err);
        return EMFA_ERR_INVALID;
    }
    *levels = P.L;
    if (level_boxes) {
        if (level_cap < P.L + 1) return EMFA_ERR_INVALID;
        for (int l = 0; l <= P.L; ++l) level_boxes[l] = (int)P.lev[l].b.size();
    }
    if (poles)
        for (size_t i = 0; i < P.poles.size(); ++i) poles[i] = P.poles[i];
    if (perm) std::copy(P.perm.begin(), P.perm.end(), perm);
    return EMFA_OK;
}

emfa_status_t emfa_mlfma_destroy(emfa_mlfma_t* M)
{
    if (!M) return EMFA_ERR_INVALID;
    cudaSetDevice(M->ctx->device);
    cudaStreamSynchronize(M->ctx->stream);
    emfa::Geom* g = M->geom;
    delete M;
    geom_release(g);
    return EMFA_OK;
}

emfa_status_t emfa_mlfma_info(const emfa_mlfma_t* M, int* levels, int* level_boxes, int* poles, size_t* near_nnz,
                              int* perm)
{
    if (!M) return EMFA_ERR_INVALID;
    if (levels) *levels = M->levels;
    if (level_boxes) std::copy(M->level_boxes.begin(), M->level_boxes.end(), level_boxes);
    if (poles) std::copy(M->poles.begin(), M->poles.end(), poles);
    if (near_nnz) *near_nnz = M->nnz;
    if (perm) std::copy(M->perm.begin(), M->perm.end(), perm);
    return EMFA_OK;
}

emfa_status_t emfa_mlfma_apply_part(emfa_mlfma_t* M, const void* x_dev, void* y_dev, int part, void* stream)
{
    if (!M || !x_dev || !y_dev || part < 0 || part > 2) return EMFA_ERR_INVALID;
    Ctx* c = M->ctx;
    EMFA_CUDA(c, cudaSetDevice(c->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
    return mlfma_apply(M, (const float2*)x_dev, (float2*)y_dev, 1, st, part);
}

emfa_status_t emfa_mlfma_apply(emfa_mlfma_t* M, const void* x_dev, void* y_dev, int n_rhs, void* stream)
{
    if (!M || !x_dev || !y_dev || n_rhs <= 0) return EMFA_ERR_INVALID;
    Ctx* c = M->ctx;
    EMFA_CUDA(c, cudaSetDevice(c->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
    MlfmaOp A;
    A.M = M;
    A.n = M->n;
    A.prec = EMFA_F32;
    return A.apply(c, x_dev, y_dev, n_rhs, st);
}

emfa_status_t emfa_mlfma_fill_v(emfa_mlfma_t* M, const double* angles_host, int n_inc, void* V_dev, void* stream)
{
    if (!M || !angles_host || n_inc <= 0 || !V_dev) return EMFA_ERR_INVALID;
    Ctx* c = M->ctx;
    EMFA_CUDA(c, cudaSetDevice(c->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
    emfa_fill_params_t fp{EMFA_CFIE, EMFA_F32, M->p.freq, M->p.alpha, 0, 0, 0};
    DevBuf tmp;
    EMFA_TRY(tmp.alloc(c, sizeof(float2) * (size_t)M->n * n_inc));
    EMFA_TRY(launch_fill_v(c, M->geom, &fp, angles_host, n_inc, tmp.ptr, st));
    size_t tot = (size_t)M->n * n_inc;
    k_gather_c64<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(dptr<float2>(tmp), dptr<int>(M->perm_d), M->n, n_inc,
                                                                (float2*)V_dev);
    c->kernel_launches += 1;
    EMFA_CUDA(c, cudaGetLastError());
    EMFA_CUDA(c, cudaStreamSynchronize(st));
    return EMFA_OK;
}

emfa_status_t emfa_mlfma_solve(emfa_mlfma_t* M, const void* B_dev, int n_rhs, void* X_dev,
                               const emfa_solver_params_t* sp, emfa_solve_info_t* info, void* stream)
{
    if (!M || !B_dev || !X_dev || !sp || n_rhs <= 0 || !(sp->tol > 0)) return EMFA_ERR_INVALID;
    Ctx* c = M->ctx;
    EMFA_CUDA(c, cudaSetDevice(c->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
    MlfmaOp A;
    A.M = M;
    A.n = M->n;
    A.prec = EMFA_F32;
    A.pre = M->precond;
    const void* B = B_dev;
    if (M->precond) {  // V <- P V (MLFMA::iterativeSolve, MLFMA.cpp:407-408)
        const size_t bytes = sizeof(float2) * (size_t)M->n * n_rhs;
        if (M->pre_b.bytes < bytes) EMFA_TRY(M->pre_b.alloc(c, bytes));
        EMFA_TRY(sai_apply(M, (const float2*)B_dev, dptr<float2>(M->pre_b), n_rhs, st));
        B = M->pre_b.ptr;
    }
    return solve_op(c, A, B, n_rhs, X_dev, sp, info, st);
}

emfa_status_t emfa_mlfma_precond_csr(const emfa_mlfma_t* M, size_t* nnz, int* ptr_host, int* col_host,
                                     void* val_host)
{
    if (!M || !nnz) return EMFA_ERR_INVALID;
    *nnz = M->precond ? M->sai_nnz : 0;
    if (!M->precond || !ptr_host) return EMFA_OK;
    Ctx* c = M->ctx;
    EMFA_CUDA(c, cudaSetDevice(c->device));
    EMFA_CUDA(c, cudaStreamSynchronize(c->stream));
    EMFA_CUDA(c, cudaMemcpy(ptr_host, M->csr_ptr.ptr, sizeof(int) * (M->n + 1), cudaMemcpyDeviceToHost));
    if (col_host) EMFA_CUDA(c, cudaMemcpy(col_host, M->csr_col.ptr, sizeof(int) * M->sai_nnz, cudaMemcpyDeviceToHost));
    if (val_host)
        EMFA_CUDA(c, cudaMemcpy(val_host, M->csr_val.ptr, sizeof(float2) * M->sai_nnz, cudaMemcpyDeviceToHost));
    return EMFA_OK;
}

emfa_status_t emfa_mlfma_precond_lists(const emfa_mlfma_t* M, int* nbox, size_t* nrows, size_t* ncols, int* rptr,
                                       int* rows, int* cptr, int* cols, int* own)
{
    if (!M || !nbox || !nrows || !ncols) return EMFA_ERR_INVALID;
    *nbox = M->precond ? (int)M->sai_own.size() : 0;
    *nrows = M->sai_rows.size();
    *ncols = M->sai_cols.size();
    if (!M->precond) return EMFA_OK;
    if (rptr) std::copy(M->sai_rptr.begin(), M->sai_rptr.end(), rptr);
    if (rows) std::copy(M->sai_rows.begin(), M->sai_rows.end(), rows);
    if (cptr) std::copy(M->sai_cptr.begin(), M->sai_cptr.end(), cptr);
    if (cols) std::copy(M->sai_cols.begin(), M->sai_cols.end(), cols);
    if (own) std::copy(M->sai_own.begin(), M->sai_own.end(), own);
    return EMFA_OK;
}

emfa_status_t emfa_mlfma_unpermute(emfa_mlfma_t* M, const void* X_box_dev, int n_rhs, void* X_rwg_dev, void* stream)
{
    if (!M || !X_box_dev || !X_rwg_dev || n_rhs <= 0) return EMFA_ERR_INVALID;
    Ctx* c = M->ctx;
    EMFA_CUDA(c, cudaSetDevice(c->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
    size_t tot = (size_t)M->n * n_rhs;
    k_scatter_c128<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>((const double2*)X_box_dev, dptr<int>(M->perm_d),
                                                                  M->n, n_rhs, (double2*)X_rwg_dev);
    c->kernel_launches += 1;
    EMFA_CUDA(c, cudaGetLastError());
    EMFA_CUDA(c, cudaStreamSynchronize(st));
    return EMFA_OK;
}

}  // extern "C"
