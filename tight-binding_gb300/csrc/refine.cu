// refine.cu -- mixed-precision form: FP64-accurate refinement of FP32 eigenpairs
// of H x = lambda S x, and the Hellmann-Feynman products of both forms.
//
// Given FP32 eigenvectors X (S-orthonormal to FP32 accuracy) and eigenvalue
// estimates l~ of FP64 H, S:
//   1. Y_H = H X, Y_S = S X to FP64 accuracy on the bf16 tensor cores
//      (exact digit splitting, ozaki.cuh; X is first rounded to 24 bits below
//      each column's largest element so that the products are exact for the
//      X used by every later step), and the diagonals T_jj = x_j^H H x_j,
//      R_jj = x_j^H S x_j by FP64 dot products.
//   2. Clusters: Rayleigh quotients T_jj / R_jj closer than delta (a fraction
//      of the spectral span) are grouped; each cluster's block (T_c, R_c) is
//      solved exactly (Cholesky + complex Jacobi, FP64), giving a rotation U_c
//      (Rayleigh-Ritz inside the cluster) and the eigenvalues l_j.
//   3. In the rotated basis X' = X U (FP64) the residuals
//      r'_j = Y_H u_j - l_j Y_S u_j (FP64; u_j column j of the block-diagonal
//      U), and G' = X'^H r' as an FP32 GEMM: r' ~ 1e-6, so G'_ij =
//      T'_ij - l_j R'_ij is accurate to ~1e-13 and uses, for every column, the
//      same l_j as the gaps below.
//   4. One Newton-type correction of the whole basis (Ogita-Aishima): for i, j
//      in different clusters E_ij = G'_ij / (l_j - l_i), E_jj = (1 - R'_jj) / 2,
//      zero inside a cluster; the eigenvalue with its second-order term
//      l_j + sum_{i not in c(j)} |G'_ij|^2 / (l_j - l_i).  Because every G'_ij
//      carries the l_j of its own gap, E + E^H = -(R' - I) exactly to first
//      order, and the Gram matrix of X'(I + E) is I - F to second order with
//      F = E^H E + E E + E^H E^H; adding F / 2 to E leaves an S-orthonormality
//      error third order in E.  F's diagonal is summed over all i; its
//      off-diagonal, where the large (small-gap) entries of E meet, over the
//      sorted neighbours within REF_BAND positions.
//   5. Z = X' (I + E) in FP64 (X' in FP64, the small X' E in FP32), columns
//      reordered by ascending eigenvalue.
// One step takes FP32-level eigenpairs (errors ~1e-6 Ry) to eigenvalue errors
// far below 1e-9 Ry; the remaining error is third order in the FP32 error.
#include <cfloat>
#include "refine.cuh"
#include "refine_cut.h"
#include "gemm.cuh"
#include "ozaki.cuh"
#include "sums.cuh"
#include "nrltb.h"

namespace nrltb {

constexpr int REF_CMAX = 16;            // largest cluster solved exactly
constexpr double REF_DELTA_REL = 5e-5;  // cluster threshold, fraction of the spectral span
// second-order Gram terms: sorted neighbours within REF_BAND positions; REF_BT
// sorted positions per CTA
constexpr int REF_BAND = 16, REF_BT = 64, REF_BR = REF_BT + 2 * REF_BAND;

static inline size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

bool refine_available() { return true; }

size_t refine_work_bytes(int n, int batch)
{
    RefineWork w;
    refine_work_carve(w, nullptr, n, batch);
    return (size_t)(uintptr_t)w.cl + 256;
}

void refine_work_carve(RefineWork &w, void *base, int n, int batch)
{
    size_t off = 0, nn = (size_t)n * n * batch, nb = (size_t)n * batch;
    char *b = (char *)base;
    auto take = [&](size_t bytes) { void *p = b + off; off = al256(off + bytes); return p; };
    w.n = n; w.batch = batch;
    w.YH = (double2 *)take(sizeof(double2) * nn);                  // H X, later X'^H and E^H E + ...
    w.YS = (double2 *)take(sizeof(double2) * nn);                  // S X, later G'^H, E^H
    w.Xd = (double2 *)take(sizeof(double2) * nn);                  // X' = X U in FP64
    w.G = (float2 *)take(sizeof(float2) * nn);                     // X'^H r', later E + E^H
    w.U = (double2 *)take(sizeof(double2) * nb * REF_CMAX);       // per column: coefficients on its cluster
    w.Ef = (float2 *)take(sizeof(float2) * nn);                    // residuals r', later E
    w.Xr = (float2 *)take(sizeof(float2) * nn);                    // X' in FP32
    w.XE = (float2 *)take(sizeof(float2) * nn);
    w.Fb = (float2 *)take(sizeof(float2) * nb * (2 * REF_BAND + 1));   // band of the Gram term
    w.oz = take(ozaki_work_bytes(n, batch));
    w.lam = (double *)take(sizeof(double) * nb * 4);               // l | R'_jj | T_jj | R_jj
    w.cl = (int *)take(sizeof(int) * nb * 4);                      // ord | pos0 | size | rank
    if (!base) w.cl = (int *)(uintptr_t)off;
}

// ---- 1. accurate diagonals -------------------------------------------------
// T_jj = x_j^H (H x_j), R_jj = x_j^H (S x_j) in FP64; warp per column
__global__ void k_ref_diag(RefineWork w, const float2 *X)
{
    const int warp = (int)((blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    const int n = w.n;
    if (warp >= n * w.batch) return;
    const int b = warp / n, j = warp % n;
    const long off = (long)b * n * n + (long)j * n;
    double t = 0, r = 0;
    for (int i = lane; i < n; i += 32) {
        const float2 x = X[off + i];
        const double2 yh = w.YH[off + i], ys = w.YS[off + i];
        const double xr = f2d_exact(x.x), xi = f2d_exact(x.y);   // widened off the FP64 pipe
        t += xr * yh.x + xi * yh.y;
        r += xr * ys.x + xi * ys.y;
    }
    t = warp_sum(t);
    r = warp_sum(r);
    if (lane == 0) {
        const long nb = (long)n * w.batch;
        w.lam[2 * nb + (long)b * n + j] = t;
        w.lam[3 * nb + (long)b * n + j] = r;
    }
}

// ---- 2. clusters: one CTA per matrix ----------------------------------------

// the rank sort takes its keys from shared memory up to this order
constexpr int REF_KEYS_MAX = 24576;

__global__ void __launch_bounds__(1024) k_ref_clusters(RefineWork w, int *status)
{
    __shared__ double red[32];
    extern __shared__ unsigned long long cl_keys[];
    const int b = blockIdx.x, n = w.n, tid = threadIdx.x, nw = blockDim.x >> 5;
    const long nb = (long)n * w.batch;
    double *l1 = w.lam + (long)b * n, *r1 = w.lam + nb + (long)b * n;
    const double *tjj = w.lam + 2 * nb + (long)b * n, *rjj = w.lam + 3 * nb + (long)b * n;
    int *ord = w.cl + (long)b * n, *pos0 = w.cl + nb + (long)b * n;
    int *csz = w.cl + 2 * nb + (long)b * n;
    double lo = 1e300, hi = -1e300;
    for (int j = tid; j < n; j += blockDim.x) {
        const double v = tjj[j] / rjj[j];
        l1[j] = v;
        r1[j] = rjj[j];
        lo = fmin(lo, v);
        hi = fmax(hi, v);
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((tid & 31) == 0) red[tid >> 5] = lo;
    __syncthreads();
    if (tid == 0) { double m = red[0]; for (int q = 1; q < nw; ++q) m = fmin(m, red[q]); red[0] = m; }
    __syncthreads();
    lo = red[0];
    __syncthreads();
    if ((tid & 31) == 0) red[tid >> 5] = hi;
    __syncthreads();
    if (tid == 0) { double m = red[0]; for (int q = 1; q < nw; ++q) m = fmax(m, red[q]); red[0] = m; }
    __syncthreads();
    hi = red[0];
    // rank sort of the estimates (ties by index); the sorted values go to a
    // scratch copy (the first n doubles of this matrix's U, written only by the
    // Rayleigh-Ritz step that follows) so the serial pass below streams them
    double *srt = (double *)(w.U + (long)b * n * REF_CMAX);
    if (n <= REF_KEYS_MAX) {
        // integer keys in shared memory: the n^2 comparisons stay off the FP64 pipe
        for (int j = tid; j < n; j += blockDim.x) cl_keys[j] = ord_key(l1[j]);
        __syncthreads();
        for (int j = tid; j < n; j += blockDim.x) {
            const unsigned long long kv = cl_keys[j];
            int r = 0;
            for (int q = 0; q < n; ++q) {
                const unsigned long long ku = cl_keys[q];
                r += (ku < kv) || (ku == kv && q < j);
            }
            ord[r] = j;
            srt[r] = l1[j];
        }
    } else {
        for (int j = tid; j < n; j += blockDim.x) {
            const double v = l1[j];
            int r = 0;
            for (int q = 0; q < n; ++q) {
                const double u = l1[q];
                r += (u < v) || (u == v && q < j);
            }
            ord[r] = j;
            srt[r] = v;
        }
    }
    __syncthreads();
    if (tid == 0) {
        // clusters: runs of sorted estimates closer than delta; a run longer than
        // REF_CMAX is cut at its largest internal gap, recursively.  Cutting a
        // gap below 1e-7 of the span would separate numerically coincident
        // eigenvalues and is reported.
        const double span = fmax(hi - lo, 1e-300);
        const double delta = REF_DELTA_REL * span;
        int forced = 0, p0 = 0;
        for (int p = 1; p <= n; ++p) {
            if (p < n && srt[p] - srt[p - 1] < delta) continue;
            forced |= ref_cut(srt, p0, p, REF_CMAX, 1e-7 * span, ord, pos0, csz);
            p0 = p;
        }
        if (forced) status[b] = NRLTB_K_NOT_CONVERGED;
    }
}

// Double-float accumulator of exact products on the FP32 pipe: x * (yh + yl)
// with x, yh, yl floats; x * yh is split into its rounded value and rounding
// error (FMA), the rounded values are summed by Knuth's two-sum, and the
// errors and the small x * yl terms go into the low word.
struct DFAcc {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add_prod(float x, float yh, float yl)
    {
        // _rn intrinsics: no contraction into FMAs, which would break the
        // exactness of the product split and of the two-sum
        const float pr = __fmul_rn(x, yh);
        const float pe = fmaf(x, yh, -pr);
        const float s = __fadd_rn(hi, pr), bp = __fsub_rn(s, hi);
        const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(pr, bp));
        hi = s;
        lo += err + fmaf(x, yl, pe);
    }
    __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// ---- 2b. Rayleigh-Ritz inside each cluster: one CTA per cluster -------------
// The cluster block T_ab = x_a^H (H x_b), R_ab = x_a^H (S x_b) is formed with
// exact products in double-float (a warp per entry); one warp then solves the
// pencil in FP64.  Column j's rotation is stored as w.U[j*CMAX + a], its
// coefficient on the cluster's a-th member (sorted position pos0 + a); the
// members' eigenvalues replace the estimates and their R'_jj becomes 1.
__global__ void __launch_bounds__(REF_CMAX * REF_CMAX) k_ref_rr(RefineWork w, const float2 *X)
{
    __shared__ double2 A[REF_CMAX][REF_CMAX + 1];   // A[col][row]
    __shared__ double2 Bm[REF_CMAX][REF_CMAX + 1];
    __shared__ double2 Vv[REF_CMAX][REF_CMAX + 1];
    const int b = blockIdx.y, p = blockIdx.x, n = w.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long nb = (long)n * w.batch;
    const int *ord = w.cl + (long)b * n, *pos0 = w.cl + nb + (long)b * n;
    const int *csz = w.cl + 2 * nb + (long)b * n;
    const int j0 = ord[p];
    if (pos0[j0] != p) return;                       // not the first member of its cluster
    const int c = csz[j0];
    double2 *U = w.U + (long)b * n * REF_CMAX;
    if (c == 1) {
        if (tid == 0) U[(long)j0 * REF_CMAX] = make_double2(1.0, 0.0);
        return;
    }
    const long mo = (long)b * n * n;
    // T_rq = x_r^H (H x_q), R_rq = x_r^H (S x_q), r <= q (Hermitian blocks: the
    // other triangle is the conjugate).  A warp per entry, its lanes over the
    // rows; the products of the FP32 x with the FP64 H x, S x are formed
    // exactly on the FP32 pipe (the FP64 factor split into two floats, the
    // leading product's rounding error recovered by an FMA) and summed in
    // double-float (Knuth's two-sum): ~2^-46 relative; the FP64 pipe takes
    // only the split's exact remainder.
    const int ne = c * (c + 1) / 2, nwarps = blockDim.x >> 5;
    for (int e = warp; e < ne; e += nwarps) {
        int q = 0, rem = e;
        while (rem > q) { rem -= q + 1; ++q; }
        const int r = rem;
        const float2 *xr = X + mo + (long)ord[p + r] * n;
        const double2 *hq = w.YH + mo + (long)ord[p + q] * n, *sq = w.YS + mo + (long)ord[p + q] * n;
        DFAcc tre, tim, rre, rim;
        for (int i = lane; i < n; i += 32) {
            const float2 x = xr[i];
            const double2 h = hq[i], sv = sq[i];
            // (conversions with integer operations: only the exact remainders
            // take the FP64 pipe)
            const float2 hh = make_float2(d2f_rn(h.x), d2f_rn(h.y)), sh = make_float2(d2f_rn(sv.x), d2f_rn(sv.y));
            const float2 hl = make_float2(d2f_rn(h.x - f2d_exact(hh.x)), d2f_rn(h.y - f2d_exact(hh.y)));
            const float2 sl = make_float2(d2f_rn(sv.x - f2d_exact(sh.x)), d2f_rn(sv.y - f2d_exact(sh.y)));
            // conj(x) y = (xr yr + xi yi) + i (xr yi - xi yr)
            tre.add_prod(x.x, hh.x, hl.x); tre.add_prod(x.y, hh.y, hl.y);
            tim.add_prod(x.x, hh.y, hl.y); tim.add_prod(-x.y, hh.x, hl.x);
            rre.add_prod(x.x, sh.x, sl.x); rre.add_prod(x.y, sh.y, sl.y);
            rim.add_prod(x.x, sh.y, sl.y); rim.add_prod(-x.y, sh.x, sl.x);
        }
        const double2 t = make_double2(warp_sum(tre.value()), warp_sum(tim.value()));
        const double2 u = make_double2(warp_sum(rre.value()), warp_sum(rim.value()));
        if (lane == 0) {
            A[q][r] = t;
            Bm[q][r] = u;
            A[r][q] = cconj(t);
            Bm[r][q] = cconj(u);
        }
    }
    __syncthreads();
    if (warp != 0) return;
    __syncwarp();
    // Hermitian by construction up to rounding: symmetrise (lanes over entries)
    for (int e = lane; e < c * c; e += 32) {
        const int r = e % c, q = e / c;
        if (r < q) continue;
        const double2 a = cscale(cadd(A[q][r], cconj(A[r][q])), 0.5), bm = cscale(cadd(Bm[q][r], cconj(Bm[r][q])), 0.5);
        A[q][r] = a; A[r][q] = cconj(a);
        Bm[q][r] = bm; Bm[r][q] = cconj(bm);
    }
    __syncwarp();
    // Cholesky Bm = L L^H (lower, in place; Bm[q][r] = element (r, q)),
    // left-looking: lane r forms element (r, k) of column k
    for (int k = 0; k < c; ++k) {
        double2 s2 = make_double2(0, 0);
        if (lane >= k && lane < c) {
            s2 = Bm[k][lane];
            for (int q = 0; q < k; ++q) s2 = csub(s2, cmul(Bm[q][lane], cconj(Bm[q][k])));
        }
        if (lane == k) Bm[k][k] = make_double2(sqrt(fmax(s2.x, 1e-300)), 0.0);
        __syncwarp();
        if (lane > k && lane < c) Bm[k][lane] = cscale(s2, 1.0 / Bm[k][k].x);
        __syncwarp();
    }
    // A <- L^{-1} A (lane per column), then A <- A L^{-H} (lane per row)
    if (lane < c) {
        const int q = lane;
        for (int r = 0; r < c; ++r) {
            double2 s2 = A[q][r];
            for (int t = 0; t < r; ++t) s2 = csub(s2, cmul(Bm[t][r], A[q][t]));
            A[q][r] = cscale(s2, 1.0 / Bm[r][r].x);
        }
    }
    __syncwarp();
    if (lane < c) {
        const int r = lane;
        for (int q = 0; q < c; ++q) {
            double2 s2 = A[q][r];
            for (int t = 0; t < q; ++t) s2 = csub(s2, cmul(A[t][r], cconj(Bm[t][q])));
            A[q][r] = cscale(s2, 1.0 / Bm[q][q].x);
        }
    }
    for (int e = lane; e < c * c; e += 32) {
        const int r = e % c, q = e / c;
        Vv[q][r] = make_double2(r == q ? 1.0 : 0.0, 0.0);
    }
    __syncwarp();
    // parallel complex Jacobi on the Hermitian A, accumulating V: a sweep is
    // c' - 1 steps of c'/2 disjoint pairs (round-robin: position 0 fixed, the
    // others rotating; c' = c rounded up to even, pairs with the extra
    // position skipped).  A step's rotations come from the same A; all their
    // column rotations (A J, V J) are applied, then all row rotations (J^H A).
    __shared__ double2 rot[REF_CMAX / 2][2];   // (cs, sn), phase conj(g) / |g| of each pair
    __shared__ int rpair[REF_CMAX / 2][2];
    const int ce = c + (c & 1), m = ce - 1, np = ce / 2;
    for (int sweep = 0; sweep < 30; ++sweep) {
        double offd = 0, dsum = 0;
        for (int e = lane; e < c * c; e += 32) {
            const int r = e % c, q = e / c;
            if (r != q) offd += A[q][r].x * A[q][r].x + A[q][r].y * A[q][r].y;
            else dsum += A[q][r].x * A[q][r].x;
        }
        offd = warp_sum(offd);
        dsum = warp_sum(dsum);
        if (!(offd > 1e-32 * dsum)) break;
        for (int st = 0; st < m; ++st) {
            if (lane < np) {
                int pa, pb;
                if (lane == 0) { pa = 0; pb = 1 + st % m; }
                else { pa = 1 + (st + lane) % m; pb = 1 + (st - lane + m) % m; }
                const int pp = min(pa, pb), qq = max(pa, pb);
                int live = qq < c;
                double2 cssn = make_double2(1.0, 0.0), phc = make_double2(1.0, 0.0);
                if (live) {
                    const double2 g = A[qq][pp];            // element (pp, qq)
                    const double ag = sqrt(g.x * g.x + g.y * g.y);
                    if (ag > 1e-300) {
                        const double app = A[pp][pp].x, aqq = A[qq][qq].x;
                        const double tau = (aqq - app) / (2.0 * ag);
                        const double t = (tau >= 0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
                        const double cs = 1.0 / sqrt(1.0 + t * t);
                        // J = diag(1, e^{-i phi}) [[cs, sn], [-sn, cs]], g = |g| e^{i phi}
                        cssn = make_double2(cs, t * cs);
                        phc = make_double2(g.x / ag, -g.y / ag);
                    } else {
                        live = 0;
                    }
                }
                rot[lane][0] = cssn;
                rot[lane][1] = phc;
                rpair[lane][0] = pp;
                rpair[lane][1] = live ? qq : -1;
            }
            __syncwarp();
            // A J and V J: columns pp, qq of every live pair, all rows
            for (int e = lane; e < np * c; e += 32) {
                const int pr = e / c, r = e % c, qq = rpair[pr][1];
                if (qq < 0) continue;
                const int pp = rpair[pr][0];
                const double cs = rot[pr][0].x, sn = rot[pr][0].y;
                const double2 phc = rot[pr][1];
                const double2 ap = A[pp][r], aq = cmul(A[qq][r], phc);
                A[pp][r] = csub(cscale(ap, cs), cscale(aq, sn));
                A[qq][r] = cadd(cscale(ap, sn), cscale(aq, cs));
                const double2 vp = Vv[pp][r], vq = cmul(Vv[qq][r], phc);
                Vv[pp][r] = csub(cscale(vp, cs), cscale(vq, sn));
                Vv[qq][r] = cadd(cscale(vp, sn), cscale(vq, cs));
            }
            __syncwarp();
            // J^H A: rows pp, qq of every live pair, all columns
            for (int e = lane; e < np * c; e += 32) {
                const int pr = e / c, q = e % c, qq = rpair[pr][1];
                if (qq < 0) continue;
                const int pp = rpair[pr][0];
                const double cs = rot[pr][0].x, sn = rot[pr][0].y;
                const double2 ph = cconj(rot[pr][1]);
                const double2 ap = A[q][pp], aq = cmul(A[q][qq], ph);
                A[q][pp] = csub(cscale(ap, cs), cscale(aq, sn));
                A[q][qq] = cadd(cscale(ap, sn), cscale(aq, cs));
            }
            __syncwarp();
            if (lane < np && rpair[lane][1] >= 0) {
                const int pp = rpair[lane][0], qq = rpair[lane][1];
                A[qq][pp] = make_double2(0, 0);
                A[pp][qq] = make_double2(0, 0);
                A[pp][pp].y = 0;
                A[qq][qq].y = 0;
            }
            __syncwarp();
        }
    }
    __syncwarp();
    // eigenvectors of the pencil: x = L^{-H} y (lane per column)
    if (lane < c) {
        const int q = lane;
        for (int r = c - 1; r >= 0; --r) {
            double2 s2 = Vv[q][r];
            for (int t = r + 1; t < c; ++t) s2 = csub(s2, cmul(cconj(Bm[r][t]), Vv[q][t]));
            Vv[q][r] = cscale(s2, 1.0 / Bm[r][r].x);
        }
    }
    __syncwarp();
    for (int e = lane; e < c * c; e += 32) {
        const int a = e % c, q = e / c;
        U[(long)ord[p + q] * REF_CMAX + a] = Vv[q][a];
    }
    for (int q = lane; q < c; q += 32) {
        const int j = ord[p + q];
        w.lam[(long)b * n + j] = A[q][q].x;        // Rayleigh-Ritz eigenvalue
        w.lam[nb + (long)b * n + j] = 1.0;         // R'_jj
    }
}

#define REF_VIEWS                                                              \
    const long nb = (long)n * w.batch;                                         \
    const int *ord = w.cl + (long)b * n, *pos0 = w.cl + nb + (long)b * n;      \
    const int *csz = w.cl + 2 * nb + (long)b * n;                              \
    const double2 *U = w.U + (long)b * n * REF_CMAX;

// 3. X' = X U in FP64 (Xd) and FP32 (Xr), and the residuals of the rotated
// basis r'_j = sum_a (Y_H[:, m_a] - l_j Y_S[:, m_a]) U_aj in FP64 (into Ef as
// FP32), m_a the members of column j's cluster; thread per element.  part:
// 0 every column, 1 the columns outside clusters (U not read), 2 the rest.
__global__ void k_ref_rotres(RefineWork w, const float2 *X, int part)
{
    const int n = w.n;
    const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    const long nn = (long)n * n;
    if (t >= nn * w.batch) return;
    const int b = (int)(t / nn);
    const long e = t - b * nn;
    const int r = (int)(e % n), j = (int)(e / n);
    REF_VIEWS
    const long mo = b * nn;
    if ((part == 1 && csz[j] != 1) || (part == 2 && csz[j] == 1)) return;
    const double l = w.lam[(long)b * n + j];
    double2 v, res;
    float2 xr;
    if (csz[j] == 1) {
        // the FP32 vector itself: widened with integer operations (exact) and
        // kept as it is for the FP32 copy, so that only the residual uses the
        // FP64 pipe
        xr = X[mo + r + (long)j * n];
        v = make_double2(f2d_exact(xr.x), f2d_exact(xr.y));
        const double2 yh = w.YH[t], ys = w.YS[t];
        res = make_double2(yh.x - l * ys.x, yh.y - l * ys.y);
    } else {
        v = make_double2(0, 0);
        double2 h = make_double2(0, 0), sx = make_double2(0, 0);
        for (int a = 0; a < csz[j]; ++a) {
            const long src = mo + r + (long)ord[pos0[j] + a] * n;
            const double2 u = U[(long)j * REF_CMAX + a];
            const float2 x = X[src];
            v = cadd(v, cmul(make_double2(f2d_exact(x.x), f2d_exact(x.y)), u));
            h = cadd(h, cmul(w.YH[src], u));
            sx = cadd(sx, cmul(w.YS[src], u));
        }
        res = make_double2(h.x - l * sx.x, h.y - l * sx.y);
        xr = make_float2(d2f_rn(v.x), d2f_rn(v.y));
    }
    w.Xd[t] = v;
    w.Xr[t] = xr;
    w.Ef[t] = make_float2(d2f_rn(res.x), d2f_rn(res.y));
}

// 4. E column j and the second-order eigenvalue term (warp per column), from
// G' (column j) and Gt = G'^H (column j = the conjugate of row j of G').  The
// gaps l_j - l_i are formed in FP64; E and the second-order terms (products of
// residual-sized FP32 entries) in FP32.  Also the diagonal of the second-order
// Gram term F = E^H (E + E^H) + E E over all i, F_jj = sum_i |E_ij|^2 +
// 2 Re(E_ij E_ji), into lam[3 nb ..] (the R_jj slots, no longer read); the
// refined eigenvalues go to lam[2 nb ..] (the T_jj slots).
__global__ void k_ref_update(RefineWork w, const float2 *Gt)
{
    const int warp = (int)((blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    const int n = w.n;
    if (warp >= n * w.batch) return;
    const int b = warp / n, j = warp % n;
    const long mo = (long)b * n * n;
    const long nb = (long)n * w.batch;
    const int *pos0 = w.cl + nb + (long)b * n;
    const double *l1 = w.lam + (long)b * n;
    const double lj = l1[j], rjj = w.lam[nb + (long)b * n + j];
    const int pj = pos0[j];
    float corr = 0.f, fjj = 0.f;
    float2 *E = w.Ef + mo + (long)j * n;
    const float2 *Gj = w.G + mo + (long)j * n, *Gtj = Gt + mo + (long)j * n;
    for (int i = lane; i < n; i += 32) {
        float2 e;
        if (i == j) {
            const float ed = (float)(0.5 * (1.0 - rjj));
            e = make_float2(ed, 0.f);
            fjj += 3.f * ed * ed;
        } else if (pos0[i] == pj) {
            e = make_float2(0.f, 0.f);
        } else {
            const float2 g = Gj[i], gt = Gtj[i];
            const float rden = 1.f / d2f_rn(lj - l1[i]);   // FP64 gap, rounded off the FP64 pipe
            e = make_float2(g.x * rden, g.y * rden);
            // E_ji = G'_ji / (l_i - l_j) = -conj(Gt_ij) rden
            const float2 c = make_float2(-gt.x * rden, gt.y * rden);
            fjj += e.x * e.x + e.y * e.y + 2.f * (e.x * c.x - e.y * c.y);
            corr += (g.x * g.x + g.y * g.y) * rden;
        }
        E[i] = e;
    }
    corr = warp_sum(corr);
    fjj = warp_sum(fjj);
    if (lane == 0) {
        w.lam[2 * nb + (long)b * n + j] = lj + (double)corr;
        w.lam[3 * nb + (long)b * n + j] = (double)fjj;
    }
}

// 4b. Off-diagonal second-order Gram terms near the diagonal of the sorted
// spectrum.  F_ij = sum_k conj(E_ki) (E_kj + conj(E_jk)) + E_ik E_kj is
// formed for the sorted neighbours i of j within REF_BAND positions, summing
// over the k within REF_BAND positions of j: the large entries of E, those of
// small gaps, all lie there (away from it |E| ~ |r| / gap is ~1e-7 and its
// products ~1e-13).  A CTA takes REF_BT consecutive sorted positions and
// gathers the (REF_BT + 2 REF_BAND)^2 block of E they need into shared memory
// (sorted coordinates); output Fb[b][j][d + REF_BAND] for i = ord[pos(j) + d].
constexpr int REF_BAND_SMEM = REF_BR * REF_BR * (int)sizeof(float2);

__global__ void __launch_bounds__(256) k_ref_band(RefineWork w, float2 *Fb)
{
    extern __shared__ float2 eb[];   // eb[c * REF_BR + r] = E[ord[q0 + r], ord[q0 + c]]
    const int n = w.n, b = blockIdx.y, p0 = blockIdx.x * REF_BT, q0 = p0 - REF_BAND, tid = threadIdx.x;
    const long mo = (long)b * n * n;
    const int *ord = w.cl + (long)b * n;
    const float2 *E = w.Ef + mo;
    for (int t = tid; t < REF_BR * REF_BR; t += blockDim.x) {
        const int c = t / REF_BR, r = t - c * REF_BR, qc = q0 + c, qr = q0 + r;
        float2 v = make_float2(0.f, 0.f);
        if (qc >= 0 && qc < n && qr >= 0 && qr < n) v = E[(long)ord[qr] + (long)ord[qc] * n];
        eb[t] = v;
    }
    __syncthreads();
    constexpr int W = 2 * REF_BAND + 1;
    for (int t = tid; t < REF_BT * W; t += blockDim.x) {
        const int pl = t / W, d = t - pl * W - REF_BAND;
        const int p = p0 + pl;
        if (p >= n) continue;
        const int cj = pl + REF_BAND, ci = cj + d;        // local sorted coordinates of j and i
        float2 f = make_float2(0.f, 0.f);
        if (d != 0 && p + d >= 0 && p + d < n) {
            for (int ck = cj - REF_BAND; ck <= cj + REF_BAND; ++ck) {
                const float2 eki = eb[ci * REF_BR + ck], ekj = eb[cj * REF_BR + ck];
                const float2 ejk = eb[ck * REF_BR + cj], eik = eb[ck * REF_BR + ci];
                const float2 pkj = make_float2(ekj.x + ejk.x, ekj.y - ejk.y);
                cfmac(f, eki, pkj);
                cfma(f, eik, ekj);
            }
        }
        Fb[((long)b * n + ord[p]) * W + d + REF_BAND] = f;
    }
}

// 4c. E += F / 2 on the band and the diagonal (thread per band entry)
__global__ void k_ref_band_apply(RefineWork w, const float2 *Fb)
{
    constexpr int W = 2 * REF_BAND + 1;
    const int n = w.n;
    const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (t >= (long)n * w.batch * W) return;
    const int d = (int)(t % W) - REF_BAND;
    const long bp = t / W;
    const int b = (int)(bp / n), p = (int)(bp - (long)b * n);   // sorted position p
    const long nb = (long)n * w.batch;
    const int *ord = w.cl + (long)b * n;
    const int j = ord[p];
    float2 *E = w.Ef + (long)b * n * n;
    if (d == 0) {
        E[j + (long)j * n].x += 0.5f * (float)w.lam[3 * nb + (long)b * n + j];
    } else if (p + d >= 0 && p + d < n) {
        const float2 f = Fb[((long)b * n + j) * W + d + REF_BAND];
        float2 &e = E[ord[p + d] + (long)j * n];
        e.x += 0.5f * f.x;
        e.y += 0.5f * f.y;
    }
}

// 5a. ascending order of the refined eigenvalues
__global__ void k_ref_rank(RefineWork w, const double *l2, double *eig, int keys)
{
    extern __shared__ unsigned long long rank_keys[];
    const int b = blockIdx.y, n = w.n;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const double *L = l2 + (long)b * n;
    const int r = rank_of(L, n, j, keys ? rank_keys : nullptr);
    if (j >= n) return;
    w.cl[(long)3 * n * w.batch + (long)b * n + j] = r;
    eig[(long)b * n + r] = L[j];
}

// 5b. Z[:, rank(j)] = X'[:, j] + (X' E)[:, j]
__global__ void k_ref_finish(RefineWork w, double2 *Z)
{
    const int n = w.n;
    const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    const long nn = (long)n * n;
    if (t >= nn * w.batch) return;
    const int b = (int)(t / nn);
    const long e = t - b * nn;
    const int r = (int)(e % n), j = (int)(e / n);
    const int dst = w.cl[(long)3 * n * w.batch + (long)b * n + j];
    const double2 x = w.Xd[t];
    const float2 d = w.XE[t];
    Z[b * nn + r + (long)dst * n] = make_double2(x.x + f2d_exact(d.x), x.y + f2d_exact(d.y));
}

void refine_eigen(cudaStream_t s, RefineWork &w, const double2 *H, const double2 *S, float2 *X,
                  double *eig, double2 *Z, int *status, const OzakiA *pre, const RefAux *ra)
{
    const int n = w.n, B = w.batch;
    const long nn = (long)n * n, nb = (long)n * B;
    const float2 onef = make_float2(1.f, 0.f), zerof = make_float2(0.f, 0.f);
    // 1. H X, S X (tensor cores, FP64-accurate), accurate diagonals
    const OzakiX ox = ozaki_prepare_x(s, X, n, B, w.oz);
    if (pre) {
        ozaki_gemm_prepared(s, ox, pre[0], w.YH);
        ozaki_gemm_prepared(s, ox, pre[1], w.YS);
    } else {
        ozaki_gemm(s, ox, H, w.YH);
        ozaki_gemm(s, ox, S, w.YS);
    }
    NRLTB_LAUNCH(k_ref_diag, cdiv(nb * 32, 256), 256, 0, s, w, X);
    // 2. clusters and their Rayleigh-Ritz rotations
    const size_t csm = n <= REF_KEYS_MAX ? sizeof(unsigned long long) * n : 0;
    if (csm > 48 * 1024) smem_attr_at_least((const void *)k_ref_clusters, (int)csm);
    NRLTB_LAUNCH(k_ref_clusters, B, 1024, csm, s, w, status);
    // 3. rotated basis, its residuals, G' = X'^H r' (X'^H formed explicitly in
    //    the YH area, free from here on: the tensor-core GEMM streams an A
    //    operand in its stored orientation twice as fast).  With a second
    //    stream the columns outside clusters are done there while the cluster
    //    solves (a few long CTAs for the largest clusters) run here.
    if (ra && ra->aux && ra->ev_a && ra->ev_b) {
        cudaEventRecord(ra->ev_a, s);
        cudaStreamWaitEvent(ra->aux, ra->ev_a, 0);
        NRLTB_LAUNCH(k_ref_rotres, cdiv(nn * B, 256), 256, 0, ra->aux, w, X, 1);
        cudaEventRecord(ra->ev_b, ra->aux);
        NRLTB_LAUNCH(k_ref_rr, dim3(n, B), REF_CMAX * REF_CMAX, 0, s, w, X);
        NRLTB_LAUNCH(k_ref_rotres, cdiv(nn * B, 256), 256, 0, s, w, X, 2);
        cudaStreamWaitEvent(s, ra->ev_b, 0);
    } else {
        NRLTB_LAUNCH(k_ref_rr, dim3(n, B), REF_CMAX * REF_CMAX, 0, s, w, X);
        NRLTB_LAUNCH(k_ref_rotres, cdiv(nn * B, 256), 256, 0, s, w, X, 0);
    }
    float2 *T1 = (float2 *)w.YH, *T2 = (float2 *)w.YS;
    conj_transpose<float>(s, w.Xr, T1, n, B);
    zgemm<float>(s, n, n, n, B, onef, T1, n, nn, 0, w.Ef, n, nn, 0, zerof, w.G, n, nn);
    // 4. E and the second-order Gram term F = E^H (E + E^H) + E E: its
    //    diagonal over all i, its off-diagonal on the band of near neighbours
    conj_transpose<float>(s, w.G, T2, n, B);
    NRLTB_LAUNCH(k_ref_update, cdiv(nb * 32, 256), 256, 0, s, w, T2);
    smem_attr_at_least((const void *)k_ref_band, REF_BAND_SMEM);
    NRLTB_LAUNCH(k_ref_band, dim3(cdiv(n, REF_BT), B), 256, REF_BAND_SMEM, s, w, w.Fb);
    NRLTB_LAUNCH(k_ref_band_apply, cdiv(nb * (2 * REF_BAND + 1), 256), 256, 0, s, w, w.Fb);
    // 5. Z = X' + X' E, reordered
    zgemm<float>(s, n, n, n, B, onef, w.Xr, n, nn, 0, w.Ef, n, nn, 0, zerof, w.XE, n, nn);
    const double *l2 = w.lam + 2 * nb;
    const size_t rsm = rank_keys_bytes(n);
    if (rsm > 48 * 1024) smem_attr_at_least((const void *)k_ref_rank, (int)rsm);
    NRLTB_LAUNCH(k_ref_rank, dim3(cdiv(n, 128), B), 128, rsm, s, w, l2, eig, rsm > 0 ? 1 : 0);
    if (Z) NRLTB_LAUNCH(k_ref_finish, cdiv(nn * B, 256), 256, 0, s, w, Z);
}

size_t hf_scratch_bytes(int n, int nkc)
{
    // FP64 form: P, Q (2 n^2 double2); mixed form: P, Q, Z as float2 and the
    // digit planes of the tensor-core products
    const size_t nn = (size_t)n * n * nkc;
    return al256(2 * sizeof(double2) * nn) + al256(sizeof(float2) * nn) + ozaki_work_bytes(n, nkc) + 512;
}

__global__ void k_to_f32(const double2 *src, float2 *dst, long count)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < count; i += (long)gridDim.x * blockDim.x) {
        const double2 v = src[i];
        dst[i] = make_float2(d2f_rn(v.x), d2f_rn(v.y));
    }
}
void launch_to_f32(cudaStream_t s, const double2 *src, float2 *dst, long count)
{
    NRLTB_LAUNCH(k_to_f32, 1184, 256, 0, s, src, dst, count);
}

int run_hf(cudaStream_t s, int n, int nkc, int prec, const double2 *dH, const double2 *dS, const double2 *Z,
           const double *eig, double *deig, void *scratch, const OzakiA *pre, const ZScratch &zs)
{
    const long nn = (long)n * n;
    double2 *P = (double2 *)scratch;
    double2 *Q = (double2 *)((char *)scratch + al256(sizeof(double2) * nn * nkc));
    if (prec == NRLTB_PREC_FP64) {
        const double2 one = make_double2(1, 0), zero = make_double2(0, 0);
        // P = triu(dH) Z, Q = triu(dS) Z
        zgemm<double>(s, n, n, n, nkc, one, dH, n, nn, 0, Z, n, nn, 0, zero, P, n, nn, 2, 0, 0, zs);
        zgemm<double>(s, n, n, n, nkc, one, dS, n, nn, 0, Z, n, nn, 0, zero, Q, n, nn, 2, 0, 0, zs);
        launch_hf_dots(s, Z, P, Q, dH, dS, eig, deig, n, nkc);
    } else {
        // Mixed form: P = dH Z', Q = dS Z' by the tensor-core digit product with
        // dH, dS rounded to 24 bits of their row scale (3 digits) and Z' = Z
        // rounded to 24 bits of its column scale, every digit pair kept: the
        // exact product of the rounded operands, so no accumulation bias (a
        // biased FP32 accumulation, as in the tensor cores' own, of ~1e-6
        // relative in P shifts the pressure coherently by ~1e-7 Ry/bohr^3);
        // then deig = Re(z^H P) - e Re(z^H Q) with FP64 Z and sums.  The
        // pressure error stays ~1e-10 Ry/bohr^3 per k against the 1e-3 kbar
        // (6.8e-9) tolerance.
        float2 *z32 = (float2 *)((char *)Q + al256(sizeof(double2) * nn * nkc));
        void *oz = (char *)z32 + al256(sizeof(float2) * nn * nkc);
        launch_to_f32(s, Z, z32, nn * nkc);
        const OzakiX ox = ozaki_prepare_x(s, z32, n, nkc, oz);
        if (pre) {
            ozaki_gemm_prepared(s, ox, pre[0], P);
            ozaki_gemm_prepared(s, ox, pre[1], Q);
        } else {
            ozaki_gemm(s, ox, dH, P, 3);
            ozaki_gemm(s, ox, dS, Q, 3);
        }
        launch_hf_dots_full(s, Z, P, Q, eig, deig, n, nkc);
    }
    return cudaGetLastError() == cudaSuccess ? NRLTB_OK : NRLTB_E_CUDA;
}

}  // namespace nrltb
