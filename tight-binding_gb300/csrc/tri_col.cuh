// tri_col.cuh -- one column of the blocked Householder tridiagonalisation
// (zhetrd/zlatrd steps) in two launches over the whole GPU.  The FP64 form takes
// this path down to its last 192 columns (its mat-vec is bound by the FP64 pipe, so every
// SM must work on every column; the rest: tri_cluster.cuh); the FP32 form where a cluster panel (tri_panel.cuh) cannot be scheduled.
//
//   k_tri_col  finishes W of the column before (w = w' + alpha v) and updates column
//              i:  a_i - V W[i,:]^H - W V[i,:]^H, with per-CTA partials of |a_i|^2.
//   k_tri_mv   derives the reflector from those partials (every CTA, same order),
//              then forms y = A v of the trailing matrix, W^H v and V^H v, and v^H y.
// alpha needs w'^H v over all rows, w' = tau (y - V (W^H v) - W (V^H v)).  With
// p1 = W^H v and p2 = V^H v it is conj(tau) (y^H v - 2 Re p1^H p2), so the sums that
// k_tri_mv leaves suffice and no third pass over the rows is needed.
//
// Every sum is per-CTA partials added by their reader in a fixed order that
// depends on n and i alone: results do not depend on the batch or on scheduling.
//
// y reads only A's lower triangle.  A warp takes 32 x 32 tiles (R, S) of the
// trailing matrix: S < R as it is (lane = row), S > R through the lower tile (S, R),
// transposed in shared memory sixteen columns at a time so that its conjugate
// products, too, are summed by a lane each (a shuffle reduction would add half as
// many FP64 operations again).  The tiles of a row block make one to a few CTAs, so
// each SM has many independent tiles whose loads are in flight together.
// Bound: the FP64 pipe (4 FMAs per element of the full trailing matrix: 12 us a
// column on average for 4 k at N = 1152, 76 for 27 k), for small batches the launches.
// The pipe also sets the shape of the rest: k_tri_col splits the panel's columns over
// the four warps of a 32-row CTA, so that 4 k already reach every SM, and the
// reflector's scalars take one root and two reciprocals per CTA.
// Against four launches per column (column update, dots, mat-vec, w update; the
// mat-vec walked all column tiles per row block in one CTA): N = 1152, 4 k 106 -> 42 us a
// column (61 in the first, 12 in the last), N = 288, 64 k 84 -> 51 us.
#pragma once
#include "eig.cuh"
#include "tri_panel.cuh"

namespace nrltb {

constexpr int TC_ROWS = 128;    // rows of k_tri_mv's dot blocks
constexpr int TC_WARPS = 8;     // warps of k_tri_mv; a CTA takes up to 16 tiles of a row block

// partials of one matrix (in w.part, tc_part_count(n) elements): |a_i|^2 of each CTA,
// W^H v | V^H v of each row block, v^H y of each tile CTA; y itself per split in w.yp
struct TcSizes {
    int m, ncol, nsp, nrb;   // trailing order, its 32-row blocks, CTAs per block, 128-row blocks
    __host__ __device__ explicit TcSizes(int m_) : m(m_)
    {
        ncol = (m + 31) / 32;
        nsp = (ncol + 2 * TC_WARPS - 1) / (2 * TC_WARPS);
        nrb = (m + TC_ROWS - 1) / TC_ROWS;
    }
};
__host__ __device__ inline int tc_part_norm(int n) { return (n + 31) / 32; }
inline size_t tc_part_count(int n)
{
    const TcSizes z(n);
    return (size_t)tc_part_norm(n) + (size_t)z.nrb * 2 * EIG_NB + (size_t)z.ncol * z.nsp;
}
inline size_t tc_y_count(int n) { return (size_t)TcSizes(n).nsp * n; }

// Roots and reciprocals that one thread needs before others can go on.  A warp's FP64
// operation takes 64 cycles of its quarter's pipe, so the library's forms (25 of them
// and more) are a microsecond and more of latency; these start from the FP32 result
// (of the argument with its exponent taken out) and take two steps of Newton's
// iteration, relative errors 2^-22 -> 2^-43 -> FP64 rounding (a few 2^-53).
__device__ __forceinline__ double tc_recip(double x)
{
    const int e = ((__double2hiint(x) >> 20) & 0x7FF) - 1023;
    if (e < -1000 || e > 1000) return 1.0 / x;
    const double m = __hiloint2double(__double2hiint(x) - (e << 20), __double2loint(x));   // [1, 2) with x's sign
    double r = f2d_exact(__frcp_rn(d2f_rn(m)));
    r = fma(r, fma(-m, r, 1.0), r);
    r = fma(r, fma(-m, r, 1.0), r);
    return __hiloint2double(__double2hiint(r) - (e << 20), __double2loint(r));
}
__device__ __forceinline__ float tc_recip(float x) { return 1.f / x; }
// s = sqrt(x), r = 1 / sqrt(x), x > 0
__device__ __forceinline__ void tc_root(double x, double &s, double &r)
{
    int e = ((__double2hiint(x) >> 20) & 0x7FF) - 1023;
    if (e < -1000 || e > 1000) {
        s = sqrt(x);
        r = 1.0 / s;
        return;
    }
    e &= ~1;
    const double m = __hiloint2double(__double2hiint(x) - (e << 20), __double2loint(x));   // [1, 4)
    double y = f2d_exact(rsqrtf(d2f_rn(m)));
    y = fma(0.5 * y, fma(-m * y, y, 1.0), y);
    y = fma(0.5 * y, fma(-m * y, y, 1.0), y);
    double g = m * y;
    g = fma(0.5 * y, fma(-g, g, m), g);
    s = __hiloint2double(__double2hiint(g) + ((e / 2) << 20), __double2loint(g));
    r = __hiloint2double(__double2hiint(y) - ((e / 2) << 20), __double2loint(y));
}
__device__ __forceinline__ void tc_root(float x, float &s, float &r)
{
    s = sqrtf(x);
    r = 1.f / s;
}

// The reflector of (al, x), |x|^2 = xn2: H (al, x) = (beta, 0) with v = (1, scale x).
// FP64: one chain of 14 operations from the FP32 root and reciprocal, each followed by
// one step of third order (relative errors 2^-22 -> 2^-64, then FP64 rounding):
//   1/sqrt(N):  y + y e (1/2 + 3/8 e),  e = 1 - N y^2;  the root N y takes the same step
//   1/D:        r + r (e + e^2),        e = 1 - D r
// with the exponents taken out, and back in, as integers.
__device__ __forceinline__ void tc_reflector(double2 al, double xn2, double2 &tau, double2 &scale, double &beta)
{
    tau = scale = make_double2(0, 0);
    beta = al.x;
    if ((xn2 == 0 && al.y == 0) || tp_vanishes(al, xn2)) return;
    const double N = fma(al.y, al.y, fma(al.x, al.x, xn2));
    int e = ((__double2hiint(N) >> 20) & 0x7FF) - 1023;
    double g, y;   // sqrt(N), 1 / sqrt(N)
    if (e < -1000 || e > 1000) {
        g = sqrt(N);
        y = 1.0 / g;
    } else {
        e &= ~1;
        const double m = __hiloint2double(__double2hiint(N) - (e << 20), __double2loint(N));   // [1, 4)
        const double y0 = f2d_exact(rsqrtf(d2f_rn(m))), g0 = m * y0, r = fma(-g0, y0, 1.0);
        const double p = fma(0.375, r, 0.5) * r, h = 0.5 * fma(m, y0, -g0);   // (half of g0's own rounding)
        g = g0 + fma(g0, p, h);
        y = fma(y0, p, y0);
        g = __hiloint2double(__double2hiint(g) + ((e / 2) << 20), __double2loint(g));
        y = __hiloint2double(__double2hiint(y) - ((e / 2) << 20), __double2loint(y));
    }
    if (al.x >= 0) { g = -g; y = -y; }
    const double2 den = make_double2(al.x - g, al.y);   // 1 / (alpha - beta)
    const double D = fma(den.x, den.x, den.y * den.y);
    const int f = ((__double2hiint(D) >> 20) & 0x7FF) - 1023;
    double rd;
    if (f < -1000 || f > 1000) {
        rd = 1.0 / D;
    } else {
        const double m = __hiloint2double(__double2hiint(D) - (f << 20), __double2loint(D));   // [1, 2)
        const double r0 = f2d_exact(__frcp_rn(d2f_rn(m))), r = fma(-m, r0, 1.0);
        rd = fma(r0, fma(r, r, r), r0);
        rd = __hiloint2double(__double2hiint(rd) - (f << 20), __double2loint(rd));
    }
    scale = make_double2(den.x * rd, -den.y * rd);
    tau = make_double2((g - al.x) * y, -al.y * y);
    beta = g;
}

// Programmatic dependent launch: a kernel lets its successor start once all its CTAs
// run, and waits for its predecessor (all of its writes visible) before it reads
// what that one wrote.
__device__ __forceinline__ void tc_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void tc_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// fin: only W of column i - 1 (the panel's last)
template <typename T>
__global__ void __launch_bounds__(128) k_tri_col(EigWork<T> w, int i, int j0, int fin)
{
    typedef typename cplx<T>::t C2;
    __shared__ C2 p1[EIG_NB], p2[EIG_NB], wi[EIG_NB], vi[EIG_NB];
    __shared__ C2 ssy[4][32], ssa[4][32];
    __shared__ T red[4];
    const int b = blockIdx.y, n = w.n, c = i - j0, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long ld = w.ld;
    const C2 zero = cmk<T>(0, 0);
    const C2 *A = w.A + b * w.mstride, *V = w.V + b * w.mstride + (long)j0 * ld;
    C2 *Wp = w.Wp + (long)b * w.wps;
    C2 *part = w.part + (long)b * w.npart;
    const int nn = tc_part_norm(n);
    const TcSizes z(n - i);   // of column i - 1
    const C2 *yp = w.yp + (long)b * w.nyp;
    const int r = i + blockIdx.x * 32 + lane;
    const bool rv = r < n;
    C2 y = zero, a = zero, vl = zero, sy = zero, sa = zero;
    if (warp == 0 && rv && !fin) a = A[r + (long)i * ld];   // (no kernel of the panel changes A)
    tc_wait();
    tc_release();
    if (warp == 0 && rv) {
        if (c > 0) {
            for (int q = 0; q < z.nsp; ++q) y = cadd(y, yp[(long)q * n + r]);
            vl = V[r + (long)(c - 1) * ld];
        }
    }
    if (c > 0) {
        const C2 tau = w.tau[(long)b * n + i - 1];
        if (tid < 2 * EIG_NB) {
            C2 s = zero;
            for (int q = 0; q < z.nrb; ++q) s = cadd(s, part[nn + q * 2 * EIG_NB + tid]);
            if (tid < EIG_NB) p1[tid] = s;
            else p2[tid - EIG_NB] = s;
        } else if (warp == 2) {
            T yv = T(0);
            const C2 *pv = part + nn + z.nrb * 2 * EIG_NB;
            for (int q = lane; q < z.ncol * z.nsp; q += 32) yv += pv[q].x;
            yv = warp_sum(yv);
            if (lane == 0) red[0] = yv;
        } else {   // row i of V and W
            if (lane < c) vi[lane] = V[i + (long)lane * ld];
            if (lane < c - 1) wi[lane] = Wp[i + (long)lane * n];
        }
        __syncthreads();
        if (warp == 1) {
            // alpha, and row i of the new column of W
            T pp = T(0);
            C2 s = zero;
            if (lane < c - 1) {
                pp = p1[lane].x * p2[lane].x + p1[lane].y * p2[lane].y;
                s = cmul(vi[lane], p1[lane]);
                cfma(s, wi[lane], p2[lane]);
            }
            pp = warp_sum(pp);
            s.x = warp_sum(s.x);
            s.y = warp_sum(s.y);
            if (lane == 0) {
                const T al = T(-0.5) * (tau.x * tau.x + tau.y * tau.y) * (red[0] - T(2) * pp);
                C2 yi = zero;
                for (int q = 0; q < z.nsp; ++q) yi = cadd(yi, yp[(long)q * n + i]);
                yi = cmul(tau, csub(yi, s));
                yi.x += al;              // v at row i is 1
                wi[c - 1] = yi;
                red[1] = al;
            }
        }
        if (rv) {   // both sums over the panel's earlier columns, eight columns' loads together
            C2 vv[8], ww[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int j = warp + 4 * u;
                vv[u] = zero;
                ww[u] = zero;
                if (j < c - 1) {
                    vv[u] = V[r + (long)j * ld];
                    ww[u] = Wp[r + (long)j * n];
                }
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int j = warp + 4 * u;
                if (j >= c - 1) break;
                cfma(sy, vv[u], p1[j]);
                cfma(sy, ww[u], p2[j]);
                if (!fin) {
                    cfma(sa, vv[u], cconj(wi[j]));
                    cfma(sa, ww[u], cconj(vi[j]));
                }
            }
        }
        ssy[warp][lane] = sy;
        ssa[warp][lane] = sa;
        __syncthreads();
        if (warp == 0 && rv) {
#pragma unroll
            for (int u = 1; u < 4; ++u) {
                sy = cadd(sy, ssy[u][lane]);
                sa = cadd(sa, ssa[u][lane]);
            }
            C2 wl = cmul(tau, csub(y, sy));
            wl = cadd(wl, cscale(vl, red[1]));
            Wp[r + (long)(c - 1) * n] = wl;
            cfma(sa, vl, cconj(wi[c - 1]));
            cfma(sa, wl, cconj(vi[c - 1]));
        }
    }
    if (fin || warp != 0) return;
    T nrm2 = T(0);
    if (rv) {
        a = csub(a, sa);
        w.col[(long)b * n + r] = a;
        if (r == i) w.d[(long)b * n + i] = (double)a.x;
        if (r >= i + 2) nrm2 = a.x * a.x + a.y * a.y;
    }
    nrm2 = warp_sum(nrm2);
    if (lane == 0) part[blockIdx.x] = cmk<T>(nrm2, T(0));
}

// v = scale u with u = column i (rows i + 2 ..) and v = 1 at row i + 1.  Every sum
// here is formed with u (zero at row i + 1) and scaled at its end, the first row's
// term added unscaled, so that no warp waits for the reflector's root and reciprocals.
template <typename T>
__global__ void __launch_bounds__(32 * TC_WARPS, 2) k_tri_mv(EigWork<T> w, int i, int j0)
{
    typedef typename cplx<T>::t C2;
    __shared__ C2 ssc;                       // the reflector's scale
    __shared__ C2 us[TC_WARPS][32];          // u of a warp's column tile
    __shared__ C2 red[TC_WARPS][32];
    extern __shared__ __align__(16) unsigned char tc_raw[];   // [warp][16][33]: transposed half tiles
    const int b = blockIdx.y, n = w.n, c = i - j0, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long ld = w.ld;
    const C2 zero = cmk<T>(0, 0);
    const C2 *A = w.A + b * w.mstride;
    const C2 *col = w.col + (long)b * n;
    C2 *part = w.part + (long)b * w.npart;
    const int nn = tc_part_norm(n), base = i + 1;
    const TcSizes z(n - base);
    // this warp's first half tile of A, which no kernel of the panel changes: its loads
    // are in flight while the column kernel before this one ends
    const int q = blockIdx.x, ntile = z.ncol * z.nsp;
    const int R = q / z.nsp, sp = q - R * z.nsp;
    int h = 2 * (sp * z.ncol / z.nsp) + warp;
    const int h_hi = q < ntile ? 2 * ((sp + 1) * z.ncol / z.nsp) : 0;
    C2 a[16];
    auto load = [&](int hh) {   // the lower half tile (R, hh / 2) or its mirror: lane = row, 16 columns
        if (hh >= h_hi) return;
        const int S = hh >> 1;
        const bool trans = S > R, diag = S == R;
        const int r = base + 32 * (trans ? S : R) + lane, c0 = base + 32 * (trans ? R : S) + 16 * (hh & 1);
        if (r - lane + 32 <= n && c0 + 16 <= n && !diag) {
#pragma unroll
            for (int u = 0; u < 16; ++u) a[u] = A[r + (long)(c0 + u) * ld];
        } else {
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                a[u] = zero;
                if (r < n && c0 + u < n && (!diag || c0 + u <= r)) a[u] = A[r + (long)(c0 + u) * ld];
            }
        }
    };
    load(h);
    tc_wait();
    tc_release();
    if (warp == TC_WARPS - 1) {
        // reflector (zlarfg) from column i's partials, the same in every CTA
        T x = T(0);
        for (int q = lane; q < (n - i + 31) / 32; q += 32) x += part[q].x;
        const T xn2 = warp_sum(x);
        if (lane == 0) {
            const C2 al = col[base];
            C2 tau = zero, scale = zero;
            T beta = al.x;
            if ((xn2 != T(0) || al.y != T(0)) && !tp_vanishes(al, xn2)) {
                T bb, rb;
                tc_root(al.x * al.x + al.y * al.y + xn2, bb, rb);
                if (al.x >= T(0)) { bb = -bb; rb = -rb; }
                const C2 den = cmk<T>(al.x - bb, al.y);   // 1 / (alpha - beta)
                const T rd = tc_recip(den.x * den.x + den.y * den.y);
                scale = cmk<T>(den.x * rd, -den.y * rd);
                tau = cmk<T>((bb - al.x) * rb, -al.y * rb);
                beta = bb;
            }
            ssc = scale;
            if (blockIdx.x == 0) {
                w.e[(long)b * n + i] = (double)beta;
                w.tau[(long)b * n + i] = tau;
            }
        }
    }
    auto urow = [&](int r) { return r > base && r < n ? col[r] : zero; };
    if (q >= ntile) {
        // ---- dots: W^H v and V^H v over 128 rows, and V[:, i] ----
        const int rb = q - ntile, r0 = base + TC_ROWS * rb;
        C2 *V = w.V + b * w.mstride;
        const C2 *Vp = V + (long)j0 * ld, *Wp = w.Wp + (long)b * w.wps;
        C2 u4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) u4[u] = urow(r0 + lane + 32 * u);
        C2 x[8];   // this warp's 8 of the 64 sums
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const int col8 = 8 * warp + t, j = col8 & (EIG_NB - 1);
            x[t] = zero;
            if (j < c) {
                const C2 *M = col8 < EIG_NB ? Wp + (long)j * n : Vp + (long)j * ld;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int r = r0 + lane + 32 * u;
                    if (r < n) cfmac(x[t], M[r], u4[u]);
                }
            }
        }
        if (((8 * warp) & (EIG_NB - 1)) < c) tp_butterfly<8>(x, lane);   // warp-uniform
        __syncthreads();
        const C2 scale = ssc;
        if ((lane & 3) == 0) {
            const int col8 = 8 * warp + (lane >> 2), j = col8 & (EIG_NB - 1);
            C2 s = zero;
            if (j < c) {
                s = cmul(x[0], scale);
                if (rb == 0)   // row i + 1
                    s = cadd(s, cconj(col8 < EIG_NB ? Wp[base + (long)j * n] : Vp[base + (long)j * ld]));
            }
            part[nn + rb * 2 * EIG_NB + col8] = s;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int r = r0 + lane + 32 * u;
            if (warp == u && r < n) V[r + (long)i * ld] = r == base ? cmk<T>(1, 0) : cmul(u4[u], scale);
        }
        if (rb == 0)
            for (int r = tid; r <= i; r += 32 * TC_WARPS) V[r + (long)i * ld] = zero;
        return;
    }
    // ---- y of row block R over the half tiles of split sp, a warp every eighth ----
    C2 (*tt)[33] = (C2 (*)[33])tc_raw + 16 * warp;
    C2 yr = zero;
    while (h < h_hi) {   // warp-uniform
        const int S = h >> 1, hf = h & 1;
        const bool trans = S > R, diag = S == R;
        const C2 uS = urow(base + 32 * S + lane);
        __syncwarp();
        us[warp][lane] = uS;
        __syncwarp();
        if (!trans) {
#pragma unroll
            for (int u = 0; u < 16; ++u) cfma(yr, a[u], us[warp][16 * hf + u]);
        }
        if (trans || diag) {
            // lane: column 16 hf + (lane mod 16), rows of its half of the tile
            const int r = 32 * (trans ? S : R) + lane, c0 = 32 * R + 16 * hf;
#pragma unroll
            for (int u = 0; u < 16; ++u) tt[u][lane] = (trans || c0 + u < r) ? a[u] : zero;
            __syncwarp();
            C2 x = zero;
#pragma unroll
            for (int u = 0; u < 16; ++u) cfmac(x, tt[lane & 15][(lane & 16) + u], us[warp][(lane & 16) + u]);
            x.x += __shfl_xor_sync(0xffffffffu, x.x, 16);
            x.y += __shfl_xor_sync(0xffffffffu, x.y, 16);
            if ((lane >> 4) == hf) yr = cadd(yr, x);
        }
        h += TC_WARPS;
        load(h);
    }
    red[warp][lane] = yr;
    __syncthreads();
    if (warp == 0) {
        C2 y = red[0][lane];
#pragma unroll
        for (int u = 1; u < TC_WARPS; ++u) y = cadd(y, red[u][lane]);
        const C2 scale = ssc;
        const int r = base + 32 * R + lane;
        y = cmul(y, scale);
        C2 vR = cmul(urow(r), scale);
        if (r == base) vR = cmk<T>(1, 0);
        if (r < n) {
            if (sp == 0) y = cadd(y, A[r + (long)base * ld]);   // column i + 1, v = 1
            w.yp[(long)b * w.nyp + (long)sp * n + r] = y;
        } else {
            y = zero;
        }
        const T yv = warp_sum(y.x * vR.x + y.y * vR.y);
        if (lane == 0) part[nn + z.nrb * 2 * EIG_NB + q] = cmk<T>(yv, T(0));
    }
}

template <typename T, typename K, typename... Args>
inline void tc_launch(cudaStream_t s, K kernel, dim3 grid, int threads, int smem, bool dependent, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = dependent ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, args...);
    if (g_launch_counter) ++*g_launch_counter;
}

// columns j0 .. j0 + jb of the panel.  The panel's first kernel follows the trailing
// update (or what else came before) in plain stream order.
template <typename T> void tri_columns(cudaStream_t s, EigWork<T> &w, int j0, int jb)
{
    const int n = w.n, B = w.batch, sm = (int)sizeof(typename cplx<T>::t) * TC_WARPS * 16 * 33;
    smem_attr_at_least((const void *)k_tri_mv<T>, sm);
    for (int i = j0; i < j0 + jb; ++i) {
        tc_launch<T>(s, k_tri_col<T>, dim3(cdiv(n - i, 32), B), 128, 0, i > j0, w, i, j0, 0);
        if (i == n - 1) return;   // the last column: d only
        const TcSizes z(n - i - 1);
        tc_launch<T>(s, k_tri_mv<T>, dim3(z.ncol * z.nsp + z.nrb, B), 32 * TC_WARPS, sm, true, w, i, j0);
    }
    const int e = j0 + jb;
    if (e < n) tc_launch<T>(s, k_tri_col<T>, dim3(cdiv(n - e, 32), B), 128, 0, true, w, e, j0, 1);
}

}  // namespace nrltb
