// tri_panel.cuh -- one panel (up to EIG_NB columns) of the blocked Householder
// tridiagonalisation A = Q T Q^H, with one thread-block cluster per matrix.
//
// The per-column chain of zhetrd/zlatrd (column update, reflector, Hermitian
// mat-vec y = A v of the trailing matrix, w = tau (y - V p1 - W p2),
// alpha = -tau/2 w^H v) is latency bound when each step is its own launch.
// Here the CL CTAs of a cluster own the matrix rows in 32-row tiles (tile t
// belongs to CTA t mod CL) and run every column of the panel in one launch,
// with three cluster barriers per column.  The cluster-wide sums (|x|^2 of
// the reflector, W^H v / V^H v, w^H v) are partials per tile in shared memory, read
// by every CTA through distributed shared memory, so all CTAs derive identical
// scalars without a further barrier.
//
// CL is chosen by how many clusters fit the device at once (tri_panel_launch), and
// the results do not depend on it: whoever owns a tile, its partials are added as
// eight ranks would, rank t mod 8 over its own tiles first (TP_RANKS), then the ranks in
// order, and a row tile's mat-vec is always cut into TP_STRIPS strips.
//
// The mat-vec reads only A's lower triangle: for an own row tile R and a
// column tile S > R, the lower tile (S, R) is read (coalesced) and its
// conjugate transpose applied with a warp butterfly (transpose-reduce), so a
// CTA forms the whole y of its own rows without cross-CTA traffic.
//
// The CTA keeps its own rows of the panel's V and W columns (and of w') in
// shared memory, so the per-column updates read no global memory but the
// current column of A, row i and the mat-vec tiles.
//
// Every CTA executes the same sequence of barriers: control flow that
// encloses a barrier depends only on kernel arguments.
#pragma once
#include <cooperative_groups.h>
#include "eig.cuh"

namespace nrltb {

constexpr int TP_STRIPS = 8;  // column strips of a row tile's mat-vec, each summed by itself
constexpr int TP_RANKS = 8;   // tiles t mod TP_RANKS are summed first, whatever the cluster size

constexpr int TP_NV = 16;     // values per lane of one butterfly (16: 16 warps fit an SM)

// A column whose elements' squares fall out of the range (2^-63 in FP32, 2^-511 in FP64) is
// left as it is: its reflector would be a quotient of zeros.  xn2: |x|^2 of the elements
// below al.  (FP64 on the exponents: the narrow pipe stays out of the column's chain.)
__device__ __forceinline__ bool tp_vanishes(float2 al, float xn2)
{
    return fmaxf(fabsf(al.x), fabsf(al.y)) < 0x1p-63f && xn2 < 0x1p-126f;
}
__device__ __forceinline__ bool tp_vanishes(double2 al, double xn2)
{
    const int hi = 0x7FFFFFFF;
    return max(__double2hiint(al.x) & hi, __double2hiint(al.y) & hi) < (1023 - 511) << 20 && __double2hiint(xn2) < 1 << 20;
}

// Transpose-reduce over the warp: lane l holds x[0..NV); afterwards x[0] of
// lane l is sum over all lanes of x[u] with u = l >> (5 - log2 NV) (lanes that
// share u hold the same total).
template <int NV, typename C2>
__device__ __forceinline__ void tp_butterfly(C2 (&x)[NV], int lane)
{
    int o = 16;
#pragma unroll
    for (int m = NV; m > 1; m >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int u = 0; u < m / 2; ++u) {
            C2 send = up ? x[u] : x[u + m / 2];
            C2 keep = up ? x[u + m / 2] : x[u];
            keep.x += __shfl_xor_sync(0xffffffffu, send.x, o);
            keep.y += __shfl_xor_sync(0xffffffffu, send.y, o);
            x[u] = keep;
        }
    }
    for (; o > 0; o >>= 1) {
        x[0].x += __shfl_xor_sync(0xffffffffu, x[0].x, o);
        x[0].y += __shfl_xor_sync(0xffffffffu, x[0].y, o);
    }
}

template <typename T> struct TpSmem {
    typedef typename cplx<T>::t C2;
    C2 *vfull;      // v of the current column, all rows (32 T_)
    C2 *acol;       // own rows: updated column, then v (32 nown)
    C2 *ypart;      // per strip: partial y of the own rows (TP_STRIPS x 32 nown)
    C2 *Vs, *Ws;    // own rows of the panel's V and W columns (EIG_NB x 32 nown each)
    C2 *wqs;        // own rows of w' of the previous column (32 nown)
    C2 *wi, *vi;    // row i of the panel's W and V
    C2 *p1, *p2;    // W^H v, V^H v (cluster sums)
    C2 *pw;         // partials of W^H v | V^H v per item (nit x 64)
    C2 *p12r;       // the same per rank of this CTA (nrk x 64)
    C2 *a0;         // element i+1 of the updated column (owner CTA)
    C2 *dotit;      // w^H v per item (nit), per rank (nrk)
    C2 *dotr;
    T *normit;      // |x|^2 per item (nit), per rank (nrk)
    T *normr;
};

// Items: the units whose partials are kept apart, one per own tile; above 64 tiles
// one per warp, which then runs over its tiles k = warp, warp + TP_WARPS, ... (the
// cluster size is TP_RANKS there).
__host__ __device__ inline bool tp_by_warp(int tiles) { return tiles > TP_RANKS * TP_STRIPS; }
__host__ __device__ inline int tp_items(int tiles, int cl)
{
    return tp_by_warp(tiles) ? TP_STRIPS : (tiles + cl - 1) / cl;
}

inline size_t tp_smem_bytes(int n, int cl, size_t c2)
{
    const int T_ = cdiv(n, 32), nown = cdiv(T_, cl), nit = tp_items(T_, cl), nrk = TP_RANKS / cl;
    return c2 * (32 * (size_t)T_ + 32 * (size_t)nown * (2 + TP_STRIPS + 2 * EIG_NB) + 4 * 32 + 64 * (size_t)(nit + nrk) +
                 1 + (size_t)(nit + nrk)) +
           (c2 / 2) * (size_t)(nit + nrk) + 64;
}

template <typename T, int CL>
__device__ __forceinline__ TpSmem<T> tp_carve(unsigned char *base, int n)
{
    typedef typename cplx<T>::t C2;
    const int T_ = (n + 31) / 32, nown = (T_ + CL - 1) / CL, nit = tp_items(T_, CL), nrk = TP_RANKS / CL;
    TpSmem<T> s;
    C2 *p = (C2 *)base;
    s.vfull = p; p += 32 * T_;
    s.acol = p; p += 32 * nown;
    s.ypart = p; p += 32 * nown * TP_STRIPS;
    s.Vs = p; p += 32 * nown * EIG_NB;
    s.Ws = p; p += 32 * nown * EIG_NB;
    s.wqs = p; p += 32 * nown;
    s.wi = p; p += 32;
    s.vi = p; p += 32;
    s.p1 = p; p += 32;
    s.p2 = p; p += 32;
    s.pw = p; p += nit * 64;
    s.p12r = p; p += nrk * 64;
    s.a0 = p; p += 1;
    s.dotit = p; p += nit;
    s.dotr = p; p += nrk;
    T *q = (T *)p;
    s.normit = q; q += nit;
    s.normr = q;
    return s;
}

// The trailing mat-vec for own row tile R over column tiles [s_lo, s_hi), one
// warp: y_R += A_RS v_S for S < R (lane = row), for S > R the lower tile (S, R)
// is read by rows and its conjugate transpose applied: the lanes' products are
// summed over all S of the strip in registers and reduced across lanes once per
// half tile (butterfly), and the diagonal tile combines both.  Tiles inside
// [lo, n) in both directions take an unmasked path.  Contributions are added to
// the strip's ypart slots of tile R.
//
// The loop is bound by the latency of the tiles' loads out of L2 (about 900 clocks), so
// the two groups of eight columns of a half tile take turns: one's loads of the next step
// are under way while the other is applied (n = 1404, 8 matrices: 33.0 -> 31.5 ms).
template <typename T>
__device__ __forceinline__ void tp_strip(const typename cplx<T>::t *A, long ld, int n, int lo, int R, int s_lo,
                                         int s_hi, const typename cplx<T>::t *vfull, typename cplx<T>::t *yp,
                                         int lane)
{
    typedef typename cplx<T>::t C2;
    constexpr int NV = TP_NV;
    // columns [u0, u0 + 8) of the half h of the strip's tile S, zero outside the trailing matrix
    auto fetch = [&](C2 (&a)[8], int S, int h, int u0) {
        const bool trans = S > R, diag = S == R;
        const int rowt = trans ? S : R, colt = trans ? R : S;
        const int r = 32 * rowt + lane, c0 = 32 * colt + h * NV;
        const unsigned off = (unsigned)(r + (c0 + u0) * (int)ld);
        const bool interior = !diag && 32 * rowt >= lo && 32 * rowt + 31 < n && c0 >= lo && c0 + NV <= n;
        if (interior) {
#pragma unroll
            for (int u = 0; u < 8; ++u) a[u] = A[off + u * (unsigned)ld];
        } else {
            const bool rv = r >= lo && r < n;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int sc = c0 + u0 + u;
                a[u] = cmk<T>(0, 0);
                if (rv && sc >= lo && sc < n && (!diag || sc <= r)) a[u] = A[off + u * (unsigned)ld];
            }
        }
    };
    C2 yr = cmk<T>(0, 0), x[NV];
    auto apply = [&](const C2 (&a)[8], int S, int h, auto part) {
        constexpr int u0 = decltype(part)::value;
        const bool trans = S > R, diag = S == R;
        if (!trans) {
            const float4 *vc = (const float4 *)(vfull + 32 * S + h * NV + u0);   // broadcast
#pragma unroll
            for (int u = 0; u < 8; u += 2) {
                const float4 v = vc[u / 2];
                cfma(yr, a[u], cmk<T>(v.x, v.y));
                cfma(yr, a[u + 1], cmk<T>(v.z, v.w));
            }
        }
        if (trans) {
            const C2 vr = vfull[32 * S + lane];
#pragma unroll
            for (int u = 0; u < 8; ++u) cfmac(x[u0 + u], a[u], vr);   // conj(a) v_r
        } else if (diag) {
            const C2 vr = vfull[32 * R + lane];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (h * NV + u0 + u < lane) cfmac(x[u0 + u], a[u], vr);
        }
    };
    const bool has_upper = s_hi - 1 >= R;   // trans or diagonal tiles in the strip (warp-uniform)
    C2 a0[8], a1[8];
    fetch(a0, s_lo, 0, 0);
    fetch(a1, s_lo, 0, 8);
#pragma unroll 1
    for (int h = 0; h < 32 / NV; ++h) {
#pragma unroll
        for (int u = 0; u < NV; ++u) x[u] = cmk<T>(0, 0);
#pragma unroll 1
        for (int S = s_lo; S < s_hi; ++S) {
            const bool wrap = S + 1 == s_hi;
            const int Sn = wrap ? s_lo : S + 1, hn = wrap ? h + 1 : h;
            apply(a0, S, h, std::integral_constant<int, 0>());
            if (hn < 32 / NV) fetch(a0, Sn, hn, 0);
            apply(a1, S, h, std::integral_constant<int, 8>());
            if (hn < 32 / NV) fetch(a1, Sn, hn, 8);
        }
        if (has_upper) {
            tp_butterfly<NV>(x, lane);
            if ((lane & 1) == 0) {   // two lanes hold each sum
                C2 &dst = yp[h * NV + (lane >> 1)];
                dst = cadd(dst, x[0]);
            }
        }
    }
    yp[lane] = cadd(yp[lane], yr);
}

template <typename T, int CL, int NW>
__global__ void __launch_bounds__(32 * NW, 16 / NW) k_tri_panel(EigWork<T> w, int j0, int jb)
{
    typedef typename cplx<T>::t C2;
    namespace cg = cooperative_groups;
    constexpr int NV = TP_NV, NR = TP_RANKS / CL;   // ranks of this CTA
    extern __shared__ __align__(16) unsigned char tp_raw[];
    cg::cluster_group cluster = cg::this_cluster();
    const int q = (int)cluster.block_rank();
    const int b = blockIdx.y, n = w.n, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long ld = w.ld;
    const C2 *A = w.A + b * w.mstride;
    C2 *V = w.V + b * w.mstride;
    C2 *Wp = w.Wp + (long)b * w.wps, *wq = w.wq + (long)b * n;
    const int T_ = cdiv(n, 32);
    const int nown = (q < T_) ? (T_ - 1 - q) / CL + 1 : 0;
    TpSmem<T> sm = tp_carve<T, CL>(tp_raw, n);
    const int ns = 32 * cdiv(T_, CL);   // row stride of Vs, Ws
    const bool bywarp = tp_by_warp(T_);
    // tiles of the row phases, one warp each; with an item per warp (tp_by_warp) the
    // first TP_STRIPS warps walk them
    const int kstep = bywarp ? TP_STRIPS : NW, k0 = (bywarp && warp >= TP_STRIPS) ? nown : warp;
    // the items of this CTA's rank v (tiles q + CL v + TP_RANKS k8) in order
    auto over_items = [&](int v, auto add) {
        if (bywarp) {
            for (int ww = 0; ww < TP_STRIPS; ++ww) add(ww);
        } else {
            for (int t = q + CL * v; t < T_; t += TP_RANKS) add(t / CL);
        }
    };
    // rank rk's entry of a per-rank array
    auto rank_at = [&](auto *r, int rk, int stride, int at) {
        return cluster.map_shared_rank(r, rk % CL)[(rk / CL) * stride + at];
    };
    // the ranks' w^H v in order: lane rk < TP_RANKS fetches one, every lane adds them
    auto sum_dot = [&]() {
        C2 mine = cmk<T>(0, 0), t = cmk<T>(0, 0);
        if (lane < TP_RANKS) mine = rank_at(sm.dotr, lane, 1, 0);
        for (int rk = 0; rk < TP_RANKS; ++rk) {
            C2 o;
            o.x = __shfl_sync(0xffffffffu, mine.x, rk);
            o.y = __shfl_sync(0xffffffffu, mine.y, rk);
            t = cadd(t, o);
        }
        return t;
    };
    // -tau dot / 2; the product's rounding is spelled out, since the compiler's choice of
    // which term to fuse would otherwise change with the code around it
    auto alpha_of = [](C2 tau, C2 dot) {
        return cmk<T>(T(-0.5) * __fmaf_rn(tau.x, dot.x, -__fmul_rn(tau.y, dot.y)),
                      T(-0.5) * __fmaf_rn(tau.x, dot.y, __fmul_rn(tau.y, dot.x)));
    };
    const C2 zero = cmk<T>(0, 0);
    auto own_from = [&](int tile) { return tile > q ? (tile - q + CL - 1) / CL : 0; };   // first own tile >= tile

    C2 tau = zero, alpha = zero;
    int c = 0;
    for (; c < jb; ++c) {
        const int i = j0 + c;
        // ---- A: alpha of the previous column; row i of V, W; update column i ----
        // the loads go out ahead of the cluster sum; a0n: column i of this warp's first tile
        C2 vin = zero, win = zero, a0n = zero;
        if (tid < c) {
            vin = V[i + (long)(j0 + tid) * ld];
            win = (tid < c - 1) ? Wp[i + (long)tid * n] : wq[i];
        }
        if (k0 < nown && 32 * (q + CL * k0) + lane < n) a0n = A[32 * (q + CL * k0) + lane + (long)i * ld];
        if (c > 0) alpha = alpha_of(tau, sum_dot());
        if (tid < c) {
            sm.vi[tid] = vin;
            sm.wi[tid] = (tid < c - 1) ? win : cadd(win, cmul(alpha, vin));
        }
        __syncthreads();
        T nrm2 = T(0);
        for (int k = k0; k < nown; k += kstep) {
            const int r = 32 * (q + CL * k) + lane;
            if (!bywarp) nrm2 = T(0);
            if (r >= i && r < n) {
                C2 a = (k == k0) ? a0n : A[r + (long)i * ld];   // before the store to Wp, which it could alias
                C2 wl = zero;
                const int slot = 32 * k + lane;
                if (c > 0) {
                    wl = cadd(sm.wqs[slot], cmul(alpha, sm.Vs[(c - 1) * ns + slot]));
                    Wp[r + (long)(c - 1) * n] = wl;
                    sm.Ws[(c - 1) * ns + slot] = wl;
                }
                // eight panel columns per round: their loads are issued together
                for (int j8 = 0; j8 < c; j8 += 8) {
                    C2 vv[8], ww[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const int j = j8 + u;
                        vv[u] = zero;
                        ww[u] = zero;
                        if (j < c) {
                            vv[u] = sm.Vs[j * ns + slot];
                            ww[u] = sm.Ws[j * ns + slot];
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (j8 + u < c) {
                            a = csub(a, cmul(vv[u], cconj(sm.wi[j8 + u])));
                            a = csub(a, cmul(ww[u], cconj(sm.vi[j8 + u])));
                        }
                }
                sm.acol[32 * k + lane] = a;
                if (r == i) w.d[(long)b * n + i] = (double)a.x;
                if (r == i + 1) *sm.a0 = a;
                if (r >= i + 2) nrm2 += a.x * a.x + a.y * a.y;
            }
            if (!bywarp) {
                const T t = warp_sum(nrm2);
                if (lane == 0) sm.normit[k] = t;
            }
        }
        if (bywarp) {
            nrm2 = warp_sum(nrm2);
            if (lane == 0 && warp < TP_STRIPS) sm.normit[warp] = nrm2;
        }
        __syncthreads();
        if (tid < NR) {   // the items of each own rank, in the order of their tiles
            T t = T(0);
            over_items(tid, [&](int it) { t += sm.normit[it]; });
            sm.normr[tid] = t;
        }
        if (i == n - 1) break;   // last column of the matrix: d only (uniform)
        cluster.sync();   // #1

        // ---- B: reflector (every CTA, same order); v; partial W^H v, V^H v ----
        T xn2 = T(0);
        {
            T mine = T(0);
            if (lane < TP_RANKS) mine = rank_at(sm.normr, lane, 1, 0);
            for (int rk = 0; rk < TP_RANKS; ++rk) xn2 += __shfl_sync(0xffffffffu, mine, rk);
        }
        const C2 al = *cluster.map_shared_rank(sm.a0, ((i + 1) / 32) % CL);
        C2 scale = zero;
        double beta;
        tau = zero;
        {
            const T xnorm = sqrt(xn2);
            if ((xnorm == T(0) && al.y == T(0)) || tp_vanishes(al, xn2)) {
                beta = (double)al.x;
            } else {
                T bb = sqrt(al.x * al.x + al.y * al.y + xnorm * xnorm);
                bb = (al.x >= T(0)) ? -bb : bb;
                tau = cmk<T>((bb - al.x) / bb, -al.y / bb);
                const C2 den = cmk<T>(al.x - bb, al.y);   // 1 / (alpha - beta)
                const T dd = den.x * den.x + den.y * den.y;
                scale = cmk<T>(den.x / dd, -den.y / dd);
                beta = (double)bb;
            }
        }
        if (q == 0 && tid == 0) {
            w.e[(long)b * n + i] = beta;
            w.tau[(long)b * n + i] = tau;
        }
        for (int k = k0; k < nown; k += kstep) {
            const int r = 32 * (q + CL * k) + lane;
            C2 v = zero;
            if (r >= i + 1 && r < n) v = (r == i + 1) ? cmk<T>(1, 0) : cmul(sm.acol[32 * k + lane], scale);
            if (r < n) V[r + (long)i * ld] = v;
            sm.acol[32 * k + lane] = v;
            sm.Vs[c * ns + 32 * k + lane] = v;
        }
        __syncthreads();
        // W^H v and V^H v over the rows of each item: a warp per item, part and half of the
        // columns, column j in butterfly slot j
        for (int un = warp; un < 4 * tp_items(T_, CL); un += NW) {
            const int item = un >> 2, part = (un >> 1) & 1, h = un & 1;
            C2 sum = zero;
            if (h * NV < c)
                for (int k = item; k < nown; k += bywarp ? TP_STRIPS : nown) {
                    const int r = 32 * (q + CL * k) + lane;
                    if (32 * (q + CL * k) + 31 < i + 1) continue;
                    const bool valid = r >= i + 1 && r < n;
                    const C2 v = sm.acol[32 * k + lane], *m = (part ? sm.Vs : sm.Ws) + h * NV * ns + 32 * k + lane;
                    C2 x[NV];
#pragma unroll
                    for (int u = 0; u < NV; ++u) {
                        x[u] = zero;
                        if (valid && h * NV + u < c) cfmac(x[u], m[u * ns], v);
                    }
                    tp_butterfly<NV>(x, lane);
                    sum = cadd(sum, x[0]);
                }
            if ((lane & 1) == 0) sm.pw[item * 64 + part * 32 + h * NV + (lane >> 1)] = sum;
        }
        __syncthreads();
        for (int e = tid; e < 64 * NR; e += 32 * NW) {
            C2 s = zero;
            over_items(e >> 6, [&](int it) { s = cadd(s, sm.pw[it * 64 + (e & 63)]); });
            sm.p12r[e] = s;
        }
        cluster.sync();   // #2

        // ---- C: cluster sums p1, p2; full v; trailing mat-vec for own rows ----
        if (tid < 64) {
            C2 o[TP_RANKS], s = zero;
#pragma unroll
            for (int rk = 0; rk < TP_RANKS; ++rk) o[rk] = rank_at(sm.p12r, rk, 64, tid);
#pragma unroll
            for (int rk = 0; rk < TP_RANKS; ++rk) s = cadd(s, o[rk]);
            if (tid < 32) sm.p1[tid] = s; else sm.p2[tid - 32] = s;
        }
        for (int s = tid; s < 32 * T_; s += 32 * NW)
            sm.vfull[s] = (s >= i + 1 && s < n) ? V[s + (long)i * ld] : zero;
        for (int e = tid; e < 32 * nown * TP_STRIPS; e += 32 * NW) sm.ypart[e] = zero;
        __syncthreads();
        {
            // each own row tile's column tiles are cut into TP_STRIPS contiguous strips
            const int tb = (i + 1) / 32, ncol = T_ - tb, st = warp % TP_STRIPS;
            const int s_lo = tb + (st * ncol) / TP_STRIPS, s_hi = tb + ((st + 1) * ncol) / TP_STRIPS;
            C2 *ys = sm.ypart + st * 32 * nown;
            if (s_lo < s_hi)
                for (int k = own_from(tb) + warp / TP_STRIPS; k < nown; k += NW / TP_STRIPS)
                    tp_strip<T>(A, ld, n, i + 1, q + CL * k, s_lo, s_hi, sm.vfull, ys + 32 * k, lane);
        }
        __syncthreads();

        // ---- D: w' = tau (y - V p1 - W p2) for own rows; partial w'^H v ----
        C2 dot = zero;
        for (int k = k0; k < nown; k += kstep) {
            const int r = 32 * (q + CL * k) + lane;
            if (!bywarp) dot = zero;
            if (r >= i + 1 && r < n) {
                C2 y = zero;
                for (int ww = 0; ww < TP_STRIPS; ++ww) y = cadd(y, sm.ypart[ww * 32 * nown + 32 * k + lane]);
                for (int j8 = 0; j8 < c; j8 += 8) {
                    C2 vv[8], ww[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const int j = j8 + u;
                        vv[u] = zero;
                        ww[u] = zero;
                        if (j < c) {
                            vv[u] = sm.Vs[j * ns + 32 * k + lane];
                            ww[u] = sm.Ws[j * ns + 32 * k + lane];
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (j8 + u < c) {
                            y = csub(y, cmul(vv[u], sm.p1[j8 + u]));
                            y = csub(y, cmul(ww[u], sm.p2[j8 + u]));
                        }
                }
                y = cmul(tau, y);
                wq[r] = y;
                sm.wqs[32 * k + lane] = y;
                cfmac(dot, y, sm.acol[32 * k + lane]);   // conj(w') v
            }
            if (!bywarp) {
                const T dx = warp_sum(dot.x), dy = warp_sum(dot.y);
                if (lane == 0) sm.dotit[k] = cmk<T>(dx, dy);
            }
        }
        if (bywarp) {
            dot.x = warp_sum(dot.x);
            dot.y = warp_sum(dot.y);
            if (lane == 0 && warp < TP_STRIPS) sm.dotit[warp] = dot;
        }
        __syncthreads();
        if (tid < NR) {
            C2 t = zero;
            over_items(tid, [&](int it) { t = cadd(t, sm.dotit[it]); });
            sm.dotr[tid] = t;
        }
        cluster.sync();   // #3
    }
    // W[:, last] = w' + alpha v of the panel's last reflected column
    if (c == jb) {
        const int i = j0 + jb - 1;
        alpha = alpha_of(tau, sum_dot());
        for (int k = warp; k < nown; k += NW) {
            const int r = 32 * (q + CL * k) + lane;
            if (r >= n) continue;
            const C2 v = (r > i) ? sm.Vs[(jb - 1) * ns + 32 * k + lane] : zero;
            const C2 qv = (r > i) ? sm.wqs[32 * k + lane] : zero;
            Wp[r + (long)(jb - 1) * n] = cadd(qv, cmul(alpha, v));
        }
    }
    cluster.sync();   // no CTA leaves while others may read its shared memory
}

template <int CL, int NW> inline cudaLaunchConfig_t tp_config(cudaLaunchAttribute *attr, int batch, size_t smem)
{
    cudaLaunchConfig_t cfg = {};
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = CL;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    cfg.gridDim = dim3(CL, batch, 1);
    cfg.blockDim = dim3(32 * NW, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Clusters of order n's panel that the device holds at once (0: none), per (device,
// shared memory) for the whole process: the answer does not depend on which thread
// asks or on what ran before.
template <int CL, int NW> inline int tp_capacity(size_t smem)
{
    static std::mutex mu;
    static std::map<std::pair<int, size_t>, int> known;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> g(mu);
    auto it = known.find(std::make_pair(dev, smem));
    if (it != known.end()) return it->second;
    int count = 0;
    const void *f = (const void *)k_tri_panel<float, CL, NW>;
    const Refusable r;   // another size, or the column kernels, take over
    bool ok = smem_attr_at_least(f, (int)smem) == cudaSuccess;
    if (ok) {
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = tp_config<CL, NW>(&attr, 1, smem);
        ok = cudaOccupancyMaxActiveClusters(&count, k_tri_panel<float, CL, NW>, &cfg) == cudaSuccess;
    }
    if (!ok) r.clear();
    return known[std::make_pair(dev, smem)] = ok ? count : 0;
}

template <int CL, int NW> inline bool tp_try(cudaStream_t s, const EigWork<float> &w, int j0, int jb, bool must_fit)
{
    const size_t smem = tp_smem_bytes(w.n, CL, sizeof(float2));
    if (smem > 200 * 1024 || tp_capacity<CL, NW>(smem) < (must_fit ? w.batch : 1)) return false;
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = tp_config<CL, NW>(&attr, w.batch, smem);
    cfg.stream = s;
    cudaEvent_t ev = kt_begin(s);
    const Refusable r;
    if (cudaLaunchKernelEx(&cfg, k_tri_panel<float, CL, NW>, w, j0, jb) != cudaSuccess) {
        r.clear();
        return false;
    }
    if (g_launch_counter) ++*g_launch_counter;
    // algorithmic bytes: the lower triangle of each column's trailing matrix, read once
    double bytes = 0;
    for (int c = 0; c < jb; ++c) {
        const double m = w.n - (j0 + c) - 1;
        bytes += 0.5 * m * (m + 1) * sizeof(float2);
    }
    kt_end(ev, s, KC_TRI_PANEL, bytes * w.batch);
    return true;
}

// Launches the panel kernel; returns false if no cluster can be scheduled.
// A column costs about 7 us of latency chain whatever CL is, plus the CTA's share of the
// mat-vec, and a second wave doubles both: so the largest cluster whose matrices all fit
// the device at once, no larger than the trailing row tiles.  16 warps fill an SM by
// themselves; where the matrices don't fit, two CTAs of eight warps share it as long as
// their memory does (five tiles), and one CTA has the whole matrix, so no partial crosses
// CTAs.  Panels of one solve, against clusters of eight CTAs of eight warps throughout:
//   n = 32,  63 matrices  (CL 1)        1.24 -> 0.28 ms
//   n = 288, 36 matrices  (CL 2)        6.9  -> 3.4 ms
//   n = 1152, 14 matrices (CL 4)        33.0 -> 30.8 ms
//   n = 1404, 8 matrices  (CL 8)        37.0 -> 31.3 ms
// and whole calls whose matrices don't fit (two waves and more): n = 72, 600 matrices:
// 11.4 ms with 16 warps, 9.4 with CL 2, 7.9 as here; n = 144, 400 matrices: 19.1, 16.1, 14.5.
// Clusters of 16 gained nothing (n = 1300, one matrix: panels 26.5 against 26.7 ms), though
// each SM then has half of the mat-vec: what the SMs of a cluster, which are neighbours,
// can read from L2 together seems to set the pace.
inline bool tri_panel_launch(cudaStream_t s, const EigWork<float> &w, int j0, int jb)
{
    const int tiles = cdiv(w.n, 32), left = cdiv(w.n - j0, 32);
    if (tp_by_warp(tiles)) return tp_try<8, 16>(s, w, j0, jb, false);
    return (left > 4 && tp_try<8, 16>(s, w, j0, jb, true)) || (left > 2 && tp_try<4, 16>(s, w, j0, jb, true)) ||
           (left > 1 && tp_try<2, 16>(s, w, j0, jb, true)) || (tiles <= 5 && tp_try<1, 8>(s, w, j0, jb, false)) || tp_try<1, 16>(s, w, j0, jb, false) ||
           tp_try<2, 16>(s, w, j0, jb, false) || tp_try<4, 16>(s, w, j0, jb, false) ||
           tp_try<8, 16>(s, w, j0, jb, false);
}

}  // namespace nrltb
