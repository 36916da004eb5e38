// tri_small.cuh -- Householder tridiagonalisation of small FP64 matrices in one launch,
// a CTA per matrix, the lower triangle resident in shared memory.
//
// The packed lower triangle fits a CTA's shared memory, so nothing is put off: each column's reflector is applied to the whole trailing matrix at once (y = A v,
// w = tau y - |tau|^2 (v^H y) v / 2, A -= v w^H + w v^H).
//
// Bound: the FP64 pipe, 8 FMAs per element of the trailing matrix and column (4 in the
// mat-vec, which takes every element twice, 8 per element of the triangle in the update);
// a warp's FP64 operation takes 64 cycles of its quarter of the SM.  What follows from it:
//  - a mat-vec thread owns a row and a share of the columns and reads both halves through
//    the one triangle, so nothing is summed across lanes; shared memory, at 1 or 2 loads
//    per 4 FMAs, has the time for the strided half;
//  - rows x shares are dealt to threads without gaps, in as many shares as leave the four
//    quarters the least time (share_count);
//  - the scalars of a column take one root and two reciprocals, by one warp, which first
//    brings the next column up to date and then works on its reflector while the other
//    warps update the rest of the triangle.
// Against two launches a column (tri_col.cuh), whole tridiagonalisations: n = 9 108 -> 43 us
// (4 matrices), 920 -> 77 us (1728); n = 36 736 -> 186 us, n = 64 1311 -> 532 us, n = 108
// 2586 -> 1395 us (36 matrices each), of which the FP64 pipe needs 820.
#pragma once
#include "eig.cuh"
#include "tri_col.cuh"

namespace nrltb {

// Above, a cluster (tri_cluster.cuh) is faster unless there are hundreds of matrices: n = 128
// 2.1 ms here, 1.13 to 1.7 ms there for 1 to 64 matrices, 3.4 for 150; below, n = 108, 1.4 ms
// against 1.1 to 1.6 and 2.3.  The rule goes by the order alone, so that a matrix has the same
// result in every batch.
constexpr int TS_MAX = 112;

inline int ts_threads(int n) { return n <= 16 ? 32 : n <= 32 ? 64 : n <= 64 ? 128 : n <= 96 ? 256 : 512; }
// triangle | v, two columns' | w | partial y | sums per warp | scalars of two columns, counter | shares per order
inline size_t ts_smem(int n, int nt)
{
    return sizeof(double2) * ((size_t)n * (n + 1) / 2 + 3 * (size_t)n + nt) + sizeof(double) * (nt / 32 + 8) +
           sizeof(int) * 2 + (size_t)n;
}

// shares of the columns for a mat-vec of order m on nt threads: above n = 96, where an SM holds two
// matrices at most, as many as there are threads, for warps to cover each other's latencies (16
// warps against 8 of the other rule, n = 108: 4 to 121 matrices 1.62 -> 1.40 ms, 300 matrices
// 2.45 -> 2.50, 600 4.89 -> 4.87); else, with other matrices to do that, the rounds of warps
// over the four quarters times the columns of a share, and the addition of the shares
__device__ inline int ts_share_count(int m, int nt)
{
    if (nt > 256) return min(nt / m, m);
    int best = 1, cost = 1 << 30;
    for (int k = 1; k * m <= nt && k <= m; ++k) {
        const int c = 8 * ((((m * k + 31) / 32) + 3) / 4) * ((m + k - 1) / k) + 4 * k * ((m + 127) / 128);
        if (c < cost) {
            cost = c;
            best = k;
        }
    }
    return best;
}

__global__ void __launch_bounds__(512) k_tri_small(EigWork<double> w)
{
    extern __shared__ __align__(16) unsigned char ts_raw[];
    const int b = blockIdx.x, n = w.n, nt = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long ld = w.ld;
    double2 *const a = (double2 *)ts_raw, *const vb = a + n * (n + 1) / 2, *const wv = vb + 2 * n, *const part = wv + n;
    double *const red = (double *)(part + nt), *const sc = red + nt / 32;   // sc[4 p ..]: tau and scale of parity p
    int *const ctr = (int *)(sc + 8);
    unsigned char *const shares = (unsigned char *)(ctr + 2);
    auto off = [&](int j) { return j * n - j * (j - 1) / 2; };   // of element (j, j)
    const double2 *A = w.A + b * w.mstride;
    double2 *V = w.V + b * w.mstride, *tau_out = w.tau + (long)b * n;
    double *d = w.d + (long)b * n, *e = w.e + (long)b * n;
    const double2 zero = make_double2(0, 0);

    for (int c = warp; c < n; c += nt / 32) {
        const int o = off(c);
        for (int r = lane; r < n; r += 32) {
            if (r >= c) a[o + r - c] = A[r + c * ld];
            if (r <= c) V[r + c * ld] = zero;
        }
    }
    for (int m = 1 + tid; m < n; m += nt) shares[m] = (unsigned char)ts_share_count(m, nt);
    __syncthreads();

    // warp 0: reflector of column i from its current elements, into buffer i & 1
    auto reflect = [&](int i) {
        const int m = n - 1 - i, p = i & 1;
        const double2 *u = a + off(i) + 1;
        if (lane == 0) d[i] = u[-1].x;
        if (m == 0) return;
        double xn2 = 0;
        for (int q = 1 + lane; q < m; q += 32) {
            xn2 = fma(u[q].x, u[q].x, xn2);
            xn2 = fma(u[q].y, u[q].y, xn2);
        }
        xn2 = warp_sum(xn2);   // (the same in every lane)
        const double2 al = u[0];
        double2 tau, scale;
        double beta;
        tc_reflector(al, xn2, tau, scale, beta);
        if (lane == 0) {
            e[i] = beta;
            tau_out[i] = tau;
            sc[4 * p] = tau.x;
            sc[4 * p + 1] = tau.y;
            sc[4 * p + 2] = scale.x;
            sc[4 * p + 3] = scale.y;
        }
    };
    // its v, by all threads
    auto scaled = [&](int i) {
        const int m = n - 1 - i, p = i & 1;
        const double2 *u = a + off(i) + 1;
        if (tid < m) {
            const double2 v = tid == 0 ? make_double2(1, 0) : cmul(u[tid], make_double2(sc[4 * p + 2], sc[4 * p + 3]));
            vb[p * n + tid] = v;
            V[i + 1 + tid + i * ld] = v;
        }
    };
    if (warp == 0) reflect(0);
    __syncthreads();
    scaled(0);
    __syncthreads();

    for (int i = 0; i < n - 1; ++i) {
        const int m = n - 1 - i, i1 = i + 1;
        const double2 *v = vb + (i & 1) * n;
        const double tx = sc[4 * (i & 1)], ty = sc[4 * (i & 1) + 1];
        const bool apply = tx != 0 || ty != 0;
        if (tid == 0) *ctr = 0;
        if (apply) {
            // y = A v: thread (row q, share) over the share's columns
            const int K = shares[m], L = (m + K - 1) / K;
            if (tid < m * K) {
                const int ch = tid / m, q = tid - ch * m, hi = min(m, ch * L + L);
                int c = ch * L;
                const int rowq = off(i1 + q) - q;                          // element (c, q) at rowq + c
                int colc = off(i1 + c) - c + q, step = n - (i1 + c) - 1;   // element (q, c); to the next column
                double2 acc = zero;
#pragma unroll 4
                for (; c < hi; ++c) {
                    const double2 x = a[c <= q ? colc : rowq + c], vc = v[c];
                    const double xy = c < q ? x.y : c == q ? 0.0 : -x.y;
                    acc.x = fma(x.x, vc.x, acc.x);
                    acc.y = fma(x.x, vc.y, acc.y);
                    acc.x = fma(-xy, vc.y, acc.x);
                    acc.y = fma(xy, vc.x, acc.y);
                    colc += step--;
                }
                part[tid] = acc;
            }
            __syncthreads();
            double2 y = zero;
            const bool row = tid < m;
            if (32 * warp < m) {
                double s = 0;
                if (row) {
                    y = part[tid];
                    for (int k = 1; k < K; ++k) y = cadd(y, part[tid + k * m]);
                    s = fma(v[tid].y, y.y, v[tid].x * y.x);
                }
                s = warp_sum(s);
                if (lane == 0) red[warp] = s;
            }
            __syncthreads();
            if (row) {
                double s = red[0];
                for (int q = 1; 32 * q < m; ++q) s += red[q];
                s *= 0.5 * (tx * tx + ty * ty);
                const double2 x = v[tid];
                wv[tid] = make_double2(fma(-s, x.x, fma(-ty, y.y, tx * y.x)), fma(-s, x.y, fma(ty, y.x, tx * y.y)));
            }
        }
        __syncthreads();
        // element (r, c) of the trailing matrix, c <= r
        auto update = [&](int at, int r, int c) {
            const double2 vr = v[r], wr = wv[r], vc = v[c], wc = wv[c];
            double2 x = a[at];
            x.x = fma(-vr.x, wc.x, x.x);
            x.x = fma(-vr.y, wc.y, x.x);
            x.x = fma(-wr.x, vc.x, x.x);
            x.x = fma(-wr.y, vc.y, x.x);
            x.y = fma(vr.x, wc.y, x.y);
            x.y = fma(-vr.y, wc.x, x.y);
            x.y = fma(wr.x, vc.y, x.y);
            x.y = fma(-wr.y, vc.x, x.y);
            if (r == c) x.y = 0;
            a[at] = x;
        };
        if (warp == 0) {
            if (apply)
                for (int r = lane; r < m; r += 32) update(off(i1) + r, r, 0);
            __syncwarp();
            reflect(i1);
        }
        // (the warps that share warp 0's quarter of the SM leave it the FP64 pipe until then)
        if (nt > 128 && warp % 4 == 0) asm volatile("bar.sync 1, %0;" :: "r"(nt / 4) : "memory");
        if (apply) {
            // columns 1 .. m - 1, c and m - c together (m elements), in turns of 64 elements
            const int tot = m * (m - 1) / 2;
            for (;;) {
                int e0 = 0;
                if (lane == 0) e0 = atomicAdd(ctr, 64);
                e0 = __shfl_sync(0xffffffffu, e0, 0);
                if (e0 >= tot) break;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int el = e0 + 32 * u + lane;
                    if (el < tot) {
                        const int pr = el / m, q = el - pr * m, len = m - 1 - pr;   // of column 1 + pr
                        const int c = q < len ? 1 + pr : len, r = q < len ? c + q : c + q - len;
                        update(off(i1 + c) + r - c, r, c);
                    }
                }
            }
        }
        __syncthreads();
        scaled(i1);
        __syncthreads();
    }
}

inline void tri_small(cudaStream_t s, const EigWork<double> &w)
{
    const int nt = ts_threads(w.n);
    const size_t sm = ts_smem(w.n, nt);
    if (sm > 48 * 1024) smem_attr_at_least((const void *)k_tri_small, (int)sm);
    NRLTB_LAUNCH(k_tri_small, w.batch, nt, sm, s, w);
}

}  // namespace nrltb
