// tri_cluster.cuh -- Householder tridiagonalisation of an FP64 matrix, or of the trailing
// part of one, in one launch: a cluster per matrix, its lower triangle resident in the
// CTAs' shared memory as 32 x 32 tiles.
//
// As in tri_small.cuh each column's reflector is applied at once (y = A v,
// w = tau y - |tau|^2 (v^H y) v / 2, A -= v w^H + w v^H), nothing is put off.  Tiles are
// numbered from the last one outwards, so that every trailing triangle is a prefix of the
// numbers, and dealt to the CTAs in turn: each has an equal share of every column's work.
// Per column:
//   A  y partials: a warp takes a row block (or a share of its tiles' columns) and sums its
//      tiles' products in registers, tiles left of the diagonal by rows, those below it by
//      columns; the CTA's sums go to every CTA                                  barrier
//   B  every CTA adds the CTAs' sums, in order, and forms v^H y and w
//   C  the next column is updated by its tiles' owners and sent to every CTA    barrier
//   D  warp 0 makes its reflector (every CTA the same); the other warps, and then it too,
//      update the rest of the triangle
// Diagonal tiles are kept whole.  A tile's element (r, c) lies at 32 c + (r ^ (c & 7)), so
// that neither direction of access has bank conflicts (16-byte elements, 8 per phase).
//
// Results don't depend on the cluster size: y's partials are kept for eight ranks, tile
// number mod 8, and added in order, whichever CTA has them.  Work is dealt to warps by a
// counter, but a unit's result does not depend on who computes it.
//
// Bound: the FP64 pipe for A and D (8 FMAs per element of the trailing matrix), and a chain
// of about 7 us a column (n = 128, eight CTAs: 9 us in all): two cluster barriers, and sums
// and scalars whose operations take 64 cycles of an SM's quarter each.
// Against two launches a column (tri_col.cuh), whole tridiagonalisations: n = 144 2.8 -> 1.5 ms
// (4 matrices), 3.6 -> 1.9 (36), 7.1 -> 5.2 (150); by columns n = 180 takes 3.6, 5.1 and 10.8 ms,
// here n = 192 2.3, 2.9 and 8.0; n = 288, the last 192 columns here: 6.4 -> 4.7 ms (4), 14.7 ->
// 11.2 (64).
#pragma once
#include <cooperative_groups.h>
#include "eig.cuh"
#include "tri_col.cuh"

namespace nrltb {

// 16 warps cover each other's latencies better than 8: n = 144 1.53 -> 1.46 ms with 15 matrices,
// 2.16 -> 1.87 with 36, 2.9 -> 2.6 with 64
constexpr int TK_THREADS = 512, TK_WARPS = TK_THREADS / 32;
constexpr int TK_RANKS = 8;     // y is summed as by eight CTAs, whatever the cluster size
constexpr int TK_MAX = 192;     // the largest order whose triangle two CTAs hold

struct TkSizes {
    int T, ntiles, slots, np;
    __host__ __device__ TkSizes(int m, int cl) : T((m + 31) / 32), ntiles(T * (T + 1) / 2), slots((ntiles + cl - 1) / cl), np(32 * T) {}
    // elements for the shares of y of one rank: what two CTAs' memory leaves beside the tiles
    __host__ __device__ int part_size() const { return T <= 5 ? 640 : 256; }
    // tiles | v of two columns | w | y of each rank | shares of y | sums per warp, scalars, counters | tile numbers
    __host__ __device__ int bytes(int cl) const
    {
        return 16 * (1024 * slots + (3 + TK_RANKS) * np + part_size() * (TK_RANKS / cl)) + 8 * (TK_WARPS + 8) + 16 + 4 * slots;
    }
};

template <int CL>
__global__ void __launch_bounds__(TK_THREADS, 1) k_tri_cluster(EigWork<double> w, int j0)
{
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char tk_raw[];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int b = blockIdx.y, n = w.n - j0, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long ld = w.ld;
    const TkSizes z(n, CL);
    const int T = z.T, np = z.np;
    double2 *const tiles = (double2 *)tk_raw, *const vb = tiles + 1024 * z.slots, *const wv = vb + 2 * np;
    constexpr int NR = TK_RANKS / CL;   // ranks of this CTA: rank + CL j
    double2 *const ybuf = wv + np, *const part = ybuf + TK_RANKS * np;
    double *const red = (double *)(part + z.part_size() * NR), *const sc = red + TK_WARPS;   // sc[4 p ..]: tau and scale of parity p
    int *const ctr = (int *)(sc + 8);
    short2 *const tab = (short2 *)(ctr + 4);   // row and column block of each own tile
    const double2 *A = w.A + b * w.mstride + j0 * (ld + 1);
    double2 *V = w.V + b * w.mstride + j0 * ld, *tau_out = w.tau + (long)b * w.n + j0;
    double *d = w.d + (long)b * w.n + j0, *e = w.e + (long)b * w.n + j0;
    const double2 zero = make_double2(0, 0);
    // number of tile (R, C), C <= R
    auto number = [&](int R, int C) { return (T - 1 - C) * (T - C) / 2 + T - 1 - R; };
    auto cell = [](int r, int c) { return 32 * c + (r ^ (c & 7)); };

    for (int C = 0; C < T; ++C)
        for (int R = C; R < T; ++R) {
            const int q = number(R, C);
            if (q % CL != rank) continue;
            if (tid == 0) tab[q / CL] = make_short2((short)R, (short)C);
            double2 *t = tiles + 1024 * (q / CL);
            for (int c = warp; c < 32; c += TK_WARPS) {
                const int gr = 32 * R + lane, gc = 32 * C + c;
                double2 x = zero;
                if (gr < n && gc < n) {
                    if (gr >= gc) x = A[gr + gc * ld];
                    else {
                        x = A[gc + gr * ld];
                        x.y = -x.y;
                    }
                    if (gr == gc) x.y = 0;
                }
                t[cell(lane, c)] = x;
            }
        }
    for (int c = rank; c < n; c += CL)
        for (int r = tid; r <= j0 + c; r += TK_THREADS) V[r + c * ld] = zero;
    for (int r = tid; r < 3 * np; r += TK_THREADS) vb[r] = zero;
    if (tid < 4) ctr[tid] = 0;
    __syncthreads();
    cluster.sync();   // the buffers are cleared before anyone sends to them

    auto send = [&](double2 *at, double2 x) {
#pragma unroll
        for (int k = 0; k < CL; ++k) *cluster.map_shared_rank(at, k) = x;
    };
    // C: column i1 of the own tiles, updated, to every CTA's v buffer of its parity
    auto head = [&](int i1, const double2 *v, bool apply) {
        const int C = i1 / 32, c = i1 % 32;
        for (int R = C + warp; R < T; R += TK_WARPS) {
            const int q = number(R, C);
            if (q % CL != rank) continue;
            double2 x = tiles[1024 * (q / CL) + cell(lane, c)];
            const int r = 32 * R + lane;
            if (apply) {
                const double2 vr = v[r], wr = wv[r], vc = v[i1], wc = wv[i1];
                x.x = fma(-vr.x, wc.x, x.x);
                x.x = fma(-vr.y, wc.y, x.x);
                x.x = fma(-wr.x, vc.x, x.x);
                x.x = fma(-wr.y, vc.y, x.x);
                x.y = fma(vr.x, wc.y, x.y);
                x.y = fma(-vr.y, wc.x, x.y);
                x.y = fma(wr.x, vc.y, x.y);
                x.y = fma(-wr.y, vc.x, x.y);
            }
            send(vb + (i1 & 1) * np + r, x);
        }
    };
    // D, warp 0: the reflector of column i in place of its elements
    auto reflect = [&](int i) {
        double2 *u = vb + (i & 1) * np;
        double xn2 = 0;
        for (int r = i + 2 + lane; r < n; r += 32) {
            xn2 = fma(u[r].x, u[r].x, xn2);
            xn2 = fma(u[r].y, u[r].y, xn2);
        }
        xn2 = warp_sum(xn2);   // (the same in every lane)
        const double dd = u[i].x;
        if (rank == 0 && lane == 0) d[i] = dd;
        if (i == n - 1) return;
        const double2 al = u[i + 1];
        double2 tau, scale;
        double beta;
        tc_reflector(al, xn2, tau, scale, beta);
        double *s = sc + 4 * (i & 1);
        if (lane == 0) {
            s[0] = tau.x;
            s[1] = tau.y;
            s[2] = scale.x;
            s[3] = scale.y;
            if (rank == 0) {
                e[i] = beta;
                tau_out[i] = tau;
            }
        }
    };
    // v of column i in place of its elements, by all threads
    auto scaled = [&](int i) {
        double2 *u = vb + (i & 1) * np;
        const double2 scale = make_double2(sc[4 * (i & 1) + 2], sc[4 * (i & 1) + 3]);
        for (int r = i / 32 * 32 + tid; r < np; r += TK_THREADS) {
            const double2 v = r <= i || r >= n ? zero : r == i + 1 ? make_double2(1, 0) : cmul(u[r], scale);
            u[r] = v;
            if (r > i && r < n && r / 32 % CL == rank) V[j0 + r + i * ld] = v;
        }
    };
    auto grab = [&](int *c) {
        int u = 0;
        if (lane == 0) u = atomicAdd(c, 1);
        return __shfl_sync(0xffffffffu, u, 0);
    };
    head(0, vb, false);
    cluster.sync();
    if (warp == 0) reflect(0);
    __syncthreads();
    scaled(0);
    __syncthreads();

    for (int i = 0; i < n - 1; ++i) {
        const int i1 = i + 1, tb = i1 / 32;
        const double2 *v = vb + (i & 1) * np;
        const double *s = sc + 4 * (i & 1);
        const double tx = s[0], ty = s[1];
        const bool apply = tx != 0 || ty != 0;   // (the same in every CTA)
        if (apply) {
            // ---- A ----
            if (tid == 0) ctr[1] = 0;
            // (shares of a row block's columns: K rows <= part_size)
            const int nb = T - tb, rows = 32 * nb, K = T <= 5 ? (nb <= 2 ? 8 : 4) : nb <= 2 ? 4 : nb <= 4 ? 2 : 1, W = 32 / K;
            for (int un = grab(ctr); un < nb * K * NR; un = grab(ctr)) {
                const int j = un % NR, k = un / NR % K, R = T - 1 - un / (NR * K), k0 = k * W, rk = rank + CL * j;
                double2 acc = zero;
                for (int X = tb; X < T; ++X) {
                    const int q = X <= R ? number(R, X) : number(X, R);
                    if (q % TK_RANKS != rk) continue;
                    const double2 *t = tiles + 1024 * (q / CL);
                    const double2 *vx = v + 32 * X;
                    const int lo = X == tb ? max(k0, i1 - 32 * tb) : k0;
                    if (X <= R) {
#pragma unroll 4
                        for (int c = lo; c < k0 + W; ++c) cfma(acc, t[cell(lane, c)], vx[c]);
                    } else {
#pragma unroll 4
                        for (int r = lo; r < k0 + W; ++r) cfmac(acc, t[cell(r, lane)], vx[r]);
                    }
                }
                if (K == 1) send(ybuf + rk * np + 32 * R + lane, acc);
                else part[(j * K + k) * rows + 32 * (R - tb) + lane] = acc;
            }
            if (K > 1) {
                __syncthreads();
                for (int t = tid; t < NR * rows; t += TK_THREADS) {
                    const int j = t / rows, r = t - j * rows;
                    double2 y = part[j * K * rows + r];
                    for (int k = 1; k < K; ++k) y = cadd(y, part[(j * K + k) * rows + r]);
                    send(ybuf + (rank + CL * j) * np + 32 * tb + r, y);
                }
            }
        }
        cluster.sync();
        if (apply) {
            // ---- B ----
            if (tid == 0) ctr[0] = 0;
            const int r = 32 * tb + tid;   // (a row a thread)
            double2 y = zero;
            if (32 * (tb + warp) < np) {
#pragma unroll
                for (int k = 0; k < TK_RANKS; ++k) y = cadd(y, ybuf[k * np + r]);
                const double dot = warp_sum(fma(v[r].y, y.y, v[r].x * y.x));
                if (lane == 0) red[warp] = dot;
            }
            __syncthreads();
            if (32 * (tb + warp) < np) {
                double sum = red[0];
                for (int q = 1; 32 * (tb + q) < np; ++q) sum += red[q];
                sum *= 0.5 * (tx * tx + ty * ty);
                const double2 x = v[r];
                wv[r] = r <= i || r >= n ? zero
                                         : make_double2(fma(-sum, x.x, fma(-ty, y.y, tx * y.x)),
                                                        fma(-sum, x.y, fma(ty, y.x, tx * y.y)));
            }
            __syncthreads();
        }
        head(i1, v, apply);
        cluster.barrier_arrive();
        // ---- D ----
        if (warp == 0) {
            cluster.barrier_wait();
            reflect(i1);
        }
        // (the warp that shares warp 0's quarter of the SM leaves it the FP64 pipe until then)
        if (warp % 4 == 0) asm volatile("bar.sync 1, %0;" :: "n"(TK_THREADS / 4) : "memory");
        if (apply) {
            const int tb2 = (i1 + 1) / 32, k2 = T - tb2, cnt = (k2 * (k2 + 1) / 2 - rank + CL - 1) / CL;
            for (int un = grab(ctr + 1); un < 8 * cnt; un = grab(ctr + 1)) {
                const short2 rc = tab[un >> 3];
                double2 *t = tiles + 1024 * (un >> 3);
                const int r = 32 * rc.x + lane, c0 = 32 * rc.y, hi = 4 * (un & 7) + 4;
                const double2 vr = v[r], wr = wv[r];
                int c = max(hi - 4, i1 + 1 - c0);
#pragma unroll 4
                for (; c < hi; ++c) {
                    const double2 vc = v[c0 + c], wc = wv[c0 + c];
                    double2 x = t[cell(lane, c)];
                    x.x = fma(-vr.x, wc.x, x.x);
                    x.x = fma(-vr.y, wc.y, x.x);
                    x.x = fma(-wr.x, vc.x, x.x);
                    x.x = fma(-wr.y, vc.y, x.x);
                    x.y = fma(vr.x, wc.y, x.y);
                    x.y = fma(-vr.y, wc.x, x.y);
                    x.y = fma(wr.x, vc.y, x.y);
                    x.y = fma(-wr.y, vc.x, x.y);
                    if (r == c0 + c) x.y = 0;
                    t[cell(lane, c)] = x;
                }
            }
        }
        if (warp != 0) cluster.barrier_wait();
        __syncthreads();
        if (i1 < n - 1) scaled(i1);
        __syncthreads();
    }
    cluster.sync();   // no CTA leaves while others may send to it
}

template <int CL> inline bool tk_try(cudaStream_t s, const EigWork<double> &w, int j0, bool must_fit)
{
    const TkSizes z(w.n - j0, CL);
    const int smem = z.bytes(CL);
    const void *f = (const void *)k_tri_cluster<CL>;
    const Refusable r;   // another size, or the column kernels, take over
    if (smem_attr_at_least(f, smem) != cudaSuccess) {
        r.clear();
        return false;
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(CL, w.batch, 1);
    cfg.blockDim = dim3(TK_THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (must_fit) {
        int count = 0;
        if (cudaOccupancyMaxActiveClusters(&count, k_tri_cluster<CL>, &cfg) != cudaSuccess) {
            r.clear();
            return false;
        }
        if (count < w.batch) return false;
    }
    if (cudaLaunchKernelEx(&cfg, k_tri_cluster<CL>, w, j0) != cudaSuccess) {
        r.clear();
        return false;
    }
    if (g_launch_counter) ++*g_launch_counter;
    return true;
}

// The columns from j0 on in one launch; false if they don't fit or no cluster can be scheduled.
// The cluster is the largest whose matrices all fit the device at once (the chain is the same,
// the shares of the FP64 work shorter): n = 144: 1.46 ms with eight CTAs (15 matrices), 1.87 with
// four (36), 2.6 with two (64).  Larger triangles need four CTAs and more, and were faster here
// only while they fit in one wave (n = 288, 8 warps: 36 matrices 7.2 ms against 10.9 by columns,
// 64 matrices 14.3 against 14.7); taking the last 192 columns alone is as fast in the first
// case (8.3) and better in the second (11.2), and goes by the order alone, so that a matrix
// has the same result in every batch.
inline bool tri_cluster(cudaStream_t s, const EigWork<double> &w, int j0)
{
    if (w.n - j0 > TK_MAX) return false;
    return tk_try<8>(s, w, j0, true) || tk_try<4>(s, w, j0, true) || tk_try<2>(s, w, j0, false);
}

}  // namespace nrltb
