// eig.cu -- batched generalized Hermitian eigensolver (see eig.cuh for the plan).
#include <algorithm>
#include <cfloat>
#include "eig.cuh"
#include "tri_col.cuh"
#include "tri_panel.cuh"
#include "tri_small.cuh"
#include "tri_cluster.cuh"

namespace nrltb {

template <typename T> __host__ __device__ inline T eps_of();
template <> __host__ __device__ inline float eps_of<float>() { return FLT_EPSILON * 0.5f; }
template <> __host__ __device__ inline double eps_of<double>() { return DBL_EPSILON * 0.5; }

static inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

template <typename T> size_t eig_work_bytes(int n, int batch)
{
    EigWork<T> w;
    eig_work_carve<T>(w, nullptr, n, batch);
    return (size_t)w.status + sizeof(int) * (size_t)batch;  // carve from 0 gives the size
}

template <typename T> void eig_work_carve(EigWork<T> &w, void *base, int n, int batch)
{
    typedef typename cplx<T>::t C2;
    size_t off = 0;
    char *b = (char *)base;
    auto take = [&](size_t bytes) { void *p = b + off; off = align256(off + bytes); return p; };
    const size_t nn = (size_t)n * n, nb = (size_t)batch;
    w.n = n; w.batch = batch; w.ld = n; w.mstride = (long)nn;
    w.L = (C2 *)take(sizeof(C2) * nn * nb);
    w.Wi = (C2 *)take(sizeof(C2) * nn * nb);
    w.A = (C2 *)take(sizeof(C2) * nn * nb);
    w.Y = (C2 *)take(sizeof(C2) * nn * nb);
    w.V = (C2 *)take(sizeof(C2) * nn * nb);
    w.VW = (C2 *)take(sizeof(C2) * n * 3 * EIG_NB * nb);
    w.wps = (long)n * 3 * EIG_NB;
    w.Wp = w.VW + (long)n * EIG_NB;
    w.wq = (C2 *)take(sizeof(C2) * n * nb);
    w.col = (C2 *)take(sizeof(C2) * n * nb);
    w.tau = (C2 *)take(sizeof(C2) * n * nb);
    w.npart = (long)tc_part_count(n);
    w.part = (C2 *)take(sizeof(C2) * w.npart * nb);
    w.nyp = (long)tc_y_count(n);
    w.yp = (C2 *)take(sizeof(C2) * w.nyp * nb);
    const size_t nbw = (size_t)std::min(EIG_WY, n), nblk = n > 1 ? (size_t)cdiv(n - 1, (int)nbw) : 0;
    w.Tt = (C2 *)take(sizeof(C2) * (EIG_NAUX + nblk) * nbw * nbw * nb);   // G per aux stream | T of each block
    w.Xt = (C2 *)take(sizeof(C2) * std::max(EIG_NB, (int)nbw) * (size_t)n * nb);
    w.d = (double *)take(sizeof(double) * n * nb);
    w.e = (double *)take(sizeof(double) * n * nb);
    w.lam = (double *)take(sizeof(double) * n * nb);
    // inverse iteration: 6 arrays of n per thread slot, 64 cdiv(n, 64) slots per matrix
    w.ylu = (double *)take(sizeof(double) * 4 * (size_t)n * (64 * (size_t)cdiv(n, 64)) * nb);
    w.yvec = (double *)take(sizeof(double) * nn * nb);
    w.perm = (int *)take(sizeof(int) * 4 * n * nb);
    w.status = (int *)take(sizeof(int) * nb);
    if (!base) w.status = (int *)(uintptr_t)off;  // size query
}

// ---------------------------------------------------------------------------
// The FP64 form solves for D H D and D S D with D_i the power of two that brings S_ii into
// [1, 4).  Its products are exact in digits of one scale per row and per column of an
// operand, but not along their inner index: in L^{-1} times L or L^{-1} times H the scale
// of the basis functions runs along it, the other way in either factor, and a basis whose
// norms differ by 1e4 would cost eight digits.  Every step is as exact with D as without;
// overlaps with a diagonal of ones, as tight binding has, are copied as they are.
// S_ii that is not a positive normal number (the factorisation will fail there): D_i = 1.
__global__ void k_unit_exp(const double2 *S, int *ex, int n, int batch)
{
    const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (t >= (long)n * batch) return;
    const long b = t / n;
    const int i = (int)(t - b * n);
    const long long bits = __double_as_longlong(S[b * n * n + i * (n + 1L)].x);
    const int e = (int)(bits >> 52);   // negative for negative numbers
    ex[t] = (e >= 1 && e <= 2046) ? -((e - 1023) >> 1) : 0;
}

// L = D S D, A = D H D
__global__ void k_to_unit(const double2 *__restrict__ S, const double2 *__restrict__ H, double2 *__restrict__ L,
                          double2 *__restrict__ A, const int *ex, int n)
{
    const unsigned nn = (unsigned)n * n, b = blockIdx.y;
    const long at = b * (long)nn;
    ex += (long)b * n;
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < nn; t += gridDim.x * blockDim.x) {
        const unsigned c = t / n, r = t - c * n;
        double2 s = S[at + t], h = H[at + t];
        const int er = ex[r], ec = ex[c];
        if (er | ec) {
            const double dr = __longlong_as_double((long long)(1023 + er) << 52);
            const double dc = __longlong_as_double((long long)(1023 + ec) << 52);
            s = make_double2(s.x * dr * dc, s.y * dr * dc);
            h = make_double2(h.x * dr * dc, h.y * dr * dc);
        }
        L[at + t] = s;
        A[at + t] = h;
    }
}

// columns of Wi by D: X = (Wi D)^H Z then has the vectors of H and S
__global__ void k_from_unit(double2 *Wi, const int *ex, int n)
{
    const int e = ex[(long)blockIdx.y * n + blockIdx.x];
    if (e == 0) return;
    const double d = __longlong_as_double((long long)(1023 + e) << 52);
    double2 *w = Wi + blockIdx.y * (long)n * n + blockIdx.x * (long)n;
    for (int r = threadIdx.x; r < n; r += blockDim.x) w[r] = make_double2(w[r].x * d, w[r].y * d);
}

__global__ void k_convert_h(const double2 *__restrict__ src, float2 *__restrict__ dst, long count)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < count; i += (long)gridDim.x * blockDim.x) {
        const double2 v = src[i];
        dst[i] = make_float2(d2f_rn(v.x), d2f_rn(v.y));   // rounded with integer operations, off the FP64 pipe
    }
}

// ---------------------------------------------------------------------------
// v s, each part rounded on its own (never contracted into a later add)
__device__ __forceinline__ float2 scale_rn(float2 v, float s) { return make_float2(__fmul_rn(v.x, s), __fmul_rn(v.y, s)); }

// Diagonal block: Cholesky L_jj L_jj^H = S_jj and its inverse, in shared memory (FP32).
__global__ void __launch_bounds__(256) k_potrf_diag(EigWork<float> w, int j0, int jb)
{
    typedef float T;
    typedef float2 C2;
    __shared__ C2 a[EIG_NB][EIG_NB + 1];   // a[c][r], updated in place
    __shared__ C2 x[EIG_NB][EIG_NB + 1];   // inverse, x[c][r]
    __shared__ int bad;
    const int b = blockIdx.x, tid = threadIdx.x;
    // lane = row r, warp = columns c = warp, warp + 8, ... (no index division)
    const int r = tid & 31, cg = tid >> 5;
    C2 *L = w.L + b * w.mstride + j0 + (long)j0 * w.ld;
    C2 *Wi = w.Wi + b * w.mstride + j0 + (long)j0 * w.ld;
    if (r < jb)
        for (int c = cg; c < jb; c += 8) a[c][r] = L[r + (long)c * w.ld];
    if (tid == 0) bad = 0;
    __syncthreads();
    // one barrier per column: every thread forms the pivot of column k itself,
    // and the scaled column k = a[k][.] / sqrt(pivot) on the fly for its
    // updates (the values the stored scaled column would hold).  Column k is
    // read but not written in step k; its finished values are written back by
    // its warp at the start of step k + 1, which reads only later columns.
    C2 held = cmk<T>(0, 0);
    int heldk = -1;
    for (int k = 0; k < jb; ++k) {
        if (heldk >= 0) { a[heldk][r] = held; heldk = -1; }
        T piv = a[k][k].x;
        const bool badk = !(piv > T(0));
        if (badk) piv = T(1);
        const T dk = sqrt(piv);
        const T inv = T(1) / dk;
        if (badk && tid == 0) bad = 1;
        if (r < jb && r >= k) {
            const C2 akr = r == k ? cmk<T>(dk, T(0)) : scale_rn(a[k][r], inv);
            if (cg == (k & 7)) { held = akr; heldk = k; }
            if (r > k) {
                int c = k + 1 + ((cg - (k + 1)) & 7);   // first column > k of this warp's group
                for (; c <= r; c += 8) a[c][r] = csub(a[c][r], cmul(akr, cconj(scale_rn(a[k][c], inv))));
            }
        }
        __syncthreads();
    }
    if (heldk >= 0) a[heldk][r] = held;
    __syncthreads();
    // inverse of the lower-triangular block, one column per thread
    if (tid < jb) {
        int c = tid;
        for (int rr = 0; rr < c; ++rr) x[c][rr] = cmk<T>(0, 0);
        x[c][c] = cmk<T>(T(1) / a[c][c].x, T(0));
        for (int rr = c + 1; rr < jb; ++rr) {
            C2 s = cmk<T>(0, 0);
            int k = c;
            for (; k + 8 <= rr; k += 8) {
                C2 av[8], xv[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    av[u] = a[k + u][rr];
                    xv[u] = x[c][k + u];
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) s = cadd(s, cmul(av[u], xv[u]));
            }
            for (; k < rr; ++k) s = cadd(s, cmul(a[k][rr], x[c][k]));
            x[c][rr] = cscale(s, -T(1) / a[rr][rr].x);
        }
    }
    __syncthreads();
    if (r < jb)
        for (int c = cg; c < jb; c += 8) {
            const C2 z = cmk<T>(0, 0);
            L[r + (long)c * w.ld] = (r >= c) ? a[c][r] : z;
            Wi[r + (long)c * w.ld] = (r >= c) ? x[c][r] : z;
        }
    if (tid == 0 && bad) w.status[b] = 1;
}

// ---------------------------------------------------------------------------
// Tridiagonal eigenvalues: Sturm-count bisection inside each unreduced block.
// The block of row r from per-row split flags (T splits between rows k and k + 1 where e[k]
// is negligible: |d_k d_(k+1)| ulp^2 + DBL_MIN >= e_k^2) in shared memory
__device__ inline void find_block_flags(const unsigned char *sp, int n, int r, int &b0, int &b1)
{
    b0 = r;
    while (b0 > 0 && !sp[b0 - 1]) --b0;
    b1 = r;
    while (b1 < n - 1 && !sp[b1]) ++b1;
}

// Quotient in the tridiagonal recurrences: FP32 takes the reciprocal-based
// quotient (2 ulp; |b| stays below 2^126 there), FP64 the IEEE one.  The FP32
// eigenpairs are refined to FP64 accuracy afterwards.
__device__ inline float tri_div(float a, float b) { return __fdividef(a, b); }
__device__ inline double tri_div(double a, double b) { return a / b; }

// Bounds of an unreduced block [b0, b1] of T: Gershgorin interval [lo, hi],
// max row sum tnorm and max e^2.  When every valid thread of the CTA is in
// the same block (the usual case: one block per matrix) the CTA computes them
// together, each thread a strided part, then min / max over the CTA (exact in
// any order, so the values equal the one-thread loop's); otherwise each
// thread loops over its own block.  Every thread of the CTA must call it.
__device__ void block_bounds(const double *d, const double *e, bool valid, int b0, int b1, double &lo, double &hi,
                             double &tnorm, double &emax2)
{
    __shared__ int sblk[2];
    __shared__ double sred[4][32];
    if (threadIdx.x == 0) { sblk[0] = b0; sblk[1] = b1; }
    __syncthreads();
    const int c0 = sblk[0], c1 = sblk[1];
    const bool all = __syncthreads_and(!valid || (b0 == c0 && b1 == c1));
    auto part = [&](int k0, int k1, int step, int kb0, int kb1) {
        for (int k = k0; k <= k1; k += step) {
            const double off = (k > kb0 ? fabs(e[k - 1]) : 0.0) + (k < kb1 ? fabs(e[k]) : 0.0);
            lo = fmin(lo, d[k] - off);
            hi = fmax(hi, d[k] + off);
            tnorm = fmax(tnorm, fabs(d[k]) + off);
            if (k < kb1) emax2 = fmax(emax2, e[k] * e[k]);
        }
    };
    if (!all) {
        if (valid) part(b0, b1, 1, b0, b1);
        return;
    }
    part(c0 + (int)threadIdx.x, c1, (int)blockDim.x, c0, c1);
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        tnorm = fmax(tnorm, __shfl_xor_sync(0xffffffffu, tnorm, o));
        emax2 = fmax(emax2, __shfl_xor_sync(0xffffffffu, emax2, o));
    }
    const int wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if ((threadIdx.x & 31) == 0) { sred[0][wid] = lo; sred[1][wid] = hi; sred[2][wid] = tnorm; sred[3][wid] = emax2; }
    __syncthreads();
    for (int q = 0; q < nw; ++q) {
        lo = fmin(lo, sred[0][q]);
        hi = fmax(hi, sred[1][q]);
        tnorm = fmax(tnorm, sred[2][q]);
        emax2 = fmax(emax2, sred[3][q]);
    }
}

// FP32 octasection (latency bound): seven independent Sturm chains per pass; the
// new interval lies between the last point counting <= j eigenvalues below it and
// the first counting more.  [a, z] shrinks to about atol.
__device__ __forceinline__ void octasect(const float *sd, const float *se2, int b0, int b1, int j, float atol,
                                         float pivmin, float &a, float &z)
{
    constexpr int NP = 7;
    const float eps = eps_of<float>();
    for (int it = 0; it < 64; ++it) {
        const float h = float(1.0 / (NP + 1)) * (z - a);
        const float tol = fmax(atol, 2.f * eps * fmax(fabs(a), fabs(z))) + pivmin;
        float m[NP];
        bool ok = z - a > tol;
#pragma unroll
        for (int i = 0; i < NP; ++i) m[i] = a + float(i + 1) * h;
        ok = ok && m[0] > a && m[NP - 1] < z;
#pragma unroll
        for (int i = 0; i + 1 < NP; ++i) ok = ok && m[i] < m[i + 1];
        if (!ok) break;
        float q[NP];
        int c[NP];
        const float d0 = sd[b0];
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            q[i] = d0 - m[i];
            if (fabs(q[i]) < pivmin) q[i] = -pivmin;
            c[i] = q[i] < 0.f;
        }
        for (int k = b0 + 1; k <= b1; ++k) {
            const float dk = sd[k], e2 = se2[k - 1];
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                q[i] = dk - m[i] - tri_div(e2, q[i]);
                if (fabs(q[i]) < pivmin) q[i] = -pivmin;
                c[i] += q[i] < 0.f;
            }
        }
        float na = a, nz = z;
        bool found = false;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            if (!found) {
                if (c[i] <= j) na = m[i];
                else { nz = m[i]; found = true; }
            }
        }
        a = na;
        z = nz;
    }
}

// One thread per (matrix, row r): eigenvalue number r - b0 of r's block, FP32.
// The matrix's d and e^2 in FP32 and the split flags of its rows are staged
// once per CTA in shared memory (2 n floats + n bytes of dynamic shared memory),
// so the Sturm chains read them without a conversion from FP64 per step and the
// block search needs no FP64 work (the values are the same).
__global__ void k_tri_bisect32(const double *dd, const double *ee, double *lamloc, int *blk, int n)
{
    extern __shared__ float bis_s[];
    const int b = blockIdx.y;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const double *d = dd + (long)b * n, *e = ee + (long)b * n;
    float *sd = bis_s, *se2 = bis_s + n;
    unsigned char *ssp = (unsigned char *)(bis_s + 2 * n);
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        sd[k] = d2f_rn(d[k]);
        const float ek = d2f_rn(e[k]);
        se2[k] = ek * ek;
        ssp[k] = k < n - 1 && fabs(d[k] * d[k + 1]) * DBL_EPSILON * DBL_EPSILON + DBL_MIN >= e[k] * e[k];
    }
    __syncthreads();
    const bool valid = r < n;
    int b0 = 0, b1 = -1;
    if (valid) find_block_flags(ssp, n, r, b0, b1);
    double tnorm = 0, lo = 1e300, hi = -1e300, emax2 = 0;
    block_bounds(d, e, valid, b0, b1, lo, hi, tnorm, emax2);
    if (!valid) return;
    const float eps = eps_of<float>();
    const float pivmin = FLT_MIN * float(fmax(1.0, emax2));
    const float atol = eps * float(tnorm);
    const int j = r - b0;
    float a = float(lo) - 2.f * atol - pivmin, z = float(hi) + 2.f * atol + pivmin;
    // Sturm count: eigenvalues of the block below x (from the shared copies, the
    // same values as converting d and e here)
    auto count = [&](float x) {
        int cnt = 0;
        float q = sd[b0] - x;
        if (fabs(q) < pivmin) q = -pivmin;
        cnt += (q < 0.f);
        for (int k = b0 + 1; k <= b1; ++k) {
            q = sd[k] - x - se2[k - 1] / q;
            if (fabs(q) < pivmin) q = -pivmin;
            cnt += (q < 0.f);
        }
        return cnt;
    };
    octasect(sd, se2, b0, b1, j, atol, pivmin, a, z);
    for (int it = 0; it < 256; ++it) {
        const float mid = 0.5f * (a + z);
        const float tol = fmax(atol, 2.f * eps * fmax(fabs(a), fabs(z))) + pivmin;
        if (!(z - a > tol) || mid == a || mid == z) break;
        if (count(mid) <= j) a = mid; else z = mid;
    }
    lamloc[(long)b * n + r] = (double)(0.5f * (a + z));
    blk[((long)b * n + r) * 2 + 0] = b0;
    blk[((long)b * n + r) * 2 + 1] = b1;
}

// FP64 eigenvalues.  The FP64 pipe is 1/64 of the FP32 one and a quotient takes a
// dozen of its operations, so (a) FP32 octasection on a scaled copy of T finds each
// eigenvalue to ~1e-7 ||T||, (b) an FP64 bracket around that is verified by Sturm
// counts, widening until it holds, and (c) it is closed on the zero of the
// characteristic polynomial by false position (Illinois weights, halved where that
// stalls or several eigenvalues share the bracket), every step kept by its count.
// Counts and polynomial values come from one recurrence without quotients,
//   p_k = (d_k - x) p_(k-1) - e_(k-1)^2 p_(k-2),
// three FP64 operations a step; sign changes count the eigenvalues below x
// (Givens), and the exponents of p_k, p_(k-1) are brought back by integer adds every
// fourth step.  A computed p_k is the exact one of entries d_k - x and e^2 changed by a
// few ulp, the same backward error as the quotient recurrence.  The bracket ends at
// the width the bisection alone ended at: max(eps ||T||, 2 eps |lambda|).
// About 9 recurrences an eigenvalue in place of 54 quotient ones:
// N = 1152, 4 k 36.7 -> 3.0 ms; N = 288, 64 k 15.8 -> 0.8 ms.
struct TriPoly {
    double m;      // mantissa part and binary exponent of p_n(x)
    int ex, cnt;   // eigenvalues of the block below x
};
// d(k), e2(k): the block's rows, scaled so that its norm is about 1 (2^-100 at least: four
// steps between two looks at the exponents must not leave the range)
template <typename D, typename E>
__device__ __forceinline__ TriPoly tri_poly(D d, E e2, int b0, int b1, double x)
{
    double p0 = 1.0, p1 = d(b0) - x;
    int ex = 0, cnt = 0;
    // an exact zero counts as a sign change (the quotient form's -pivmin)
    auto nz = [](double p, double prev) {
        if ((__double_as_longlong(p) << 1) == 0)
            p = __longlong_as_double((__double_as_longlong(prev) & (long long)0x8000000000000000ull) ^
                                     (long long)0x8000000000000000ull ^ (0x200ll << 52));
        return p;
    };
    auto step = [&](double dk, double ek2) {
        const double t = (dk - x) * p1;
        double p = fma(-ek2, p0, t);
        p = nz(p, p1);
        cnt += (int)((unsigned)(__double2hiint(p) ^ __double2hiint(p1)) >> 31);
        p0 = p1;
        p1 = p;
    };
    p1 = nz(p1, p0);
    cnt = (int)((unsigned)__double2hiint(p1) >> 31);
    int k = b0 + 1;
    for (; k + 4 <= b1 + 1; k += 4) {
        double dk[4], ek[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) { dk[u] = d(k + u); ek[u] = e2(k + u - 1); }
#pragma unroll
        for (int u = 0; u < 4; ++u) step(dk[u], ek[u]);
        const int e1 = (__double2hiint(p1) >> 20) & 0x7FF, e0 = (__double2hiint(p0) >> 20) & 0x7FF;
        const int em = max(e0, e1);
        if (em > 1023 + 300 || em < 1023 - 300) {
            // both by 2^(1023 - em); one that would leave the normal range goes to a signed 2^-1000
            const int sft = 1023 - em;
            auto sc = [&](double p, int ep) {
                const int en = ep + sft;
                const int keep = __double2hiint(p) & (int)0x800FFFFFu;
                return en > 20 ? __hiloint2double(keep | (en << 20), __double2loint(p))
                               : __hiloint2double((keep & (int)0x80000000u) | (23 << 20), 0);
            };
            p1 = sc(p1, e1);
            p0 = sc(p0, e0);
            ex -= sft;
        }
    }
    for (; k <= b1; ++k) step(d(k), e2(k - 1));
    TriPoly r;
    const int e1 = (__double2hiint(p1) >> 20) & 0x7FF;
    r.m = __hiloint2double((__double2hiint(p1) & (int)0x800FFFFFu) | (1023 << 20), __double2loint(p1));
    r.ex = ex + e1 - 1023;
    r.cnt = cnt;
    return r;
}

// Eigenvalue j of the block [b0, b1], known to lie in [glo, ghi] and thought to lie in [a, z],
// to `atol`.
template <typename D, typename E>
__device__ __forceinline__ double tri_close(D d, E e2, int b0, int b1, int j, double a, double z, double glo, double ghi,
                                            double tnorm, double atol)
{
    const double eps = eps_of<double>(), pivmin = DBL_MIN;
    TriPoly pa = tri_poly(d, e2, b0, b1, a), pz = tri_poly(d, e2, b0, b1, z);
    double h = 64.0 * (double)eps_of<float>() * tnorm;
    for (int t = 0; t < 16 && pa.cnt > j && a > glo; ++t, h *= 64.0) {
        z = a;
        pz = pa;
        a = fmax(glo, a - h);
        pa = tri_poly(d, e2, b0, b1, a);
    }
    h = 64.0 * (double)eps_of<float>() * tnorm;
    for (int t = 0; t < 16 && pz.cnt <= j && z < ghi; ++t, h *= 64.0) {
        a = z;
        pa = pz;
        z = fmin(ghi, z + h);
        pz = tri_poly(d, e2, b0, b1, z);
    }
    double wa = 1.0, wz = 1.0;   // Illinois weights of the two values
    int side = 0;                // which end moved last (+1 a, -1 z), doubled when twice in a row
    double width2 = 2.0 * (z - a);   // width two steps ago
    for (int it = 0; it < 256; ++it) {
        const double width = z - a, mid = a + 0.5 * width;
        const double tol = fmax(atol, 2.0 * eps * fmax(fabs(a), fabs(z))) + pivmin;
        if (!(width > tol) || mid <= a || mid >= z) break;
        double x = mid;
        const bool one = pz.cnt - pa.cnt == 1;
        if (one && !(it & 1 && width > 0.5 * width2)) {
            // zero of the line through the weighted values (they differ in sign)
            const int de = max(-1000, min(1000, pz.ex - pa.ex));
            const double fa = fabs(pa.m) * wa, fz = scalbn(fabs(pz.m) * wz, de);
            x = a + width * (fa / (fa + fz));
            // at least half a tolerance inside, so that the far end comes in too
            x = fmin(fmax(x, a + 0.5 * tol), z - 0.5 * tol);
            if (!(x > a && x < z)) x = mid;
        }
        if (it & 1) width2 = width;
        const TriPoly p = tri_poly(d, e2, b0, b1, x);
        if (p.cnt <= j) {
            a = x;
            pa = p;
            wa = 1.0;
            if (side > 0) wz *= 0.5;
            side = 1;
        } else {
            z = x;
            pz = p;
            wz = 1.0;
            if (side < 0) wa *= 0.5;
            side = -1;
        }
    }
    return a + 0.5 * (z - a);
}

// The same for a block that is smaller than the matrix by more than the shared copies' scale
// can serve: from d and e themselves, scaled by 2^-sx for this block (whose numbers
// lo, hi, tnorm are in that scale).
__device__ __noinline__ double tri_close_small(const double *dg, const double *eg, int sx, int b0, int b1, int j, double lo,
                                               double hi, double tnorm)
{
    const double sc = scalbn(1.0, -sx), atol = eps_of<double>() * tnorm;
    const double glo = lo - 2.0 * atol - DBL_MIN, ghi = hi + 2.0 * atol + DBL_MIN;
    auto d = [&](int k) { return dg[k] * sc; };
    auto e2 = [&](int k) {
        const double e = eg[k] * sc;
        return e * e;
    };
    return tri_close(d, e2, b0, b1, j, glo, ghi, glo, ghi, tnorm, atol);
}

// Scaled copies of d and e^2 in FP64 and FP32 and the split flags, 25 n bytes: in
// shared memory, or in `work` (32 n bytes per matrix) where that is too little;
// there every CTA of a matrix writes the same values and reads its own.
__global__ void k_tri_bisect64(const double *dd, const double *ee, double *lamloc, int *blk, int n, double *work)
{
    extern __shared__ __align__(16) unsigned char bis64_s[];
    __shared__ double smax[32];
    double *d = work ? work + 4 * (long)n * blockIdx.y : (double *)bis64_s, *e2 = d + n;
    float *sd = (float *)(e2 + n), *se2 = sd + n;
    unsigned char *ssp = (unsigned char *)(se2 + n);
    const int b = blockIdx.y, tid = threadIdx.x;
    const int r = blockIdx.x * blockDim.x + tid;
    const double *dg = dd + (long)b * n, *eg = ee + (long)b * n;
    // scale: a power of two that brings the largest element to [1/2, 1)
    double mx = 0;
    for (int k = tid; k < n; k += blockDim.x) mx = fmax(mx, fmax(fabs(dg[k]), k < n - 1 ? fabs(eg[k]) : 0.0));
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((tid & 31) == 0) smax[tid >> 5] = mx;
    __syncthreads();
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) mx = fmax(mx, smax[q]);
    int sx = 0;
    if (mx > 0 && mx < 1e300) frexp(mx, &sx);
    sx = max(-900, min(900, sx));
    const double sc = scalbn(1.0, -sx);
    for (int k = tid; k < n; k += blockDim.x) {
        const double dk = dg[k] * sc, ek = k < n - 1 ? eg[k] * sc : 0.0;
        d[k] = dk;
        e2[k] = ek * ek;
        sd[k] = (float)dk;
        const float ef = (float)ek;
        se2[k] = ef * ef;
        ssp[k] = k < n - 1 && fabs(dg[k] * dg[k + 1]) * DBL_EPSILON * DBL_EPSILON + DBL_MIN >= eg[k] * eg[k];
    }
    __syncthreads();
    const bool valid = r < n;
    int b0 = 0, b1 = -1;
    if (valid) find_block_flags(ssp, n, r, b0, b1);
    double tnorm = 0, lo = 1e300, hi = -1e300, emax2 = 0;
    block_bounds(dg, eg, valid, b0, b1, lo, hi, tnorm, emax2);
    if (!valid) return;
    const int j = r - b0;
    double lam;
    if (b0 != b1 && tnorm > 0 && tnorm * sc < 0x1p-100) {
        frexp(tnorm, &sx);
        sx = max(-900, sx);
        const double bs = scalbn(1.0, -sx);
        lam = tri_close_small(dg, eg, sx, b0, b1, j, lo * bs, hi * bs, tnorm * bs);
    } else if (b0 == b1) {
        lam = d[b0];
    } else {
        lo *= sc;
        hi *= sc;
        tnorm *= sc;
        const double eps = eps_of<double>(), atol = eps * tnorm, pivmin = DBL_MIN;
        const double glo = lo - 2.0 * atol - pivmin, ghi = hi + 2.0 * atol + pivmin;
        double a = glo, z = ghi;
        if (tnorm > 1e-30) {   // FP32's range holds the block
            float fa = (float)glo, fz = (float)ghi;
            const float w = 4.f * eps_of<float>() * (float)tnorm;
            fa -= w;
            fz += w;
            octasect(sd, se2, b0, b1, j, eps_of<float>() * (float)tnorm, FLT_MIN, fa, fz);
            // the FP32 interval widened by its own error, then checked
            const double m = 4.0 * (double)eps_of<float>() * tnorm;
            a = fmax(glo, (double)fa - m);
            z = fmin(ghi, (double)fz + m);
        }
        lam = tri_close([&](int k) { return d[k]; }, [&](int k) { return e2[k]; }, b0, b1, j, a, z, glo, ghi, tnorm, atol);
    }
    lamloc[(long)b * n + r] = scalbn(lam, sx);
    blk[((long)b * n + r) * 2 + 0] = b0;
    blk[((long)b * n + r) * 2 + 1] = b1;
}

// Global ascending order: rank of (lamloc[r], r).
__global__ void k_tri_rank(const double *lamloc, int *rank, double *lam, int n, int keys)
{
    extern __shared__ unsigned long long trk_keys[];
    const int b = blockIdx.y;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const double *L = lamloc + (long)b * n;
    const int cnt = rank_of(L, n, r, keys ? trk_keys : nullptr);
    if (r >= n) return;
    rank[(long)b * n + r] = cnt;
    lam[(long)b * n + cnt] = L[r];
}

__device__ inline unsigned hash_bits(unsigned a, unsigned b)
{
    unsigned h = a * 0x9E3779B1u ^ (b + 0x7F4A7C15u) * 0x85EBCA77u;
    h ^= h >> 15; h *= 0x2C1B3C6Du; h ^= h >> 12; h *= 0x297A2D39u; h ^= h >> 15;
    return h & 0xFFFFFFu;
}
// (m 2^-23 - 1) size in [-size, size) for a 24-bit m and a power of two: exact in FP32 as in
// FP64, so the FP32 form gives the same values without the FP64 pipe
template <typename TB> __device__ inline TB hash_unit(unsigned a, unsigned b, TB size)
{
    return (TB)hash_bits(a, b) * (size * TB(1.0 / 8388608.0)) - size;
}
// 2^e, |e| < 1000 (FP32: 120)
template <typename TB> __device__ inline TB pow2_of(int e)
{
    if constexpr (sizeof(TB) == 8) return __hiloint2double((1023 + e) << 20, 0);
    else return __int_as_float((127 + e) << 23);
}

// An array of one thread whose elements are `st` apart (thread-interleaved
// scratch: a warp's accesses to the same element index are coalesced).
template <typename TB> struct Strided {
    TB *p;
    long st;
    __device__ Strided(TB *p_, long st_) : p(p_), st(st_) {}
    __device__ TB &operator[](long k) const { return p[k * st]; }
    __device__ Strided operator+(long k) const { return Strided(p + k * st, st); }
};

// Tridiagonal eigenvectors by inverse iteration in TB arithmetic (FP64 for
// the FP64 form, FP32 for the FP32 solve of the mixed form), one thread per
// eigenvalue (dstein's dgttrf/dgtts2 steps, 3 iterations from a pseudo-random
// start in FP64, 2 in FP32), written to the eigenvalue's column of Y.  Members of a cluster of
// close eigenvalues iterate independently; k_tri_cluster_orth then
// orthonormalises each cluster.  An exactly degenerate cluster's iterates are
// independent random combinations inside its invariant subspace, and a member
// separated by g from the others keeps only ~eps ||T|| / g of their
// directions, so orthonormalising after the iteration spans the same subspace
// as re-orthogonalising during it.
//
// Each iteration is two sweeps.  The forward sweep factors T_block - lam I =
// P L U (dgttrf, the running row in registers) and applies P and L at the
// same time; the multipliers are used as they are made and never stored, and
// U's three diagonals are stored in the first iteration only (every
// iteration recomputes the same factor).  The backward sweep solves with U
// and accumulates the norm and the largest component; the normalisation is
// applied as the next sweep reads the vector.  Scratch: 4 arrays of n TB per
// thread, interleaved across the launch's threads (a warp's accesses to one
// element index are one coalesced line); the backward sweep loads INV_BLK
// steps' operands at once so that their latencies overlap.
constexpr int INV_BLK = 8;

template <typename TB>
__global__ void k_tri_invit(const double *dd, const double *ee, const double *lamloc, const int *blk,
                            const int *rank, double *yvec, TB *scratch, int n)
{
    const int b = blockIdx.y;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = r < n;
    const double *d = dd + (long)b * n, *e = ee + (long)b * n, *L = lamloc + (long)b * n;
    const int b0 = valid ? blk[((long)b * n + r) * 2] : 0, b1 = valid ? blk[((long)b * n + r) * 2 + 1] : -1;
    const int len = b1 - b0 + 1;
    // the block's max row sum: by the whole CTA when its threads share one
    // block (max is exact in any order), else per thread
    double tnorm = 0;
    {
        __shared__ int iblk[2];
        __shared__ double ired[32];
        if (threadIdx.x == 0) { iblk[0] = b0; iblk[1] = b1; }
        __syncthreads();
        const int c0 = iblk[0], c1 = iblk[1];
        const bool all = __syncthreads_and(!valid || (b0 == c0 && b1 == c1));
        const int k0 = all ? c0 + (int)threadIdx.x : b0, step = all ? (int)blockDim.x : 1;
        if (all || valid)
            for (int k = k0; k <= (all ? c1 : b1); k += step)
                tnorm = fmax(tnorm, fabs(d[k]) + (k > (all ? c0 : b0) ? fabs(e[k - 1]) : 0.0) +
                                        (k < (all ? c1 : b1) ? fabs(e[k]) : 0.0));
        if (all) {
            for (int o = 16; o > 0; o >>= 1) tnorm = fmax(tnorm, __shfl_xor_sync(0xffffffffu, tnorm, o));
            if ((threadIdx.x & 31) == 0) ired[threadIdx.x >> 5] = tnorm;
            __syncthreads();
            for (int q = 0; q < (int)((blockDim.x + 31) >> 5); ++q) tnorm = fmax(tnorm, ired[q]);
        }
    }
    // FP32: the matrix's d and e rounded once per CTA into shared memory (the
    // same values as converting at each step, without the FP64 pipe)
    extern __shared__ float invit_s[];
    const float *sdf = invit_s, *sef = invit_s + n;
    if (sizeof(TB) == 4) {
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            invit_s[k] = d2f_rn(d[k]);
            invit_s[n + k] = d2f_rn(e[k]);
        }
        __syncthreads();
    }
    auto Dk = [&](int k) { return sizeof(TB) == 4 ? TB(sdf[k]) : TB(d[k]); };
    auto Ek = [&](int k) { return sizeof(TB) == 4 ? TB(sef[k]) : TB(e[k]); };
    if (!valid) return;
    const long NT = (long)gridDim.y * gridDim.x * blockDim.x;
    Strided<TB> S(scratch + ((long)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x, NT);
    // 1 / pivots, first and second super-diagonals of U, iterate
    Strided<TB> RG = S, DU = S + n, DU2 = S + 2 * n, v = S + 3 * n;
    // A solve multiplies its right-hand side by up to 1 / tiny, and the norm squares that.  A block
    // whose norm is so far from one that this leaves the range (one of zeros, above all) takes
    // right-hand sides of the size of `tiny`; the factor is a power of two and goes with the norm.
    constexpr int range = sizeof(TB) == 8 ? 400 : 40;
    const double tn = fmax(tnorm, sizeof(TB) == 8 ? 0x1p-900 : 0x1p-80);
    const TB tiny = eps_of<TB>() * TB(2) * TB(tn);
    const int ex = (__double2hiint(tn) >> 20) - 1023;
    const TB size = (ex < -range || ex > range) ? pow2_of<TB>(ex - (sizeof(TB) == 8 ? 51 : 22)) : TB(1);
    const TB lam = TB(L[r]);
    auto pivot = [&](TB g) { return (fabs(g) < tiny) ? ((g < TB(0)) ? -tiny : tiny) : g; };
    const unsigned seed = (unsigned)(b * 7919 + r);
    // dstein's one converging solve and two extra (FP64); the FP32 solve of the
    // mixed form is refined afterwards, so one extra suffices there
    const int iters = sizeof(TB) == 8 ? 3 : 2;
    TB inv = TB(1);
    int kmax = 0;
    TB vmax = TB(-1), vkmax = TB(0);
    for (int it = 0; it < iters; ++it) {
        // forward: factor (dgttrf) and apply P, L; element k + 1 of the
        // right-hand side is the previous iterate scaled by inv (the random
        // start in the first iteration)
        auto rhs = [&](int k) { return it == 0 ? hash_unit<TB>(seed, (unsigned)k, size) : v[k] * inv; };
        TB dcur = Dk(b0) - lam, ducur = (len > 1) ? Ek(b0) : TB(0);
        TB vc = rhs(0);
        for (int kb = 0; kb < len - 1; kb += INV_BLK) {
            TB vn[INV_BLK], rgv[INV_BLK];
#pragma unroll
            for (int u = 0; u < INV_BLK; ++u)
                if (kb + u < len - 1) {
                    vn[u] = rhs(kb + u + 1);
                    if (sizeof(TB) == 8 && it > 0) rgv[u] = RG[kb + u];
                }
#pragma unroll
            for (int u = 0; u < INV_BLK; ++u) {
                const int k = kb + u;
                if (k >= len - 1) break;
                const TB dlk = Ek(b0 + k);
                TB dnext = Dk(b0 + k + 1) - lam;
                TB dunext = (k < len - 2) ? Ek(b0 + k + 1) : TB(0);
                if (sizeof(TB) == 8) {
                    // FP64 takes a dozen operations of its narrow pipe for a quotient: one
                    // per step, 1 / pivot, which also gives the multiplier and which the
                    // later iterations read back.  The rows are exchanged by selection, so
                    // that a warp whose threads differ pays for one form (N = 1152, 4
                    // matrices 3.72 -> 3.46 ms, N = 144, 15 matrices 0.43 -> 0.34)
                    const bool sw = fabs(dcur) < fabs(dlk);
                    const TB p = sw ? dlk : dcur, q = sw ? dcur : dlk, g1 = sw ? dnext : ducur, g2 = sw ? ducur : dnext;
                    const TB rp = it == 0 ? tri_div(TB(1), pivot(p)) : rgv[u];
                    const TB f = q * rp, vk = sw ? vn[u] : vc, vo = sw ? vc : vn[u];
                    if (it == 0) { RG[k] = rp; DU[k] = g1; DU2[k] = sw ? dunext : TB(0); }
                    dnext = g2 - f * g1;
                    if (sw) dunext = -f * dunext;
                    v[k] = vk;
                    vc = vo - f * vk;
                } else if (fabs(dcur) >= fabs(dlk)) {
                    const TB f = (dcur != TB(0)) ? tri_div(dlk, dcur) : TB(0);
                    if (it == 0) { RG[k] = tri_div(TB(1), pivot(dcur)); DU[k] = ducur; DU2[k] = TB(0); }
                    dnext -= f * ducur;
                    v[k] = vc;
                    vc = vn[u] - f * vc;
                } else {
                    const TB f = tri_div(dcur, dlk);
                    if (it == 0) { RG[k] = tri_div(TB(1), pivot(dlk)); DU[k] = dnext; DU2[k] = dunext; }
                    dnext = ducur - f * dnext;
                    dunext = -f * dunext;
                    v[k] = vn[u];
                    vc = vc - f * vn[u];
                }
                dcur = dnext;
                ducur = dunext;
            }
        }
        if (it == 0) RG[len - 1] = tri_div(TB(1), pivot(dcur));
        // backward: U solve (the two following elements in registers), the
        // norm and the largest component (first in increasing k on ties)
        TB x1 = vc * RG[len - 1], x2 = TB(0);
        v[len - 1] = x1;
        TB nrm = x1 * x1;
        vmax = fabs(x1); kmax = len - 1; vkmax = x1;
        for (int kb = len - 2; kb >= 0; kb -= INV_BLK) {
            TB du[INV_BLK], du2[INV_BLK], rg[INV_BLK], vv[INV_BLK];
#pragma unroll
            for (int u = 0; u < INV_BLK; ++u) {
                const int k = kb - u;
                if (k >= 0) { du[u] = DU[k]; du2[u] = DU2[k]; rg[u] = RG[k]; vv[u] = v[k]; }
            }
#pragma unroll
            for (int u = 0; u < INV_BLK; ++u) {
                const int k = kb - u;
                if (k >= 0) {
                    const TB xk = (vv[u] - du[u] * x1 - du2[u] * x2) * rg[u];
                    v[k] = xk;
                    nrm += xk * xk;
                    if (fabs(xk) >= vmax) { vmax = fabs(xk); kmax = k; vkmax = xk; }
                    x2 = x1;
                    x1 = xk;
                }
            }
        }
        nrm = sqrt(nrm);
        inv = (nrm > TB(0)) ? (it < iters - 1 ? size : TB(1)) / nrm : TB(0);
    }
    // sign convention: largest component positive
    (void)kmax;
    // (widening and the sign with integer operations: the same values as
    // sg * (double) x, off the FP64 pipe)
    const long long sgbit = (vkmax < TB(0)) ? (long long)0x8000000000000000ull : 0ll;
    double *z = yvec + (long)b * n * n + (long)rank[(long)b * n + r] * n;
    // eight elements' loads before their stores (a load after a store to z
    // could alias it and would wait for it)
    for (int k8 = 0; k8 < n; k8 += 8) {
        TB vv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int k = k8 + u;
            vv[u] = (k < n && k >= b0 && k <= b1) ? v[k - b0] : TB(0);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int k = k8 + u;
            if (k >= n) break;
            double x = 0.0;
            if (k >= b0 && k <= b1) {
                if constexpr (sizeof(TB) == 4) x = f2d_exact(vv[u] * inv);
                else x = (double)(vv[u] * inv);
                x = __longlong_as_double(__double_as_longlong(x) ^ sgbit);
            }
            z[k] = x;
        }
    }
}

// Orthonormalise each cluster of eigenvalues closer than ctol ||T|| (within
// an unreduced block) by modified Gram-Schmidt, twice; one warp per
// eigenvalue, the warp of a cluster's first member does the work.
__global__ void __launch_bounds__(256) k_tri_cluster_orth(const double *dd, const double *ee, const double *lamloc,
                                                          const int *blk, const int *rank, double *yvec, int n,
                                                          double ctol)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.y, r = blockIdx.x * 8 + warp;
    if (r >= n) return;   // warp-uniform
    const double *d = dd + (long)b * n, *e = ee + (long)b * n, *L = lamloc + (long)b * n;
    const int b0 = blk[((long)b * n + r) * 2], b1 = blk[((long)b * n + r) * 2 + 1];
    const int len = b1 - b0 + 1;
    double tnorm = 0;
    for (int k = b0 + lane; k <= b1; k += 32)
        tnorm = fmax(tnorm, fabs(d[k]) + (k > b0 ? fabs(e[k - 1]) : 0.0) + (k < b1 ? fabs(e[k]) : 0.0));
    for (int o = 16; o > 0; o >>= 1) tnorm = fmax(tnorm, __shfl_xor_sync(0xffffffffu, tnorm, o));
    const double gap = ctol * fmax(tnorm, DBL_MIN);
    if (r > b0 && L[r] - L[r - 1] < gap) return;   // not the first member
    int rend = r;
    while (rend < b1 && L[rend + 1] - L[rend] < gap) ++rend;
    if (rend == r) return;
    double *Y = yvec + (long)b * n * n;
    for (int m = r; m <= rend; ++m) {
        double *v = Y + (long)rank[(long)b * n + m] * n + b0;
        for (int pass = 0; pass < 2; ++pass) {
            for (int p = r; p < m; ++p) {
                const double *zp = Y + (long)rank[(long)b * n + p] * n + b0;
                double sdot = 0;
                for (int k = lane; k < len; k += 32) sdot += zp[k] * v[k];
                sdot = warp_sum(sdot);
                for (int k = lane; k < len; k += 32) v[k] -= sdot * zp[k];
                __syncwarp();
            }
        }
        double nrm = 0;
        for (int k = lane; k < len; k += 32) nrm += v[k] * v[k];
        nrm = sqrt(warp_sum(nrm));
        const double inv = (nrm > 0) ? 1.0 / nrm : 0.0;
        // sign convention: the first largest component positive
        double vmax = -1.0;
        int kmax = 0;
        for (int k = lane; k < len; k += 32) {
            const double a = fabs(v[k]);
            if (a > vmax) { vmax = a; kmax = k; }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, vmax, o);
            const int ok = __shfl_xor_sync(0xffffffffu, kmax, o);
            if (ov > vmax || (ov == vmax && ok < kmax)) { vmax = ov; kmax = ok; }
        }
        const double sg = (v[kmax] < 0) ? -inv : inv;
        __syncwarp();
        for (int k = lane; k < len; k += 32) v[k] *= sg;
        __syncwarp();
    }
}

// real eigenvector matrix -> complex working precision
template <typename C2>
__global__ void k_real_to_cplx(const double *y, C2 *z, long count)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < count; i += (long)gridDim.x * blockDim.x) {
        C2 o;
        if constexpr (sizeof(o.x) == 4) o.x = d2f_rn(y[i]);
        else o.x = y[i];
        o.y = 0;
        z[i] = o;
    }
}

// compact-WY T factor of a block of jb <= EIG_WY reflectors (G = Vb^H Vb and T
// column-major nbw x nbw per matrix): column by column,
// T[0:c, c] = -tau_c T[0:c, 0:c] G[0:c, c], T[c, c] = tau_c (LAPACK's larft,
// forward columnwise).  FP32: one CTA of EIG_WY threads per matrix, thread = row;
// T is built in shared memory (128 x 129 complex = 132 KB, dynamic).  Row r of T
// depends only on row r and on G, so the threads need no barrier between
// columns: the columns of G (and the taus) come in groups of LARFT_GC through
// shared memory, with a barrier per group.  The lanes of a warp walk k together
// from the warp's first row, so that their reads of T are consecutive and G[k, c]
// is one broadcast; row r adds its terms k >= r in order of k (the
// one-row-at-a-time sums).
constexpr int LARFT_GC = 8;
__global__ void __launch_bounds__(EIG_WY) k_larft_wy(const float2 *G, float2 *Tm, const float2 *tau, int n, int j0,
                                                     int jb, int nbw)
{
    __shared__ float2 g[LARFT_GC][EIG_WY];
    __shared__ float2 tg[LARFT_GC];
    extern __shared__ __align__(16) unsigned char larft_smem[];
    const int b = blockIdx.x, r = threadIdx.x, kw = r & ~31;
    const float2 *Gb = G + (long)b * nbw * nbw;
    float2 *Tb = Tm + (long)b * nbw * nbw;
    constexpr int lt = EIG_WY + 1;   // column stride of the working T
    float2 *Tw = (float2 *)larft_smem;
    for (int c0 = 0; c0 < jb; c0 += LARFT_GC) {
        const int cn = min(LARFT_GC, jb - c0);
        __syncthreads();   // every thread is done with the previous group's columns
        for (int q = 0; q < cn; ++q)
            if (r < c0 + q) g[q][r] = Gb[r + (long)(c0 + q) * nbw];
        if (r < cn) tg[r] = tau[(long)b * n + j0 + c0 + r];
        __syncthreads();
        for (int q = 0; q < cn; ++q) {
            const int c = c0 + q;
            const float2 tc = tg[q];
            if (kw < c) {   // warp-uniform
                float2 acc = make_float2(0.f, 0.f);
                int k = kw;
                for (; k + 8 <= c; k += 8) {
                    float2 tv[8], gv[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        tv[u] = Tw[r + (k + u) * lt];
                        gv[u] = g[q][k + u];
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (k + u >= r) cfma(acc, tv[u], gv[u]);
                }
                for (; k < c; ++k)
                    if (k >= r) cfma(acc, Tw[r + k * lt], g[q][k]);
                if (r < c) Tw[r + (long)c * lt] = cscale(cmul(tc, acc), -1.f);
            }
            if (r == c) Tw[c + (long)c * lt] = tc;
        }
    }
    __syncthreads();
    for (int c = 0; c < jb; ++c)
        if (r <= c) Tb[r + (long)c * nbw] = Tw[r + (long)c * lt];
}

// The same T factor for FP64, whose T does not fit the shared memory of one SM and
// whose dots are bound by the FP64 pipe: row r of T depends on row r and G alone, so
// a matrix's rows are spread over CTAs of 16, a warp holding four rows with eight
// lanes over k each (fewer lanes a row leave a longer chain, more a longer
// reduction); the columns of G come through shared memory eight at a time.
// One CTA per matrix with T in global memory took 1.38 ms a block of 128 at 4 k, this
// 0.28; at 64 k 0.95 against 0.54.
constexpr int LARFT_RC = 8;
// T = [T1, -T1 G12 T2; 0, T2] for the reflectors before and from LARFT_HALF on: only T1
// and T2 are formed here, which is a quarter of the operations and half of the chain, the
// corner by two digit products (wy_block): a block of 128 with these products, n = 144 218 ->
// 150 us (charges of 16 atoms), n = 288, 64 matrices 543 -> 310.
constexpr int LARFT_HALF = 64;
__global__ void __launch_bounds__(128) k_larft_rows(const double2 *G, double2 *Tm, const double2 *tau, int n, int j0,
                                                    int jb, int nbw)
{
    __shared__ double2 g[LARFT_RC][EIG_WY];
    __shared__ double2 trow[16][EIG_WY];
    const int b = blockIdx.y, lane = threadIdx.x & 31, kp = lane & 7, rl = threadIdx.x >> 3;
    const int cbeg = 16 * blockIdx.x, r = cbeg + rl;   // the CTA's first row: earlier columns are zero
    const int rw = cbeg + 4 * (threadIdx.x >> 5);      // the warp's first row
    const double2 *Gb = G + (long)b * nbw * nbw;
    double2 *Tb = Tm + (long)b * nbw * nbw;
    const double2 *tb = tau + (long)b * n + j0;
    double2 *t = trow[rl];
    if (cbeg < LARFT_HALF) jb = min(jb, LARFT_HALF);   // a multiple of the CTA's rows
    for (int c0 = cbeg / LARFT_RC * LARFT_RC; c0 < jb; c0 += LARFT_RC) {
        const int cn = min(LARFT_RC, jb - c0);
        __syncthreads();
#pragma unroll 8
        for (int q = 0; q < cn; ++q) {
            const int k = threadIdx.x;
            if (k < c0 + q && k >= cbeg) g[q][k] = Gb[k + (long)(c0 + q) * nbw];
        }
        __syncthreads();
        for (int q = 0; q < cn; ++q) {
            const int c = c0 + q;
            if (c < rw) continue;   // warp-uniform
            double2 acc = make_double2(0, 0);
            for (int k = rw + kp; k < c; k += 8)
                if (k >= r) cfma(acc, t[k], g[q][k]);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
                acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
                acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
            }
            if (kp == 0 && r <= c && r < jb) {
                const double2 tc = tb[c], m = cmul(tc, acc);
                const double2 v = c > r ? make_double2(-m.x, -m.y) : tc;
                t[c] = v;
                Tb[r + (long)c * nbw] = v;
            }
            __syncwarp();
        }
    }
}

// The same for FP64, where operations of the FP64 pipe are the cost (a warp's takes 64
// cycles of its quarter of the SM).  Factor and inverse X advance together: after
// column k of L and row k of X, row r > k of the block takes
//   a(r, c) -= l_rk conj(l_ck)  for columns c > k,
//   y(r, c) += l_rk x_kc        for c <= k,  then x_r = -y_r / l_rr,
// one FMA for all 32 lanes (lane = column, c > k of the factor, c <= k of the
// inverse), rows dealt over the warps.  The pivot's root and reciprocal are formed by
// one warp (tc_root).
// 32 x 32: 187 us by the FP32 kernel's scheme in FP64 (every warp forming the root
// and reciprocal, one warp the inverse), 53 here.
__global__ void __launch_bounds__(256) k_potrf_diag64(EigWork<double> w, int j0, int jb)
{
    __shared__ double2 m[EIG_NB][EIG_NB + 1];    // m[r][c]: a (c > k) | y (c <= k)
    __shared__ double2 lo[EIG_NB][EIG_NB + 1];   // L, lo[c][r]
    __shared__ double2 xo[EIG_NB][EIG_NB + 1];   // X, xo[r][c]
    __shared__ int bad;
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double2 *L = w.L + b * w.mstride + j0 + (long)j0 * w.ld;
    double2 *Wi = w.Wi + b * w.mstride + j0 + (long)j0 * w.ld;
    const double2 z = make_double2(0, 0);
    for (int c = warp; c < EIG_NB; c += 8) m[lane][c] = lane < jb && c < jb ? L[lane + (long)c * w.ld] : z;
    if (tid == 0) bad = 0;
    __syncthreads();
    for (int k = 0; k < jb; ++k) {
        if (warp == (k & 7)) {
            double piv = m[k][k].x;
            const bool badk = !(piv > 0.0);
            if (badk) piv = 1.0;
            double dk, inv;
            tc_root(piv, dk, inv);
            const double2 y = m[k][lane], a = m[lane][k];   // row k, column k
            xo[k][lane] = lane < k ? cscale(y, -inv) : lane == k ? make_double2(inv, 0.0) : z;
            lo[k][lane] = lane > k ? cscale(a, inv) : lane == k ? make_double2(dk, 0.0) : z;
            if (badk && lane == 0) bad = 1;
        }
        __syncthreads();
        double2 o = xo[k][lane];
        if (lane > k) {
            o = lo[k][lane];
            o.x = -o.x;   // -conj
        }
        for (int r = k + 1 + ((warp - (k + 1)) & 7); r < jb; r += 8) {
            double2 t = lane == k ? z : m[r][lane];
            cfma(t, lo[k][r], o);
            if (lane <= r) m[r][lane] = t;
        }
        __syncthreads();
    }
    if (lane < jb)
        for (int c = warp; c < jb; c += 8) {
            L[lane + (long)c * w.ld] = lo[c][lane];
            Wi[lane + (long)c * w.ld] = xo[lane][c];
        }
    if (tid == 0 && bad) w.status[b] = 1;
}

// Join the inverted 32 x 32 diagonal blocks of L pairwise: for the 64-block at
// j0 = 64 t, W(j0+32.., j0..) = -W11 L10 W00 (W00, W11 the blocks' inverses,
// lower triangular; L10 the 32 x 32 block of L below W00).  One CTA per
// (pair, matrix); the three 32 x 32 blocks in shared memory.
template <typename T>
__global__ void __launch_bounds__(256) k_inv_pair(EigWork<T> w)
{
    typedef typename cplx<T>::t C2;
    __shared__ C2 a0[32][32], b1[32][32], lt[32][32];   // [col][row]
    const int b = blockIdx.y, n = w.n, tid = threadIdx.x;
    const int j0 = 2 * EIG_NB * blockIdx.x, j1 = j0 + EIG_NB;
    if (j1 >= n) return;
    const int m1 = min(EIG_NB, n - j1);
    const long ld = w.ld;
    const C2 *Wi = w.Wi + b * w.mstride, *L = w.L + b * w.mstride;
    C2 *Wo = w.Wi + b * w.mstride;
    const C2 z = cmk<T>(0, 0);
    for (int e = tid; e < 1024; e += 256) {
        const int r = e & 31, c = e >> 5;
        a0[c][r] = (r >= c) ? Wi[(j0 + r) + (long)(j0 + c) * ld] : z;
        b1[c][r] = (r >= c && r < m1) ? Wi[(j1 + r) + (long)(j1 + c) * ld] : z;
        lt[c][r] = (r < m1) ? L[(j1 + r) + (long)(j0 + c) * ld] : z;
    }
    __syncthreads();
    // T1 = W11 L10 (W11 lower: k <= r), four entries per thread
    C2 t1[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int e = tid + 256 * u, r = e & 31, c = e >> 5;
        C2 acc = z;
        for (int k = 0; k <= r; ++k) cfma(acc, b1[k][r], lt[c][k]);
        t1[u] = acc;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int e = tid + 256 * u;
        lt[e >> 5][e & 31] = t1[u];
    }
    __syncthreads();
    // W10 = -T1 W00 (W00 lower: k >= c)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int e = tid + 256 * u, r = e & 31, c = e >> 5;
        C2 acc = z;
        for (int k = c; k < 32; ++k) cfma(acc, lt[k][r], a0[c][k]);
        if (r < m1) Wo[(j1 + r) + (long)(j0 + c) * ld] = cscale(acc, T(-1));
    }
}

// Rows t0.. of the panel's V columns j0..j0+jb into columns 0..jb and
// 2 EIG_NB.. of VW (W sits in between), for the merged trailing update
__global__ void k_copy_vpanel(const float2 *V, long ld, long ms, float2 *VW, long ldw, long wps, int t0, int j0, int jb,
                              int rem)
{
    const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= (long)rem * jb) return;
    const int b = blockIdx.y, r = (int)(e % rem), c = (int)(e / rem);
    const float2 v = V[b * ms + t0 + r + (long)(j0 + c) * ld];
    float2 *o = VW + b * wps + t0 + r;
    o[(long)c * ldw] = v;
    o[(long)(2 * EIG_NB + c) * ldw] = v;
}

// The FP64 form's copy.  Its product takes each row of [V W] as digits of one scale, and
// V's entries are at most 1 while W's go as the norm of A: left as they are, a matrix of
// norm 1e6 or 1e-6 would lose 20 bits of V or W.  So column c's pair is brought to one
// size by powers of two, V_c 2^a and W_c 2^-a with a half the difference of their largest
// exponents, which leaves V_c W_c^H + W_c V_c^H as it is; a pair whose V or W is zero adds
// nothing and is cleared.  A CTA per column: a few us beside a product of 20 to 400.
__global__ void __launch_bounds__(256) k_scale_vpanel(const double2 *V, long ld, long ms, double2 *VW, long ldw, long wps,
                                                      int t0, int j0, int rem)
{
    __shared__ unsigned long long smx[2][8];
    const int b = blockIdx.y, c = blockIdx.x, tid = threadIdx.x;
    const double2 *v = V + b * ms + t0 + (long)(j0 + c) * ld;
    double2 *o = VW + b * wps + t0 + (long)c * ldw, *wc = o + (long)EIG_NB * ldw, *o2 = wc + (long)EIG_NB * ldw;
    auto part = [](double2 x) {   // as integers, so that a NaN is the largest
        return max((unsigned long long)__double_as_longlong(fabs(x.x)), (unsigned long long)__double_as_longlong(fabs(x.y)));
    };
    unsigned long long mv = 0, mw = 0;
    for (int r = tid; r < rem; r += 256) {
        mv = max(mv, part(v[r]));
        mw = max(mw, part(wc[r]));
    }
    for (int q = 16; q > 0; q >>= 1) {
        mv = max(mv, (unsigned long long)__shfl_xor_sync(0xffffffffu, mv, q));
        mw = max(mw, (unsigned long long)__shfl_xor_sync(0xffffffffu, mw, q));
    }
    if ((tid & 31) == 0) {
        smx[0][tid >> 5] = mv;
        smx[1][tid >> 5] = mw;
    }
    __syncthreads();
    for (int q = 0; q < 8; ++q) {
        mv = max(mv, smx[0][q]);
        mw = max(mw, smx[1][q]);
    }
    const int ev = (int)(mv >> 52), ew = (int)(mw >> 52);
    const bool keep = mv != 0 && mw != 0;
    const int a = (ev < 2047 && ew < 2047) ? (ew - ev) >> 1 : 0;   // |a| <= 1023
    const double up = a > -1023 ? __longlong_as_double((long long)(1023 + a) << 52) : 0x1p-1023;
    const double dn = a < 1023 ? __longlong_as_double((long long)(1023 - a) << 52) : 0x1p-1023;
    for (int r = tid; r < rem; r += 256) {
        double2 x = v[r], y = wc[r];
        x = keep ? make_double2(x.x * up, x.y * up) : make_double2(0, 0);
        y = keep ? make_double2(y.x * dn, y.y * dn) : make_double2(0, 0);
        o[r] = x;
        o2[r] = x;
        wc[r] = y;
    }
}

__global__ void k_fill_int(int *p, int v, int count)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) p[i] = v;
}

// ---------------------------------------------------------------------------
template <typename T>
void eig_solve(cudaStream_t s, EigWork<T> &w, const double2 *H, const double2 *S, double *eig,
               typename cplx<T>::t *X, bool vectors, cudaEvent_t tri_start, const EigAux *ax)
{
    typedef typename cplx<T>::t C2;
    const int n = w.n, B = w.batch;
    const long ld = w.ld, ms = w.mstride;
    const C2 one = cmk<T>(1, 0), mone = cmk<T>(-1, 0), zero = cmk<T>(0, 0);
    const long cnt = (long)n * n * B;
    cudaMemsetAsync(w.status, 0, sizeof(int) * B, s);
    // 0. inputs in working precision: S -> L, H -> A (A is free until step 3)
    int *const ex = (int *)w.d;   // FP64: exponents of D, until step 4
    if constexpr (sizeof(T) == 4) {
        NRLTB_LAUNCH(k_convert_h, 1184, 256, 0, s, S, w.L, cnt);
        NRLTB_LAUNCH(k_convert_h, 1184, 256, 0, s, H, w.A, cnt);
    } else {
        NRLTB_LAUNCH(k_unit_exp, cdiv((long)n * B, 128), 128, 0, s, S, ex, n, B);
        NRLTB_LAUNCH(k_to_unit, dim3((unsigned)std::min(cdiv((long)n * n, 256), 512), B), 256, 0, s, S, H, w.L, w.A, ex, n);
    }
    // 1. Cholesky S = L L^H
    for (int j0 = 0; j0 < n; j0 += EIG_NB) {
        const int jb = std::min(EIG_NB, n - j0), rem = n - j0 - jb;
        if constexpr (sizeof(T) == 4) NRLTB_LAUNCH(k_potrf_diag, B, 256, 0, s, w, j0, jb);
        else NRLTB_LAUNCH(k_potrf_diag64, B, 256, 0, s, w, j0, jb);
        if (rem > 0) {
            C2 *P = w.L + (j0 + jb) + (long)j0 * ld;
            zgemm<T>(s, rem, jb, jb, B, one, P, ld, ms, 0, w.Wi + j0 + (long)j0 * ld, ld, ms, 1, zero, P, ld, ms,
                     0, 1, 0, w.zs);
            zgemm<T>(s, rem, rem, jb, B, mone, P, ld, ms, 0, P, ld, ms, 1, one,
                     w.L + (j0 + jb) + (long)(j0 + jb) * ld, ld, ms, 0, 0, 1, w.zs);
        }
    }
    // 2. Wi = L^{-1}, bottom-up blocked: the 32 x 32 diagonal blocks are already
    //    inverted; pairs of them are joined into 64 x 64 diagonal inverses, then
    //    the 64-wide block columns are filled from the bottom (GEMMs with n = 64,
    //    wide enough for the tensor-core tile)
    {
        const int npair = cdiv(n, 2 * EIG_NB);
        NRLTB_LAUNCH(k_inv_pair<T>, dim3(npair, B), 256, 0, s, w);
        constexpr int NB2 = 2 * EIG_NB;
        int jlast = ((n - 1) / NB2) * NB2;
        for (int j0 = jlast; j0 >= 0; j0 -= NB2) {
            const int jb = std::min(NB2, n - j0), rem = n - j0 - jb;
            if (rem <= 0) continue;
            const long ldx = n;
            zgemm<T>(s, rem, jb, rem, B, one, w.Wi + (long)(j0 + jb) * (ld + 1), ld, ms, 0,
                     w.L + (j0 + jb) + (long)j0 * ld, ld, ms, 0, zero, w.Xt, ldx, (long)NB2 * n, 1, 0, 0, w.zs);
            zgemm<T>(s, rem, jb, jb, B, mone, w.Xt, ldx, (long)NB2 * n, 0, w.Wi + (long)j0 * (ld + 1), ld, ms, 0,
                     zero, w.Wi + (j0 + jb) + (long)j0 * ld, ld, ms, 0, 2, 0, w.zs);
        }
    }
    // 3. A = Wi H Wi^H (lower tiles); FP32: Wi^H formed explicitly in L (free
    //    after step 2) so that both tensor-core GEMMs stream stored operands
    if (sizeof(T) == 4) {
        conj_transpose<T>(s, w.Wi, w.L, n, B);
        zgemm<T>(s, n, n, n, B, one, w.A, ld, ms, 0, w.L, ld, ms, 0, zero, w.Y, ld, ms, 0, 1, 0, w.zs);
    } else {
        zgemm<T>(s, n, n, n, B, one, w.A, ld, ms, 0, w.Wi, ld, ms, 1, zero, w.Y, ld, ms, 0, 1, 0, w.zs);
    }
    zgemm<T>(s, n, n, n, B, one, w.Wi, ld, ms, 0, w.Y, ld, ms, 0, zero, w.A, ld, ms, 1, 0, 1, w.zs);
    if constexpr (sizeof(T) == 8) {
        if (vectors) NRLTB_LAUNCH(k_from_unit, dim3(n, B), 128, 0, s, w.Wi, ex, n);
    }
    if (tri_start) cudaEventRecord(tri_start, s);
    // 4. tridiagonalisation: FP32 one cluster launch per panel (tri_panel.cuh); FP64 one
    //    launch for a small matrix (tri_small.cuh) or for the last TK_MAX columns of a
    //    larger one (tri_cluster.cuh).  The other columns, and all of them where a cluster
    //    cannot be scheduled, two launches each (tri_col.cuh)
    bool clusters = sizeof(T) == 4;
    int from = 0;   // the columns that are left to the loop
    if constexpr (sizeof(T) == 8) {
        if (n <= TS_MAX) {
            tri_small(s, w);
            from = n;
        }
    }
    for (int j0 = from; j0 < n; j0 += EIG_NB) {
        if constexpr (sizeof(T) == 8) {
            if (tri_cluster(s, w, j0)) break;
        }
        const int jb = std::min(EIG_NB, n - j0);
        if constexpr (sizeof(T) == 4) clusters = clusters && tri_panel_launch(s, w, j0, jb);
        if (!clusters) tri_columns<T>(s, w, j0, jb);
        if (std::min(j0 + jb - 1, n - 2) < j0) break;
        const int t0 = j0 + jb, rem = n - t0;
        if (rem > 0) {
            C2 *Vp = w.V + t0 + (long)j0 * ld, *Wpp = w.Wp + t0;
            C2 *At = w.A + (long)t0 * (ld + 1);
            if (jb == EIG_NB) {
                // A -= [Vp Wp] [Wp Vp]^H in one rank-64 update: Vp copied on both sides of W
                if constexpr (sizeof(T) == 4)
                    NRLTB_LAUNCH(k_copy_vpanel, dim3(cdiv((long)rem * jb, 256), B), 256, 0, s, w.V, ld, ms, w.VW,
                                 (long)n, w.wps, t0, j0, jb, rem);
                else
                    NRLTB_LAUNCH(k_scale_vpanel, dim3(jb, B), 256, 0, s, w.V, ld, ms, w.VW, (long)n, w.wps, t0, j0, rem);
                zgemm<T>(s, rem, rem, 2 * EIG_NB, B, mone, w.VW + t0, n, w.wps, 0, w.VW + t0 + (long)n * EIG_NB, n,
                         w.wps, 1, one, At, ld, ms, 0, 0, 1, w.zs);
            } else {
                zgemm<T>(s, rem, rem, jb, B, mone, Vp, ld, ms, 0, Wpp, n, w.wps, 1, one, At, ld, ms, 0, 0, 1, w.zs);
                zgemm<T>(s, rem, rem, jb, B, mone, Wpp, n, w.wps, 0, Vp, ld, ms, 1, one, At, ld, ms, 0, 0, 1, w.zs);
            }
        }
    }
    // the back-transform's WY factors need only V and tau: with the auxiliary
    // streams they are formed there, a block on each in turn, while this one
    // solves the tridiagonal problem
    const int nbw = std::min(EIG_WY, n), nref = n - 1;
    const long sG = (long)nbw * nbw;
    auto Tf_of = [&](int j0) { return w.Tt + (long)(EIG_NAUX + j0 / nbw) * sG * B; };
    // block j0's G and T on stream st, with G buffer g
    auto wy_block = [&](cudaStream_t st, int g, int j0) {
        C2 *const G = w.Tt + (long)g * sG * B;
        const int jb = std::min(nbw, nref - j0), mb = n - j0 - 1;
        const C2 *Vb = w.V + (j0 + 1) + (long)j0 * ld;
        zgemm<T>(st, jb, jb, mb, B, one, Vb, ld, ms, 1, Vb, ld, ms, 0, zero, G, nbw, sG, 0, 0, 0, w.zs);
        if (sizeof(T) == 4) {
            const int sm = (int)(sizeof(C2) * EIG_WY * (EIG_WY + 1));
            smem_attr_at_least((const void *)k_larft_wy, sm);
            NRLTB_LAUNCH(k_larft_wy, B, EIG_WY, sm, st, (const float2 *)G, (float2 *)Tf_of(j0), (const float2 *)w.tau, n,
                         j0, jb, nbw);
        } else {
            C2 *const Tf = Tf_of(j0);
            NRLTB_LAUNCH(k_larft_rows, dim3(cdiv(jb, 16), B), 128, 0, st, (const double2 *)G, (double2 *)Tf,
                         (const double2 *)w.tau, n, j0, jb, nbw);
            if (jb > LARFT_HALF) {   // T1 G12, then that times T2, in T's corner
                const int h = LARFT_HALF, j2 = jb - h;
                C2 *const T12 = Tf + (long)h * nbw;
                zgemm<T>(st, h, j2, h, B, one, Tf, nbw, sG, 0, G + (long)h * nbw, nbw, sG, 0, zero, T12, nbw, sG, 2, 0, 0,
                         w.zs);
                zgemm<T>(st, h, j2, j2, B, mone, T12, nbw, sG, 0, T12 + h, nbw, sG, 0, zero, T12, nbw, sG, 0, 1, 0, w.zs);
            }
        }
    };
    const int j0last = nref >= 1 ? ((nref - 1) / nbw) * nbw : -1;
    bool on_aux = vectors && ax && ax->tri_done;
    for (int q = 0; q < EIG_NAUX; ++q) on_aux = on_aux && ax->aux[q] && ax->wy_done[q];
    if (on_aux) {
        cudaEventRecord(ax->tri_done, s);
        for (int q = 0; q < EIG_NAUX; ++q) cudaStreamWaitEvent(ax->aux[q], ax->tri_done, 0);
        for (int j0 = j0last, q = 0; j0 >= 0; j0 -= nbw, q = (q + 1) % EIG_NAUX) wy_block(ax->aux[q], q, j0);
        for (int q = 0; q < EIG_NAUX; ++q) cudaEventRecord(ax->wy_done[q], ax->aux[q]);
    }
    // 5. tridiagonal eigenproblem (FP64 inverse iteration; bisection in T)
    double *lamloc = (double *)w.Xt;   // free at this point: n doubles per matrix fit
    int *blk = w.perm, *rank = w.perm + 2 * (long)n * B;
    {
        dim3 g(cdiv(n, 128), B);
        if (sizeof(T) == 4) {
            const size_t bsm = 2 * sizeof(float) * n + n;
            if (bsm > 48 * 1024) smem_attr_at_least((const void *)k_tri_bisect32, (int)bsm);
            NRLTB_LAUNCH(k_tri_bisect32, g, 128, bsm, s, w.d, w.e, lamloc, blk, n);
        } else {
            // a warp per CTA while that leaves CTAs to every SM (the FP64 pipe is the SM's)
            const int nt = (long)n * B < 64L * 152 * 8 ? 32 : 64;
            size_t bsm = 25 * (size_t)n + 16;
            double *work = nullptr;
            if (bsm > 200 * 1024) {
                work = w.ylu;   // inverse iteration's scratch, free until then
                bsm = 0;
            }
            if (bsm > 48 * 1024) smem_attr_at_least((const void *)k_tri_bisect64, (int)bsm);
            NRLTB_LAUNCH(k_tri_bisect64, dim3(cdiv(n, nt), B), nt, bsm, s, w.d, w.e, lamloc, blk, n, work);
        }
        const size_t rsm = rank_keys_bytes(n);
        if (rsm > 48 * 1024) smem_attr_at_least((const void *)k_tri_rank, (int)rsm);
        NRLTB_LAUNCH(k_tri_rank, g, 128, rsm, s, lamloc, rank, w.lam, n, rsm > 0 ? 1 : 0);
        cudaMemcpyAsync(eig, w.lam, sizeof(double) * n * B, cudaMemcpyDeviceToDevice, s);
    }
    if (!vectors) return;
    {
        // eigenvalues closer than ctol ||T|| are orthonormalised as one cluster
        // (LAPACK's dstein uses 1e-3 ||T||; outside a cluster the vectors'
        // overlap is ~ eps ||T|| / gap <= 1e-11 for FP64)
        const double ctol = 1e-5;
        // 64 threads per CTA: cdiv(n, 64) * 64 * B thread slots <= the scratch carve's 64 cdiv(n, 64) n B
        const size_t ism = sizeof(T) == 4 ? 2 * sizeof(float) * n : 0;
        if (ism > 48 * 1024)
            smem_attr_at_least((const void *)k_tri_invit<T>, (int)ism);
        NRLTB_LAUNCH(k_tri_invit<T>, dim3(cdiv(n, 64), B), 64, ism, s, w.d, w.e, lamloc, blk, rank, w.yvec,
                     (T *)w.ylu, n);
        NRLTB_LAUNCH(k_tri_cluster_orth, dim3(cdiv(n, 8), B), 256, 0, s, w.d, w.e, lamloc, blk, rank, w.yvec, n,
                     ctol);
        NRLTB_LAUNCH(k_real_to_cplx<C2>, 1184, 256, 0, s, w.yvec, w.Y, cnt);
    }
    // 6. Z = Q Y: blocks of EIG_WY reflectors applied last to first as
    //    Y[j0+1:, :] -= Vb (Tb (Vb^H Y[j0+1:, :])), Vb = V[j0+1:, j0:j0+jb] (the
    //    reflectors of the block vanish above row j0+1); then X = Wi^H Z.
    //    A (free after step 4) holds Vb^H Y, L (free after step 2) holds Tb Vb^H Y.
    {
        if (on_aux)
            for (int q = 0; q < EIG_NAUX; ++q) cudaStreamWaitEvent(s, ax->wy_done[q], 0);
        else
            for (int j0 = j0last; j0 >= 0; j0 -= nbw) wy_block(s, 0, j0);
        const long sX = (long)nbw * n;
        for (int j0 = (nref >= 1 ? ((nref - 1) / nbw) * nbw : -1); j0 >= 0; j0 -= nbw) {
            const int jb = std::min(nbw, nref - j0), mb = n - j0 - 1;
            const C2 *Vb = w.V + (j0 + 1) + (long)j0 * ld;
            C2 *Yb = w.Y + (j0 + 1);
            const C2 *Tf = Tf_of(j0);
            if (sizeof(T) == 4) {
                // Vb^H formed explicitly in Xt: the tensor-core GEMM streams an A
                // operand in its stored orientation twice as fast
                conj_transpose<T>(s, Vb, ld, ms, w.Xt, nbw, sX, mb, jb, B);
                zgemm<T>(s, jb, n, mb, B, one, w.Xt, nbw, sX, 0, Yb, ld, ms, 0, zero, w.A, nbw, sX, 0, 0, 0, w.zs);
            } else {
                zgemm<T>(s, jb, n, mb, B, one, Vb, ld, ms, 1, Yb, ld, ms, 0, zero, w.A, nbw, sX, 0, 0, 0, w.zs);
            }
            zgemm<T>(s, jb, n, jb, B, one, Tf, nbw, sG, 0, w.A, nbw, sX, 0, zero, w.L, nbw, sX, 2, 0, 0, w.zs);
            zgemm<T>(s, mb, n, jb, B, mone, Vb, ld, ms, 0, w.L, nbw, sX, 0, one, Yb, ld, ms, 0, 0, 0, w.zs);
        }
        if (sizeof(T) == 4) {
            // Wi^H formed explicitly in L (free again): the tensor-core GEMM
            // streams an A operand in its stored orientation twice as fast
            conj_transpose<T>(s, w.Wi, w.L, n, B);
            zgemm<T>(s, n, n, n, B, one, w.L, ld, ms, 0, w.Y, ld, ms, 0, zero, X, ld, ms, 2, 0, 0, w.zs);
        } else {
            zgemm<T>(s, n, n, n, B, one, w.Wi, ld, ms, 1, w.Y, ld, ms, 0, zero, X, ld, ms, 2, 0, 0, w.zs);
        }
    }
}

template size_t eig_work_bytes<double>(int, int);
template size_t eig_work_bytes<float>(int, int);
template void eig_work_carve<double>(EigWork<double> &, void *, int, int);
template void eig_work_carve<float>(EigWork<float> &, void *, int, int);
template void eig_solve<double>(cudaStream_t, EigWork<double> &, const double2 *, const double2 *, double *,
                                double2 *, bool, cudaEvent_t, const EigAux *);
template void eig_solve<float>(cudaStream_t, EigWork<float> &, const double2 *, const double2 *, double *,
                               float2 *, bool, cudaEvent_t, const EigAux *);

}  // namespace nrltb
