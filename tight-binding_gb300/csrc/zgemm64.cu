// zgemm64.cu -- FP64 complex GEMM C = alpha op(A) op(B) + beta C (alpha = +-1,
// beta = 0 or 1) as exact digit products on the bf16 tensor cores.
//
// GB300 has no FP64 tensor path and two FP64 FMAs a cycle per SM, so the FMA-pipe
// kernel (gemm.cuh) needs 2 M cycles for 64 x 64 x 128 complex multiply-adds.
// Here every row of op(A) and every column of op(B) is scaled by a power of two
// and written as an integer below 2^55 in ZD = 7 balanced base-256 digits (one
// rounding, 2^-56 of the row's or column's largest element, as against 2^-53 of
// the element itself).  A digit product is an integer that FP32 accumulation
// sums exactly, so the further errors are the dropped digit pairs s + t > 7
// (below 2^-58 of row maximum x column maximum per term), the unit of the
// 64-bit sums, to which every chunk of 32 k is rounded twice (below), and the
// last rounding.  In all below K 2^-51 row maximum x column maximum, which
// tests/test_gpu_kernel_edges.py holds against extended precision; an FMA chain
// has K 2^-52 of the sum of |a| |b|.  So an element far below its row's largest
// keeps fewer bits than FP64's 53, and below 2^-56 of it none: what a solve
// needs is accuracy against the norm, and there the two agree (eig.cu's k_unit_exp
// and k_scale_vpanel see to the scales that would not cancel).
//
// Layout.  A chunk is 32 k.  Plane s of A's 128 rows is one 16 KB tile of the
// 128-byte-swizzled K-major layout, row i = [re digits of 32 k | im digits]; plane
// t of X = op(B), 64 columns, is one 16 KB tile of 128 rows, row j = [re | -im],
// row 64 + j = [im | re].  So a digit pair of a chunk is a plain real product
// of depth 64 giving [Re | Im] in 128 accumulator columns: four 128 x 128 x 16
// MMAs.  A chunk takes 34 pairs.  Its planes are all resident (7 slots of A_p and
// X_p, 224 KB), so the pairs go level by level, L = s + t from 7 down to 0: a
// level needs one accumulator, four of them fill tensor memory, and slot p is
// last read by level p, so the next chunk's copies refill the slots in the order
// 6, 5, .. 0 behind the MMAs.
//
// Exactness: a level sums at most 7 pairs x 64 products of at most 2^14, below
// 2^22.9.  Two levels make a 32-bit integer (256 v_(L-1) + v_L, below 1.9e9) and the
// four of a chunk are shifted into one 64-bit integer per element, whose unit
// 2^(e_i + f_j + d - 62) leaves room for the whole sum (d from the row's or the
// columns' sums of magnitudes, whichever is less), so that it never overflows.  The two
// higher pairs of levels fall below the unit and are rounded to it: half a unit each, K / 32
// units in all (at K = 1152 36 units of 2^-62 of the bound on the result).
//
// Bound: the MMAs, issued by one thread; sixteen fold warps and the producer run
// beside them.  Measured figures are at zgemm64_supported below.
#include <algorithm>
#include <climits>
#include <cuda_bf16.h>
#include "common.cuh"
#include "digits.cuh"
#include "gemm.cuh"

namespace nrltb {

namespace {
constexpr int ZD = 7;                       // digits of each operand
constexpr int ZL = 8;                       // levels s + t = 0 .. 7
constexpr int Z_BM = 128, Z_BN = 64, Z_BK = 32;
constexpr int Z_TILE = 128 * 128;           // one plane tile, bytes
constexpr int Z_SLOT = 2 * Z_TILE;          // planes A_p and X_p
constexpr int Z_FOLD = 16;                  // fold warps: 4 per 32-lane quarter, 16 columns each
constexpr int Z_THREADS = 32 * (Z_FOLD + 2);   // + producer warp + MMA warp
constexpr int Z_NBAR = 2 * ZD + 9;          // slot full / empty, level full / empty, MMAs at the end
constexpr int Z_SMEM = ZD * Z_SLOT + 1024 + 8 * Z_NBAR + 16;
constexpr int Z_BAD = INT_MAX;              // exponent of a row or column with an infinity or a NaN
static_assert(Z_SMEM <= 227 * 1024, "planes of a chunk fit the shared memory of an SM");

// op(A) as rows r x k, op(B) as columns r x k: element P[r sr + k sk]
struct ZOperand {
    const double2 *P;
    long sr, sk, sb;      // strides of rows, of k and between matrices
    int R, K, conj, tri;  // tri 1: k <= r, 2: k >= r, the rest reads as zero
    int rp, kc;           // padded rows, chunks
    unsigned char *D;     // planes: [matrix][row tile][chunk][plane]
    int *ex, *la;         // per row: largest element < 2^ex; sum of magnitudes < 2^la
    int tile_rows;        // rows of a tile: 128 (A), 64 (X)
};

// Longest rows whose exponents the digit kernel forms: each of their up to four chunks reads the
// whole row again.  Against a launch for them, a preparation of K = 64 or 128: N = 288, 64
// matrices 56 -> 36 us, N = 144, 15 matrices 28 -> 16; rows up to 192 lost (charges of 16
// atoms, K = 144: 11.30 -> 11.45 ms a call).
constexpr int Z_FUSE = 128;
enum ZOrder { Z_BY_MATRIX, Z_ROWS_UP, Z_ROWS_DOWN, Z_COLS_UP, Z_COLS_DOWN, Z_LOWER };
constexpr int Z_GROUP = 4;   // matrices whose tiles are dealt together (see z_tile)

struct ZProduct {
    const unsigned char *DA, *DX;
    const int *exA, *laA, *exX, *laX;
    int m, n, k, batch, mt, nt, kc;
    int neg, beta1, triA, triB, triC;
    int order, per, gb;   // tile order, tiles of one matrix, matrices of a group
    double2 *C;
    long ldc, sC;
    int hold;             // ZScratch
};
}  // namespace

__device__ unsigned g_z64_fault;

// smallest e with v < 2^e for v > 0 (from the exponent field; subnormals by their own bits)
__device__ __forceinline__ int z_exp_above(unsigned long long bits)
{
    const int E = (int)(bits >> 52) & 0x7FF;
    if (E) return E - 1022;
    const unsigned long long m = bits & 0xFFFFFFFFFFFFFull;
    return m ? -1073 + (63 - __clzll((long long)m)) : 0;
}

__device__ __forceinline__ bool z_in(int tri, int r, int k) { return tri == 0 || (tri == 1 ? k <= r : k >= r); }

__device__ __forceinline__ void z_stat(double2 v, unsigned long long &mx, double &sum)
{
    const double ar = fabs(v.x), ai = fabs(v.y);
    mx = max(mx, max((unsigned long long)__double_as_longlong(ar), (unsigned long long)__double_as_longlong(ai)));
    sum += ar + ai;
}
// the exponents ex, la of a row's largest magnitude and sum
__device__ __forceinline__ int2 z_row_exps(unsigned long long mx, double sum)
{
    const bool bad = mx >= (0x7FFull << 52);
    const int e = bad ? Z_BAD : z_exp_above(mx);
    // the sum's own rounding (K 2^-53 relative) widens it by 2^-30
    const double s = sum * (1.0 + 0x1p-30);
    int l = (mx && !bad && s < 0x1p1000) ? z_exp_above((unsigned long long)__double_as_longlong(s)) : e;
    if (!bad && s >= 0x1p1000) l = e + 19;   // more than the 2^17 elements of a row can add
    return make_int2(e, bad ? Z_BAD : max(l, e));
}

// Largest magnitude and sum of magnitudes of every row.  One CTA per 32 rows, a
// warp's lanes over rows (BYROW: rows are contiguous) or over k.
template <bool BYROW>
__device__ __forceinline__ void z_stats_rows(const ZOperand &o, int block, int b, unsigned long long (*smx)[33],
                                             double (*ssum)[33])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double2 *P = o.P + b * o.sb;
    const int r0 = block * 32;
    const int r = BYROW ? r0 + lane : r0 + warp;
    unsigned long long mx = 0;
    double sum = 0;
    if (r < o.R) {
        int k = BYROW ? warp : lane;
        for (; k + 96 < o.K; k += 128) {
            double2 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                v[u] = make_double2(0, 0);
                if (z_in(o.tri, r, k + 32 * u)) v[u] = P[r * o.sr + (k + 32 * u) * o.sk];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) z_stat(v[u], mx, sum);
        }
        for (; k < o.K; k += 32) {
            if (z_in(o.tri, r, k)) z_stat(P[r * o.sr + k * o.sk], mx, sum);
        }
    }
    if (BYROW) {   // warps hold parts of the same 32 rows: transpose, then a warp per row
        smx[warp][lane] = mx;
        ssum[warp][lane] = sum;
        __syncthreads();
        mx = smx[lane][warp];
        sum = ssum[lane][warp];
    }
    for (int q = 16; q > 0; q >>= 1) {
        mx = max(mx, (unsigned long long)__shfl_xor_sync(0xffffffffu, (long long)mx, q));
        sum += __shfl_xor_sync(0xffffffffu, sum, q);
    }
    if (lane == 0 && r0 + warp < o.rp) {
        const long at = (long)b * o.rp + r0 + warp;
        const int2 x = z_row_exps(mx, sum);
        o.ex[at] = x.x;
        o.la[at] = x.y;
    }
}

// Both operands in one launch, here and for the digits: most products are of a panel with
// something, and a grid of a few CTAs costs its latency, not its work.  Preparing a
// product, four launches -> two: N = 144, 15 matrices 39 -> 28 us, N = 1152, 4 matrices
// 46 -> 33 us on average.
__global__ void __launch_bounds__(1024) k_z_stats(ZOperand a, ZOperand x)
{
    __shared__ unsigned long long smx[32][33];
    __shared__ double ssum[32][33];
    const int na = a.rp / 32, q = blockIdx.x, b = blockIdx.y;
    if (q < na) {
        if (a.sr == 1) z_stats_rows<true>(a, q, b, smx, ssum);
        else z_stats_rows<false>(a, q, b, smx, ssum);
    } else {
        if (x.sr == 1) z_stats_rows<true>(x, q - na, b, smx, ssum);
        else z_stats_rows<false>(x, q - na, b, smx, ssum);
    }
}

// Digit planes.  One CTA per 64 rows and chunk; thread = row and 8 consecutive k
// (four threads hold a row's chunk, so that they write 64 contiguous bytes).
// XOP: the tile rows [re | -im] and [im | re] of op(B); else [re | im] of op(A).
// STATS: the rows' exponents are formed here, by every chunk's CTA from the whole row
// (Z_FUSE: short rows, which then are read again from L2 by their few chunks), instead of
// by a launch before.
template <bool XOP, bool STATS> __device__ __forceinline__ void z_digits_rows(const ZOperand &o, int block, int kc, int b)
{
    const int g = threadIdx.x & 3, r = block * 64 + (threadIdx.x >> 2), k0 = kc * Z_BK + 8 * g;
    if (r >= o.rp) return;
    const int t0 = r / o.tile_rows * o.tile_rows;   // first row of the tile
    const double2 *P = o.P + b * o.sb;
    int2 x;
    if (STATS) {
        // the sum in integers, 2^-30 of the largest magnitude and rounded up (the FP64 pipe would
        // take 128 clocks an element and warp)
        unsigned long long mx = 0, sum = 0;
        auto each = [&](auto use) {
            if (r < o.R)
                for (int k = g; k < o.K; k += 16) {
                    double2 v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        v[u] = make_double2(0, 0);
                        if (k + 4 * u < o.K && z_in(o.tri, r, k + 4 * u)) v[u] = P[r * o.sr + (k + 4 * u) * o.sk];
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        use((unsigned long long)__double_as_longlong(v[u].x) & ~(1ull << 63));
                        use((unsigned long long)__double_as_longlong(v[u].y) & ~(1ull << 63));
                    }
                }
        };
        each([&](unsigned long long a) { mx = max(mx, a); });
#pragma unroll
        for (int q = 1; q < 4; q <<= 1)   // the row's four threads (o.rp is a multiple of the block's rows)
            mx = max(mx, (unsigned long long)__shfl_xor_sync(0xffffffffu, (long long)mx, q));
        const bool bad = mx >= (0x7FFull << 52);
        x.x = bad ? Z_BAD : z_exp_above(mx);
        each([&](unsigned long long a) {
            const int E = max((int)(a >> 52), 1), sh = 23 + x.x + 1022 - E;
            const unsigned long long m = (a & 0xFFFFFFFFFFFFFull) | ((a >> 52) ? 1ull << 52 : 0);
            if (m) sum += ((unsigned)sh < 64u ? m >> sh : 0) + 1;
        });
#pragma unroll
        for (int q = 1; q < 4; q <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, q);
        x.y = bad ? Z_BAD : max(x.x, sum ? x.x - 30 + 64 - __clzll((long long)sum) : x.x);
        if (kc == 0 && g == 0) {
            o.ex[(long)b * o.rp + r] = x.x;
            o.la[(long)b * o.rp + r] = x.y;
        }
    }
    // chunks that a triangular operand's tile never reads
    if (o.tri == 1 && kc * Z_BK >= t0 + o.tile_rows) return;
    if (o.tri == 2 && (kc + 1) * Z_BK <= t0 / Z_BK * Z_BK) return;
    const int e = STATS ? x.x : o.ex[(long)b * o.rp + r];
    const int p = 8 * ZD - 1 - e;
    const bool use = r < o.R && e != Z_BAD;
    uint32_t wr[ZD][4], wi[ZD][4];
#pragma unroll
    for (int u2 = 0; u2 < 4; ++u2) {
        float fr[2][ZD], fi[2][ZD];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = k0 + 2 * u2 + h;
            double2 v = make_double2(0.0, 0.0);
            if (use && k < o.K && z_in(o.tri, r, k)) v = P[r * o.sr + k * o.sk];
            if (o.conj) v.y = -v.y;
            long long U = oz_scaled_rint(v.x, p), W = oz_scaled_rint(v.y, p);
#pragma unroll
            for (int s = ZD - 1; s >= 0; --s) {
                // balanced digit; the top one takes what is left (at most 128)
                const int dr = s ? (int)((U + 128) & 255) - 128 : (int)U;
                const int di = s ? (int)((W + 128) & 255) - 128 : (int)W;
                U = (U - dr) >> 8;
                W = (W - di) >> 8;
                fr[h][s] = __int_as_float(0x4B400000 + dr) - 12582912.0f;   // small integer to float
                fi[h][s] = __int_as_float(0x4B400000 + di) - 12582912.0f;
            }
        }
#pragma unroll
        for (int s = 0; s < ZD; ++s) {
            __nv_bfloat162 a = __floats2bfloat162_rn(fr[0][s], fr[1][s]), c = __floats2bfloat162_rn(fi[0][s], fi[1][s]);
            wr[s][u2] = *reinterpret_cast<uint32_t *>(&a);
            wi[s][u2] = *reinterpret_cast<uint32_t *>(&c);
        }
    }
    const int rt = r - t0;
    unsigned char *T = o.D + (((long)b * (o.rp / o.tile_rows) + r / o.tile_rows) * o.kc + kc) * ZD * Z_TILE;
#pragma unroll
    for (int s = 0; s < ZD; ++s, T += Z_TILE) {
        const uint4 re = make_uint4(wr[s][0], wr[s][1], wr[s][2], wr[s][3]);
        const uint4 im = make_uint4(wi[s][0], wi[s][1], wi[s][2], wi[s][3]);
        *(uint4 *)(T + oz_swz(rt, g)) = re;
        if (!XOP) {
            *(uint4 *)(T + oz_swz(rt, 4 + g)) = im;
        } else {
            const uint4 ng = make_uint4(im.x ^ 0x80008000u, im.y ^ 0x80008000u, im.z ^ 0x80008000u, im.w ^ 0x80008000u);
            *(uint4 *)(T + oz_swz(rt, 4 + g)) = ng;
            *(uint4 *)(T + oz_swz(64 + rt, g)) = im;
            *(uint4 *)(T + oz_swz(64 + rt, 4 + g)) = re;
        }
    }
}

template <bool STATS> __global__ void __launch_bounds__(256) k_z_digits(ZOperand a, ZOperand x)
{
    const int na = a.rp / 64, q = blockIdx.x;
    if (q < na) z_digits_rows<false, STATS>(a, q, blockIdx.y, blockIdx.z);
    else z_digits_rows<true, STATS>(x, q - na, blockIdx.y, blockIdx.z);
}

// the results that leave the normal range (a call, so that its FP64-pipe
// operations stay out of the common path)
__device__ __noinline__ double z_scaled_slow(long long a, int k) { return scalbn((double)a, k); }

// a 2^k rounded to nearest even, with integer operations
__device__ __forceinline__ double z_to_double(long long a, int k)
{
    if (a == 0) return 0.0;
    const unsigned long long u = a < 0 ? 0ull - (unsigned long long)a : (unsigned long long)a;
    const int lz = __clzll((long long)u);
    const unsigned long long mm = u << lz;   // top bit at 63
    unsigned long long q = mm >> 11;
    const unsigned long long rem = mm & 0x7FFull;
    q += (rem > 0x400ull || (rem == 0x400ull && (q & 1ull))) ? 1ull : 0ull;
    const int E = 63 - lz + k + 1023;        // a carry out of q moves into the exponent
    if (E <= 0 || E >= 0x7FE) return z_scaled_slow(a, k);
    return __longlong_as_double((long long)(((unsigned long long)E << 52) + (q - (1ull << 52)) +
                                            (a < 0 ? 0x8000000000000000ull : 0ull)));
}

// chunks [c0, c1) that tile (it, jt) sums over
__device__ __forceinline__ void z_range(const ZProduct &g, int it, int jt, int &c0, int &c1)
{
    int lo = 0, hi = g.k;
    if (g.triA == 1) hi = min(hi, (it + 1) * Z_BM);
    if (g.triA == 2) lo = max(lo, it * Z_BM);
    if (g.triB == 1) hi = min(hi, (jt + 1) * Z_BN);
    if (g.triB == 2) lo = max(lo, jt * Z_BN);
    c0 = lo / Z_BK;
    c1 = (hi + Z_BK - 1) / Z_BK;
    if (c1 < c0) c1 = c0;
}
// Tile t of a launch.  The tiles of a triangular product differ in work by their
// row (triA, triC) or column (triB): those with the most chunks come first, over
// gb matrices at a time (few enough for their planes to meet in L2), so that the
// static deal over the CTAs ends evenly; triC = 1 has only the tiles that touch
// the lower triangle.  N = 1152, 4 matrices, against matrix by matrix: triA = 2
// 1016 -> 797 us, triB = 1 895 -> 786 us.
__device__ __forceinline__ void z_tile(const ZProduct &g, int t, int &b, int &it, int &jt)
{
    const int grp = t / (g.per * g.gb), nb = min(g.gb, g.batch - grp * g.gb);
    int r = t - grp * g.per * g.gb;
    b = grp * g.gb;
    if (g.order == Z_BY_MATRIX) {
        const int q = r / g.per;
        b += q;
        r -= q * g.per;
        it = r / g.nt;
        jt = r - it * g.nt;
    } else if (g.order == Z_LOWER) {
        int cnt = 0;
        for (it = g.mt - 1; it > 0; --it) {
            cnt = min(g.nt, 2 * it + 2);
            if (r < cnt * nb) break;
            r -= cnt * nb;
        }
        cnt = min(g.nt, 2 * it + 2);
        const int q = r / cnt;
        b += q;
        jt = r - q * cnt;
    } else {
        const bool rows = g.order == Z_ROWS_UP || g.order == Z_ROWS_DOWN, down = g.order == Z_ROWS_DOWN || g.order == Z_COLS_DOWN;
        const int major = rows ? g.mt : g.nt, minor = rows ? g.nt : g.mt;
        int x = r / (minor * nb);
        r -= x * minor * nb;
        if (down) x = major - 1 - x;
        const int q = r / minor;
        b += q;
        it = rows ? x : r - q * minor;
        jt = rows ? r - q * minor : x;
    }
}
__device__ __forceinline__ bool z_skip(const ZProduct &g, int it, int jt)
{
    return g.triC == 2 && jt * Z_BN + Z_BN - 1 < it * Z_BM;
}

// Persistent: one CTA per SM, tiles blockIdx.x, + gridDim.x, ..; barrier phases
// run on across tiles, so the next tile's copies and MMAs start while the fold
// warps write the last one.  18 warps: at most 5 per SM sub-partition, 96
// registers a thread (32 accumulators of a fold thread take 64).
__global__ void __maxnreg__(96) k_z_gemm(ZProduct g, unsigned *fault)
{
    extern __shared__ __align__(16) unsigned char z_raw[];
    const uint32_t raw_s = oz_saddr(z_raw);
    unsigned char *base = z_raw + (((raw_s + 1023u) & ~1023u) - raw_s);
    uint64_t *bars = (uint64_t *)(base + ZD * Z_SLOT);
    uint32_t *tslot = (uint32_t *)(bars + Z_NBAR);
    volatile int *abort = (volatile int *)(tslot + 1);
    const uint32_t bar0 = oz_saddr(bars);
    auto full = [&](int p) { return bar0 + 8u * p; };
    auto empty = [&](int p) { return bar0 + 8u * (ZD + p); };
    auto tfull = [&](int q) { return bar0 + 8u * (2 * ZD + q); };
    auto tempty = [&](int q) { return bar0 + 8u * (2 * ZD + 4 + q); };
    const uint32_t last = bar0 + 8u * (2 * ZD + 8);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(oz_saddr(tslot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int q = 0; q < Z_NBAR; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar0 + 8u * q),
                         "r"(q >= 2 * ZD + 4 && q < 2 * ZD + 8 ? Z_FOLD + g.hold : 1) : "memory");
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;
    const int ntiles = g.per * g.batch;

    if (warp == Z_FOLD) {
        // ---- producer: slots 6, 5, .. 0 of every chunk ----
        if (lane == 0) {
            bool ok = true;
            int c = 0, stop = 0;   // chunks of this CTA so far; slot at which it gave up
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
                int b, it, jt;
                z_tile(g, t, b, it, jt);
                if (z_skip(g, it, jt)) continue;
                int c0, c1;
                z_range(g, it, jt, c0, c1);
                const unsigned char *pa = g.DA + (((long)b * g.mt + it) * g.kc) * ZD * Z_TILE;
                const unsigned char *px = g.DX + (((long)b * g.nt + jt) * g.kc) * ZD * Z_TILE;
                for (int kc = c0; kc < c1 && ok; ++kc, ++c)
                    for (int p = ZD - 1; p >= 0; --p) {
                        if (c > 0 && !(ok = oz_wait(empty(p), (c - 1) & 1, abort))) {
                            stop = p + 1;
                            break;
                        }
                        const uint32_t dst = oz_saddr(base + p * Z_SLOT);
                        const long off = ((long)kc * ZD + p) * Z_TILE;
                        oz_expect(full(p), Z_SLOT);
                        oz_bulk(dst, pa + off, Z_TILE, full(p));
                        oz_bulk(dst + Z_TILE, px + off, Z_TILE, full(p));
                        if (kc + 1 < c1) {   // the next chunk's planes into L2
                            oz_prefetch_l2(pa + off + (long)ZD * Z_TILE, Z_TILE);
                            oz_prefetch_l2(px + off + (long)ZD * Z_TILE, Z_TILE);
                        }
                    }
            }
            if (!ok) { *abort = 1; atomicOr(fault ? fault : &g_z64_fault, 1u); }
            // every copy has landed (c counts the chunk it gave up in: slots stop .. 6 were sent)
            for (int p = 0; p < ZD; ++p) {
                const int sent = p < stop ? c - 1 : c;
                if (sent > 0) oz_drain(full(p), (sent - 1) & 1);
            }
        }
    } else if (warp == Z_FOLD + 1) {
        // ---- MMA issue ----
        if (lane == 0) {
            bool ok = true;
            const uint64_t da0 = oz_desc(oz_saddr(base)), dx0 = da0 + (Z_TILE >> 4);
            constexpr uint64_t SL = Z_SLOT >> 4;   // slot stride in the descriptor's address field
            int c = 0;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
                int b, it, jt;
                z_tile(g, t, b, it, jt);
                if (z_skip(g, it, jt)) continue;
                int c0, c1;
                z_range(g, it, jt, c0, c1);
                for (int kc = c0; kc < c1 && ok; ++kc, ++c) {
                    // (unrolled: the issuing thread must stay ahead of 64 cycles an MMA)
#pragma unroll
                    for (int L = ZL - 1; L >= 0; --L) {
                        if (!ok) break;
                        const int q = 7 - L, buf = q & 3, use = 2 * c + (q >> 2);
                        if (use > 0) ok = oz_wait(tempty(buf), (use - 1) & 1, abort);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t tl = tmem + 128u * buf;
                        // pairs (sd, L - sd) from the middle outwards: the slots that the
                        // chunk refills last are read last
                        const int smin = L > ZD - 1 ? L - (ZD - 1) : 0, smax = L - smin, mid = (smin + smax + 1) / 2;
#pragma unroll
                        for (int u = 0; u < ZD; ++u) {
                            if (u > smax - smin) break;
                            const int sd = (u & 1) ? mid - (u + 1) / 2 : mid + u / 2, td = L - sd;
                            if (L == ZL - 1 || (L == ZL - 2 && (sd == 0 || td == 0))) {
                                // first reads of this chunk's slots
                                if (ok) ok = oz_wait(full(sd), c & 1, abort) && oz_wait(full(td), c & 1, abort);
                                if (!ok) break;
                                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            }
                            const uint64_t da = da0 + sd * SL, dx = dx0 + td * SL;
                            oz_mma(tl, da, dx, u > 0 ? 1u : 0u);
                            oz_mma(tl, da + 2, dx + 2, 1u);
                            oz_mma(tl, da + 4, dx + 4, 1u);
                            oz_mma(tl, da + 6, dx + 6, 1u);
                        }
                        if (!ok) break;
                        oz_commit(tfull(buf));
                        if (L < ZD) oz_commit(empty(L));
                    }
                }
            }
            if (ok && c > 0) ok = oz_wait(empty(0), (c - 1) & 1, abort);   // every MMA has finished
            if (!ok) {
                *abort = 1;
                atomicOr(fault ? fault : &g_z64_fault, 1u);
                oz_commit(last);
                oz_drain(last, 0);
            }
        }
    } else if (warp < Z_FOLD) {
        // ---- fold warps ----
        const int q4 = warp & 3, h = warp >> 2;
        const uint32_t trow = tmem + ((uint32_t)(32 * q4) << 16) + 16u * h;
        bool ok = true;
        int c = 0;
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
            int b, it, jt;
            z_tile(g, t, b, it, jt);
            if (z_skip(g, it, jt)) continue;
            int c0, c1;
            z_range(g, it, jt, c0, c1);
            // bits that the sum over k can reach above row maximum x column maximum: by
            // the row's sum of magnitudes, or by those of the warp's 16 columns
            int del;
            {
                const long ai = (long)b * g.mt * Z_BM + it * Z_BM + 32 * q4 + lane;
                const int e = g.exA[ai];
                del = e == Z_BAD ? 0 : g.laA[ai] - e;
                int dj = 0;
                if (lane < 16) {
                    const long aj = (long)b * g.nt * Z_BN + jt * Z_BN + 16 * h + lane;
                    const int f = g.exX[aj];
                    dj = f == Z_BAD ? 0 : g.laX[aj] - f;
                }
                dj = __reduce_max_sync(0xffffffffu, dj);
                del = __reduce_max_sync(0xffffffffu, del);
                del = min(min(del, dj), 19);
                // the old C into L2 while the products run
                if (g.beta1 && (lane & 7) == 0 && it * Z_BM + 32 * q4 + lane < g.m) {
                    const double2 *cp = g.C + b * g.sC + it * Z_BM + 32 * q4 + lane;
                    for (int x = 0; x < 16; ++x)
                        if (jt * Z_BN + 16 * h + x < g.n)
                            asm volatile("prefetch.global.L2 [%0];" :: "l"(cp + (long)(jt * Z_BN + 16 * h + x) * g.ldc));
                }
            }
            long long acc[32];
#pragma unroll
            for (int x = 0; x < 32; ++x) acc[x] = 0;
            for (c1 += c - c0; c < c1 && ok; ++c) {
#pragma unroll
                for (int lp = 0; lp < 4; ++lp) {
                    const int buf = (2 * lp) & 3, use = 2 * c + (lp >> 1);
                    if (ok) ok = oz_wait(tfull(buf), use & 1, abort) && oz_wait(tfull(buf + 1), use & 1, abort);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int hf = 0; hf < 8; ++hf) {
                        float lo[4], hi[4];
                        const uint32_t c4 = trow + 128u * buf + 64u * (hf >> 2) + 4u * (hf & 3);
                        oz_ld4(c4, lo);
                        oz_ld4(c4 + 128u, hi);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        if (hf == 7) {
                            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                            __syncwarp();
                            if (lane == 0) { oz_arrive(tempty(buf)); oz_arrive(tempty(buf + 1)); }
                        }
#pragma unroll
                        for (int x = 0; x < 4; ++x) {
                            long long &a = acc[4 * hf + x];
                            const int w = lp < 2 ? 256 * __float2int_rn(hi[x]) + __float2int_rn(lo[x])
                                                 : (int)(256u * __float_as_uint(hi[x] + 12582912.0f) + __float_as_uint(lo[x] + 12582912.0f) - (256u * 0x4B400000u + 0x4B400000u));
                            if (lp == 0) a += (w + (1 << (7 + del))) >> (8 + del);
                            else if (lp == 1) a += ((long long)w * 65536 + (1ll << (7 + del))) >> (8 + del);
                            else if (lp == 2) a += (long long)w * (1 << (24 - del));
                            else a += (long long)((unsigned long long)(long long)w << (40 - del));
                        }
                    }
                }
            }
            if (!ok) break;
            // C[i, j], j = 16 consecutive columns, four at a time (the old C of the
            // four loaded before their stores)
            // (the tile decoded again: its coordinates would take registers from the fold)
            int t2 = t;
            asm volatile("" : "+r"(t2));
            z_tile(g, t2, b, it, jt);
            const int i = it * Z_BM + 32 * q4 + lane, j0 = jt * Z_BN + 16 * h;
            const int ei = g.exA[(long)b * g.mt * Z_BM + i];
            const bool badrow = ei == Z_BAD;
            double2 *cp = g.C + b * g.sC + i;
            double2 old[2];
#pragma unroll
            for (int x = 0; x < 16; ++x) {
                const int j = j0 + x;
                if (g.beta1 && i < g.m) {   // the old C one column ahead
                    if (x == 0) old[0] = cp[(long)min(j, g.n - 1) * g.ldc];
                    if (x < 15) old[(x + 1) & 1] = cp[(long)min(j + 1, g.n - 1) * g.ldc];
                }
                if (i < g.m && j < g.n) {
                    const int f = g.exX[(long)b * g.nt * Z_BN + j];
                    double2 *o = cp + (long)j * g.ldc;
                    double2 v;
                    if (badrow || f == Z_BAD) {
                        v.x = v.y = __longlong_as_double(0x7FF8000000000000ll);
                    } else {
                        v.x = z_to_double(g.neg ? -acc[x] : acc[x], ei + f + del - 62);
                        v.y = z_to_double(g.neg ? -acc[16 + x] : acc[16 + x], ei + f + del - 62);
                    }
                    if (g.beta1) v = cadd(old[x & 1], v);
                    *o = v;
                }
                __syncwarp();
            }
            __syncwarp();
        }
        if (!ok && lane == 0) { *abort = 1; atomicOr(fault ? fault : &g_z64_fault, 1u); }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512u) : "memory");
    }
}

// Digit path for m, n, k >= 16 of this form; the FMA-pipe kernel keeps
// the rest, where its one or two 64 x 64 tiles of k < 16 take no longer than the five
// launches here (about 25 us).  The rule is on m, n, k alone, so that a matrix takes
// the same route in every batch.
// Measured, 4 matrices, operands' digits included: 1152^3 1.65 ms against 42 on the
// FMA pipe; 1152 x 1152 x 64 0.17 against 2.4; the FP64 step of 4 k at N = 1152 spends
// 22 ms in products against 277, 64 k at N = 288 9 against 82.  The product kernel
// takes 15 000 cycles a chunk (tensor pipe 60 % busy, 8 700 cycles of MMAs), the
// rest waiting on the folds, whose conversions and 64-bit adds come to 6 000 issue
// slots a chunk; a tile's entry and write-back add about 20 000 cycles.
constexpr int Z_MIN = 16;
bool zgemm64_supported(const GemmArgs<double> &g)
{
    const bool al = g.alpha.y == 0.0 && (g.alpha.x == 1.0 || g.alpha.x == -1.0);
    const bool be = g.beta.y == 0.0 && (g.beta.x == 0.0 || g.beta.x == 1.0);
    return al && be && g.m >= Z_MIN && g.n >= Z_MIN && g.k >= Z_MIN && g.k <= 131072;
}

static inline size_t z_al(size_t x) { return (x + 255) & ~size_t(255); }
static int z_sms()
{
    static std::mutex m;
    static std::map<int, int> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(m);
    auto f = cache.find(dev);
    if (f != cache.end()) return f->second;
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return cache[dev] = sms > 0 ? sms : 1;
}

// scratch for one matrix of an m x n x k product: planes of both operands, exponents
static size_t z_bytes_per_matrix(int m, int n, int k)
{
    const size_t mt = cdiv(m, Z_BM), nt = cdiv(n, Z_BN), kc = cdiv(k, Z_BK);
    return (mt + nt) * kc * ZD * Z_TILE + sizeof(int) * 2 * (mt * Z_BM + nt * Z_BN);
}

size_t zgemm64_scratch_bytes(int n, int batch)
{
    // enough for every matrix of a batch at once, or as many as ZGEMM64_SCRATCH_MAX holds:
    // a larger batch goes in parts, and one matrix above it takes the FMA pipe, as
    // every product of an order below Z_MIN does
    if (n < Z_MIN) return 0;
    const size_t per = z_bytes_per_matrix(n, n, n);
    if (per > ZGEMM64_SCRATCH_MAX) return 0;
    return std::min<size_t>(per * batch, ZGEMM64_SCRATCH_MAX) + 4 * 256;
}

bool zgemm64_launch(cudaStream_t s, const GemmArgs<double> &g, const ZScratch &zs)
{
    const size_t per = z_bytes_per_matrix(g.m, g.n, g.k);
    if (!zs.p || zs.bytes < per + 4 * 256) return false;
    const int nb = (int)std::min<size_t>(g.batch, (zs.bytes - 4 * 256) / per);
    const Refusable r;   // the FMA-pipe kernel takes over
    if (smem_attr_at_least((const void *)k_z_gemm, Z_SMEM) != cudaSuccess) {
        r.clear();
        return false;
    }
    const int mt = cdiv(g.m, Z_BM), nt = cdiv(g.n, Z_BN), kc = cdiv(g.k, Z_BK);
    unsigned char *base = (unsigned char *)zs.p;
    unsigned char *DA = base, *DX = DA + (size_t)nb * mt * kc * ZD * Z_TILE;
    int *exA = (int *)(DX + (size_t)nb * nt * kc * ZD * Z_TILE);
    int *laA = (int *)((char *)exA + z_al(sizeof(int) * (size_t)nb * mt * Z_BM));
    int *exX = (int *)((char *)laA + z_al(sizeof(int) * (size_t)nb * mt * Z_BM));
    int *laX = (int *)((char *)exX + z_al(sizeof(int) * (size_t)nb * nt * Z_BN));
    for (int b0 = 0; b0 < g.batch; b0 += nb) {
        const int bn = std::min(nb, g.batch - b0);
        ZOperand a = {}, x = {};
        a.P = g.A + b0 * g.sA;
        a.sr = g.opA ? g.lda : 1;
        a.sk = g.opA ? 1 : g.lda;
        a.sb = g.sA;
        a.R = g.m;
        a.K = g.k;
        a.conj = g.opA;
        a.tri = g.triA;
        a.rp = mt * Z_BM;
        a.kc = kc;
        a.D = DA;
        a.ex = exA;
        a.la = laA;
        a.tile_rows = Z_BM;
        x.P = g.B + b0 * g.sB;
        x.sr = g.opB ? 1 : g.ldb;
        x.sk = g.opB ? g.ldb : 1;
        x.sb = g.sB;
        x.R = g.n;
        x.K = g.k;
        x.conj = g.opB;
        x.tri = g.triB;
        x.rp = nt * Z_BN;
        x.kc = kc;
        x.D = DX;
        x.ex = exX;
        x.la = laX;
        x.tile_rows = Z_BN;
        const dim3 gd((a.rp + x.rp) / 64, kc, bn);
        if (g.k <= Z_FUSE) {
            NRLTB_LAUNCH(k_z_digits<true>, gd, 256, 0, s, a, x);
        } else {
            NRLTB_LAUNCH(k_z_stats, dim3((a.rp + x.rp) / 32, bn), 1024, 0, s, a, x);
            NRLTB_LAUNCH(k_z_digits<false>, gd, 256, 0, s, a, x);
        }
        ZProduct p = {};
        p.DA = DA;
        p.DX = DX;
        p.exA = exA;
        p.laA = laA;
        p.exX = exX;
        p.laX = laX;
        p.m = g.m;
        p.n = g.n;
        p.k = g.k;
        p.batch = bn;
        p.mt = mt;
        p.nt = nt;
        p.kc = kc;
        p.neg = g.alpha.x < 0;
        p.beta1 = g.beta.x != 0.0;
        p.triA = g.triA;
        p.triB = g.triB;
        p.triC = g.triC;
        p.C = g.C + b0 * g.sC;
        p.ldc = g.ldc;
        p.sC = g.sC;
        p.hold = zs.hold;
        p.order = g.triC == 1   ? Z_LOWER
                  : g.triA == 1 ? Z_ROWS_DOWN
                  : g.triA == 2 ? Z_ROWS_UP
                  : g.triB == 1 ? Z_COLS_DOWN
                  : g.triB == 2 ? Z_COLS_UP
                                : Z_BY_MATRIX;
        p.per = mt * nt;
        if (p.order == Z_LOWER) {
            p.per = 0;
            for (int it = 0; it < mt; ++it) p.per += std::min(nt, 2 * it + 2);
        }
        p.gb = p.order == Z_BY_MATRIX ? 1 : std::min(bn, Z_GROUP);
        const int grid = (int)std::min<long>((long)p.per * bn, z_sms());
        NRLTB_LAUNCH(k_z_gemm, grid, Z_THREADS, Z_SMEM, s, p, g_fault_word);
    }
    return true;
}

unsigned zgemm64_fault(bool clear)
{
    unsigned v = 0;
    cudaMemcpyFromSymbol(&v, g_z64_fault, sizeof(v));
    if (clear) {
        const unsigned z = 0;
        cudaMemcpyToSymbol(g_z64_fault, &z, sizeof(z));
    }
    return v;
}

}  // namespace nrltb
