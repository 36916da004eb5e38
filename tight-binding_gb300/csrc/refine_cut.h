/*
 * refine_cut.h -- runs of close eigenvalues cut into clusters (k_ref_clusters), as a
 * plain C function that a host-compiled check runs too.
 */
#pragma once
#ifdef __CUDACC__
#define RC_FN static __device__ inline
#else
#define RC_FN static inline
#endif

/* The sorted values srt[a0 .. e0) become clusters of at most cmax: a longer run is cut
 * at its largest gap (the first of equal ones), recursively.  pos0 and csz of a value's
 * column ord[q] take its cluster's first position and size.  Returns 1 if a gap below
 * `least` had to be cut.
 * Pieces wait on a stack with the smaller one on top, so that each level holds at most
 * half of the one below and 32 levels are enough for any run.  (With the right piece
 * always on top, a run of equal values, whose cuts take one value at a time off the
 * left, fills any stack; what is left over then exceeds the cluster solve's arrays.) */
RC_FN int ref_cut(const double *srt, int a0, int e0, int cmax, double least, const int *ord, int *pos0, int *csz)
{
    int stk[33][2], sp = 1, forced = 0;
    stk[0][0] = a0;
    stk[0][1] = e0;
    while (sp > 0) {
        --sp;
        const int a = stk[sp][0], e = stk[sp][1];
        if (e - a <= cmax) {
            for (int q = a; q < e; ++q) {
                pos0[ord[q]] = a;
                csz[ord[q]] = e - a;
            }
            continue;
        }
        int cut = a + 1;
        double best = -1.0;
        for (int q = a + 1; q < e; ++q) {
            const double g = srt[q] - srt[q - 1];
            if (g > best) {
                best = g;
                cut = q;
            }
        }
        if (best < least) forced = 1;
        const int left = cut - a > e - cut;   /* the larger piece goes below */
        stk[sp][0] = left ? a : cut;
        stk[sp][1] = left ? cut : e;
        ++sp;
        stk[sp][0] = left ? cut : a;
        stk[sp][1] = left ? e : cut;
        ++sp;
    }
    return forced;
}
