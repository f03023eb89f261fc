// Column solves of the scalar big-n kernels (bigsolve.cu): a column's rows spread over G adjacent lanes
// (G a power of two), lane g holding rows i = G r + g in y[r], r < RM.
//
// A sweep over the row slots is a switch fall-through chain: it enters at the block of 8 slots that holds
// the highest row, each case has compile-time register indices, and a `break` ends the sweep at the
// active range's edge, so no dynamic register index is formed.  Control flow is uniform over the group
// (rows are predicated), so partial results combine with one shuffle; every lane of the warp must call.
//
// Packed lower-triangular tiles use column-major packing: A(i, j), i >= j, at P[pk(j, n) + i - j]
// (pk in stages.cuh).
#pragma once

#include "stages.cuh"

// Row-slot sequences.  SBG_DESC64(C) expands to C(63) C(62) ... C(0) (a one-jump
// select, e.g. of a pivot); SBG_BLOCKS(K) expands to K(7) ... K(0), one `case` per block
// of 8 rows, so that the rows of a block are straight-line code the scheduler can
// interleave, and SBG_ROWS8(S, B) expands to S(8B+7) ... S(8B) inside a block.
#define SBG_DESC64(C) C(63) C(62) C(61) C(60) C(59) C(58) C(57) C(56) C(55) C(54) C(53) C(52) C(51) C(50) C(49) C(48) C(47) C(46) C(45) C(44) C(43) C(42) C(41) C(40) C(39) C(38) C(37) C(36) C(35) C(34) C(33) C(32) C(31) C(30) C(29) C(28) C(27) C(26) C(25) C(24) C(23) C(22) C(21) C(20) C(19) C(18) C(17) C(16) C(15) C(14) C(13) C(12) C(11) C(10) C(9) C(8) C(7) C(6) C(5) C(4) C(3) C(2) C(1) C(0)
#define SBG_BLOCKS(K) K(7) K(6) K(5) K(4) K(3) K(2) K(1) K(0)
#define SBG_ROWS8(S, B) S((B) * 8 + 7) S((B) * 8 + 6) S((B) * 8 + 5) S((B) * 8 + 4) \
                        S((B) * 8 + 3) S((B) * 8 + 2) S((B) * 8 + 1) S((B) * 8 + 0)

namespace sbg {

// y <- L^{-1} y (forward substitution) with L packed by columns (Lp, order n): lane g of the
// group holds rows G r + g.  Each solved w_k stays in its slot of the owning lane.
template <int G, int RM, typename R>
__device__ __forceinline__ void grp_trsm_lower_packed(const cplx<R>* Lp, const R* invd, cplx<R> (&y)[RM], int n,
                                                      int g) {
    using C = cplx<R>;
    const int lane = threadIdx.x & 31;
    const int nb = ((n - 1) / G) >> 3;
    for (int k = 0; k < n; ++k) {
        const int rk = k / G, gk = k - rk * G;
        C piv = y[0];
#define SBG_SEL(I) case I: if constexpr ((I) < RM) piv = y[I]; break;
        switch (rk) { SBG_DESC64(SBG_SEL) default: break; }
#undef SBG_SEL
        if constexpr (G > 1) piv = cshfl(piv, (lane & ~(G - 1)) | gk);
        const C wk = cscale(piv, invd[k]);
        if (g == gk) {
#define SBG_SET(I) case I: if constexpr ((I) < RM) y[I] = wk; break;
            switch (rk) { SBG_DESC64(SBG_SET) default: break; }
#undef SBG_SET
        }
        const C* lk = Lp + pk(k, n) - k;             // lk[i] = L(i, k)
        const int kb = (k + 1) / G - 1;              // slots <= kb are inactive on every lane
#define SBG_S(I) if constexpr ((I) < RM) { const int i = G * (I) + g; if (i > k && i < n) y[I] = cfms(lk[i], wk, y[I]); }
#define SBG_K(B) case B: if ((B) * 8 + 7 <= kb) break; SBG_ROWS8(SBG_S, B)
        switch (nb) { SBG_BLOCKS(SBG_K) default: break; }
#undef SBG_K
#undef SBG_S
    }
}

}  // namespace sbg
