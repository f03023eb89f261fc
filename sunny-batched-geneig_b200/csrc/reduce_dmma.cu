// Cholesky of B and the reduction C = L^{-1} A L^{-H} on the FP64 tensor cores (k_reduce_dmma), one CTA
// per pair, n <= kReduceDmmaMaxN.
//
// L stays in shared memory as 8 x 8 blocks, factored right-looking, a column block at a time: a lane per
// row in registers (the diagonal block's rows repeated in every warp that takes part), then the trailing
// blocks as products.
// The two solves then run as in the back-transform (back_dmma.cu): a warp holds eight columns,
// transposed, as accumulators of mma.sync.m8n8k4.f64 -- lane (g, t) has column g, rows 8 I + 2t and
// 8 I + 2t + 1 of every tile I -- which are the next product's A operand as they stand when its
// contraction runs over the rows in the order 0 2 4 6, 1 3 5 7:
//   W_I^T = (A_I^T - sum_{J < I} W_J^T L_IJ^T) (L_II^{-1})^T,
// and again with W^H (transposed through shared memory, the output buffer or, above n = 56, the pair's
// rotation-log region, free until the eigensolve) in place of A.  The second solve forms all of C, of which the lower triangle is kept: 8 n^3 flops for
// both against 16/3 n^3 with C's symmetry, but no warp waits for another inside a solve.
//
// Half of a CTA's time at n = 54 is the Cholesky's chain of pivots (2.9 K cycles per block of eight
// columns, 47 K in all), which the other CTAs of the SM cover; the products need 15 K cycles per pair and SM,
// the kernel takes 31 K.  Microseconds per 1,000 pairs, the kernels it replaces (a warp per pair for the
// Cholesky and a thread per column for the solves up to 56, tile products through L2 above) -> now: n = 24
// 33 -> 14, 32 41 -> 24, 47 178 -> 71, 54 213 -> 105, 64 362 -> 141, 72 711 -> 210, 96 784 -> 490, 128 1,615 ->
// 1,170; 8 pairs of n = 54 135 -> 25 us.
#include "kernels.cuh"
#include "stages.cuh"
#include "tiles.cuh"

namespace sbg {

namespace {

constexpr int kBlkLd = 9;                   // an 8 x 8 block in shared memory: (i, j) at i + 9 j, so that
constexpr int kBlk = 8 * kBlkLd;            // the 16-byte fragment loads are free of bank conflicts

template <int NT>
struct ReduceDmmaSmem {
    static constexpr size_t l = 0;
    static constexpr size_t linv = l + 16 * static_cast<size_t>(kBlk) * (NT * (NT + 1) / 2);
    static constexpr size_t flag = linv + 16 * static_cast<size_t>(kBlk) * NT;
    // W, (r, c) at r + kLdw c, where as many CTAs fit an SM with it as without (MINB below).  n = 49 .. 56, two CTAs
    // either way: 104 us per 1,000 pairs at n = 49 against 128 through the output buffer; 41 .. 48, three instead
    // of four: 76 against 71 at n = 47.
    static constexpr int kLdw = 8 * NT + 1;
    static constexpr bool kW = NT <= 7 && NT != 6;
    static constexpr size_t wt = flag + 16;
    static constexpr size_t total = wt + (kW ? 16 * static_cast<size_t>(kLdw) * 8 * NT : 0);
};

// (dr, di) += (ar + i ai)(br + i bi): four real products; nai = -ai.
__device__ __forceinline__ void cmma(double (&dr)[2], double (&di)[2], double ar, double ai, double nai, double2 b) {
    dmma(dr[0], dr[1], ar, b.x);
    dmma(di[0], di[1], ai, b.x);
    dmma(dr[0], dr[1], nai, b.y);
    dmma(di[0], di[1], ar, b.y);
}

// One step of the Cholesky for the rows of column block K that this warp's lanes hold, lanes 0 .. 7 the
// diagonal block's (every warp that takes part), the others 24 rows below it: zpotrf's steps, column by
// column, the pivot row's entries by shuffles, so the panel below costs nothing beside the diagonal
// block.  Returns 0, or the local order of the first leading minor that is not positive (also NaN), the
// same on every lane.
__device__ __forceinline__ int factor_rows(double2 (&a)[8]) {
    const int lane = threadIdx.x & 31;
    int f = 0;                                                    // (no early exit: a branch per column cost
#pragma unroll                                                    // as much as the column)
    for (int k = 0; k < 8; ++k) {
        const double dkk = __shfl_sync(0xffffffffu, a[k].x, k);
        if (!(dkk > 0.0) && f == 0) f = k + 1;
        const double rs = rsqrt(dkk);
        double dsq = dkk * rs;                                    // sqrt(dkk) after one Newton step
        dsq = fma(fma(-dsq, dsq, dkk), 0.5 * rs, dsq);
        a[k] = cscale(a[k], rs);
#pragma unroll
        for (int j = k + 1; j < 8; ++j) a[j] = cfmsc(a[k], cshfl(a[k], j), a[j]);
        if (lane == k) a[k] = make_double2(dsq, 0.0);
    }
    return f;
}

template <int NT, int NW, int MINB>
__global__ void __launch_bounds__(32 * NW, MINB) k_reduce_dmma(int mode, const double2* __restrict__ A,
                                                               const double2* __restrict__ B, int n, int batch,
                                                               Workspace ws, double2* __restrict__ out,
                                                               int* __restrict__ info) {
    using Sm = ReduceDmmaSmem<NT>;
    const int b = blockIdx.x;
    if (b >= batch || !pair_selected(ws, b)) return;
    extern __shared__ __align__(16) unsigned char smem[];
    double2* Lt = reinterpret_cast<double2*>(smem + Sm::l);       // block (I, J), J <= I, at I (I + 1) / 2 + J
    double2* Li = reinterpret_cast<double2*>(smem + Sm::linv);
    int* fail = reinterpret_cast<int*>(smem + Sm::flag);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    const size_t mat = static_cast<size_t>(n) * n;
    const double2 zero = make_double2(0.0, 0.0);
    auto block = [&](int I, int J) { return Lt + (I * (I + 1) / 2 + J) * kBlk; };
    auto entry = [&](int i, int j) -> double2& { return block(i >> 3, j >> 3)[(i & 7) + kBlkLd * (j & 7)]; };
    // ---- B's lower triangle, padded with the identity
    {
        const double2* Bb = B + mat * b;
        for (int j = w; j < 8 * NT; j += NW)
            for (int i = (j & ~7) + lane; i < 8 * NT; i += 32) {
                double2* e = &entry(i, j);
                if (i < n && j < n && i >= j) cp_async16(e, Bb + i + static_cast<size_t>(j) * n);
                else *e = make_double2(i == j ? 1.0 : 0.0, 0.0);
            }
        if (tid == 0) *fail = 0;
        if (mode == kReduceFull || mode == kReduceHegst) {        // A into L2 while the Cholesky runs
            const char* a = reinterpret_cast<const char*>(A + mat * b);
            for (size_t o = 128 * static_cast<size_t>(tid); o < 16 * mat; o += 128 * 32 * NW)
                asm volatile("prefetch.global.L2 [%0];" :: "l"(a + o));
        }
        cp_async_wait();
    }
    __syncthreads();
    // ---- Cholesky, a column block at a time
    if (mode != kReduceFromLM) {
        for (int K = 0; K < NT; ++K) {
            if (w == 0 || 8 * (K + 1) + 24 * w < 8 * NT) {
                const int r = lane < 8 ? 8 * K + lane : 8 * (K + 1) + 24 * w + lane - 8;
                const bool in = r < 8 * NT;
                double2* row = block(in ? r >> 3 : K, K) + (r & 7);
                double2 a[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) a[k] = row[kBlkLd * k];
                const int f = factor_rows(a);
                if (f) {
                    if (tid == 0) *fail = 8 * K + f;
                } else if (in && (lane >= 8 || w == 0)) {
                    // (another warp may still read the diagonal block: its L is stored after the barrier)
                    if (lane >= 8) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) row[kBlkLd * k] = a[k];
                    }
                }
                if (w == 0 && lane < 8) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) Li[K * kBlk + lane + kBlkLd * k] = a[k];
                }
            }
            __syncthreads();
            if (*fail) {                                          // uniform
                if (tid == 0) info[b] = mode == kReduceFull ? n + *fail : *fail;
                return;
            }
            // T(I, J) -= L(I, K) L(J, K)^H, K < J <= I, the blocks dealt to the warps
            const int m = NT - K - 1, tiles = m * (m + 1) / 2;
            int i = 0, j = w;                                     // tile w + NW s of the triangle, row by row
            for (int p = w; p < tiles; p += NW, j += NW) {
                while (j > i) { j -= i + 1; ++i; }
                const double2* P = block(K + 1 + i, K);
                const double2* Q = block(K + 1 + j, K);
                double2* T = block(K + 1 + i, K + 1 + j);
                double dr[2], di[2], er[2] = {0.0, 0.0}, ei[2] = {0.0, 0.0};
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const double2 v = T[g + kBlkLd * (2 * t + q)];
                    dr[q] = v.x;
                    di[q] = v.y;
                }
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const double2 a = P[g + kBlkLd * (2 * t + q)];
                    double2 c = Q[g + kBlkLd * (2 * t + q)];
                    c.y = -c.y;
                    if (q == 0) cmma(dr, di, -a.x, -a.y, a.y, c);
                    else cmma(er, ei, -a.x, -a.y, a.y, c);
                }
#pragma unroll
                for (int q = 0; q < 2; ++q) T[g + kBlkLd * (2 * t + q)] = make_double2(dr[q] + er[q], di[q] + ei[q]);
            }
            __syncthreads();
        }
    }
    // ---- the diagonal blocks, factored in Li, to their place, and their inverses over them in Li
    for (int K = w; K < NT; K += NW) {
        double2* D = block(K, K);
        double2* I8 = Li + K * kBlk;
        if (mode != kReduceFromLM) {
            for (int e = lane; e < 64; e += 32)
                if ((e & 7) > (e >> 3)) D[(e & 7) + kBlkLd * (e >> 3)] = I8[(e & 7) + kBlkLd * (e >> 3)];
            if (lane < 8) {
                // (the root of an infinite pivot came out as NaN, 0 inf; its column below is zero: the row drops out)
                const double root = I8[10 * lane].x;
                D[10 * lane] = make_double2(root == root ? root : __longlong_as_double(0x7ff0000000000000ll), 0.0);
            }
            __syncwarp();
        }
        if (lane < 8) {                                           // lane j: column j of the inverse
            double2 x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                double2 s = make_double2(i == lane ? 1.0 : 0.0, 0.0);
#pragma unroll
                for (int l = 0; l < i; ++l) s = cfms(D[i + l * kBlkLd], x[l], s);
                x[i] = cscale(s, 1.0 / D[i + i * kBlkLd].x);
                I8[i + kBlkLd * lane] = x[i];
            }
        }
    }
    __syncthreads();
    auto store_l = [&]() {
        double2* dst = mode == kReduceChol ? out + mat * b : ws.LV + mat * b;
        for (int j = w; j < n; j += NW)
            for (int i = (mode == kReduceChol ? 0 : j & ~31) + lane; i < n; i += 32) {
                if (i >= j) dst[i + static_cast<size_t>(j) * n] = entry(i, j);
                else if (mode == kReduceChol) dst[i + static_cast<size_t>(j) * n] = zero;
            }
    };
    if (mode == kReduceChol || mode == kReduceFromLM) {
        store_l();
        if (tid == 0) info[b] = 0;
        return;
    }
    // ---- W = L^{-1} A, then C = L^{-1} W^H
    const double2* Ab = A + mat * b;
    double2* Ob = out + mat * b;
    // W goes through shared memory where it fits, else through out itself when every warp has one tile of
    // columns (all of W is read before any of C is stored), else through the rotation-log region
    double2* Wg = Sm::kW ? reinterpret_cast<double2*>(smem + Sm::wt)
                         : (NW == NT ? Ob : static_cast<double2*>(ws.log) + static_cast<size_t>(ws.log_stride) * b);
    const int ldw = Sm::kW ? Sm::kLdw : n;
    auto store_w = [&](int r, int c, double2 v) { Wg[r + static_cast<size_t>(c) * ldw] = v; };
    for (int pass = 0; pass < 2; ++pass) {
        for (int ct = w; ct < NT; ct += NW) {
            const int col = 8 * ct + g;
            double yr[NT][2], yi[NT][2];
#pragma unroll
            for (int I = 0; I < NT; ++I)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int r = 8 * I + 2 * t + q;
                    double2 v = zero;
                    if (r < n && col < n) {
                        if (pass == 0) v = Ab[r + static_cast<size_t>(col) * n];
                        else {
                            v = Wg[col + static_cast<size_t>(r) * ldw];
                            v.y = -v.y;
                        }
                    }
                    yr[I][q] = v.x;
                    yi[I][q] = v.y;
                }
            if (pass == 0 && ct == w && mode == kReduceFull) store_l();            // while A arrives
            if (!Sm::kW && NW == NT && pass == 1) __syncthreads();
#pragma unroll
            for (int I = 0; I < NT; ++I) {
#pragma unroll
                for (int J = 0; J < I; ++J) {
                    const double2* P = Lt + (I * (I + 1) / 2 + J) * kBlk;
#pragma unroll
                    for (int q = 0; q < 2; ++q)
                        cmma(yr[I], yi[I], -yr[J][q], -yi[J][q], yi[J][q], P[g + kBlkLd * (2 * t + q)]);
                }
                double xr[2] = {0.0, 0.0}, xi[2] = {0.0, 0.0};
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    cmma(xr, xi, yr[I][q], yi[I][q], -yi[I][q], Li[I * kBlk + g + kBlkLd * (2 * t + q)]);
                yr[I][0] = xr[0]; yr[I][1] = xr[1];
                yi[I][0] = xi[0]; yi[I][1] = xi[1];
            }
            if (col < n) {
#pragma unroll
                for (int I = 0; I < NT; ++I)
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int r = 8 * I + 2 * t + q;
                        if (r >= n) continue;
                        if (pass == 0) store_w(r, col, make_double2(yr[I][q], yi[I][q]));
                        else if (r >= col) Ob[r + static_cast<size_t>(col) * n] = make_double2(yr[I][q], r == col ? 0.0 : yi[I][q]);
                        else if (mode == kReduceHegst) Ob[r + static_cast<size_t>(col) * n] = zero;
                    }
            }
        }
        __syncthreads();                                          // W is complete (this CTA wrote all of it)
    }
    if (tid == 0) info[b] = 0;
}

template <int NT, int NW, int MINB>
cudaError_t run_reduce_dmma(int mode, const double2* A, const double2* B, int n, int batch, const Workspace& ws,
                            double2* out, int* info, cudaStream_t stream) {
    const size_t smem = ReduceDmmaSmem<NT>::total;
    if (smem > static_cast<size_t>(max_smem_optin())) return cudaErrorInvalidValue;
    static SmemOptIn f;
    set_smem_limit(reinterpret_cast<const void*>(k_reduce_dmma<NT, NW, MINB>), f, static_cast<int>(smem));
    k_reduce_dmma<NT, NW, MINB><<<batch, 32 * NW, smem, stream>>>(mode, A, B, n, batch, ws, out, info);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_reduce_dmma(int mode, const double2* A, const double2* B, int n, int batch, const Workspace& ws,
                               double2* out, int* info, cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (n < 1 || n > kReduceDmmaMaxN || !B || !info) return cudaErrorInvalidValue;
    if ((mode == kReduceFull || mode == kReduceHegst) && (!A || !out)) return cudaErrorInvalidValue;
    if ((mode == kReduceFull || mode == kReduceFromLM) && !ws.LV) return cudaErrorInvalidValue;
    if (mode == kReduceChol && !out) return cudaErrorInvalidValue;
    if (n > 56 && mode != kReduceChol && mode != kReduceFromLM &&
        (!ws.log || static_cast<size_t>(ws.log_stride) < static_cast<size_t>(n) * n))
        return cudaErrorInvalidValue;
    // (column tiles, warps, CTAs per SM): as many CTAs as shared memory leaves room for, some registers spilled for it
    // (stores up to 224 bytes a thread, 692 for 18 tiles).  A warp per tile up to 56; above, fewer warps with two or more tiles
    // each and more CTAs, so that other pairs' solves run beside a pair's Cholesky (n = 64: 8 warps x 2 CTAs
    // 161 us per 1,000 pairs, 4 x 4 136; n = 72: 5 x 2 255, 5 x 3 215, 9 x 1 343)
#define SBG_CASE(NT, NW, MINB) case NT: return run_reduce_dmma<NT, NW, MINB>(mode, A, B, n, batch, ws, out, info, stream)
    const int nt = (n + 7) / 8;
    switch (nt <= 12 ? nt : (nt + 1) / 2 * 2) {
        SBG_CASE(1, 1, 16);
        SBG_CASE(2, 2, 16);
        SBG_CASE(3, 3, 10);
        SBG_CASE(4, 4, 6);
        SBG_CASE(5, 5, 4);
        SBG_CASE(6, 6, 4);
        SBG_CASE(7, 7, 2);
        SBG_CASE(8, 4, 4);
        SBG_CASE(9, 5, 3);
        SBG_CASE(10, 5, 2);
        SBG_CASE(11, 6, 2);
        SBG_CASE(12, 6, 2);
        SBG_CASE(14, 7, 1);
        SBG_CASE(16, 8, 1);
        SBG_CASE(18, 9, 1);
        default: return cudaErrorInvalidValue;
    }
#undef SBG_CASE
}

size_t reduce_dmma_smem_bytes(int n) {
    const int nt = (n + 7) / 8;
    switch (nt <= 12 ? nt : (nt + 1) / 2 * 2) {
#define SBG_CASE(NT) case NT: return ReduceDmmaSmem<NT>::total
        SBG_CASE(1); SBG_CASE(2); SBG_CASE(3); SBG_CASE(4); SBG_CASE(5); SBG_CASE(6); SBG_CASE(7); SBG_CASE(8);
        SBG_CASE(9); SBG_CASE(10); SBG_CASE(11); SBG_CASE(12); SBG_CASE(14); SBG_CASE(16); SBG_CASE(18);
        default: return 0;
#undef SBG_CASE
    }
}

}  // namespace sbg
