// Back-transform X = L^{-H} Q Z on the FP64 tensor cores with the columns in REGISTERS (k_back_dmma),
// one CTA per pair, one warp per eight columns, n <= kBackDmmaMaxN.
//
// A warp holds its columns transposed, Y^T (8 columns x n rows), as accumulators of
// mma.sync.m8n8k4.f64: lane (g, t) = (lane / 4, lane % 4) has column g, rows 8 I + 2t and 8 I + 2t + 1
// of every 8-row tile I.  The same registers are the A operand of the next product if its
// contraction runs over the rows in the order 0 2 4 6, 1 3 5 7 -- a sum in another order -- so no
// element of Y ever moves: only V and L, shared by all warps, are read from shared memory.  There
// row k of the LV tile (LV(k, i) = v_k(i), i > k; L below and on the diagonal) has an odd leading
// dimension, which keeps the 16-byte fragment loads free of bank conflicts in both orders.
//
//   Q    blocks of 8 reflectors in compact WY form (zlarft's T), last to first:
//        W^T = Y^T conj(V), W^T <- W^T T^T, Y^T -= W^T V^T
//   L    X_I^T = (Y_I^T - sum_{J > I} X_J^T conj(L_JI)) conj(L_II^{-1}), tile by tile from the last
//
// Bound by the tensor pipe and its latency: the products alone take 20.4 K cycles per pair and SM at
// n = 54 (NT = 7), the kernel 33 K.  It replaced a thread per column (n <= 56: one 16-byte broadcast per
// complex FMA, FP64 pipe 29 % busy), 4 or 8 lanes per column (57 .. 84) and, for 85 .. 96, tile products
// through L2.  Microseconds per 1,000 pairs before -> now: n = 24 22 -> 12, 32 29 -> 22, 47 178 -> 67, 54
// 174 -> 108, 64 472 -> 140, 72 1,286 -> 237, 96 1,441 -> 454; 8 pairs of n = 54: 87 -> 30 us.
#include "kernels.cuh"
#include "stages.cuh"
#include "tiles.cuh"

namespace sbg {

namespace {

constexpr int kBlkLd = 9;                   // an 8 x 8 block (T, L_II^{-1}) in shared memory: (i, j) at i + 9 j
constexpr int kBlk = 8 * kBlkLd;

template <int NT>
struct BackDmmaSmem {
    static constexpr int kLd = 8 * NT + 1;
    static constexpr size_t lv = 0;
    static constexpr size_t t = lv + 16 * static_cast<size_t>(kLd) * 8 * NT;
    static constexpr size_t linv = t + 16 * static_cast<size_t>(kBlk) * NT;
    static constexpr size_t tau = linv + 16 * static_cast<size_t>(kBlk) * NT;
    static constexpr size_t total = tau + 16 * 8 * NT;
};

// (dr, di) += (ar + i ai)(br + i bi): four real products; nai = -ai.
__device__ __forceinline__ void cmma(double (&dr)[2], double (&di)[2], double ar, double ai, double nai, double2 b) {
    dmma(dr[0], dr[1], ar, b.x);
    dmma(di[0], di[1], ai, b.x);
    dmma(dr[0], dr[1], nai, b.y);
    dmma(di[0], di[1], ar, b.y);
}

template <int NT, int MINB>
__global__ void __launch_bounds__(32 * NT, MINB) k_back_dmma(int mode, int n, int batch, Workspace ws,
                                                             double2* __restrict__ X, const int* __restrict__ info) {
    using Sm = BackDmmaSmem<NT>;
    constexpr int kLd = Sm::kLd, kThreads = 32 * NT;
    const int b = blockIdx.x;
    if (b >= batch || !pair_selected(ws, b)) return;
    const size_t mat = static_cast<size_t>(n) * n;
    double2* Xb = X + mat * b;
    const int tid = threadIdx.x;
    if (info[b] > n || info[b] < 0) {                             // uniform: B was not positive definite
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
        for (size_t idx = tid; idx < mat; idx += kThreads) Xb[idx] = make_double2(nan, nan);
        return;
    }
    extern __shared__ __align__(16) unsigned char smem[];
    double2* LV = reinterpret_cast<double2*>(smem + Sm::lv);
    double2* Tm = reinterpret_cast<double2*>(smem + Sm::t);
    double2* Li = reinterpret_cast<double2*>(smem + Sm::linv);
    double2* tau = reinterpret_cast<double2*>(smem + Sm::tau);
    const int lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    const double2 zero = make_double2(0.0, 0.0);
    // ---- LV into shared memory, padded with the identity
    {
        const double2* LVg = ws.LV + mat * b;
        const bool cols = n > kSmallMaxN;                         // reflectors along LV's columns
        for (int j = w; j < 8 * NT; j += NT)
            for (int i = lane; i < 8 * NT; i += 32) {
                double2* e = LV + i + j * kLd;
                if (i < n && j < n) {
                    // (v_i(j) above the diagonal)
                    cp_async16(e, i >= j || !cols ? LVg + i + static_cast<size_t>(j) * n
                                                  : LVg + (j - i - 1) + static_cast<size_t>(n - 1 - i) * n);
                } else {
                    *e = make_double2(i == j ? 1.0 : 0.0, 0.0);
                }
            }
        for (int i = tid; i < 8 * NT; i += kThreads) tau[i] = i < n ? ws.tau[static_cast<size_t>(n) * b + i] : zero;
    }
    // ---- the warp's columns
    double yr[NT][2], yi[NT][2];
    const int col = 8 * w + g;
    const double* Zg = reinterpret_cast<const double*>(Xb);
#pragma unroll
    for (int I = 0; I < NT; ++I)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int r = 8 * I + 2 * t + q;
            double2 v = zero;
            if (r < n && col < n) {
                if (mode == kBackLOnly) v = Xb[r + static_cast<size_t>(col) * n];
                else v.x = Zg[r + static_cast<size_t>(col) * n];
            }
            yr[I][q] = v.x;
            yi[I][q] = v.y;
        }
    cp_async_wait();
    __syncthreads();                                              // every Z is read before any X is stored
    // V(8 I + i, 8 B + k): zero on and above the diagonal of the tile I == B
    auto vat = [&](int I, int B, int i, int k) {
        double2 v = LV[(8 * B + k) + (8 * I + i) * kLd];
        if (I == B && i <= k) v = zero;
        return v;
    };
    // ---- warp w: T of block w of reflectors, the inverse of diagonal block w of L
    if (mode != kBackLOnly) {
        double gr[2] = {0.0, 0.0}, gi[2] = {0.0, 0.0};            // G(g, 2t + q) = v_g^H v_{2t+q}
        for (int I = w; I < NT; ++I)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const double2 v = vat(I, w, 2 * t + q, g);
                cmma(gr, gi, v.x, -v.y, v.y, v);
            }
        double2* T = Tm + w * kBlk;
#pragma unroll
        for (int q = 0; q < 2; ++q) T[g + kBlkLd * (2 * t + q)] = make_double2(gr[q], gi[q]);
        __syncwarp();
        if (lane < 8) {                                           // lane i: row i of T
            double2 row[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                double2 s = zero;
#pragma unroll
                for (int l = 0; l < j; ++l) s = cfma(row[l], T[l + kBlkLd * j], s);
                const double2 tj = tau[8 * w + j];
                row[j] = j == lane ? tj : j > lane ? cmul(s, make_double2(-tj.x, -tj.y)) : zero;
            }
            __syncwarp(0xffu);
#pragma unroll
            for (int j = 0; j < 8; ++j) T[lane + kBlkLd * j] = row[j];
        }
    }
    if (mode != kBackQOnly && lane < 8) {                         // lane j: column j of L_ww^{-1}
        const double2* D = LV + 8 * w + 8 * w * kLd;
        double2 x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            double2 s = make_double2(i == lane ? 1.0 : 0.0, 0.0);
#pragma unroll
            for (int l = 0; l < i; ++l) s = cfms(D[i + l * kLd], x[l], s);
            x[i] = cscale(s, 1.0 / D[i + i * kLd].x);
            Li[w * kBlk + i + kBlkLd * lane] = x[i];
        }
    }
    __syncthreads();
    // ---- Y <- Q Y
    if (mode != kBackLOnly) {
        for (int B = NT - 1; B >= 0; --B) {
            if (8 * B + 1 >= n) continue;                         // no reflector in the block
            double wr[2] = {0.0, 0.0}, wi[2] = {0.0, 0.0};
#pragma unroll
            for (int I = 0; I < NT; ++I) {
                if (I < B) continue;                              // uniform
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    double2 v = vat(I, B, 2 * t + q, g);
                    v.y = -v.y;
                    cmma(wr, wi, yr[I][q], yi[I][q], -yi[I][q], v);
                }
            }
            double ur[2] = {0.0, 0.0}, ui[2] = {0.0, 0.0};
#pragma unroll
            for (int q = 0; q < 2; ++q)
                cmma(ur, ui, wr[q], wi[q], -wi[q], Tm[B * kBlk + g + kBlkLd * (2 * t + q)]);
#pragma unroll
            for (int I = 0; I < NT; ++I) {
                if (I < B) continue;
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    cmma(yr[I], yi[I], -ur[q], -ui[q], ui[q], vat(I, B, g, 2 * t + q));
            }
        }
    }
    // ---- Y <- L^{-H} Y
    if (mode != kBackQOnly) {
#pragma unroll
        for (int I = NT - 1; I >= 0; --I) {
#pragma unroll
            for (int J = NT - 1; J > I; --J)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    double2 l = LV[(8 * J + 2 * t + q) + (8 * I + g) * kLd];
                    l.y = -l.y;
                    cmma(yr[I], yi[I], -yr[J][q], -yi[J][q], yi[J][q], l);
                }
            double xr[2] = {0.0, 0.0}, xi[2] = {0.0, 0.0};
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                double2 l = Li[I * kBlk + (2 * t + q) + kBlkLd * g];
                l.y = -l.y;
                cmma(xr, xi, yr[I][q], yi[I][q], -yi[I][q], l);
            }
            yr[I][0] = xr[0]; yr[I][1] = xr[1];
            yi[I][0] = xi[0]; yi[I][1] = xi[1];
        }
    }
    if (col < n) {
#pragma unroll
        for (int I = 0; I < NT; ++I)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int r = 8 * I + 2 * t + q;
                if (r < n) Xb[r + static_cast<size_t>(col) * n] = make_double2(yr[I][q], yi[I][q]);
            }
    }
}

// ----------------------------------------------------------------------------- k_back_dmma_stream
// The same for kBackDmmaMaxN < n <= kBackStreamMaxN, where the LV tile no longer fits shared memory: V and
// L pass through it in panels of 8 columns (a block of reflectors, then a block column of L), two
// buffers, the next panel copied (cp.async) while one is used.  kStreamWarps warps hold 8 columns each and
// make as many passes over the panels as the columns take.  The first pass's X would overwrite Z (real, in
// the first half of the X slot), so Z is first copied to the pair's rotation-log region.  A warp's columns
// take 8 registers per 8 rows: 24 tiles (n = 192) are the most.  us per 1,000 pairs, tile products through L2
// (k_back_q_tc + k_back_tc) -> this: n = 128 3,200 -> 1,530, 160 5,800 -> 2,980, 192 9,200 -> 4,500.
constexpr int kStreamWarps = 8;

template <int NT>
struct BackStreamSmem {
    static constexpr size_t panel = 16 * static_cast<size_t>(kBlkLd) * 8 * NT;   // (i, k) at k + 9 i
    static constexpr size_t t = 2 * panel;
    static constexpr size_t linv = t + 16 * static_cast<size_t>(kBlk) * NT;
    static constexpr size_t total = linv + 16 * static_cast<size_t>(kBlk) * NT;
};

template <int NT>
__global__ void __launch_bounds__(32 * kStreamWarps, 1) k_back_dmma_stream(int mode, int n, int batch, Workspace ws,
                                                                           double2* __restrict__ X,
                                                                           const int* __restrict__ info) {
    using Sm = BackStreamSmem<NT>;
    constexpr int kThreads = 32 * kStreamWarps;
    const int b = blockIdx.x;
    if (b >= batch || !pair_selected(ws, b)) return;
    const size_t mat = static_cast<size_t>(n) * n;
    double2* Xb = X + mat * b;
    const int tid = threadIdx.x;
    if (info[b] > n || info[b] < 0) {                             // uniform: B was not positive definite
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
        for (size_t idx = tid; idx < mat; idx += kThreads) Xb[idx] = make_double2(nan, nan);
        return;
    }
    extern __shared__ __align__(16) unsigned char smem[];
    double2* Tm = reinterpret_cast<double2*>(smem + Sm::t);
    double2* Li = reinterpret_cast<double2*>(smem + Sm::linv);
    const int lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    const double2 zero = make_double2(0.0, 0.0);
    const double2* LVg = ws.LV + mat * b;
    const double2* taug = ws.tau + static_cast<size_t>(n) * b;
    double* Zc = reinterpret_cast<double*>(static_cast<double2*>(ws.log) + static_cast<size_t>(ws.log_stride) * b);
    const bool do_q = mode != kBackLOnly, do_l = mode != kBackQOnly;
    const int nt = (n + 7) / 8;
    auto panel_at = [&](int p) { return reinterpret_cast<double2*>(smem + (p & 1) * Sm::panel); };
    // panel p of a pass: p < nq, the reflectors of block B = nq - 1 - p (rows 8 B ..); then block column I =
    // nt - 1 - (p - nq) of L, rows 8 (I + 1) ..
    const int nq = do_q ? (n + 6) / 8 : 0, npan = nq + (do_l ? nt : 0);      // reflectors 0 .. n - 2
    auto fetch = [&](int p) {
        double2* P = panel_at(p);
        const bool q = p < nq;
        const int c0 = 8 * (q ? nq - 1 - p : nt - 1 - (p - nq)), r0 = q ? c0 : c0 + 8;
        const int c = c0 + w;                                     // a column per warp
        for (int i = r0 + lane; i < 8 * NT; i += 32) {
            double2* e = P + w + kBlkLd * i;
            if (i < n && c < n && (!q || i > c))
                cp_async16(e, q ? LVg + (i - c - 1) + static_cast<size_t>(n - 1 - c) * n
                                : LVg + i + static_cast<size_t>(c) * n);
            else
                *e = zero;
        }
    };
    if (npan > 0) fetch(0);
    if (do_q) {
        const double* Zg = reinterpret_cast<const double*>(Xb);
        for (size_t idx = tid; idx < mat; idx += kThreads) Zc[idx] = Zg[idx];
    }
    // ---- T of every block of reflectors and the inverse of every diagonal block of L, a block per warp at a time
    for (int B = w; B < nt; B += kStreamWarps) {
        if (do_q) {
            double gr[2] = {0.0, 0.0}, gi[2] = {0.0, 0.0};        // G(g, 2t + q) = v_g^H v_{2t+q}
            const int k = 8 * B + g;
#pragma unroll 2
            for (int I = B; I < nt; ++I)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int i = 8 * I + 2 * t + q;
                    const double2 v = i > k && i < n && k + 1 < n ? LVg[(i - k - 1) + static_cast<size_t>(n - 1 - k) * n] : zero;
                    cmma(gr, gi, v.x, -v.y, v.y, v);
                }
            double2* T = Tm + B * kBlk;
#pragma unroll
            for (int q = 0; q < 2; ++q) T[g + kBlkLd * (2 * t + q)] = make_double2(gr[q], gi[q]);
            __syncwarp();
            if (lane < 8) {                                       // lane i: row i of T
                double2 row[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    double2 s = zero;
#pragma unroll
                    for (int l = 0; l < j; ++l) s = cfma(row[l], T[l + kBlkLd * j], s);
                    const double2 tj = 8 * B + j < n ? taug[8 * B + j] : zero;
                    row[j] = j == lane ? tj : j > lane ? cmul(s, make_double2(-tj.x, -tj.y)) : zero;
                }
                __syncwarp(0xffu);
#pragma unroll
                for (int j = 0; j < 8; ++j) T[lane + kBlkLd * j] = row[j];
            }
        }
        if (do_l && lane < 8) {                                   // lane j: column j of L_BB^{-1}
            double2 x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                double2 s = make_double2(i == lane ? 1.0 : 0.0, 0.0);
                const int r = 8 * B + i;
#pragma unroll
                for (int l = 0; l < i; ++l)
                    s = cfms(r < n ? LVg[r + static_cast<size_t>(8 * B + l) * n] : zero, x[l], s);
                x[i] = cscale(s, r < n ? 1.0 / LVg[r + static_cast<size_t>(r) * n].x : 1.0);
                Li[B * kBlk + i + kBlkLd * lane] = x[i];
            }
        }
    }
    cp_async_wait();
    __syncthreads();                                              // also: Z is copied before any X is stored
    for (int c0 = 0; c0 < nt; c0 += kStreamWarps) {
        const int col = 8 * (c0 + w) + g;
        double yr[NT][2], yi[NT][2];
#pragma unroll
        for (int I = 0; I < NT; ++I)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int r = 8 * I + 2 * t + q;
                double2 v = zero;
                if (r < n && col < n) {
                    if (do_q) v.x = Zc[r + static_cast<size_t>(col) * n];
                    else v = Xb[r + static_cast<size_t>(col) * n];
                }
                yr[I][q] = v.x;
                yi[I][q] = v.y;
            }
        // the panel after p: of this pass, or the first of the next
        auto advance = [&](int p) {
            if (p + 1 < npan) fetch(p + 1);
        };
        for (int p = 0; p < nq; ++p) {
            const int B = nq - 1 - p;
            advance(p);
            const double2* V = panel_at(p);
            double wr[2] = {0.0, 0.0}, wi[2] = {0.0, 0.0};
#pragma unroll
            for (int I = 0; I < NT; ++I) {
                if (I < B) continue;                              // uniform
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    double2 v = V[g + kBlkLd * (8 * I + 2 * t + q)];
                    v.y = -v.y;
                    cmma(wr, wi, yr[I][q], yi[I][q], -yi[I][q], v);
                }
            }
            double ur[2] = {0.0, 0.0}, ui[2] = {0.0, 0.0};
#pragma unroll
            for (int q = 0; q < 2; ++q)
                cmma(ur, ui, wr[q], wi[q], -wi[q], Tm[B * kBlk + g + kBlkLd * (2 * t + q)]);
#pragma unroll
            for (int I = 0; I < NT; ++I) {
                if (I < B) continue;
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    cmma(yr[I], yi[I], -ur[q], -ui[q], ui[q], V[(2 * t + q) + kBlkLd * (8 * I + g)]);
            }
            cp_async_wait();
            __syncthreads();
        }
        if (do_l) {
#pragma unroll
            for (int I = NT - 1; I >= 0; --I) {
                if (I >= nt) continue;                            // uniform
                const int p = nq + nt - 1 - I;
                advance(p);
                const double2* P = panel_at(p);
#pragma unroll
                for (int J = NT - 1; J > I; --J)
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        double2 l = P[g + kBlkLd * (8 * J + 2 * t + q)];
                        l.y = -l.y;
                        cmma(yr[I], yi[I], -yr[J][q], -yi[J][q], yi[J][q], l);
                    }
                double xr[2] = {0.0, 0.0}, xi[2] = {0.0, 0.0};
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    double2 l = Li[I * kBlk + (2 * t + q) + kBlkLd * g];
                    l.y = -l.y;
                    cmma(xr, xi, yr[I][q], yi[I][q], -yi[I][q], l);
                }
                yr[I][0] = xr[0]; yr[I][1] = xr[1];
                yi[I][0] = xi[0]; yi[I][1] = xi[1];
                cp_async_wait();
                __syncthreads();
            }
        }
        if (c0 + kStreamWarps < nt) fetch(0);                     // for the next pass
        if (col < n) {
#pragma unroll
            for (int I = 0; I < NT; ++I)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int r = 8 * I + 2 * t + q;
                    if (r < n) Xb[r + static_cast<size_t>(col) * n] = make_double2(yr[I][q], yi[I][q]);
                }
        }
        cp_async_wait();
        __syncthreads();
    }
}

template <int NT>
cudaError_t run_back_stream(int mode, int n, int batch, const Workspace& ws, double2* X, const int* info,
                            cudaStream_t stream) {
    const size_t smem = BackStreamSmem<NT>::total;
    if (smem > static_cast<size_t>(max_smem_optin())) return cudaErrorInvalidValue;
    static SmemOptIn f;
    set_smem_limit(reinterpret_cast<const void*>(k_back_dmma_stream<NT>), f, static_cast<int>(smem));
    k_back_dmma_stream<NT><<<batch, 32 * kStreamWarps, smem, stream>>>(mode, n, batch, ws, X, info);
    return cudaGetLastError();
}

template <int NT, int MINB>
cudaError_t run_back_dmma(int mode, int n, int batch, const Workspace& ws, double2* X, const int* info,
                          cudaStream_t stream) {
    const size_t smem = BackDmmaSmem<NT>::total;
    if (smem > static_cast<size_t>(max_smem_optin())) return cudaErrorInvalidValue;
    static SmemOptIn f;
    set_smem_limit(reinterpret_cast<const void*>(k_back_dmma<NT, MINB>), f, static_cast<int>(smem));
    k_back_dmma<NT, MINB><<<batch, 32 * NT, smem, stream>>>(mode, n, batch, ws, X, info);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_back_dmma(int mode, int n, int batch, const Workspace& ws, double2* X, const int* info,
                             cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (n < 1 || n > kBackDmmaMaxN || !X || !info || !ws.LV || !ws.tau) return cudaErrorInvalidValue;
#define SBG_CASE(NT, MINB) case NT: return run_back_dmma<NT, MINB>(mode, n, batch, ws, X, info, stream)
    // (column tiles = warps, CTAs per SM): as many CTAs as shared memory and the columns' registers allow; for nine
    // tiles two are worth 964 bytes of spill stores a thread (n = 72: 271 us per 1,000 pairs with one CTA and none, 237
    // with two)
    switch ((n + 7) / 8) {
        SBG_CASE(1, 16);
        SBG_CASE(2, 16);
        SBG_CASE(3, 8);
        SBG_CASE(4, 6);
        SBG_CASE(5, 4);
        SBG_CASE(6, 3);
        SBG_CASE(7, 2);
        SBG_CASE(8, 2);
        SBG_CASE(9, 2);
        SBG_CASE(10, 1);
        SBG_CASE(11, 1);
        SBG_CASE(12, 1);
        default: return cudaErrorInvalidValue;
    }
#undef SBG_CASE
}

cudaError_t launch_back_stream(int mode, int n, int batch, const Workspace& ws, double2* X, const int* info,
                               cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (n <= kSmallMaxN || n > kBackStreamMaxN || !X || !info || !ws.LV || !ws.tau || !ws.log)
        return cudaErrorInvalidValue;
    if (2 * static_cast<size_t>(ws.log_stride) < static_cast<size_t>(n) * n) return cudaErrorInvalidValue;
#define SBG_CASE(NT) if (n <= 8 * (NT)) return run_back_stream<NT>(mode, n, batch, ws, X, info, stream)
    SBG_CASE(14);
    SBG_CASE(16);
    SBG_CASE(18);
    SBG_CASE(20);
    SBG_CASE(22);
    SBG_CASE(24);
#undef SBG_CASE
    return cudaErrorInvalidValue;
}

size_t back_stream_smem_bytes(int n) {
    const size_t nt = static_cast<size_t>((n <= 112 ? 112 : (n + 15) / 16 * 16) / 8);      // as the cases above
    return 16 * kBlk * (2 * nt + 2 * nt);
}

size_t back_dmma_smem_bytes(int n) {
    const size_t nt = static_cast<size_t>((n + 7) / 8);
    return 16 * (8 * nt * (8 * nt + 1) + 2 * kBlk * nt + 8 * nt);
}

}  // namespace sbg
