// Householder tridiagonalisation with the matrix in REGISTERS and shared memory (k_hetrd_reg), NW
// warps per pair, for n <= kHetrdRegMaxN.
//
// zhetd2's steps (LAPACK's reflectors, p = tau A v, w = p - tau/2 (p^H v) v, A -= v w^H + w v^H) on
// the full Hermitian matrix: warp w holds the columns j = w (mod NW), lane l of it the rows
// l, l + RS, .. (RS = ceil(n / R) <= 32).  The warp's last NS columns, which live longest, stay in
// its registers (R x NS complex entries a thread); the earlier ones are in shared memory, each lane
// reading and writing its own rows.  Keeping both triangles costs 12 m^2 FMAs a step instead of 8, but every row sum
// of the matvec is then a sum over a thread's own registers and NW partials: no column walk, no
// reduction per column, and the only operands read are the vectors' entries v_j, w_j of the warp's
// column -- one address for the whole warp (a broadcast, half the cost of a 16-byte load with
// distinct addresses), used for R rows.
//
// One pass per step: step k - 1's update is applied to each live column just before the column's
// part of the matvec with v_k; column k alone is updated ahead, for the reflector formed from it.
//
// The kernels it replaces walked the packed triangle in shared memory (a warp per pair, each lane
// its own row: 47 K shared-memory wavefronts per pair at n = 54, 62 % of the load/store unit's rate),
// a full tile in shared memory by 256 threads (66 <= n <= 84), or the triangle in L2 (n > 84).
// Microseconds per 1,000 pairs before -> now: n = 24 48 -> 20, 32 80 -> 31, 47 191 -> 113, 54 284 -> 141,
// 72 1,197 -> 422, 96 2,013 -> 737, 128 4,600 -> 2,070.  It is bound by the latency of a step's chain
// (column sum, norm, square root, reflector) at the few pairs an SM holds and by the load/store unit (62 % at
// n = 54); FP64 pipe 47 % busy.
//
// The mixed form's complex64 Householder (n <= kMixedMaxN) is the same kernel in FP32: C (FP64, in the X
// buffer) is rounded as it is read, and the outputs go where the FP64 form's go, promoted: reflectors, d, e,
// and tau rescaled in FP64 so that each H = I - tau v v^H is unitary to FP64 rounding for the promoted v
// (|tau|^2 ||v||^2 = 2 Re tau; the FP32 tau satisfies it only to ~1e-7), which keeps the refinement's
// Y = Q Z orthonormal to the level of Z.  C itself also goes to the pair's stash in the refinement's tile
// format, since X is overwritten before the refinement runs.  It replaced a warp per pair on the packed
// triangle: microseconds per 4,096 pairs n = 8 34 -> 21, 16 93 -> 50, 24 185 -> 104, 32 310 -> 186, 40 505 -> 325,
// 54 790 -> 574.
#include "kernels.cuh"
#include "stages.cuh"

#include <type_traits>

namespace sbg {

namespace {

// Shared memory: v of this step and the next, w per warp, the matvec's partial row sums and v^H A v
// per warp, (tau, beta) of two steps, and the columns of the first `off` slots.  The vectors have rv + 1 rows:
// every thread's rows and every slot's column, and one spare row for the lanes that hold no row; a
// column has rn + 1.
template <typename F, int R, int NW>
struct RegHetrdSmem {
    int rs, rn, rv, off;
    size_t v, w, part, spart, tau, cols, total;
    __host__ __device__ RegHetrdSmem(int n, int ns) {
        const int slots = (n + NW - 1) / NW;
        rs = (n + R - 1) / R;
        rn = R * rs;
        off = slots > ns ? slots - ns : 0;
        rv = NW * (off + ns) > rn ? NW * (off + ns) : rn;
        const size_t row = sizeof(cplx<F>) * static_cast<size_t>(rv + 1);
        size_t o = 0;
        v = o;     o += 2 * row;
        w = o;     o += NW * row;
        part = o;  o += NW > 1 ? NW * row : 0;
        spart = o; o += 8 * ((NW + 1) & ~1);
        tau = o;   o += sizeof(cplx<F>) * 4;
        cols = o;  o += sizeof(cplx<F>) * static_cast<size_t>(off) * NW * (rn + 1);
        total = o;
    }
};

template <typename F> __device__ __forceinline__ cplx<F> as(double2 z);
template <> __device__ __forceinline__ double2 as<double>(double2 z) { return z; }
template <> __device__ __forceinline__ float2 as<float>(double2 z) {
    return make_float2(static_cast<float>(z.x), static_cast<float>(z.y));
}
template <typename F> __device__ __forceinline__ double2 as(float2 z) { return make_double2(z.x, z.y); }
__device__ __forceinline__ void stage(double2* dst, const double2* src) { cp_async16(dst, src); }
__device__ __forceinline__ void stage(float2* dst, const double2* src) { *dst = as<float>(*src); }

template <int NW>
__device__ __forceinline__ void pair_sync() {
    if constexpr (NW == 1) __syncwarp(); else __syncthreads();
}

// The reflector that zeroes column c below row c + 1, formed by the warp that holds the column
// (x[s]: its entry of row s RS + lane, zero outside the matrix; la: the lane of row c + 1): v into
// vnext at the thread's rows (at[s]; zero up to row c), tau and beta into stau[0..1], d[c] to dg.
template <typename F, int R>
__device__ __forceinline__ void form_reflector(int c, int RS, int la, const double2 (&x)[R], const int (&at)[R],
                                               double2* vnext, double2* stau, double* dg) {
    const int lane = threadIdx.x & 31;
    const bool in = lane < RS;
    double2 alpha = make_double2(0.0, 0.0);
    double s2 = 0.0;
#pragma unroll
    for (int s = 0; s < R; ++s) {
        const int r = s * RS + lane;
        const double t = fma(x[s].x, x[s].x, x[s].y * x[s].y);
        s2 += r > c + 1 && in ? t : 0.0;
        if (r == c + 1) alpha = x[s];                             // (lanes >= RS hold row r + .. of no slot: not read)
    }
    alpha = cshfl(alpha, la);
    s2 = warp_sum(s2);
    // beta = -sign(Re alpha) ||(alpha, x)||, tau = (beta - alpha) / beta, scale = 1 / (alpha - beta);
    // H = I for a zero tail and a real alpha.  The norm is n2 rsqrt(n2) after one Newton step.
    // (An n2 or a reciprocal outside the normal range gives NaN, or a norm of 2^510 and more: k_tridiag_values sees
    // either in d and e and has the pair formed again, scaled.)
    const bool id = s2 == 0.0 && alpha.y == 0.0;
    const double n2 = fma(alpha.x, alpha.x, fma(alpha.y, alpha.y, s2));
    const double rn = rsqrt(n2);
    double nrm = n2 * rn;
    nrm = fma(fma(-nrm, nrm, n2), 0.5 * rn, nrm);
    const double beta = alpha.x >= 0.0 ? -nrm : nrm, ib = alpha.x >= 0.0 ? -rn : rn;
    const double ar = alpha.x - beta, ai = alpha.y;
    const double rd = recip_nr(fma(ar, ar, ai * ai));
    const double2 scale = id ? make_double2(0.0, 0.0) : make_double2(ar * rd, -ai * rd);
    const double2 tk = id ? make_double2(0.0, 0.0) : make_double2((beta - alpha.x) * ib, -alpha.y * ib);
    double2 v[R];
#pragma unroll
    for (int s = 0; s < R; ++s) {
        const int r = s * RS + lane;
        v[s] = cmul(x[s], scale);
        if (r <= c + 1 || !in) v[s] = make_double2(r == c + 1 && in ? 1.0 : 0.0, 0.0);
        vnext[at[s]] = v[s];
    }
    if (lane == 0) { stau[0] = tk; stau[1] = make_double2(id ? alpha.x : beta, 0.0); }
#pragma unroll
    for (int s = 0; s < R; ++s)
        if (in && s * RS + lane == c) dg[c] = x[s].x;
}

// The same in FP32.  Apart from the FP64 form, whose code one template for both made 2 % slower (32,768
// pairs of n = 54: 4.66 -> 4.75 ms).
template <typename F, int R>
__device__ __forceinline__ void form_reflector(int c, int RS, int la, const float2 (&x)[R], const int (&at)[R],
                                               float2* vnext, float2* stau, double* dg) {
    const int lane = threadIdx.x & 31;
    const bool in = lane < RS;
    using F2 = cplx<F>;
    const F2 zero = mk<F>(F(0), F(0));
    F2 alpha = zero;
    F s2 = F(0);
#pragma unroll
    for (int s = 0; s < R; ++s) {
        const int r = s * RS + lane;
        const F t = fma(x[s].x, x[s].x, x[s].y * x[s].y);
        s2 += r > c + 1 && in ? t : F(0);
        if (r == c + 1) alpha = x[s];                             // (lanes >= RS hold row r + .. of no slot: not read)
    }
    alpha = cshfl(alpha, la);
    s2 = warp_sum(s2);
    // beta = -sign(Re alpha) ||(alpha, x)||, tau = (beta - alpha) / beta, scale = 1 / (alpha - beta);
    // H = I for a zero tail and a real alpha.  The norm is n2 rsqrt(n2) after one Newton step.
    const bool id = s2 == F(0) && alpha.y == F(0);
    const F n2 = fma(alpha.x, alpha.x, fma(alpha.y, alpha.y, s2));
    const F rn = rsqrtf(n2);
    F nrm = n2 * rn;
    nrm = fma(fma(-nrm, nrm, n2), F(0.5) * rn, nrm);
    const F beta = alpha.x >= F(0) ? -nrm : nrm, ib = alpha.x >= F(0) ? -rn : rn;
    const F ar = alpha.x - beta, ai = alpha.y;
    const F rd = 1.0f / fma(ar, ar, ai * ai);
    const F2 scale = id ? zero : mk<F>(ar * rd, -ai * rd);
    const F2 tk = id ? zero : mk<F>((beta - alpha.x) * ib, -alpha.y * ib);
    F2 v[R];
#pragma unroll
    for (int s = 0; s < R; ++s) {
        const int r = s * RS + lane;
        v[s] = cmul(x[s], scale);
        if (r <= c + 1 || !in) v[s] = mk<F>(r == c + 1 && in ? F(1) : F(0), F(0));
        vnext[at[s]] = v[s];
    }
    if (lane == 0) { stau[0] = tk; stau[1] = mk<F>(id ? alpha.x : beta, F(0)); }
#pragma unroll
    for (int s = 0; s < R; ++s)
        if (in && s * RS + lane == c) dg[c] = x[s].x;
}

// One case per column slot: a sweep over the live slots q0 .. NS - 1 jumps into the sequence once
// and falls through.  The columns of slot q0 that are dead already meet v = w = 0.
#define SBG_ASC32(C) C(0) C(1) C(2) C(3) C(4) C(5) C(6) C(7) C(8) C(9) C(10) C(11) C(12) C(13) C(14) C(15) \
    C(16) C(17) C(18) C(19) C(20) C(21) C(22) C(23) C(24) C(25) C(26) C(27) C(28) C(29) C(30) C(31)

// kBlock: register columns between two tests for live ones
template <typename F, int R, int NW, int NS, int MINB, int kBlock>
__global__ void __launch_bounds__(32 * NW, MINB) k_hetrd_reg(int n, int batch, const double2* __restrict__ C,
                                                             Workspace ws, const int* __restrict__ info) {
    const int b = blockIdx.x;
    if (b >= batch || !pair_selected(ws, b)) return;
    if (info[b] != 0) return;                                     // uniform
    extern __shared__ __align__(16) unsigned char smem[];
    using F2 = cplx<F>;
    constexpr bool kSingle = sizeof(F) == 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const RegHetrdSmem<F, R, NW> lay(n, NS);
    const int RS = lay.rs, RV = lay.rv, CR = lay.rn + 1, off = lay.off;
    F2* vbuf = reinterpret_cast<F2*>(smem + lay.v);
    F2* wb = reinterpret_cast<F2*>(smem + lay.w) + warp * (RV + 1);
    F2* part = reinterpret_cast<F2*>(smem + lay.part);
    F* spart = reinterpret_cast<F*>(smem + lay.spart);
    F2* stau = reinterpret_cast<F2*>(smem + lay.tau);
    F2* cols = reinterpret_cast<F2*>(smem + lay.cols) + warp * CR;       // slot q's column: + q NW CR
    const size_t mat = static_cast<size_t>(n) * n;
    const double2* Cb = C + mat * b;
    double* dg = ws.d + static_cast<size_t>(n) * b;
    double* eg = ws.e + static_cast<size_t>(n) * b;
    double2* taug = ws.tau + static_cast<size_t>(n) * b;
    double2* LVg = ws.LV + mat * b;
    const bool lv_cols = n > kSmallMaxN;
    const F2 zero = mk<F>(F(0), F(0));
    const bool in = lane < RS;
    // where the thread's rows are in the vectors and columns; lanes without a row use the spare row (zero)
    int at[R], ac[R];
#pragma unroll
    for (int s = 0; s < R; ++s) {
        at[s] = in ? s * RS + lane : RV;
        ac[s] = in ? s * RS + lane : CR - 1;
    }

    if constexpr (kSingle) {
        // C itself, full Hermitian, to the pair's stash (refine_stash_entries: re plane, im plane, zero padded)
        const int NP = refine_np(n), LD = refine_ld(n);
        double* sre = reinterpret_cast<double*>(static_cast<char*>(ws.log) + 16 * static_cast<size_t>(ws.log_stride) * b);
        double* sim = sre + static_cast<size_t>(NP) * LD;
        for (int j = warp; j < NP; j += NW)
            for (int i = j + lane; i < NP; i += 32) {
                double2 v = i < n && j < n ? Cb[i + static_cast<size_t>(j) * n] : make_double2(0.0, 0.0);
                if (i == j) v.y = 0.0;
                sre[j * LD + i] = v.x;
                sim[j * LD + i] = v.y;
                if (i != j) { sre[i * LD + j] = v.x; sim[i * LD + j] = -v.y; }
            }
    }
    // C's lower triangle, mirrored: the shared-memory columns' lower parts by cp.async and the register
    // columns' by loads that are all in flight together, then the upper parts from shared memory (row j of
    // an earlier column; only the register columns' own corner is read transposed from global memory)
    F2* col0 = cols - warp * CR;                             // column j < off NW at col0 + j CR
    const int jr = off * NW;                                      // first register column
    for (int q = 0; q < off; ++q) {
        const int j = q * NW + warp;
#pragma unroll
        for (int s = 0; s < R; ++s) {
            const int r = s * RS + lane;
            if (in && r >= j && r < n) stage(col0 + j * CR + r, Cb + r + static_cast<size_t>(j) * n);
            else if (!in || r >= n) col0[j * CR + ac[s]] = zero;
        }
    }
    F2 a[R][NS];
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        const int j = (off + q) * NW + warp;
#pragma unroll
        for (int s = 0; s < R; ++s) {
            const int r = s * RS + lane;
            a[s][q] = zero;
            if (in && r < n && j < n && r >= jr)
                a[s][q] = as<F>(r >= j ? Cb[r + static_cast<size_t>(j) * n] : Cb[j + static_cast<size_t>(r) * n]);
        }
    }
    if constexpr (!kSingle) cp_async_wait();
    pair_sync<NW>();
    for (int q = 0; q < off; ++q) {
        const int j = q * NW + warp;
#pragma unroll
        for (int s = 0; s < R; ++s) {
            const int r = s * RS + lane;
            if (in && r < j) {
                const F2 z = col0[r * CR + j];
                col0[j * CR + r] = mk<F>(z.x, -z.y);
            }
            if (in && r == j) col0[j * CR + r].y = F(0);
        }
    }
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        const int j = (off + q) * NW + warp;
#pragma unroll
        for (int s = 0; s < R; ++s) {
            const int r = s * RS + lane;
            if (in && r < jr && j < n) a[s][q] = col0[r * CR + j];
            if (r < j) a[s][q].y = -a[s][q].y;
            if (r == j) a[s][q].y = F(0);
        }
    }
    for (int i = threadIdx.x; i < 2 * (RV + 1); i += 32 * NW) vbuf[i] = zero;    // rows n .. RV stay zero
    for (int i = lane; i <= RV; i += 32) wb[i] = zero;
    pair_sync<NW>();
    if (warp == 0) {
        F2 x[R];
#pragma unroll
        for (int s = 0; s < R; ++s) x[s] = off > 0 ? cols[ac[s]] : a[s][0];
        form_reflector<F, R>(0, RS, RS > 1 ? 1 : 0, x, at, vbuf, stau, dg);
    }
    pair_sync<NW>();

    F2 vr[R], wr[R];                                         // v, w of the pending update: the thread's rows
#pragma unroll
    for (int s = 0; s < R; ++s) vr[s] = wr[s] = zero;
    // rows below s0 RS are done from step s0 RS - 1 on: a phase per number of live row slots
    auto phase = [&](auto first, int k0, int k1) {
        constexpr int S0 = decltype(first)::value;
        for (int k = k0; k < k1; ++k) {
            const F2* v = vbuf + (k & 1) * (RV + 1);
            const F2* vp = vbuf + ((k + 1) & 1) * (RV + 1);
            const F2 tk = stau[2 * (k & 1)];
            const int q0 = (k + 1) / NW, q0r = q0 - off;          // the first live column's slot, register slot
            // ---- one pass over the live columns: step k - 1's update, then the warp's share of A v
            F2 acc[R], am[R];                                // the two products of each part apart:
#pragma unroll
            for (int s = S0; s < R; ++s) acc[s] = am[s] = zero;   // half as long a dependent chain
            {
                F2* c = cols + q0 * (NW * CR);
                const F2 *pv = v + q0 * NW + warp, *pp = vp + q0 * NW + warp, *pw = wb + q0 * NW + warp;
#pragma unroll 2
                for (int left = off - q0; left > 0; --left) {
                    const F2 pj = *pp, wj = *pw, vj = *pv;
#pragma unroll
                    for (int s = S0; s < R; ++s) {
                        const F2 t = cfmsc(wr[s], pj, cfmsc(vr[s], wj, c[ac[s]]));
                        c[ac[s]] = t;
                        acc[s].x = fma(t.x, vj.x, acc[s].x);
                        acc[s].y = fma(t.x, vj.y, acc[s].y);
                        am[s].x = fma(t.y, vj.y, am[s].x);
                        am[s].y = fma(t.y, vj.x, am[s].y);
                    }
                    c += NW * CR;
                    pv += NW;
                    pp += NW;
                    pw += NW;
                }
            }
#pragma unroll
            for (int q = 0; q < NS; q += kBlock) {
                if (q0r < q + kBlock) {                           // uniform
                    F2 vj[kBlock], wj[kBlock], pj[kBlock];
#pragma unroll
                    for (int u = 0; u < kBlock; ++u)
                        if (q + u < NS) {
                            pj[u] = vp[(off + q + u) * NW + warp];
                            wj[u] = wb[(off + q + u) * NW + warp];
                            vj[u] = v[(off + q + u) * NW + warp];
                        }
#pragma unroll
                    for (int u = 0; u < kBlock; ++u)
                        if (q + u < NS) {
#pragma unroll
                            for (int s = S0; s < R; ++s) {
                                const F2 t = cfmsc(wr[s], pj[u], cfmsc(vr[s], wj[u], a[s][q + u]));
                                a[s][q + u] = t;
                                acc[s].x = fma(t.x, vj[u].x, acc[s].x);
                                acc[s].y = fma(t.x, vj[u].y, acc[s].y);
                                am[s].x = fma(t.y, vj[u].y, am[s].x);
                                am[s].y = fma(t.y, vj[u].x, am[s].y);
                            }
                        }
                }
            }
#pragma unroll
            for (int s = S0; s < R; ++s) {
                acc[s].x -= am[s].x;
                acc[s].y += am[s].y;
                vr[s] = v[at[s]];
            }
            // ---- v^H A v (real) and the row sums over the warps
            F vav = F(0);
#pragma unroll
            for (int s = S0; s < R; ++s) vav = fma(vr[s].x, acc[s].x, fma(vr[s].y, acc[s].y, vav));
            if constexpr (NW > 1) {
#pragma unroll
                for (int s = S0; s < R; ++s) part[warp * (RV + 1) + at[s]] = acc[s];
                vav = warp_sum(vav);
                if (lane == 0) spart[warp] = vav;
                __syncthreads();
                F2 pt[R][NW];
#pragma unroll
                for (int s = S0; s < R; ++s)
#pragma unroll
                    for (int u = 0; u < NW; ++u) pt[s][u] = part[u * (RV + 1) + at[s]];
                vav = F(0);
#pragma unroll
                for (int u = 0; u < NW; ++u) vav += spart[u];
#pragma unroll
                for (int s = S0; s < R; ++s) {
#pragma unroll
                    for (int u = 1; u < NW; ++u) pt[s][0] = cadd(pt[s][0], pt[s][u]);
                    acc[s] = pt[s][0];
                }
            } else {
                vav = warp_sum(vav);
            }
            // ---- w = p + a2 v, p = tau A v, a2 = -tau/2 (p^H v) = -|tau|^2 / 2 (v^H A v); every warp all rows
            const F a2 = F(-0.5) * cabs2(tk) * vav;
#pragma unroll
            for (int s = S0; s < R; ++s) {
                const F2 p = cmul(tk, acc[s]);
                const bool live = in && s * RS + lane > k;
                wr[s] = live ? mk<F>(fma(a2, vr[s].x, p.x), fma(a2, vr[s].y, p.y)) : zero;
                wb[at[s]] = wr[s];
            }
            __syncwarp();
            // ---- column k + 1 (slot q0) takes the update at once and gives the next reflector
            if (k + 1 - q0 * NW == warp) {
                F2 x[R];
#pragma unroll
                for (int s = 0; s < R; ++s) x[s] = zero;
#define SBG_S(I) case I: if constexpr ((I) < NS) { _Pragma("unroll") for (int s = S0; s < R; ++s) x[s] = a[s][I]; } break;
                if (q0r < 0) {
#pragma unroll
                    for (int s = S0; s < R; ++s) x[s] = cols[q0 * NW * CR + ac[s]];
                } else {
                    switch (q0r) { SBG_ASC32(SBG_S) default: break; }
                }
#undef SBG_S
                const F2 vj = v[k + 1], wj = wb[k + 1];
#pragma unroll
                for (int s = S0; s < R; ++s) x[s] = cfmsc(wr[s], vj, cfmsc(vr[s], wj, x[s]));
                const int la = k + 2 - S0 * RS == RS ? 0 : k + 2 - S0 * RS;       // the lane of row k + 2
                form_reflector<F, R>(k + 1, RS, la, x, at, vbuf + ((k + 1) & 1) * (RV + 1), stau + 2 * ((k + 1) & 1), dg);
            }
            if (NW == 1 || k + 2 - (k + 2) / NW * NW == warp) {   // meanwhile another warp stores reflector k
#pragma unroll
                for (int s = S0; s < R; ++s) {
                    const int r = s * RS + lane;
                    if (in && r > k && r < n) {
                        if (lv_cols) LVg[(r - k - 1) + static_cast<size_t>(n - 1 - k) * n] = as<double>(vr[s]);
                        else LVg[k + static_cast<size_t>(r) * n] = as<double>(vr[s]);
                    }
                }
                if constexpr (kSingle) {                          // unitary in FP64: |tau|^2 ||v||^2 = 2 Re tau
                    double s2 = 0.0;
#pragma unroll
                    for (int s = S0; s < R; ++s) {
                        const double x = vr[s].x, y = vr[s].y;
                        s2 = fma(x, x, fma(y, y, s2));
                    }
                    s2 = warp_sum(s2);
                    const double tr = tk.x, ti = tk.y, t2 = tr * tr + ti * ti, sc = t2 > 0.0 ? 2.0 * tr / (t2 * s2) : 0.0;
                    if (lane == 0) { taug[k] = make_double2(tr * sc, ti * sc); eg[k] = stau[2 * (k & 1) + 1].x; }
                } else {
                    if (lane == 0) { taug[k] = tk; eg[k] = stau[2 * (k & 1) + 1].x; }
                }
            }
            pair_sync<NW>();
        }
    };
    auto from = [&](int s) { return s == 0 ? 0 : s == R ? n - 1 : min(n - 1, s * RS - 1); };
    phase(std::integral_constant<int, 0>{}, from(0), from(1));
    if constexpr (R > 1) phase(std::integral_constant<int, 1>{}, from(1), from(2));
    if constexpr (R > 2) phase(std::integral_constant<int, 2>{}, from(2), from(3));
    if constexpr (R > 3) phase(std::integral_constant<int, 3>{}, from(3), from(4));
    if constexpr (R > 4) phase(std::integral_constant<int, 4>{}, from(4), from(5));
    if (threadIdx.x == 0) { eg[n - 1] = 0.0; taug[n - 1] = make_double2(0.0, 0.0); }
}

// (rows per lane, warps per pair, column slots in registers, pairs per SM, block) by n.  Measured over the
// neighbouring shapes, microseconds per 1,000 pairs: few warps and many pairs per SM win (n = 48: 1 warp 113, 2
// 122; n = 54: 2 warps 141, 1 warp 170, and in an earlier form 3 warps 185, 4 227, 8 327) until a
// pair's columns no longer fit beside others in shared memory; fewer register slots than these make the
// shared-memory part the bound (n = 54: 8 slots 162, 10 147, 12 141).  A block of 4 where it measured better (n = 32: 33.2
// with 2, 30.6 with 4), 2 elsewhere.  Above n = 128 nine slots of five rows spill 740 bytes a thread (stores).
#define SBG_HETRD_REG_BY_N(n, F)                                                       \
    do {                                                                               \
        if ((n) <= 24) F(1, 1, 8, 24, 2);                                              \
        if ((n) <= 32) F(1, 1, 16, 16, 4);                                             \
        if ((n) <= 40) F(2, 1, 10, 10, 2);                                             \
        if ((n) <= 48) F(2, 1, 16, 8, 2);                                              \
        if ((n) <= 56) F(2, 2, 12, 5, 4);                                              \
        if ((n) <= 64) F(2, 2, 16, 4, 2);                                              \
        if ((n) <= 76) F(3, 4, 7, 3, 2);                                               \
        if ((n) <= 96) F(3, 4, 8, 2, 2);                                               \
        if ((n) <= 128) F(4, 8, 8, 1, 2);                                              \
        F(5, 8, 9, 1, 2);                                                              \
    } while (0)

// The complex64 form (n <= kMixedMaxN): half the registers and shared memory an entry, so more pairs per SM.
// Microseconds per 4,096 pairs (n = 54): 2 warps x 12 slots 574, 2 x 16 615, 1 x 24 718, 1 x 32 752; n = 32:
// 24 slots 186, 32 194, 16 207; n = 24: 8 slots at 28 pairs per SM 104, 24 at 16 117.
#define SBG_HETRD_C64_BY_N(n, F)                                                       \
    do {                                                                               \
        if ((n) <= 24) F(1, 1, 8, 28, 2);                                              \
        if ((n) <= 32) F(1, 1, 24, 16, 4);                                             \
        F(2, 2, 12, 10, 4);                                                            \
    } while (0)

template <typename F, int R, int NW, int NS, int MINB, int kBlock>
cudaError_t run_hetrd_reg(int n, int batch, const double2* C, const Workspace& ws, const int* info,
                          cudaStream_t stream) {
    const size_t smem = RegHetrdSmem<F, R, NW>(n, NS).total;
    if (smem > static_cast<size_t>(max_smem_optin())) return cudaErrorInvalidValue;
    static SmemOptIn f;
    set_smem_limit(reinterpret_cast<const void*>(k_hetrd_reg<F, R, NW, NS, MINB, kBlock>), f, static_cast<int>(smem));
    k_hetrd_reg<F, R, NW, NS, MINB, kBlock><<<batch, 32 * NW, smem, stream>>>(n, batch, C, ws, info);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_hetrd_reg(int n, int batch, const double2* C, const Workspace& ws, const int* info,
                             cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (n < 1 || n > kHetrdRegMaxN || !C || !info || !ws.LV || !ws.d || !ws.e || !ws.tau) return cudaErrorInvalidValue;
#define SBG_RUN(R, NW, NS, MINB, KB) return run_hetrd_reg<double, R, NW, NS, MINB, KB>(n, batch, C, ws, info, stream)
    SBG_HETRD_REG_BY_N(n, SBG_RUN);
#undef SBG_RUN
}

size_t hetrd_reg_smem_bytes(int n) {
#define SBG_SIZE(R, NW, NS, MINB, KB) return RegHetrdSmem<double, R, NW>(n, NS).total
    SBG_HETRD_REG_BY_N(n, SBG_SIZE);
#undef SBG_SIZE
}

cudaError_t launch_hetrd_c64(int n, int batch, const double2* C, const Workspace& ws, int* info, cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (n < 1 || n > kMixedMaxN || !C || !info || !ws.LV || !ws.d || !ws.e || !ws.tau || !ws.log ||
        ws.log_stride < refine_stash_entries(n))
        return cudaErrorInvalidValue;
#define SBG_RUN(R, NW, NS, MINB, KB) return run_hetrd_reg<float, R, NW, NS, MINB, KB>(n, batch, C, ws, info, stream)
    SBG_HETRD_C64_BY_N(n, SBG_RUN);
#undef SBG_RUN
}

size_t hetrd_c64_smem_bytes(int n) {
#define SBG_SIZE(R, NW, NS, MINB, KB) return RegHetrdSmem<float, R, NW>(n, NS).total
    SBG_HETRD_C64_BY_N(n, SBG_SIZE);
#undef SBG_SIZE
}

}  // namespace sbg
