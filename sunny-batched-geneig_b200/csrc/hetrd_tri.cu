// Householder tridiagonalisation for n > kHetrdRegMaxN (k_hetrd_tri): one CTA of 8 warps per pair on the
// packed lower triangle, as many of its last columns as fit in shared memory and the first ones in the
// pair's rotation-log region (free until the eigensolve, in L2 while the CTA works on it).
//
// zhetd2's steps with ONE pass over the trailing triangle per step: step k-1's rank-2 update is
// applied lazily, to column k by warp 0 just before it forms reflector k from that column, and to
// columns k+1.. by all warps in the same walk that forms the Hermitian matvec with reflector k.  The walk
// goes down columns, a long and a short one per warp at a time, 32 consecutive rows per load; lane l owns
// the rows l (mod 32), so its entries of v, w and the matvec's row sums stay in registers and only the
// two columns' sums need a reduction, done together.
//
// With the whole triangle in L2 (3 CTAs per SM, 444 triangles of 295 KB at n = 192: more than L2 holds)
// the walks were bound by that traffic, 2.6 TB/s: 14.4 us per pair at n = 192.  The last 154
// columns of n = 192 take part in all but 2 % of it.  Now 8.6 us per pair; 83 % of a step is the walk,
// ~1,450 cycles per two columns where the FP64 pipe needs 440: the latency of two columns' chains, of the step's
// barriers and of shared memory with two warps per scheduler (issue slots 30 % used, FP64 pipe 18 %).  us per 1,000 pairs before -> now: n = 160 7,500 -> 5,600, 192 14,400 -> 8,600.
#include "kernels.cuh"
#include "stages.cuh"

#include <type_traits>

namespace sbg {

namespace {

constexpr int kTriThreads = 256, kTriWarps = kTriThreads / 32;
constexpr size_t kTriSmem = 227 * 1024;

struct TriSmem {
    int j0;                     // first column in shared memory
    size_t v, w, col, rows, red, tau, tri, total;
    __host__ __device__ explicit TriSmem(int n) {
        const size_t nv = 16 * static_cast<size_t>(n);
        size_t o = 0;
        v = o;    o += 2 * nv;                  // reflectors k and k-1, by row
        w = o;    o += nv;                      // w of the pending update
        col = o;  o += nv;                      // column sums of the matvec, then p
        rows = o; o += kTriWarps * nv;          // row sums, per warp
        red = o;  o += 8 * kTriWarps;
        tau = o;  o += 16 * 2;
        tri = o;
        const size_t room = (kTriSmem - o) / 16;
        int m = 0;
        while (m < n && static_cast<size_t>(m + 1) * (m + 2) / 2 <= room) ++m;
        j0 = n - m;
        total = o + 16 * (static_cast<size_t>(m) * (m + 1) / 2);
    }
};

template <int S>
__global__ void __launch_bounds__(kTriThreads, 1) k_hetrd_tri(int n, int batch, const double2* __restrict__ C,
                                                              Workspace ws, const int* __restrict__ info) {
    const int b = blockIdx.x;
    if (b >= batch || !pair_selected(ws, b)) return;
    if (info[b] != 0) return;                                     // the Cholesky failed (uniform)
    extern __shared__ __align__(16) unsigned char smem[];
    const TriSmem L(n);
    const int j0 = L.j0;
    double2* vbuf = reinterpret_cast<double2*>(smem + L.v);
    double2* wb = reinterpret_cast<double2*>(smem + L.w);
    double2* colp = reinterpret_cast<double2*>(smem + L.col);
    double2* prow = reinterpret_cast<double2*>(smem + L.rows);
    double* red = reinterpret_cast<double*>(smem + L.red);
    double2* s_tk = reinterpret_cast<double2*>(smem + L.tau);
    double2* Ps = reinterpret_cast<double2*>(smem + L.tri);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t mat = static_cast<size_t>(n) * n;
    const double2* Cb = C + mat * b;
    double2* Pg = static_cast<double2*>(ws.log) + static_cast<size_t>(ws.log_stride) * b;
    double* dout = ws.d + static_cast<size_t>(n) * b;
    double* eout = ws.e + static_cast<size_t>(n) * b;
    double2* tout = ws.tau + static_cast<size_t>(n) * b;
    const double2 zero = make_double2(0.0, 0.0);
    // column j: entry of row i at column(j)[i], i >= j
    auto col_s = [&](int j) { return Ps + (pk(j, n) - pk(j0, n)) - j; };
    auto col_g = [&](int j) { return Pg + pk(j, n) - j; };
    auto column = [&](int j) { return j >= j0 ? col_s(j) : col_g(j); };
    for (int j = warp; j < n; j += kTriWarps) {                   // (C's diagonal is real as the reduction left it)
        double2* cj = column(j);
        const double2* c = Cb + static_cast<size_t>(j) * n;
        for (int i = j + lane; i < n; i += 32) {
            if (j >= j0) cp_async16(cj + i, c + i);
            else cj[i] = c[i];
        }
    }
    cp_async_wait();
    // (finite before their first step: the walk multiplies them by zeros while nothing is pending)
    for (int i = tid; i < 3 * n; i += kTriThreads) (i < 2 * n ? vbuf : wb - 2 * n)[i] = zero;
    __syncthreads();
    bool upd = false;                                             // step k-1's update pending (uniform)
    for (int k = 0; k + 1 < n; ++k) {
        double2* vb = vbuf + (k & 1) * n;                         // reflector k, vb[i] for rows i > k
        const double2* vp = vbuf + ((k + 1) & 1) * n;             // reflector k-1 (while upd)
        if (warp == 0) {
            double2* ck = column(k);
            double2 x[S];
            double s2 = 0.0;
            const double2 wk = upd ? wb[k] : zero, vk = upd ? vp[k] : zero;
            double2 alpha = zero;
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const int i = 32 * s + lane;
                const bool in = i >= k && i < n;
                x[s] = in ? ck[i] : zero;
                const double2 wi = in && upd ? wb[i] : zero, pi = in && upd ? vp[i] : zero;
                x[s] = cfmsc(wi, vk, cfmsc(pi, wk, x[s]));
                if (i == k) dout[k] = x[s].x;
                if (i == k + 1) alpha = x[s];
                const double t = fma(x[s].x, x[s].x, x[s].y * x[s].y);
                s2 += i > k + 1 ? t : 0.0;
            }
            alpha = cshfl(alpha, (k + 1) & 31);
            s2 = warp_sum(s2);
            // as k_hetrd_reg's reflector: beta = -sign(Re alpha) ||.||, H = I for a zero tail and a real alpha
            const bool id = s2 == 0.0 && alpha.y == 0.0;
            const double n2 = fma(alpha.x, alpha.x, fma(alpha.y, alpha.y, s2));
            const double rn = rsqrt(n2);
            double nrm = n2 * rn;
            nrm = fma(fma(-nrm, nrm, n2), 0.5 * rn, nrm);
            const double beta = alpha.x >= 0.0 ? -nrm : nrm, ib = alpha.x >= 0.0 ? -rn : rn;
            const double ar = alpha.x - beta, ai = alpha.y;
            const double rd = recip_nr(fma(ar, ar, ai * ai));
            const double2 scale = id ? zero : make_double2(ar * rd, -ai * rd);
            const double2 tk = id ? zero : make_double2((beta - alpha.x) * ib, -alpha.y * ib);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const int i = 32 * s + lane;
                const double2 v = i == k + 1 ? make_double2(1.0, 0.0) : cmul(x[s], scale);
                if (i > k && i < n) {
                    vb[i] = v;
                    ck[i] = v;
                }
            }
            if (lane == 0) {
                s_tk[k & 1] = tk;
                eout[k] = id ? alpha.x : beta;
                tout[k] = tk;
            }
        }
        __syncthreads();
        const double2 tk = s_tk[k & 1];
        const bool mv = tk.x != 0.0 || tk.y != 0.0;
        if (!upd && !mv) continue;                                // nothing to apply or form (uniform)
        // ---- the walk: the lane's rows of v_{k-1}, w and v_k in registers (zero where there are none)
        double2 acc[S], rp[S], rw[S], rv[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int i = 32 * s + lane;
            const bool live = i > k && i < n;
            acc[s] = zero;
            rp[s] = live && upd ? vp[i] : zero;
            rw[s] = live && upd ? wb[i] : zero;
            rv[s] = live && mv ? vb[i] : zero;
        }
        // one column, whose diagonal lies in chunk SJ: its update, its part of the row sums, its own sum.
        // Only that chunk and the last need masks, and there is no branch inside, so that the chunks'
        // loads and chains overlap (with masks everywhere three quarters of the instructions were selects).
        auto walk_from = [&](auto first, double2* cj, int j) {
            constexpr int SJ = decltype(first)::value;
            const double2 vj = vb[j], wj = wb[j], pj = vp[j];     // (w and v_{k-1} are zero in rp, rw without upd)
            double2 a[S];
#pragma unroll
            for (int s = SJ; s < S; ++s) {
                const int i = 32 * s + lane;
                if (s == SJ) a[s] = i >= j && i < n ? cj[i] : zero;
                else if (s == S - 1) a[s] = i < n ? cj[i] : zero;
                else a[s] = cj[i];
            }
#pragma unroll
            for (int s = SJ; s < S; ++s) a[s] = cfmsc(rw[s], pj, cfmsc(rp[s], wj, a[s]));
            double2 cs, cm;                                       // the two products of each part apart
            {
                const int i = 32 * SJ + lane;
                if (i == j) a[SJ].y = 0.0;
                if (i >= j && i < n) cj[i] = a[SJ];
                if (i < j) a[SJ] = zero;
                acc[SJ] = cfma(a[SJ], vj, acc[SJ]);
                if (i == j) a[SJ] = zero;
                cs = make_double2(a[SJ].x * rv[SJ].x, a[SJ].x * rv[SJ].y);
                cm = make_double2(a[SJ].y * rv[SJ].y, a[SJ].y * rv[SJ].x);
            }
#pragma unroll
            for (int s = SJ + 1; s < S; ++s) {
                const int i = 32 * s + lane;
                if (s < S - 1 || i < n) cj[i] = a[s];
                acc[s] = cfma(a[s], vj, acc[s]);
                cs.x = fma(a[s].x, rv[s].x, cs.x);
                cs.y = fma(a[s].x, rv[s].y, cs.y);
                cm.x = fma(a[s].y, rv[s].y, cm.x);
                cm.y = fma(a[s].y, rv[s].x, cm.y);
            }
            return make_double2(cs.x + cm.x, cs.y - cm.y);        // sum conj(a_ij) v_i, i > j
        };
        auto walk_at = [&](double2* cj, int j) {
            switch (j >> 5) {
                case 0: return walk_from(std::integral_constant<int, 0>{}, cj, j);
                case 1: return walk_from(std::integral_constant<int, 1>{}, cj, j);
                case 2: return walk_from(std::integral_constant<int, 2>{}, cj, j);
                case 3: return walk_from(std::integral_constant<int, 3>{}, cj, j);
                case 4: return walk_from(std::integral_constant<int, 4>{}, cj, j);
                case 5: if constexpr (S > 5) return walk_from(std::integral_constant<int, 5>{}, cj, j);
                case 6: if constexpr (S > 6) return walk_from(std::integral_constant<int, 6>{}, cj, j);
                default: return walk_from(std::integral_constant<int, S - 1>{}, cj, j);
            }
        };
        auto walk = [&](int j) { return j >= j0 ? walk_at(col_s(j), j) : walk_at(col_g(j), j); };
        const int m = n - k - 1, npair = (m + 1) >> 1;            // columns k+1+q and n-1-q
        for (int q = warp; q < npair; q += kTriWarps) {
            const int ja = k + 1 + q, jb = n - 1 - q;
            const double2 sa = walk(ja);
            const double2 sb = jb == ja ? zero : walk(jb);
            // both columns' sums over the warp: lanes 0 8 16 24 end with sa.x sa.y sb.x sb.y
            const bool hi = lane & 16, hj = lane & 8;
            double2 keep = hi ? sb : sa;
            const double2 send = hi ? sa : sb;
            keep.x += shfl_xor(send.x, 16);
            keep.y += shfl_xor(send.y, 16);
            double one = (hj ? keep.y : keep.x) + shfl_xor(hj ? keep.x : keep.y, 8);
#pragma unroll
            for (int h = 4; h >= 1; h >>= 1) one += shfl_xor(one, h);
            if ((lane & 7) == 0 && (!hi || jb != ja))
                reinterpret_cast<double*>(colp + (hi ? jb : ja))[hj ? 1 : 0] = one;
        }
        if (mv) {
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const int i = 32 * s + lane;
                if (i > k && i < n) prow[warp * n + i] = acc[s];
            }
        }
        __syncthreads();
        if (!mv) { upd = false; continue; }                       // H_k = I: nothing pending (uniform)
        // ---- p = tau A22 v, then w = p + a2 v, a2 = -|tau|^2 / 2 (v^H A22 v)
        double vav = 0.0;
        const int i = k + 1 + tid;                                // (m <= 255: one row per thread)
        double2 p = zero, vi = zero;
        if (i < n) {
            double2 sum = colp[i];
#pragma unroll
            for (int w8 = 0; w8 < kTriWarps; ++w8) sum = cadd(sum, prow[w8 * n + i]);
            vi = vb[i];
            vav = fma(vi.x, sum.x, vi.y * sum.y);
            p = cmul(tk, sum);
        }
        vav = warp_sum(vav);
        if (lane == 0) red[warp] = vav;
        __syncthreads();
        vav = 0.0;
#pragma unroll
        for (int w8 = 0; w8 < kTriWarps; ++w8) vav += red[w8];
        const double a2 = -0.5 * cabs2(tk) * vav;
        if (i < n) wb[i] = make_double2(fma(a2, vi.x, p.x), fma(a2, vi.y, p.y));
        __syncthreads();
        upd = true;
    }
    if (tid == 0) {
        double2 a = column(n - 1)[n - 1];
        if (upd) {                                                // step n-2's update of A(n-1, n-1)
            const double2* vl = vbuf + ((n - 2) & 1) * n;
            a = cfmsc(wb[n - 1], vl[n - 1], cfmsc(vl[n - 1], wb[n - 1], a));
        }
        dout[n - 1] = a.x;
        eout[n - 1] = 0.0;
        tout[n - 1] = zero;
    }
    double2* LVb = ws.LV + mat * b;
    for (int k = warp; k + 1 < n; k += kTriWarps) {               // reflector k along LV's column n-1-k
        const double2* ck = column(k);
        for (int i = k + 1 + lane; i < n; i += 32) LVb[(i - k - 1) + static_cast<size_t>(n - 1 - k) * n] = ck[i];
    }
}

template <int S>
cudaError_t run_hetrd_tri(int n, int batch, const double2* C, const Workspace& ws, const int* info,
                          cudaStream_t stream) {
    const size_t smem = TriSmem(n).total;
    if (smem > static_cast<size_t>(max_smem_optin())) return cudaErrorInvalidValue;
    static SmemOptIn f;
    set_smem_limit(reinterpret_cast<const void*>(k_hetrd_tri<S>), f, static_cast<int>(smem));
    k_hetrd_tri<S><<<batch, kTriThreads, smem, stream>>>(n, batch, C, ws, info);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_hetrd_tri(int n, int batch, const double2* C, const Workspace& ws, const int* info,
                             cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (n < 2 || n > kBigMaxN || !C || !info || !ws.LV || !ws.d || !ws.e || !ws.tau || !ws.log)
        return cudaErrorInvalidValue;
    const TriSmem L(n);
    if (static_cast<size_t>(ws.log_stride) < static_cast<size_t>(pk(L.j0, n))) return cudaErrorInvalidValue;
    switch ((n + 31) / 32) {
        case 5: return run_hetrd_tri<5>(n, batch, C, ws, info, stream);
        case 6: return run_hetrd_tri<6>(n, batch, C, ws, info, stream);
        case 7: return run_hetrd_tri<7>(n, batch, C, ws, info, stream);
        case 8: return run_hetrd_tri<8>(n, batch, C, ws, info, stream);
        default: return cudaErrorInvalidValue;
    }
}

size_t hetrd_tri_smem_bytes(int n) { return TriSmem(n).total; }

}  // namespace sbg
