// Two pieces of the eigensolve of the real symmetric tridiagonals T (d, e) that the Householder kernels
// leave in the workspace: the eigenvalues, and the orthonormalisation of close eigenvectors.  (The
// eigenvectors themselves come from k_tridiag_invit.)
//
// k_tridiag_values: bisection on Sturm counts (LAPACK dstebz's method).
//
// The implicit-QL recurrence is one dependent chain of ~1.2 n^2 rotations per pair, each ~200 cycles
// of FP64 latency; with one thread per pair it took 846 us for ANY batch up to ~19,000 pairs at
// n = 54 and 4.1 ms at n = 128.  Here every eigenvalue has a thread (two when n > 32, whose two
// recurrences overlap), and the dependent chain of one Sturm count is n FMAs.  The recurrence is the
// product form p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2} (no division: three FP64 operations and
// one broadcast load of (d_i, e_{i-1}^2) a row), rescaled by powers of two every eight rows; its
// count is exact for a T whose entries are perturbed by a few eps each, so the eigenvalues carry an
// error of a few eps ||T||, as QL's.  Once an eigenvalue is alone in its bracket, the recurrence's last
// value (the characteristic polynomial) places the next shift.  Kernel time, QL -> halving only -> now: 8 pairs of n = 54
// 846 -> 69 -> 46 us, 32,768 pairs 4.0 -> 1.95 -> 1.3 ms, 65,536 of n = 32 1.18 -> 1.2 -> 0.84 ms, 2,048 of n = 128
// 9.9 -> 0.65 -> 0.37 ms.  Issue-bound when the GPU is full (FP64, sign and load instructions in equal parts).
//
// k_tridiag_ortho: pairs with many eigenvalues closer than inverse iteration can keep orthogonal by
// itself (near a Goldstone point one huge eigenvalue makes all others a cluster) get their vectors Z
// from plain inverse iteration and are orthonormalised here, all at once, by the Newton-Schulz
// iteration for the polar factor, Z <- Z (3 I - Z^T Z) / 2 (the nearest orthonormal matrix; symmetric
// in the vectors, so none of them takes another's error).  Inverse iteration leaves
// z_i^T z_j ~ eps ||T|| / |lambda_i - lambda_j|, so the mixing moves each residual by a few eps ||T||
// only, and one step squares the defect: for gaps above 1e-7 ||T|| one step is enough.  Products on
// the FP64 tensor cores (mma.sync.m8n8k4.f64).  The rotation-log QL these pairs took before cost
// 17 of 29 ms per 4,096 pairs of n = 96.
#include "kernels.cuh"
#include "stages.cuh"
#include "tiles.cuh"

namespace sbg {

namespace {

constexpr int kRows = 8;                    // rows between two rescalings
constexpr double kPadD = 8.0;               // padding rows: d - x > 0, no sign change
// Floor of e^2 (T scaled to norm ~1): an exact zero would leave p at zero once x hits an eigenvalue
// of a leading block exactly; 1e-20 off the diagonal moves no eigenvalue by more than that.
constexpr double kMinE2 = 1e-40;

struct ValuesSmem {
    size_t de, lam, p, cnt, red, total;
    __host__ __device__ ValuesSmem(int n, int points) {
        const size_t rows = static_cast<size_t>((n + kRows - 1) / kRows * kRows);
        size_t o = 0;
        de = o;  o += 16 * rows;
        lam = o; o += 8 * ((static_cast<size_t>(n) + 1) & ~size_t(1));
        p = o;   o += 8 * static_cast<size_t>(points);
        cnt = o; o += 8 * static_cast<size_t>(points);
        red = o; o += 16 * 8;
        total = o;
    }
};

// Number of eigenvalues of T below x[s], s < NE, and det(T - x[s] I) up to sign and one common factor as
// p[s] 2^e[s].
template <int NE>
__device__ __forceinline__ void sturm(const double2* __restrict__ de, int rows, const double (&x)[NE], int (&cnt)[NE],
                                      double (&p)[NE], int (&e)[NE]) {
    double pm[NE];
#pragma unroll
    for (int s = 0; s < NE; ++s) { p[s] = 1.0; pm[s] = 0.0; cnt[s] = 0; e[s] = 0; }
    double2 next[kRows];
#pragma unroll
    for (int u = 0; u < kRows; ++u) next[u] = de[u];
    for (int i0 = 0; i0 < rows; i0 += kRows) {
        double2 r[kRows];
#pragma unroll
        for (int u = 0; u < kRows; ++u) r[u] = next[u];
        const int i1 = i0 + kRows < rows ? i0 + kRows : 0;        // the next block, in flight meanwhile
#pragma unroll
        for (int u = 0; u < kRows; ++u) next[u] = de[i1 + u];
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
#pragma unroll
            for (int s = 0; s < NE; ++s) {
                const double pn = fma(r[u].x - x[s], p[s], -(r[u].y * pm[s]));
                cnt[s] += static_cast<unsigned>(__double2hiint(pn) ^ __double2hiint(p[s])) >> 31;
                pm[s] = p[s];
                p[s] = pn;
            }
        }
#pragma unroll
        for (int s = 0; s < NE; ++s) {      // bring the larger of the two to [1, 2)
            const int ex = max(__double2hiint(p[s]) & 0x7ff00000, __double2hiint(pm[s]) & 0x7ff00000);
            const double f = __hiloint2double(0x7fe00000 - ex, 0);
            p[s] *= f;
            pm[s] *= f;
            e[s] += ex >> 20;
        }
    }
}

// One end of an eigenvalue's bracket: the shift, the count there, and det(T - x I) = p 2^e (none at the
// ends of the Gershgorin interval: p is NaN).
struct End {
    double x, p;
    int c, e;
};

// 2^k, for k clamped to the normal range.
__device__ __forceinline__ double pow2_clamped(int k) {
    return __hiloint2double((min(max(k, -1000), 1000) + 1023) << 20, 0);
}

// The sum of x over the CTA, in every thread (red: a slot per warp).
__device__ __forceinline__ double block_sum(double x, double* red) {
    x = warp_sum(x);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    x = 0.0;
    for (int w = 0; w < static_cast<int>(blockDim.x) >> 5; ++w) x += red[w];
    __syncthreads();
    return x;
}

// The FP64 Householder again, by this CTA, for a pair with a column whose squared norm left the normal range: one of
// norm below 1.5e-154 comes out of k_hetrd_reg and k_hetrd_tri as NaN, one above 3e153 can come out wrong.  LAPACK's zlarfg
// rescales such a column as it meets it; a test for it there, never true, made every step's chain longer (the
// kernel 3 % slower at n = 54, 10 % at 24 and 32, 20 % at 40), while here it is part of a norm that is
// formed anyway.  C (lower triangle) times a power of two, its largest entry in [1, 2), goes to S (n x n, full); a column
// that is below 2^-450 then is taken as zero.  zhetd2's steps, each a pass over S in L2: milliseconds at n = 128.
// v, w: n entries of shared memory each.  Loops stay rolled, for the registers of
// the kernel.  Nothing is written if C is not finite.
__device__ __noinline__ void hetrd_scaled(int n, const double2* C, double2* S, double2* v, double2* w, double* red,
                                          double* d, double* e, double2* tau, double2* LV, bool lv_cols) {
    const int tid = threadIdx.x, T = blockDim.x;
    int most = 0;                                                 // high word of the largest |part| of C's triangle
#pragma unroll 1
    for (int j = 0; j < n; ++j)
#pragma unroll 1
        for (int i = j + (tid & 31); i < n; i += 32) {            // (every warp all of it)
            const double2 z = C[i + static_cast<size_t>(j) * n];
            most = max(most, max(__double2hiint(z.x) & 0x7fffffff, i == j ? 0 : __double2hiint(z.y) & 0x7fffffff));
        }
    most = __reduce_max_sync(0xffffffffu, most);
    if (most >= 0x7ff00000) return;                               // uniform
    const int hi = min(max(0x7fe00000 - (most & 0x7ff00000), 0x00100000), 0x7fd00000);
    const double by = __hiloint2double(hi, 0), back = __hiloint2double(0x7fe00000 - hi, 0);
#pragma unroll 1
    for (int idx = tid; idx < n * n; idx += T) {
        const int j = idx / n, i = idx - j * n;
        double2 z = cscale(C[max(i, j) + static_cast<size_t>(min(i, j)) * n], by);
        if (i <= j) z.y = i < j ? -z.y : 0.0;
        S[idx] = z;
    }
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k + 1 < n; ++k) {
        const double2* ck = S + static_cast<size_t>(k) * n;
        const double2 alpha = ck[k + 1];
        double s2 = 0.0;
#pragma unroll 1
        for (int i = k + 2 + tid; i < n; i += T) s2 += cabs2(ck[i]);
        s2 = fma(alpha.y, alpha.y, block_sum(s2, red));
        const bool id = s2 <= 0x1p-900;                           // uniform
        const double nrm = sqrt(fma(alpha.x, alpha.x, s2)), beta = alpha.x >= 0.0 ? -nrm : nrm;
        const double ar = alpha.x - beta, den = fma(ar, ar, alpha.y * alpha.y);
        const double2 zero = make_double2(0.0, 0.0);
        const double2 tk = id ? zero : make_double2((beta - alpha.x) / beta, -alpha.y / beta);
        const double2 scale = id ? zero : make_double2(ar / den, -alpha.y / den);
        if (tid == 0) {
            d[k] = ck[k].x * back;
            e[k] = (id ? alpha.x : beta) * back;
            tau[k] = tk;
        }
#pragma unroll 1
        for (int i = k + 1 + tid; i < n; i += T) {
            v[i] = i == k + 1 ? make_double2(1.0, 0.0) : id ? zero : cmul(ck[i], scale);
            if (lv_cols) LV[(i - k - 1) + static_cast<size_t>(n - 1 - k) * n] = v[i];
            else LV[k + static_cast<size_t>(i) * n] = v[i];
        }
        __syncthreads();
        if (id) continue;
        // w = p + a2 v, p = tau A22 v, a2 = -|tau|^2 / 2 (v^H A22 v); then A22 -= v w^H + w v^H
        double vav = 0.0;
#pragma unroll 1
        for (int i = k + 1 + tid; i < n; i += T) {
            double2 sum = zero;
#pragma unroll 1
            for (int j = k + 1; j < n; ++j) sum = cfma(S[i + static_cast<size_t>(j) * n], v[j], sum);
            vav = fma(v[i].x, sum.x, fma(v[i].y, sum.y, vav));
            w[i] = cmul(tk, sum);
        }
        const double a2 = -0.5 * cabs2(tk) * block_sum(vav, red);
#pragma unroll 1
        for (int i = k + 1 + tid; i < n; i += T) w[i] = make_double2(fma(a2, v[i].x, w[i].x), fma(a2, v[i].y, w[i].y));
        __syncthreads();
#pragma unroll 1
        for (int i = k + 1 + tid; i < n; i += T)
#pragma unroll 1
            for (int j = k + 1; j < n; ++j) {
                double2 z = cfmsc(w[i], v[j], cfmsc(v[i], w[j], S[i + static_cast<size_t>(j) * n]));
                if (i == j) z.y = 0.0;
                S[i + static_cast<size_t>(j) * n] = z;
            }
        __syncthreads();
    }
    if (tid == 0) {
        d[n - 1] = S[static_cast<size_t>(n) * n - 1].x * back;
        e[n - 1] = 0.0;
        tau[n - 1] = make_double2(0.0, 0.0);
    }
    __syncthreads();
}

// One pair per CTA of ceil(n / (32 NE)) warps; thread t holds the eigenvalues of index t + T s.
// A T that is not finite, or so large that a reflector may have been wrong, is formed again from C (where there is
// one) by hetrd_scaled and goes through the QL recurrence (one thread), whose info code it gets.
// (At most 72 registers for NE = 1, one warp: hetrd_scaled alone would take 80, and 28 pairs fit an SM as 25.)
template <int NE>
__global__ void __launch_bounds__(NE == 1 ? 32 : 128, NE == 1 ? 28 : 4)
    k_tridiag_values(int n, int batch, Workspace ws, double* __restrict__ W, int* __restrict__ info,
                     const double2* __restrict__ C) {
    const int b = blockIdx.x;
    if (b >= batch || !pair_selected(ws, b)) return;
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int points = T * NE, rows = (n + kRows - 1) / kRows * kRows;
    const ValuesSmem lay(n, points);
    double2* de = reinterpret_cast<double2*>(smem + lay.de);
    double* lam = reinterpret_cast<double*>(smem + lay.lam);
    double* gp = reinterpret_cast<double*>(smem + lay.p);
    int2* cnt = reinterpret_cast<int2*>(smem + lay.cnt);
    double* red = reinterpret_cast<double*>(smem + lay.red);
    const double* dg = ws.d + static_cast<size_t>(n) * b;
    const double* eg = ws.e + static_cast<size_t>(n) * b;
    double* Wb = W + static_cast<size_t>(n) * b;
    if (info[b] != 0) {                                           // uniform
        for (int i = tid; i < n; i += T) Wb[i] = __longlong_as_double(0x7ff8000000000000ll);
        return;
    }
    // ---- norm, Gershgorin interval, any off-diagonal entry
    double amax = 0.0, gl = __longlong_as_double(0x7ff0000000000000ll), gu = -gl, esum = 0.0;
    bool finite = true;
    for (int i = tid; i < n; i += T) {
        const double di = dg[i], el = i > 0 ? fabs(eg[i - 1]) : 0.0, er = i + 1 < n ? fabs(eg[i]) : 0.0;
        finite = finite && isfinite(di) && isfinite(er);
        amax = fmax(amax, fmax(fabs(di), er));
        gl = fmin(gl, di - (el + er));
        gu = fmax(gu, di + (el + er));
        esum = fmax(esum, er);
    }
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
        amax = fmax(amax, shfl_xor(amax, m));
        gl = fmin(gl, shfl_xor(gl, m));
        gu = fmax(gu, shfl_xor(gu, m));
        esum = fmax(esum, shfl_xor(esum, m));
    }
    if (T > 32) {
        if (lane == 0) { red[4 * warp] = amax; red[4 * warp + 1] = gl; red[4 * warp + 2] = gu; red[4 * warp + 3] = esum; }
        finite = __syncthreads_and(finite);
        for (int w = 0; w < T / 32; ++w) {
            amax = fmax(amax, red[4 * w]);
            gl = fmin(gl, red[4 * w + 1]);
            gu = fmax(gu, red[4 * w + 2]);
            esum = fmax(esum, red[4 * w + 3]);
        }
    } else {
        finite = __all_sync(0xffffffffu, finite);
    }
    if (!finite || amax >= 0x1p508) {                             // uniform
        double* d = reinterpret_cast<double*>(smem + lay.de);     // 2 rows doubles: d, then e
        if (C) {
            const size_t nn = static_cast<size_t>(n) * n, at = static_cast<size_t>(n) * b;
            double2* v = reinterpret_cast<double2*>(smem);        // (de, lam, p, cnt: 40 n bytes)
            hetrd_scaled(n, C + nn * b, static_cast<double2*>(ws.log) + static_cast<size_t>(ws.log_stride) * b, v, v + n,
                         red, ws.d + at, ws.e + at, ws.tau + at, ws.LV + nn * b, n > kSmallMaxN);
        }
        double* e = d + rows;
        for (int i = tid; i < n; i += T) { d[i] = dg[i]; e[i] = eg[i]; }
        __syncthreads();
        if (tid == 0) {
            const int r = ql_chain<double, false>(n, d, e, 1, nullptr, 0, nullptr, Wb);
            if (r > 0) info[b] = r;
        }
        return;
    }
    if (!(esum > 0.0)) {                                          // T diagonal: its entries, sorted
        for (int i = tid; i < n; i += T) lam[i] = dg[i];
        __syncthreads();
        for (int i = tid; i < n; i += T) {
            int rank = 0;
            for (int j = 0; j < n; ++j) rank += (lam[j] < lam[i] || (lam[j] == lam[i] && j < i)) ? 1 : 0;
            Wb[rank] = lam[i];
        }
        return;
    }
    // ---- T scaled by a power of two to max-norm in [1/2, 1)
    const double us = pow2_norm(amax), sc = 1.0 / us;
    for (int i = tid; i < rows; i += T) {
        double2 r = make_double2(kPadD, 0.0);
        if (i < n) {
            const double e = i > 0 ? eg[i - 1] * sc : 0.0;
            r = make_double2(dg[i] * sc, i > 0 ? fmax(e * e, kMinE2) : 0.0);
        }
        de[i] = r;
    }
    gl = fmax(gl * sc, -6.0) - 1e-15;                             // (gl, gu may have overflowed)
    gu = fmin(gu * sc, 6.0) + 1e-15;
    const double w0 = (gu - gl) / (points + 1);
    __syncthreads();
    // ---- counts on a grid of `points` shifts bracket every eigenvalue to one cell
    double x[NE], px[NE];
    int c[NE], ex[NE];
#pragma unroll
    for (int s = 0; s < NE; ++s) x[s] = fma(static_cast<double>(tid * NE + s + 1), w0, gl);
    sturm<NE>(de, rows, x, c, px, ex);
#pragma unroll
    for (int s = 0; s < NE; ++s) {
        gp[tid * NE + s] = px[s];
        cnt[tid * NE + s] = make_int2(c[s], ex[s]);
    }
    __syncthreads();
    // ---- then every cell down to the spacing of the numbers at it (eps ||T|| and no less): halved while it
    // holds more than one eigenvalue, and else by the zero of the chord through det(T - x I) at its ends
    // (regula falsi with Anderson & Bjorck's reduction of an end that stays): 14 to 23 counts in all for the
    // slowest eigenvalue of a warp where halving takes 49.  The counts alone decide which end moves; a step
    // that is too close to an end is moved off it by that spacing, so that the other end follows, and a
    // cell that three steps did not halve is halved (two: 28 to 32 counts).  Where det(T - x I) nearly
    // vanishes at an end (another eigenvalue just outside the cell), every chord lands there and that end alone
    // creeps: the step after such a step halves (T = tridiag(1, h |i - c|, 1), n = 40 .. 128: 87 counts at most
    // instead of 151).  Any four steps halve a cell, whatever the chords do, and the widest grid cell (n <= 32,
    // 12 / 33 of the scaled norm) is 52 halvings from its last width: 208 steps, so the limit is never met.
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    End lo[NE], hi[NE];
    double wa[NE], wb[NE], wc[NE];                                // its width one, two and three steps ago
    int side[NE];
    bool open[NE];
#pragma unroll
    for (int s = 0; s < NE; ++s) {
        const int j = tid + s * T;
        int a = 0, z = points;                                    // first grid point with count > j
        while (a < z) {
            const int m = (a + z) >> 1;
            if (cnt[m].x > j) z = m; else a = m + 1;
        }
        lo[s] = a > 0 ? End{fma(static_cast<double>(a), w0, gl), gp[a - 1], cnt[a - 1].x, cnt[a - 1].y}
                      : End{gl, nan, 0, 0};
        hi[s] = a < points ? End{fma(static_cast<double>(a + 1), w0, gl), gp[a], cnt[a].x, cnt[a].y}
                           : End{gu, nan, n, 0};
        wa[s] = wb[s] = wc[s] = 4.0 * (hi[s].x - lo[s].x);
        side[s] = 0;
        open[s] = j < n;
    }
    for (int step = 0; step < 256; ++step) {
        bool any = false;
#pragma unroll
        for (int s = 0; s < NE; ++s) {
            const int j = tid + s * T;
            const double w = hi[s].x - lo[s].x, mid = lo[s].x + 0.5 * w;
            const double least = 1.1102230246251565e-16 * fmax(1.0, 2.0 * fabs(mid));
            double t = mid;
            if (lo[s].c == j && hi[s].c == j + 1 && w <= 0.5 * wc[s]) {
                const double r = fabs(lo[s].p) * pow2_clamped(lo[s].e - hi[s].e);
                const double q = fma(w, r / (r + fabs(hi[s].p)), lo[s].x);
                if (q == q) t = fmin(fmax(q, lo[s].x + least), hi[s].x - least);
            }
            open[s] = open[s] && w > least && t > lo[s].x && t < hi[s].x;
            wc[s] = wb[s];
            wb[s] = wa[s];
            wa[s] = w;
            x[s] = open[s] ? t : lo[s].x;
            any = any || open[s];
        }
        if (!__any_sync(0xffffffffu, any)) break;
        sturm<NE>(de, rows, x, c, px, ex);
#pragma unroll
        for (int s = 0; s < NE; ++s) {
            if (!open[s]) continue;
            const bool up = c[s] <= tid + s * T;
            End& moved = up ? lo[s] : hi[s];
            End& stays = up ? hi[s] : lo[s];
            const int way = up ? -1 : 1;
            // (its own end moved by less than 2^-51: about the spacing that a step is held off an end by)
            if ((__double2hiint(x[s] - moved.x) & 0x7fffffff) < (1023 - 51) << 20) wc[s] = 0.0;
            if (side[s] == way) {
                const double m = 1.0 - fabs(px[s] / moved.p) * pow2_clamped(ex[s] - moved.e);
                stays.p *= m > 0.0 ? m : 0.5;                     // (also where the end had no value)
            }
            moved = End{x[s], px[s], c[s], ex[s]};
            side[s] = way;
        }
    }
#pragma unroll
    for (int s = 0; s < NE; ++s) {
        const int j = tid + s * T;
        if (j < n) lam[j] = (lo[s].x + 0.5 * (hi[s].x - lo[s].x)) * us;
    }
    __syncthreads();
    // ---- ascending (close eigenvalues may come out swapped in their last bits)
    bool sorted = true;
    for (int j = tid; j + 1 < n; j += T) sorted = sorted && lam[j] <= lam[j + 1];
    sorted = T > 32 ? __syncthreads_and(sorted) : __all_sync(0xffffffffu, sorted);
    if (!sorted) {
        if (tid == 0)
            for (int j = 1; j < n; ++j) lam[j] = fmax(lam[j], lam[j - 1]);
        __syncthreads();
    }
    for (int j = tid; j < n; j += T) Wb[j] = lam[j];
}

// ----------------------------------------------------------------------------- k_tridiag_ortho
constexpr int kOrthoThreads = 128;          // 4 warps, each a 16 x 16 quarter of a 32 x 32 tile
constexpr int kOrthoLdA = 36;               // A(i, k) at k * 36 + i, B(k, j) at j * 20 + k: fragment loads of
constexpr int kOrthoLdB = 20;               // 8 bytes by lanes (g, t) are then free of bank conflicts
constexpr int kOrthoKP = 16;
static_assert(kOrthoLdA % 16 == 4 && kOrthoLdB % 16 == 4, "fragment strides");
constexpr int kOrthoSteps = 6;
constexpr double kOrthoMost = 0.3;          // a larger defect: vectors of one eigenspace, left to the QL

struct OrthoSmem {
    size_t rows, bs, red, total;
    // rows: a block of 32 rows of Z (all columns); the first product's A panel and the warp QL's Z tile share it
    __host__ __device__ explicit OrthoSmem(int n, bool with_ql) {
        const size_t nk = static_cast<size_t>((n + kOrthoKP - 1) / kOrthoKP * kOrthoKP);
        size_t r = 8 * kOrthoLdA * nk;
        const size_t ql = 8 * (static_cast<size_t>(n) * tile_ld(n) + 2 * static_cast<size_t>(n));
        if (with_ql && ql > r) r = ql;
        size_t o = 0;
        rows = o; o += (r + 15) & ~size_t(15);
        bs = o;   o += 8 * kOrthoLdB * 32;
        red = o;  o += 8 * 4;
        total = o;
    }
};

// acc += A(32 x 16) B(16 x 32) of two panels in shared memory, the warp's quarter.
__device__ __forceinline__ void panel_mma(double (&acc)[2][2][2], const double* as, const double* bs) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int wr = w >> 1, wc = w & 1;
#pragma unroll
    for (int k0 = 0; k0 < kOrthoKP; k0 += 4) {
        double a[2], b[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            a[h] = as[(k0 + t) * kOrthoLdA + 16 * wr + 8 * h + g];
            b[h] = bs[(16 * wc + 8 * h + g) * kOrthoLdB + k0 + t];
        }
#pragma unroll
        for (int br = 0; br < 2; ++br)
#pragma unroll
            for (int bc = 0; bc < 2; ++bc) dmma(acc[br][bc][0], acc[br][bc][1], a[br], b[bc]);
    }
}

// Pairs with ws.flag == kFlagOrtho only.  Z (n x n, column-major) is the first half of the pair's X slot,
// G = Z^T Z goes to the second.  A pair it cannot orthonormalise: with_ql, the warp QL here (n <= 63:
// Z in shared memory); otherwise ws.flag = kFlagRedo, for the rotation-log QL.
__global__ void __launch_bounds__(kOrthoThreads) k_tridiag_ortho(int n, int batch, Workspace ws,
                                                                 double* __restrict__ W, double2* __restrict__ X,
                                                                 int* __restrict__ info, int with_ql) {
    const int b = blockIdx.x;
    if (b >= batch || !pair_selected(ws, b)) return;
    if (ws.flag[b] != kFlagOrtho) return;                         // uniform
    extern __shared__ __align__(16) unsigned char smem[];
    const OrthoSmem lay(n, with_ql != 0);
    double* zr = reinterpret_cast<double*>(smem + lay.rows);
    double* bs = reinterpret_cast<double*>(smem + lay.bs);
    double* red = reinterpret_cast<double*>(smem + lay.red);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    const size_t nn = static_cast<size_t>(n) * n;
    double* Z = reinterpret_cast<double*>(X + nn * b);
    double* G = Z + nn;
    const int nk = (n + kOrthoKP - 1) / kOrthoKP * kOrthoKP;
    bool done = false;
    for (int step = 0; step < kOrthoSteps && !done; ++step) {
        // ---- G = Z^T Z: lower tiles, mirrored; the largest entry of |G - I|
        double off = 0.0;
        for (int i0 = 0; i0 < n; i0 += 32)
            for (int j0 = 0; j0 <= i0; j0 += 32) {
                double acc[2][2][2] = {};
                for (int k0 = 0; k0 < n; k0 += kOrthoKP) {
                    __syncthreads();
                    for (int e = tid; e < 32 * kOrthoKP; e += kOrthoThreads) {
                        const int k = e % kOrthoKP, c = e / kOrthoKP;
                        const bool row = k0 + k < n;
                        zr[k * kOrthoLdA + c] = row && i0 + c < n ? __ldcg(Z + static_cast<size_t>(i0 + c) * n + k0 + k) : 0.0;
                        bs[c * kOrthoLdB + k] = row && j0 + c < n ? __ldcg(Z + static_cast<size_t>(j0 + c) * n + k0 + k) : 0.0;
                    }
                    __syncthreads();
                    panel_mma(acc, zr, bs);
                }
#pragma unroll
                for (int br = 0; br < 2; ++br)
#pragma unroll
                    for (int bc = 0; bc < 2; ++bc)
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const int i = i0 + 16 * (w >> 1) + 8 * br + g, j = j0 + 16 * (w & 1) + 8 * bc + 2 * t + q;
                            if (i >= n || j >= n) continue;
                            const double v = acc[br][bc][q];
                            __stcg(G + i + static_cast<size_t>(j) * n, v);
                            if (i0 != j0) __stcg(G + j + static_cast<size_t>(i) * n, v);
                            const double d = fabs(v - (i == j ? 1.0 : 0.0));
                            off = d > off || !(d == d) ? d : off;             // (a NaN stays)
                        }
            }
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) {
            const double o = shfl_xor(off, m);
            off = o > off || !(o == o) ? o : off;
        }
        __syncthreads();
        if (lane == 0) red[w] = off;
        __syncthreads();
        for (int u = 0; u < 4; ++u) off = red[u] > off || !(red[u] == red[u]) ? red[u] : off;
        if (!(off <= kOrthoMost)) break;                          // uniform; also NaN
        if (off <= 1e-14) { done = true; break; }
        // ---- Z <- Z (3 I - G) / 2, a block of 32 rows at a time (in place: a block reads its own rows)
        for (int r0 = 0; r0 < n; r0 += 32) {
            __syncthreads();
            for (int e = tid; e < 32 * nk; e += kOrthoThreads) {
                const int r = e & 31, c = e >> 5;
                zr[c * kOrthoLdA + r] = r0 + r < n && c < n ? __ldcg(Z + static_cast<size_t>(c) * n + r0 + r) : 0.0;
            }
            for (int j0 = 0; j0 < n; j0 += 32) {
                double acc[2][2][2] = {};
                for (int k0 = 0; k0 < n; k0 += kOrthoKP) {
                    __syncthreads();
                    for (int e = tid; e < 32 * kOrthoKP; e += kOrthoThreads) {
                        const int k = e % kOrthoKP, c = e / kOrthoKP;
                        bs[c * kOrthoLdB + k] =
                            k0 + k < n && j0 + c < n ? __ldcg(G + static_cast<size_t>(j0 + c) * n + k0 + k) : 0.0;
                    }
                    __syncthreads();
                    panel_mma(acc, zr + k0 * kOrthoLdA, bs);
                }
#pragma unroll
                for (int br = 0; br < 2; ++br)
#pragma unroll
                    for (int bc = 0; bc < 2; ++bc)
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const int r = 16 * (w >> 1) + 8 * br + g, j = j0 + 16 * (w & 1) + 8 * bc + 2 * t + q;
                            if (r0 + r < n && j < n)
                                __stcg(Z + static_cast<size_t>(j) * n + r0 + r,
                                       fma(1.5, zr[j * kOrthoLdA + r], -0.5 * acc[br][bc][q]));
                        }
            }
        }
        __syncthreads();
        done = off * off * n <= 1e-15;                            // the next defect is below ||E||_2^2
    }
    if (done) return;
    if (!with_ql) {
        if (tid == 0) ws.flag[b] = kFlagRedo;
        return;
    }
    // ---- the warp QL, Z row-major in shared memory
    __syncthreads();
    if (w != 0) return;
    const int ldz = tile_ld(n);
    double* dd = zr + static_cast<size_t>(n) * ldz;
    double* ee = dd + n;
    for (int r = lane; r < n; r += 32)
        for (int c = 0; c < n; ++c) zr[r * ldz + c] = (r == c) ? 1.0 : 0.0;
    for (int i = lane; i < n; i += 32) {
        dd[i] = ws.d[static_cast<size_t>(n) * b + i];
        ee[i] = ws.e[static_cast<size_t>(n) * b + i];
    }
    __syncwarp();
    const int unconv = tridiag_ql<double>(n, dd, ee, zr, ldz);
    __syncwarp();
    for (int i = lane; i < n; i += 32) W[static_cast<size_t>(n) * b + i] = dd[i];
    for (int r = lane; r < n; r += 32)
        for (int k = 0; k < n; ++k) Z[r + static_cast<size_t>(k) * n] = zr[r * ldz + k];
    if (lane == 0) info[b] = unconv;
}

// ----------------------------------------------------------------------------- k_tridiag_tiny
// n <= kTridiagTinyMaxN: eigenvalues and eigenvectors by the warp QL, Z row-major in shared memory; one launch,
// where bisection, inverse iteration and k_tridiag_ortho are three that cost more than their work.  The
// eigensolve of 65,536 pairs, those three -> this, in us: n = 1 145 -> 41, 2 281 -> 76, 3 298 -> 154, 4 315 -> 240, 5
// 338 -> 344, 6 355 -> 463; of one pair 13 -> 6, 19 -> 8, 19 -> 10, 19 -> 14, 19 -> 18, 19 -> 23.
__global__ void __launch_bounds__(32) k_tridiag_tiny(int n, int batch, Workspace ws, double* __restrict__ W,
                                                     double2* __restrict__ X, int* __restrict__ info,
                                                     const double2* __restrict__ C) {
    const int b = blockIdx.x, lane = threadIdx.x;
    if (b >= batch || !pair_selected(ws, b)) return;
    __shared__ __align__(16) double2 vw[2 * kTridiagTinyMaxN];
    __shared__ double z[kTridiagTinyMaxN * (kTridiagTinyMaxN + 1)], d[kTridiagTinyMaxN], e[kTridiagTinyMaxN], red[1];
    const size_t nn = static_cast<size_t>(n) * n, at = static_cast<size_t>(n) * b;
    if (lane == 0) ws.flag[b] = kFlagDone;
    if (info[b] != 0) {                                           // uniform
        if (lane < n) W[at + lane] = __longlong_as_double(0x7ff8000000000000ll);
        return;
    }
    double x = lane < n ? ws.d[at + lane] : 0.0, y = lane + 1 < n ? ws.e[at + lane] : 0.0;
    if (C && __any_sync(0xffffffffu, !(fabs(x) < 0x1p508 && fabs(y) < 0x1p508))) {
        hetrd_scaled(n, C + nn * b, static_cast<double2*>(ws.log) + static_cast<size_t>(ws.log_stride) * b, vw, vw + n, red,
                     ws.d + at, ws.e + at, ws.tau + at, ws.LV + nn * b, false);
        x = lane < n ? ws.d[at + lane] : 0.0;
        y = lane + 1 < n ? ws.e[at + lane] : 0.0;
    }
    const int ld = n + 1;
    if (lane < n) {
        d[lane] = x;
        e[lane] = y;
        for (int c = 0; c < n; ++c) z[lane * ld + c] = lane == c ? 1.0 : 0.0;
    }
    __syncwarp();
    const int unconv = tridiag_ql<double>(n, d, e, z, ld);
    __syncwarp();
    if (lane < n) {
        double* Z = reinterpret_cast<double*>(X + nn * b);
        W[at + lane] = d[lane];
        for (int k = 0; k < n; ++k) Z[lane + k * n] = z[lane * ld + k];
    }
    if (lane == 0 && unconv) info[b] = unconv;
}

template <int NE>
cudaError_t run_values(int n, int batch, const Workspace& ws, double* W, int* info, const double2* C,
                       cudaStream_t stream) {
    const int T = 32 * ((n + 32 * NE - 1) / (32 * NE));
    k_tridiag_values<NE><<<batch, T, ValuesSmem(n, T * NE).total, stream>>>(n, batch, ws, W, info, C);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_tridiag_values(int n, int batch, const Workspace& ws, double* W, int* info, const double2* C,
                                  cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (n < 1 || n > kBigMaxN || !W || !info || !ws.d || !ws.e) return cudaErrorInvalidValue;
    if (C && (!ws.LV || !ws.tau || !ws.log || ws.log_stride < n * n)) return cudaErrorInvalidValue;
    return n <= 32 ? run_values<1>(n, batch, ws, W, info, C, stream) : run_values<2>(n, batch, ws, W, info, C, stream);
}

cudaError_t launch_tridiag_tiny(int n, int batch, const Workspace& ws, double* W, double2* X, int* info,
                                const double2* C, cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (n < 1 || n > kTridiagTinyMaxN || !W || !X || !info || !ws.d || !ws.e || !ws.flag) return cudaErrorInvalidValue;
    if (C && (!ws.LV || !ws.tau || !ws.log || ws.log_stride < n * n)) return cudaErrorInvalidValue;
    k_tridiag_tiny<<<batch, 32, 0, stream>>>(n, batch, ws, W, X, info, C);
    return cudaGetLastError();
}

cudaError_t launch_tridiag_ortho(int n, int batch, const Workspace& ws, double* W, double2* X, int* info,
                                 bool with_ql, cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (n < 1 || n > kBigMaxN || !W || !X || !info || !ws.d || !ws.e || !ws.flag) return cudaErrorInvalidValue;
    const size_t smem = OrthoSmem(n, with_ql).total;
    if (smem > static_cast<size_t>(max_smem_optin())) return cudaErrorInvalidValue;
    static SmemOptIn f;
    set_smem_limit(reinterpret_cast<const void*>(k_tridiag_ortho), f, max_smem_optin());
    k_tridiag_ortho<<<batch, kOrthoThreads, smem, stream>>>(n, batch, ws, W, X, info, with_ql ? 1 : 0);
    return cudaGetLastError();
}

size_t tridiag_values_smem_bytes(int n) {
    const int NE = n <= 32 ? 1 : 2;
    return ValuesSmem(n, 32 * ((n + 32 * NE - 1) / (32 * NE)) * NE).total;
}

size_t tridiag_ortho_smem_bytes(int n, bool with_ql) { return OrthoSmem(n, with_ql).total; }

}  // namespace sbg
