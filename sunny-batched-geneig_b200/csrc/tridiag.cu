// Eigenvalues of the real symmetric tridiagonals T (d, e) that the Householder kernels leave in the
// workspace, by bisection on Sturm counts (LAPACK dstebz's method): k_tridiag_values.
//
// The implicit-QL recurrence is one dependent chain of ~1.2 n^2 rotations per pair, each ~200 cycles
// of FP64 latency; with one thread per pair it took 846 us for ANY batch up to ~19,000 pairs at
// n = 54 and 4.1 ms at n = 128.  Here every eigenvalue has a thread (two when n > 32, whose two
// recurrences overlap), and the dependent chain of one Sturm count is n FMAs.  The recurrence is the
// product form p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2} (no division: three FP64 operations and
// one broadcast load of (d_i, e_{i-1}^2) a row), rescaled by powers of two every eight rows; its
// count is exact for a T whose entries are perturbed by a few eps each, so the eigenvalues carry an
// error of a few eps ||T||, as QL's.  Whole solves, QL -> bisection (FP64 form): 8 pairs of n = 54
// 1,421 -> 628 us, 1,024 pairs 1,955 -> 944 us, 32,768 pairs 30.4 -> 28.3 ms; 2,048 pairs of n = 128
// 30.4 -> 21.1 ms; 65,536 pairs of n = 32, which fill the GPU with either, 12.64 -> 12.63 ms.
#include "kernels.cuh"
#include "stages.cuh"

namespace sbg {

namespace {

constexpr int kRows = 8;                    // rows between two rescalings
constexpr double kPadD = 8.0;               // padding rows: d - x > 0, no sign change
// Floor of e^2 (T scaled to norm ~1): an exact zero would leave p at zero once x hits an eigenvalue
// of a leading block exactly; 1e-20 off the diagonal moves no eigenvalue by more than that.
constexpr double kMinE2 = 1e-40;

struct ValuesSmem {
    size_t de, lam, cnt, ql, red, total;
    __host__ __device__ ValuesSmem(int n, int points) {
        const size_t rows = static_cast<size_t>((n + kRows - 1) / kRows * kRows);
        size_t o = 0;
        de = o;  o += 16 * rows;
        lam = o; o += 8 * ((static_cast<size_t>(n) + 1) & ~size_t(1));
        cnt = o; o += 4 * static_cast<size_t>(points);
        red = o; o += 16 * 8;
        total = o;
    }
};

// Number of eigenvalues of T below x[s], s < NE.
template <int NE>
__device__ __forceinline__ void sturm(const double2* __restrict__ de, int rows, const double (&x)[NE], int (&cnt)[NE]) {
    double p[NE], pm[NE];
#pragma unroll
    for (int s = 0; s < NE; ++s) { p[s] = 1.0; pm[s] = 0.0; cnt[s] = 0; }
    for (int i0 = 0; i0 < rows; i0 += kRows) {
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            const double2 r = de[i0 + u];
#pragma unroll
            for (int s = 0; s < NE; ++s) {
                const double pn = fma(r.x - x[s], p[s], -(r.y * pm[s]));
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
        }
    }
}

// One pair per CTA of ceil(n / (32 NE)) warps; thread t holds the eigenvalues of index t + T s.
// A T that is not finite goes through the QL recurrence (one thread), whose info code it gets.
template <int NE>
__global__ void __launch_bounds__(128) k_tridiag_values(int n, int batch, Workspace ws, double* __restrict__ W,
                                                        int* __restrict__ info) {
    const int b = blockIdx.x;
    if (b >= batch || !pair_selected(ws, b)) return;
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int points = T * NE, rows = (n + kRows - 1) / kRows * kRows;
    const ValuesSmem lay(n, points);
    double2* de = reinterpret_cast<double2*>(smem + lay.de);
    double* lam = reinterpret_cast<double*>(smem + lay.lam);
    int* cnt = reinterpret_cast<int*>(smem + lay.cnt);
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
    if (!finite) {                                                // uniform
        double* d = reinterpret_cast<double*>(smem + lay.de);     // 2 rows doubles: d, then e
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
    double x[NE];
    int c[NE];
#pragma unroll
    for (int s = 0; s < NE; ++s) x[s] = fma(static_cast<double>(tid * NE + s + 1), w0, gl);
    sturm<NE>(de, rows, x, c);
#pragma unroll
    for (int s = 0; s < NE; ++s) cnt[tid * NE + s] = c[s];
    __syncthreads();
    double lo[NE];
#pragma unroll
    for (int s = 0; s < NE; ++s) {
        const int j = tid + s * T;
        int a = 0, z = points;                                    // first grid point with count > j
        while (a < z) {
            const int m = (a + z) >> 1;
            if (cnt[m] > j) z = m; else a = m + 1;
        }
        lo[s] = fma(static_cast<double>(a), w0, gl);
    }
    // ---- halve every cell to below eps ||T|| / 2 (the same number of steps for all)
    double w = w0;
    while (w > 1.1102230246251565e-16) {
        w *= 0.5;
#pragma unroll
        for (int s = 0; s < NE; ++s) x[s] = lo[s] + w;
        sturm<NE>(de, rows, x, c);
#pragma unroll
        for (int s = 0; s < NE; ++s)
            if (c[s] <= tid + s * T) lo[s] = x[s];
    }
#pragma unroll
    for (int s = 0; s < NE; ++s) {
        const int j = tid + s * T;
        if (j < n) lam[j] = (lo[s] + 0.5 * w) * us;
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

template <int NE>
cudaError_t run_values(int n, int batch, const Workspace& ws, double* W, int* info, cudaStream_t stream) {
    const int T = 32 * ((n + 32 * NE - 1) / (32 * NE));
    k_tridiag_values<NE><<<batch, T, ValuesSmem(n, T * NE).total, stream>>>(n, batch, ws, W, info);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_tridiag_values(int n, int batch, const Workspace& ws, double* W, int* info, cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (n < 1 || n > kBigMaxN || !W || !info || !ws.d || !ws.e) return cudaErrorInvalidValue;
    return n <= 32 ? run_values<1>(n, batch, ws, W, info, stream) : run_values<2>(n, batch, ws, W, info, stream);
}

}  // namespace sbg
