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
// error of a few eps ||T||, as QL's.  Whole solves, QL -> bisection (FP64 form): 8 pairs of n = 54
// 1,421 -> 628 us, 1,024 pairs 1,955 -> 944 us, 32,768 pairs 30.4 -> 28.3 ms; 2,048 pairs of n = 128
// 30.4 -> 21.1 ms; 65,536 pairs of n = 32, which fill the GPU with either, 12.64 -> 12.63 ms.
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

size_t tridiag_ortho_smem_bytes(int n, bool with_ql) { return OrthoSmem(n, with_ql).total; }

}  // namespace sbg
