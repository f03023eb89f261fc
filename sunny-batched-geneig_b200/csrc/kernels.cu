// Stage kernels of the batched generalized eigensolve for n <= 84, and the launchers
// that route larger n to the cluster kernels of bigsolve.cu.
//
//   reduce   k_reduce_dmma (reduce_dmma.cu): B = L L^H and C = L^{-1} A L^{-H}; L into the
//            workspace, C into the caller's X buffer.
//   hetrd    k_hetrd_reg (hetrd_reg.cu): Householder tridiagonalisation of C, reflectors and
//            (d, e, tau) into the workspace; the mixed form (n <= 63) runs it in
//            complex64.
//   eig      k_tridiag_values (tridiag.cu: bisection on Sturm counts), k_tridiag_invit
//            (eigenvectors by inverse iteration, one warp per pair) and k_tridiag_ortho
//            (tridiag.cu: pairs with large clusters); k_ql_chain + k_ql_apply_rows (n > 63) or a
//            warp QL inside those kernels for the pairs they cannot take; n <= 4 k_tridiag_tiny, the
//            warp QL alone.  The mixed form refines
//            Y = Q Z against C afterwards (refine.cu).
//   back     k_back_dmma (back_dmma.cu): X = L^{-H} Q Z, written over Z (the mixed form:
//            Y = Q Z, then X = L^{-H} Y after the refinement).
//
// Every stage gives a pair one warp or one CTA.  The redo QL's recurrence is a dependent scalar chain per
// pair, so it runs a thread per pair.
#include "kernels.cuh"
#include "stages.cuh"

#include <algorithm>
#include <cstdlib>
#include <atomic>
#include <mutex>

namespace sbg {

namespace {

__host__ __device__ inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// ----------------------------------------------------------------------------- k_ql_chain
// The rotation-log QL's first half, for the pairs flagged kFlagRedo only (they keep the flag, or get 3
// on a log overflow): one THREAD per pair, the scalar QL recurrence with (d, e) in shared memory
// interleaved over the CTA, rotations appended to the pair's log.
__global__ void k_ql_chain(int n, int batch, Workspace ws, double* __restrict__ W, int* __restrict__ info) {
    const int tid = threadIdx.x, T = blockDim.x;
    const int b = blockIdx.x * T + tid;
    extern __shared__ __align__(16) unsigned char smem[];
    double* d = reinterpret_cast<double*>(smem) + tid;
    double* e = reinterpret_cast<double*>(smem) + static_cast<size_t>(n) * T + tid;
    if (b >= batch || !pair_selected(ws, b)) return;
    if (ws.flag[b] != kFlagRedo) return;
    if (info[b] > 0 && info[b] <= n) info[b] = 0;              // QL non-convergence: run it again here
    double* Wb = W + static_cast<size_t>(n) * b;
    double2* log = reinterpret_cast<double2*>(ws.log) + static_cast<size_t>(ws.log_cap) * b;
    if (info[b] != 0) {
        for (int i = 0; i < n; ++i) Wb[i] = __longlong_as_double(0x7ff8000000000000ll);
        log[0] = make_double2(-1.0, 0.0);
        return;
    }
    for (int i = 0; i < n; ++i) {
        d[i * T] = ws.d[static_cast<size_t>(n) * b + i];
        e[i * T] = ws.e[static_cast<size_t>(n) * b + i];
    }
    const int r = ql_chain<double>(n, d, e, T, log, ws.log_cap, ws.perm + static_cast<size_t>(n) * b, Wb);
    if (r < 0) ws.flag[b] = 3;
    else if (r > 0) info[b] = r;
}

// ----------------------------------------------------------------------------- k_tridiag_invit
// Eigenvectors of the tridiagonal T (d, e) from its FP64 eigenvalues (k_tridiag_values) by inverse
// iteration, one warp per pair, one lane per eigenvector at a time (LAPACK dstein's method):
// T - lambda_j I = L U without pivoting, a pivot below eps ||T|| replaced by that size, two
// solves, each followed by normalisation.  That is O(n) work
// per vector against the O(n^2) of applying every QL rotation to it.  Vectors of
// eigenvalues closer than kInvitOrtol ||T|| (a cluster) are then orthogonalised in order (Gram-Schmidt);
// where two of them overlap too much for that, the cluster's members are computed again, one lane per
// member, with three solves each orthogonalised against the cluster's earlier vectors.  The other
// vectors' orthogonality is ~eps ||T|| / gap.  A pair with a
// cluster of more than kInvitMaxCluster eigenvalues (a spectrum dominated by one huge eigenvalue) or
// more cluster members than lanes gets every vector as if it stood alone, and k_tridiag_ortho
// orthonormalises them.  Every vector must pass ||T z - lambda z|| <= kInvitTol ||T||; a pair with a
// failed vector or a T that is not finite is recomputed by the QL instead.
// Bound by the latency of the lanes' recurrences with the pairs that the lane scratch leaves room for (8 per
// SM at n = 54; FP64 pipe 13 % busy).  32,768 pairs at n = 54: 1.95 -> 1.12 ms with the backward-only first solve,
// the lane count below, running pointers, and cluster members in the main batches instead of three rounds of
// their own for one close pair of eigenvalues in a spectrum.
// Per-lane scratch (1/u and the vector) is interleaved [i * ld + lane]: lane-parallel
// recurrences read consecutive words, and the warp's column-by-column copy to the caller's X
// buffer (Z, column k = vector k) reads it across lanes without bank conflicts.
constexpr double kInvitOrtol = 3e-4;
constexpr int kInvitMaxCluster = 8;
constexpr double kInvitTol = 256.0 * 1.1102230246251565e-16;
// Vectors (lanes) at a time, the same for every batch, and the odd stride of the lane scratch
// [i * ld + lane], which both the lanes' recurrences and the reads across lanes take without conflicts:
// 27 and 27 at n = 54 instead of 32 and 33, 22 % less scratch and two more pairs per SM.
__host__ __device__ constexpr int invit_lanes(int n) { return (n + (n + 31) / 32 - 1) / ((n + 31) / 32); }
__host__ __device__ constexpr int invit_ld(int n) { return invit_lanes(n) | 1; }

struct InvitSmem {
    size_t scr, dd, ee, lam, cls, mem, flag, per_warp;
    // with_tile: the scratch also holds the in-kernel fallback QL's Z tile
    __host__ __device__ explicit InvitSmem(int n, bool with_tile = true) {
        size_t o = 0;
        const size_t lanes = 2 * static_cast<size_t>(invit_ld(n)) * n, tile = static_cast<size_t>(n) * tile_ld(n);
        scr = o;  o += 8 * (with_tile && tile > lanes ? tile : lanes);
        dd = o;   o += 8 * static_cast<size_t>(n);
        ee = o;   o += 8 * static_cast<size_t>(n);
        lam = o;  o += 8 * static_cast<size_t>(n);
        cls = o;  o += align_up(4 * static_cast<size_t>(n), 16);
        mem = o;  o += 4 * 32;
        flag = o; o += 16;
        per_warp = o;
    }
};

__device__ __forceinline__ double invit_start(int j, int i) {
    unsigned h = static_cast<unsigned>(i + 1) * 0x9E3779B1u ^ static_cast<unsigned>(j + 1) * 0x85EBCA77u;
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 12;
    return static_cast<double>(h & 0xFFFFFu) * (2.0 / 1048575.0) - 1.0;
}

// Per-lane pieces of inverse iteration on T - lam I; iu and z are the lane's columns of the interleaved
// scratch (element i at i * ld).  Operands are loaded a step ahead, so each dependent chain is only the
// recurrence itself.
// T - lam I = L U without pivoting (pivots below `tiny` raised to it): keeps 1/u_i.
__device__ __forceinline__ void invit_factor(int n, int ld, double lam, const double* __restrict__ dd,
                                             const double* __restrict__ ee, double tiny, double* __restrict__ iu) {
    double u = dd[0] - lam;
    if (fabs(u) < tiny) u = copysign(tiny, u);
    double r = recip_nr(u);
    *iu = r;
    double dn = n > 1 ? dd[1] - lam : 0.0, en = n > 1 ? ee[0] * ee[0] : 0.0;
    for (int i = 1; i < n; ++i) {
        const double di = dn, e2 = en;
        if (i + 1 < n) { dn = dd[i + 1] - lam; en = ee[i] * ee[i]; }
        u = fma(-e2, r, di);
        if (fabs(u) < tiny) u = copysign(tiny, u);
        r = recip_nr(u);
        iu += ld;
        *iu = r;
    }
}
// z <- U^{-1} y, y in z (ONES: y = 1, whatever z holds); returns ||z||^2.
template <bool ONES>
__device__ __forceinline__ double invit_back(int n, int ld, const double* __restrict__ ee, const double* __restrict__ iu,
                                             double* __restrict__ z) {
    z += static_cast<size_t>(n - 1) * ld;
    iu += static_cast<size_t>(n - 1) * ld;
    double zn = (ONES ? 1.0 : *z) * *iu;                   // U z = y  (U(i, i+1) = e_i)
    *z = zn;
    double s2 = zn * zn;
    double yp = 1.0, ep = 0.0, ip = 0.0;
    if (n > 1) {
        if (!ONES) yp = z[-ld];
        ep = ee[n - 2];
        ip = iu[-ld];
    }
    for (int i = n - 2; i >= 0; --i) {
        z -= ld;
        iu -= ld;
        const double yi = yp, ei = ep, ii = ip;
        if (i > 0) { if (!ONES) yp = z[-ld]; ep = ee[i - 1]; ip = iu[-ld]; }
        zn = fma(-ei, zn, yi) * ii;
        *z = zn;
        s2 = fma(zn, zn, s2);
    }
    return s2;
}
// z <- (T - lam I)^{-1} x with the factors above, x = sc z, or (GEN) the start vector of eigenvalue
// j; returns ||z||^2 (summed in the backward pass).
template <bool GEN>
__device__ __forceinline__ double invit_solve(int n, int ld, const double* __restrict__ ee,
                                              const double* __restrict__ iu, double* __restrict__ z, double sc, int j) {
    double* zi = z;
    const double* ui = iu;
    double y = GEN ? invit_start(j, 0) : sc * *zi;
    *zi = y;
    double xn = 0.0, cn = 0.0;
    if (n > 1) { xn = GEN ? invit_start(j, 1) : sc * zi[ld]; cn = ee[0] * *ui; }
    for (int i = 1; i < n; ++i) {                      // L y = x  (L(i, i-1) = e_{i-1} / u_{i-1})
        zi += ld;
        ui += ld;
        const double x = xn, c = cn;
        if (i + 1 < n) { xn = GEN ? invit_start(j, i + 1) : sc * zi[ld]; cn = ee[i] * *ui; }
        y = fma(-c, y, x);
        *zi = y;
    }
    return invit_back<false>(n, ld, ee, iu, z);
}
// z <- sc z in place; returns ||T z - lam z||^2 of the scaled vector (one pass).
__device__ __forceinline__ double invit_scale_residual(int n, int ld, double lam, const double* __restrict__ dd,
                                                       const double* __restrict__ ee, double* __restrict__ z,
                                                       double sc) {
    double zp = 0.0, zc = *z, r2 = 0.0, el = 0.0;
    for (int i = 0; i < n; ++i) {
        const double zx = i + 1 < n ? z[ld] : 0.0, er = i + 1 < n ? ee[i] : 0.0;
        const double v = fma(er, zx, fma(el, zp, (dd[i] - lam) * zc));
        r2 = fma(v, v, r2);
        *z = zc * sc;
        z += ld;
        zp = zc;
        zc = zx;
        el = er;
    }
    return r2 * sc * sc;
}

// flag_redo: a pair the kernel cannot take gets ws.flag = 2 and no output (the rotation-log QL is
// then run for the flagged pairs); otherwise the warp QL runs here, on a Z tile in the scratch.
__global__ void __launch_bounds__(32) k_tridiag_invit(int n, int batch, Workspace ws, double* __restrict__ W,
                                                      double2* __restrict__ X, int* __restrict__ info,
                                                      int flag_redo) {
    const int b = blockIdx.x, lane = threadIdx.x & 31;
    if (b >= batch || !pair_selected(ws, b)) return;
    if (lane == 0) ws.flag[b] = kFlagDone;
    const int inf = info[b];
    if (inf > n || inf < 0) return;                   // an earlier stage failed: W and X are NaN
    extern __shared__ __align__(16) unsigned char smem[];
    const InvitSmem lay(n, !flag_redo);
    double* scr = reinterpret_cast<double*>(smem + lay.scr);
    double* dd = reinterpret_cast<double*>(smem + lay.dd);
    double* ee = reinterpret_cast<double*>(smem + lay.ee);
    double* lam = reinterpret_cast<double*>(smem + lay.lam);
    int* cls = reinterpret_cast<int*>(smem + lay.cls);
    int* members = reinterpret_cast<int*>(smem + lay.mem);
    int* sflag = reinterpret_cast<int*>(smem + lay.flag);
    double* Wb = W + static_cast<size_t>(n) * b;
    double* Zg = reinterpret_cast<double*>(X + static_cast<size_t>(n) * n * b);
    double rs = 0.0;
    for (int i = lane; i < n; i += 32) {
        dd[i] = ws.d[static_cast<size_t>(n) * b + i];
        ee[i] = ws.e[static_cast<size_t>(n) * b + i];
        lam[i] = Wb[i];
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
        double v = fabs(dd[i]);
        if (i > 0) v += fabs(ee[i - 1]);
        if (i + 1 < n) v += fabs(ee[i]);
        rs = fmax(rs, v);
    }
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) rs = fmax(rs, shfl_xor(rs, m));
    const double tnorm = rs > 0.0 && isfinite(rs) ? rs : 1.0;
    const double tiny = 1.1102230246251565e-16 * tnorm;
    if (lane == 0) {                                  // clusters: cls[j] = index of the first member
        int start = 0, biggest = 1, cnt = 0;
        for (int j = 0; j < n; ++j) {
            if (j > 0 && !(lam[j] - lam[j - 1] <= kInvitOrtol * tnorm)) start = j;
            cls[j] = start;
            biggest = max(biggest, j - start + 1);
            if (start != j) { if (cnt < 32) members[cnt] = j; ++cnt; }
        }
        sflag[0] = biggest;
        sflag[1] = cnt;
    }
    __syncwarp();
    const int cnt = sflag[1], nl = invit_lanes(n), ld = invit_ld(n);
    bool fallback = inf != 0;
    const bool together = sflag[0] > kInvitMaxCluster || cnt > nl;    // all vectors here, then k_tridiag_ortho
    if (!fallback) {
        bool ok = true;
        double* invu = scr;
        double* zs = scr + ld * n;
        double *iu = invu + lane, *z = zs + lane;     // (lanes >= nl have no column and never touch them)
        // (1) every vector as if it stood alone: factor, two solves, residual test; nl at a time, then
        // copied out column by column.  The first solve starts from L 1, so that only its backward half is
        // left (EISPACK tinvit's start); for k_tridiag_ortho from a pseudo-random vector of its own
        // (L times one saves its forward half too, but the vectors come out closer to one another: n = 96 with
        // a dominating eigenvalue, k_tridiag_ortho 833 -> 915 us against 629 -> 581 us here).
        for (int base = 0; base < n; base += nl) {
            const int j = base + lane;
            if (lane < nl && j < n) {
                invit_factor(n, ld, lam[j], dd, ee, tiny, iu);
                double s2 = together ? invit_solve<true>(n, ld, ee, iu, z, 1.0, j) : invit_back<true>(n, ld, ee, iu, z);
                const bool f1 = s2 > 0.0 && isfinite(s2);
                s2 = invit_solve<false>(n, ld, ee, iu, z, f1 ? 1.0 / sqrt(s2) : 1.0, j);
                const bool f2 = s2 > 0.0 && isfinite(s2);
                const double r2 = invit_scale_residual(n, ld, lam[j], dd, ee, z, f2 ? 1.0 / sqrt(s2) : 1.0);
                ok &= f1 && f2 && sqrt(r2) <= kInvitTol * tnorm;
            }
            __syncwarp();
            const int top = min(nl, n - base);
            for (int L = 0; L < top; ++L) {
                const int jj = base + L;
                double* zc = Zg + static_cast<size_t>(jj) * n;
                for (int i = lane; i < n; i += 32) zc[i] = zs[i * ld + L];
            }
            __syncwarp();
        }
        ok = __all_sync(0xffffffffu, ok);              // from here on `ok` is the same on every lane
        // (2) cluster members, in index order: Gram-Schmidt against the cluster's earlier vectors.  Vectors
        // of eigenvalues a gap apart overlap by eps ||T|| / gap only, and taking that out moves the residual
        // by eps ||T||; if an overlap is larger than 1e-6, the eigenvalues are too close for vectors
        // computed alone and (3) computes the members again.  (Each lane reads and writes its own rows.)
        bool again = false;
        if (ok && !together) {
            for (int m = 0; m < cnt && !again; ++m) {
                const int j = members[m];
                double* zj = Zg + static_cast<size_t>(j) * n;
                for (int q = cls[j]; q < j && !again; ++q) {
                    const double* zq = Zg + static_cast<size_t>(q) * n;
                    double c = 0.0;
                    for (int i = lane; i < n; i += 32) c = fma(zq[i], zj[i], c);
                    c = warp_sum(c);
                    again = !(fabs(c) <= 1e-6);                   // uniform
                    for (int i = lane; i < n; i += 32) zj[i] = fma(-c, zq[i], zj[i]);
                }
                double s2 = 0.0;
                for (int i = lane; i < n; i += 32) s2 = fma(zj[i], zj[i], s2);
                const double inv = 1.0 / sqrt(warp_sum(s2));
                for (int i = lane; i < n; i += 32) zj[i] *= inv;
            }
        }
        // (3) such clusters' members, one lane each, all at once: three rounds of a solve
        // (every lane its own member) and modified Gram-Schmidt in index order (the whole warp,
        // lanes over rows) against the cluster's first vector and its earlier members
        if (again) {
            const int jm = lane < cnt ? members[lane] : -1;
            if (jm >= 0) {
                invit_factor(n, ld, lam[jm], dd, ee, tiny, iu);
            }
            for (int it = 0; it < 3 && ok; ++it) {        // each round's input is unit (Gram-Schmidt below)
                if (jm >= 0) {
                    if (it == 0) invit_solve<true>(n, ld, ee, iu, z, 1.0, jm);
                    else invit_solve<false>(n, ld, ee, iu, z, 1.0, jm);
                }
                __syncwarp();
                for (int m = 0; m < cnt && ok; ++m) {
                    const int j = members[m], s0 = cls[j];
                    const double* q0 = Zg + static_cast<size_t>(s0) * n;
                    double c = 0.0;
                    for (int i = lane; i < n; i += 32) c = fma(q0[i], zs[i * ld + m], c);
                    c = warp_sum(c);
                    for (int i = lane; i < n; i += 32) zs[i * ld + m] = fma(-c, q0[i], zs[i * ld + m]);
                    for (int m2 = 0; m2 < m; ++m2) {
                        if (cls[members[m2]] != s0) continue;     // uniform
                        double c2 = 0.0;
                        for (int i = lane; i < n; i += 32) c2 = fma(zs[i * ld + m2], zs[i * ld + m], c2);
                        c2 = warp_sum(c2);
                        for (int i = lane; i < n; i += 32)
                            zs[i * ld + m] = fma(-c2, zs[i * ld + m2], zs[i * ld + m]);
                    }
                    double s2 = 0.0;
                    for (int i = lane; i < n; i += 32) s2 = fma(zs[i * ld + m], zs[i * ld + m], s2);
                    s2 = warp_sum(s2);
                    if (!(s2 > 0.0) || !isfinite(s2)) { ok = false; break; }     // uniform
                    const double inv = 1.0 / sqrt(s2);
                    for (int i = lane; i < n; i += 32) zs[i * ld + m] *= inv;
                }
                __syncwarp();
            }
            if (jm >= 0 && ok) ok &= sqrt(invit_scale_residual(n, ld, lam[jm], dd, ee, z, 1.0)) <= kInvitTol * tnorm;
            for (int m = 0; m < cnt; ++m) {
                double* zc = Zg + static_cast<size_t>(members[m]) * n;
                for (int i = lane; i < n; i += 32) zc[i] = zs[i * ld + m];
            }
        }
        fallback = !__all_sync(0xffffffffu, ok);
    }
    if (!fallback && together && lane == 0) ws.flag[b] = kFlagOrtho;
    if (fallback && flag_redo) {
        if (lane == 0) ws.flag[b] = kFlagRedo;
        return;
    }
    if (fallback) {                                   // the warp QL, Z tile over the lane scratch
        const int ldz = tile_ld(n);
        __syncwarp();
        for (int r = lane; r < n; r += 32)
            for (int c = 0; c < n; ++c) scr[r * ldz + c] = (r == c) ? 1.0 : 0.0;
        for (int i = lane; i < n; i += 32) {
            dd[i] = ws.d[static_cast<size_t>(n) * b + i];
            ee[i] = ws.e[static_cast<size_t>(n) * b + i];
        }
        __syncwarp();
        const int unconv = tridiag_ql<double>(n, dd, ee, scr, ldz);
        __syncwarp();
        for (int i = lane; i < n; i += 32) Wb[i] = dd[i];
        for (int r = lane; r < n; r += 32)
            for (int k = 0; k < n; ++k) Zg[r + static_cast<size_t>(k) * n] = scr[r * ldz + k];
        if (lane == 0) info[b] = unconv;
    }
}

template <class K>
void set_max_smem_once(K kernel, SmemOptIn& rec) {
    set_smem_limit(reinterpret_cast<const void*>(kernel), rec, max_smem_optin());
}

}  // namespace

// ============================================================================== host side

int ql_log_capacity(int n) {
    const int dflt = (3 * n * n) / 2 + 8 * n + 16;
    if (const char* v = std::getenv("SBG_QL_LOG_CAPACITY")) {
        const int c = std::atoi(v);
        if (c >= 16 && c < dflt) return c;
    }
    return dflt;
}

size_t workspace_bytes_per_pair(int n, bool mixed) {
    const size_t nn = static_cast<size_t>(n) * n;
    // the default (largest) rotation-log capacity, or the mixed form's stash if that is larger
    const size_t cap = static_cast<size_t>(std::max((3 * n * n) / 2 + 8 * n + 16, refine_stash_entries(n)));
    const size_t refine = mixed_big(n, mixed) ? 5 * 16 * nn + 4 : 0;
    return 16 * nn + 16 * n + 8 * n * 2 + 16 * cap + 4 * n + 4 + refine;
}

namespace {
// Byte offsets of the workspace's regions from its base, each rounded up to 256 bytes: seven,
// and for the mixed form above kMixedMaxN six more (the refinement's matrices and status).
struct WorkspaceLayout {
    size_t LV, tau, d, e, log, perm, flag, rfC = 0, rfY = 0, rfP = 0, rfG = 0, rfS = 0, rstat = 0, end;
    int log_cap, log_stride;
    bool refine;
    WorkspaceLayout(int n, int capacity, bool mixed) {
        const size_t nn = static_cast<size_t>(n) * n, cap = static_cast<size_t>(capacity);
        log_cap = ql_log_capacity(n);
        log_stride = std::max(std::max(log_cap, refine_stash_entries(n)), tc_scratch_entries(n));
        refine = mixed_big(n, mixed);
        size_t o = 0;
        auto take = [&](size_t bytes) { const size_t q = o; o += align_up(bytes, 256); return q; };
        LV = take(16 * nn * cap);
        tau = take(16 * n * cap);
        d = take(8 * n * cap);
        e = take(8 * n * cap);
        log = take(16 * static_cast<size_t>(log_stride) * cap);
        perm = take(4 * n * cap);
        flag = take(4 * cap);
        if (refine) {
            rfC = take(16 * nn * cap);
            rfY = take(16 * nn * cap);
            rfP = take(16 * nn * cap);
            rfG = take(16 * nn * cap);
            rfS = take(16 * nn * cap);
            rstat = take(4 * cap);
        }
        end = o;
    }
};
}  // namespace

size_t workspace_bytes(int n, int capacity, bool mixed) { return WorkspaceLayout(n, capacity, mixed).end; }

Workspace carve_workspace(void* base, int n, int capacity, bool mixed) {
    const WorkspaceLayout lay(n, capacity, mixed);
    char* p = static_cast<char*>(base);
    Workspace w;
    w.n = n;
    w.capacity = capacity;
    w.LV = reinterpret_cast<double2*>(p + lay.LV);
    w.tau = reinterpret_cast<double2*>(p + lay.tau);
    w.d = reinterpret_cast<double*>(p + lay.d);
    w.e = reinterpret_cast<double*>(p + lay.e);
    w.log_cap = lay.log_cap;
    w.log_stride = lay.log_stride;
    w.log = p + lay.log;
    w.perm = reinterpret_cast<int*>(p + lay.perm);
    w.flag = reinterpret_cast<int*>(p + lay.flag);
    if (lay.refine) {
        w.rfC = reinterpret_cast<double2*>(p + lay.rfC);
        w.rfY = reinterpret_cast<double2*>(p + lay.rfY);
        w.rfP = reinterpret_cast<double2*>(p + lay.rfP);
        w.rfG = reinterpret_cast<double2*>(p + lay.rfG);
        w.rfS = reinterpret_cast<double2*>(p + lay.rfS);
        w.rstat = reinterpret_cast<int*>(p + lay.rstat);
    }
    return w;
}

int max_smem_optin() {
    // per device ordinal (devices can differ); 0 = not yet queried
    static std::atomic<int> cache[SmemOptIn::kDevices];
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return 0; }
    if (dev >= 0 && dev < SmemOptIn::kDevices && (v = cache[dev].load(std::memory_order_relaxed)) > 0) return v;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (dev >= 0 && dev < SmemOptIn::kDevices) cache[dev].store(v, std::memory_order_relaxed);
    return v;
}

void set_smem_limit(const void* kernel, SmemOptIn& rec, int bytes) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return; }
    const bool tracked = dev >= 0 && dev < SmemOptIn::kDevices;
    if (tracked && rec.raised[dev].load(std::memory_order_acquire) >= bytes) return;
    // Idempotent: two threads that race here both set the same limit.  A failure is left for
    // the launch to report (it fails with the limit unraised).
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    if (!tracked) return;
    int cur = rec.raised[dev].load(std::memory_order_relaxed);
    while (cur < bytes && !rec.raised[dev].compare_exchange_weak(cur, bytes, std::memory_order_acq_rel)) {
    }
}

size_t invit_smem_bytes(int n, bool with_tile) { return InvitSmem(n, with_tile).per_warp; }

cudaError_t launch_reduce(int mode, const double2* A, const double2* B, int n, int batch,
                          const Workspace& ws, double2* out, int* info, const LaunchShape& shape, cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    // kReduceMixed is kReduceFull that, above kSmallMaxN, stops before the tridiagonalisation
    // (below it the reduction never tridiagonalises)
    const bool hegst_only = mode == kReduceMixed;
    if (hegst_only) mode = kReduceFull;
    if (n <= kSmallMaxN) return launch_reduce_dmma(mode, A, B, n, batch, ws, out, info, stream);
    if (mode != kReduceFull) return cudaErrorInvalidValue;
    if (!shape.reduce_tc)
        return launch_reduce_big(A, B, n, batch, ws, out, info, stream, hegst_only ? kBigHegstOnly : kBigFull);
    // tensor-core Cholesky + reduction, then the Householder
    const cudaError_t err = n <= kReduceDmmaMaxN ? launch_reduce_dmma(mode, A, B, n, batch, ws, out, info, stream)
                                                 : launch_reduce_tc(A, B, n, batch, ws, out, info, stream);
    if (err != cudaSuccess || hegst_only) return err;
    return launch_reduce_big(A, B, n, batch, ws, out, info, stream, kBigHetrdOnly);
}

cudaError_t launch_hetrd(int n, int batch, const double2* C, const Workspace& ws, int* info, cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (n > kSmallMaxN) return big_path(n) ? cudaSuccess : cudaErrorInvalidValue;   // done by the reduce launch
    return launch_hetrd_reg(n, batch, C, ws, info, stream);
}

size_t ql_chain_smem_bytes(int n, int threads) { return 8 * 2 * static_cast<size_t>(n) * threads; }
size_t ql_warps_bound_bytes(int n, int pairs_per_cta) {
    const size_t rows = (static_cast<size_t>(n) + 31) / 32;
    return (align_up(8 * static_cast<size_t>(n) * tile_ld(n), 16) + rows * 2 * 32 * 16 + align_up(16 * static_cast<size_t>(n), 16)) *
           pairs_per_cta;
}

size_t eig_smem_bytes(int n, int chain_threads) {
    const bool ql_here = n <= kInvitQlMaxN;
    const size_t m = std::max(tridiag_values_smem_bytes(n), std::max(invit_smem_bytes(n, ql_here), tridiag_ortho_smem_bytes(n, ql_here)));
    return ql_here ? m : std::max(m, std::max(ql_chain_smem_bytes(n, chain_threads), ql_rows_smem_bytes(n)));
}

cudaError_t launch_ql_chain(int n, int batch, const Workspace& ws, double* W, int* info, int chain_threads,
                            cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (!W || !info || !ws.d || !ws.e || !ws.log || !ws.perm || !ws.flag) return cudaErrorInvalidValue;
    const size_t cs = ql_chain_smem_bytes(n, chain_threads);
    if (cs > static_cast<size_t>(max_smem_optin())) return cudaErrorInvalidValue;
    static SmemOptIn f;
    set_max_smem_once(k_ql_chain, f);
    k_ql_chain<<<(batch + chain_threads - 1) / chain_threads, chain_threads, cs, stream>>>(n, batch, ws, W, info);
    return cudaGetLastError();
}

cudaError_t launch_eig_invit(int n, int batch, const Workspace& ws, double* W, double2* X, int* info,
                             const double2* C, bool flag_redo, cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (!W || !X || !info || !ws.d || !ws.e || !ws.flag) return cudaErrorInvalidValue;
    if (n <= kTridiagTinyMaxN) return launch_tridiag_tiny(n, batch, ws, W, X, info, C, stream);
    const size_t is = InvitSmem(n, !flag_redo).per_warp;
    if (is > static_cast<size_t>(max_smem_optin())) return cudaErrorInvalidValue;
    static SmemOptIn fi;
    set_max_smem_once(k_tridiag_invit, fi);
    const cudaError_t err = launch_tridiag_values(n, batch, ws, W, info, C, stream);
    if (err != cudaSuccess) return err;
    k_tridiag_invit<<<batch, 32, is, stream>>>(n, batch, ws, W, X, info, flag_redo ? 1 : 0);
    return launch_tridiag_ortho(n, batch, ws, W, X, info, !flag_redo, stream);
}

cudaError_t launch_eig(int n, int batch, const Workspace& ws, double* W, double2* X, int* info, const double2* C,
                       int chain_threads, cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (n > kInvitQlMaxN) return launch_ql_rows(n, batch, ws, W, X, info, C, chain_threads, stream);
    return launch_eig_invit(n, batch, ws, W, X, info, C, false, stream);
}

// ----------------------------------------------------------------------------- k_pull_pairs
// Pairs are walked grid-stride, each by the whole CTA; every thread keeps 4 independent 16-byte
// loads in flight (their latency is the host link's, about a microsecond), then stores them.
constexpr int kPullThreads = 256;
constexpr int kPullDepth = 4;

__global__ void __launch_bounds__(kPullThreads) k_pull_pairs(const double2* __restrict__ src,
                                                             double2* __restrict__ dst, int count, int n,
                                                             int lower) {
    const int nn = n * n;
    for (int p = blockIdx.x; p < count; p += gridDim.x) {
        const double2* s = src + static_cast<size_t>(nn) * p;
        double2* d = dst + static_cast<size_t>(nn) * p;
        for (int base = 0; base < nn; base += kPullDepth * kPullThreads) {
            double2 v[kPullDepth];
            int at[kPullDepth];
#pragma unroll
            for (int u = 0; u < kPullDepth; ++u) {
                const int e = base + u * kPullThreads + threadIdx.x;
                const int col = e / n, row = e - col * n;
                at[u] = (e < nn && (!lower || row >= col)) ? e : -1;
                if (at[u] >= 0) v[u] = s[e];
            }
#pragma unroll
            for (int u = 0; u < kPullDepth; ++u)
                if (at[u] >= 0) d[at[u]] = v[u];
        }
    }
}

cudaError_t launch_pull_pairs(const double2* src, double2* dst, int count, int n, bool lower, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    k_pull_pairs<<<std::min(count, sms), kPullThreads, 0, stream>>>(src, dst, count, n, lower ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_back(int mode, int n, int batch, const Workspace& ws, double2* X, int* info,
                        const LaunchShape& shape, cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    if (!X || !info || !ws.LV || !ws.tau) return cudaErrorInvalidValue;
    if (n <= kSmallMaxN || (n <= kBackDmmaMaxN && shape.reduce_tc))
        return launch_back_dmma(mode, n, batch, ws, X, info, stream);
    if (!shape.reduce_tc) return launch_back_big(mode, n, batch, ws, X, info, stream);
    if (n <= kBackStreamMaxN) return launch_back_stream(mode, n, batch, ws, X, info, stream);
    if (mode != kBackLOnly) {                           // Q Z and L^{-H} as products through L2
        const cudaError_t err = launch_back_q_tc(n, batch, ws, X, info, stream);
        if (err != cudaSuccess || mode == kBackQOnly) return err;
    }
    return launch_back_tc(n, batch, ws, X, info, stream);
}

// Device self-test of recip_nr (the inverse iteration's reciprocal): r[i] = recip_nr(u[i]).
__global__ void k_selftest_recip(const double* __restrict__ u, double* __restrict__ r, int count) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) r[i] = recip_nr(u[i]);
}

cudaError_t launch_selftest_recip(const double* u, double* r, int count, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    const int blocks = std::min((count + 255) / 256, 148 * 8);
    k_selftest_recip<<<blocks, 256, 0, stream>>>(u, r, count);
    return cudaGetLastError();
}

// FP64 FMA throughput probe: every thread runs kFmaChains independent dependent chains of
// fma(a, x, y) (x, y runtime values, so nothing folds) for `iters` rounds and stores their sum.
// Flops = 2 * kFmaChains * iters * threads.  Enough independent chains per warp cover the FMA
// latency, so the FP64 pipe, not the chain, bounds it.
constexpr int kFmaChains = 8;
__global__ void __launch_bounds__(256) k_selftest_fp64_fma(double* __restrict__ out, int iters, double x, double y) {
    double a[kFmaChains];
#pragma unroll
    for (int c = 0; c < kFmaChains; ++c) a[c] = threadIdx.x * 1e-3 + c;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
#pragma unroll
            for (int c = 0; c < kFmaChains; ++c) a[c] = fma(a[c], x, y);
        }
    }
    double sum = 0.0;
#pragma unroll
    for (int c = 0; c < kFmaChains; ++c) sum += a[c];
    out[blockIdx.x * blockDim.x + threadIdx.x] = sum;
}

cudaError_t launch_selftest_fp64_fma(double* out, int blocks, int iters, cudaStream_t stream) {
    if (blocks <= 0 || iters <= 0) return cudaErrorInvalidValue;
    k_selftest_fp64_fma<<<blocks, 256, 0, stream>>>(out, iters, 0.999999, 1e-7);
    return cudaGetLastError();
}

}  // namespace sbg
