// Stage device functions of the generalized Hermitian-definite eigensolve
//   A x = lambda B x,  B = L L^H,  C = L^{-1} A L^{-H} = Q T Q^H,  T Z = Z Lambda,
//   X = L^{-H} Q Z.
//
// Each function runs on one CTA ("team") over tiles that live in shared memory
// (column-major, leading dimension ld = n | 1 so row walks are bank-conflict
// free).  The stage boundaries are the reference's (src/geneig_fixed.cu:455-464):
// potrf on B, the two-sided triangular reduction, the Hermitian eigensolve and
// the back substitution; the eigensolve is split into Householder
// tridiagonalisation, implicit QL on the real tridiagonal, and the reflector
// back-application.
#pragma once

#include "common.cuh"

namespace sbg {

// ============================================================================ hetrd (lower)
// Householder reduction of the Hermitian tile A (lower triangle valid) to real
// symmetric tridiagonal form T = Q^H A Q, Q = H_0 H_1 ... H_{n-2},
// H_k = I - tau_k v_k v_k^H with v_k = (0_{k+1}, 1, A(k+2:n, k)) stored in place.
// Outputs d[0:n], e[0:n-1] (real), tau[0:n-1].  The steps are LAPACK zhetd2's
// (reflector as zlarfg, p = tau A22 v, w = p - tau/2 (p^H v) v,
// A22 -= v w^H + w v^H).  Two CTA barriers per step: every warp computes the
// reflector and w itself (into its own slices of vw / ww, n complex per warp), so no
// warp waits on another for those; the barriers only separate the Hermitian matvec
// (a row walk over the lower part and a column walk over the mirrored upper part,
// partial sums in pbuf, 2n complex) from the rank-2 update, and the update from the
// next step.
template <typename R>
__device__ void hetrd_lower(cplx<R>* A, int lda, int n, R* d, R* e, cplx<R>* tau,
                            cplx<R>* vw_all, cplx<R>* pbuf, cplx<R>* ww_all) {
    using C = cplx<R>;
    const int tid = threadIdx.x, T = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5;
    C* vw = vw_all + warp * n;
    C* ww = ww_all + warp * n;
    for (int k = 0; k + 1 < n; ++k) {
        const int m = n - k - 1;
        C* x = A + (k + 1) + k * lda;                    // x[0..m) = A(k+1:n, k)
        // ---- reflector (every warp)
        R s2 = R(0);
        for (int i = 1 + lane; i < m; i += 32) s2 += cabs2(x[i]);
        s2 = warp_sum(s2);
        const C alpha = x[0];
        C tk, scale;
        R beta;
        if (s2 == R(0) && alpha.y == R(0)) {
            tk = mk<R>(R(0), R(0)); beta = alpha.x; scale = mk<R>(R(0), R(0));
        } else {
            const R nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + s2);
            beta = alpha.x >= R(0) ? -nrm : nrm;
            tk = mk<R>((beta - alpha.x) / beta, -alpha.y / beta);
            const R ar = alpha.x - beta, ai = alpha.y;   // scale = 1 / (alpha - beta)
            const R den = ar * ar + ai * ai;
            scale = mk<R>(ar / den, -ai / den);
        }
        if (tid == 0) { e[k] = beta; tau[k] = tk; }
        if (tk.x == R(0) && tk.y == R(0)) continue;      // H_k = I (uniform: same value in every warp)
        for (int i = lane; i < m; i += 32) vw[i] = (i == 0) ? mk<R>(R(1), R(0)) : cmul(x[i], scale);
        __syncwarp();
        // ---- p partial sums: part 0 = sum_{j<=r} A22(r,j) v_j, part 1 = sum_{j>r} conj(A22(j,r)) v_j
        C* A22 = A + (k + 1) + (k + 1) * lda;
        for (int t = tid; t < 2 * m; t += T) {
            const int part = t >= m, r = t - part * m;
            C acc0 = mk<R>(R(0), R(0)), acc1 = mk<R>(R(0), R(0));
            if (part == 0) {
                int j = 0;
                for (; j + 1 < r; j += 2) {
                    acc0 = cfma(A22[r + j * lda], vw[j], acc0);
                    acc1 = cfma(A22[r + (j + 1) * lda], vw[j + 1], acc1);
                }
                for (; j < r; ++j) acc0 = cfma(A22[r + j * lda], vw[j], acc0);
                const R drr = A22[r + r * lda].x;
                acc0.x = fma(drr, vw[r].x, acc0.x);
                acc0.y = fma(drr, vw[r].y, acc0.y);
            } else {
                const C* col = A22 + r * lda;
                int j = r + 1;
                for (; j + 1 < m; j += 2) {
                    acc0 = cfmac(col[j], vw[j], acc0);
                    acc1 = cfmac(col[j + 1], vw[j + 1], acc1);
                }
                for (; j < m; ++j) acc0 = cfmac(col[j], vw[j], acc0);
            }
            pbuf[t] = cadd(acc0, acc1);
        }
        __syncthreads();
        // the scaled reflector replaces x (nobody reads column k after the barrier above)
        if (warp == 0)
            for (int i = 1 + lane; i < m; i += 32) x[i] = vw[i];
        // ---- p = tau (part0 + part1); alpha2 = -tau/2 (p^H v); w = p + alpha2 v (every warp)
        C dot = mk<R>(R(0), R(0));
        for (int r = lane; r < m; r += 32) {
            const C p = cmul(tk, cadd(pbuf[r], pbuf[m + r]));
            ww[r] = p;
            dot = cfmac(p, vw[r], dot);
        }
        dot.x = warp_sum(dot.x);
        dot.y = warp_sum(dot.y);
        const C a2 = cscale(cmul(tk, dot), R(-0.5));
        for (int r = lane; r < m; r += 32) ww[r] = cfma(a2, vw[r], ww[r]);
        __syncwarp();
        // ---- A22 -= v w^H + w v^H on the lower triangle; thread (row r, column chunk c)
        {
            const int chunks = max(1, T / m);
            const int cw = (m + chunks - 1) / chunks;
            for (int t = tid; t < m * chunks; t += T) {
                const int r = t % m, c = t / m;
                const C vr = vw[r], wr = ww[r];
                const int j0 = c * cw, j1 = min(r + 1, (c + 1) * cw);
                for (int j = j0; j < j1; ++j) {
                    C a = A22[r + j * lda];
                    a = cfmsc(vr, ww[j], a);
                    a = cfmsc(wr, vw[j], a);
                    if (j == r) a.y = R(0);
                    A22[r + j * lda] = a;
                }
            }
        }
        __syncthreads();
    }
    for (int i = tid; i < n; i += T) d[i] = A[i + i * lda].x;
    if (tid == 0 && n >= 1) e[n - 1] = R(0);
    __syncthreads();
}

// ============================================================================ tridiagonal QL
// The power of two that scales a T of max-norm anorm to [1/2, 1) (exactly: a diagonal T keeps its
// entries); 1 for a zero or non-finite norm.  Kept within the normal range, as is its reciprocal.
template <typename R>
__device__ __forceinline__ R pow2_norm(R anorm) {
    if (!(anorm > R(0)) || !isfinite(anorm)) return R(1);
    int ex;
    frexp(anorm, &ex);
    constexpr int kMost = sizeof(R) == 8 ? 1022 : 126;
    return scalbn(R(1), min(max(ex, -kMost), kMost));
}

// Eigen-decomposition of the real symmetric tridiagonal (d, e) by implicit QL
// with Wilkinson-type shifts, accumulating the rotations into Z (row-major,
// Z[r * ldz + c], initialised to I by the caller).  One warp per problem: every
// lane runs the same scalar recurrence (so no broadcast is needed) and applies
// each rotation to the rows it owns (r = lane + 32 q).  The deflation test is
// LAPACK dsteqr's relative one, |e_m|^2 <= eps^2 |d_m| |d_{m+1}| + safmin, and the
// matrix is scaled by a power of two to max-norm in [1/2, 1) first (dsteqr scales only at the range
// limits; scaling always keeps the single-precision variant safe).
// Eigenvalues come back ascending with Z's columns permuted alike (dsteqr's
// final selection sort).  Returns the number of off-diagonals that had not
// converged after 30 n iterations (0 on success; n - 1, with NaN in d and Z, for a T that is not finite).
// d, e live in shared memory private to the warp; only lane 0 writes them.
template <typename R>
__device__ int tridiag_ql(int n, R* d, R* e, R* Z, int ldz) {
    const int lane = threadIdx.x & 31;
    const R eps = sizeof(R) == 8 ? R(1.1102230246251565e-16) : R(5.9604645e-08);
    const R eps2 = eps * eps;
    const R safmin = sizeof(R) == 8 ? R(2.2250738585072014e-308) : R(1.17549435e-38);
    // scale to max-norm in [1/2, 1)
    R anorm = R(0);
    bool finite = true;
    for (int i = 0; i < n; ++i) { anorm = fmax(anorm, fabs(d[i])); finite = finite && isfinite(d[i]); }
    for (int i = 0; i + 1 < n; ++i) { anorm = fmax(anorm, fabs(e[i])); finite = finite && isfinite(e[i]); }
    if (!finite) {                                           // uniform: no sweep would converge
        const R nan = static_cast<R>(__longlong_as_double(0x7ff8000000000000ll));
        __syncwarp();
        for (int i = lane; i < n; i += 32) d[i] = nan;
        for (int row = lane; row < n; row += 32)
            for (int k = 0; k < n; ++k) Z[row * ldz + k] = nan;
        __syncwarp();
        return n - 1;
    }
    anorm = pow2_norm(anorm);
    const R sc = R(1) / anorm;
    __syncwarp();
    if (lane == 0) {
        for (int i = 0; i < n; ++i) d[i] *= sc;
        for (int i = 0; i + 1 < n; ++i) e[i] *= sc;
        e[n - 1] = R(0);
    }
    __syncwarp();
    int unconverged = 0, iter = 0;
    const int maxit = 30 * n;                                // in all, as dsteqr
    for (int l = 0; l < n && unconverged == 0; ++l) {
        for (;;) {
            int m = l;
            for (; m < n - 1; ++m) {
                const R em = e[m];
                if (em * em <= (eps2 * fabs(d[m])) * fabs(d[m + 1]) + safmin) break;
            }
            if (m == l) break;
            if (iter == maxit) {
                for (int i = l; i + 1 < n; ++i) unconverged += e[i] != R(0) ? 1 : 0;
                break;
            }
            ++iter;
            const R el = e[l], dl = d[l];
            R g = (d[l + 1] - dl) / (R(2) * el);
            R r = sqrt(fma(g, g, R(1)));
            g = d[m] - dl + el / (g + copysign(r, g));
            R s = R(1), c = R(1), p = R(0);
            bool early = false;
            for (int i = m - 1; i >= l; --i) {
                const R ei = e[i];
                const R f = s * ei, b = c * ei;
                const R rr = fma(f, f, g * g);
                if (rr == R(0)) {
                    __syncwarp();
                    if (lane == 0) { d[i + 1] -= p; e[m] = R(0); }
                    __syncwarp();
                    early = true;
                    break;
                }
                const R ri = rsqrt(rr);
                r = rr * ri;
                s = f * ri;
                c = g * ri;
                const R di1 = d[i + 1];
                g = di1 - p;
                r = fma(d[i] - g, s, R(2) * c * b);
                p = s * r;
                __syncwarp();
                if (lane == 0) { e[i + 1] = rr * ri; d[i + 1] = g + p; }
                g = fma(c, r, -b);
                // rotate columns i, i+1 of the rows this lane owns
                for (int row = lane; row < n; row += 32) {
                    R* zr = Z + row * ldz;
                    const R zi = zr[i], zi1 = zr[i + 1];
                    zr[i + 1] = fma(s, zi, c * zi1);
                    zr[i] = fma(c, zi, -s * zi1);
                }
                __syncwarp();
            }
            if (early) continue;
            __syncwarp();
            if (lane == 0) { d[l] -= p; e[l] = g; e[m] = R(0); }
            __syncwarp();
        }
    }
    // sort ascending (selection sort, as dsteqr)
    for (int i = 0; i + 1 < n; ++i) {
        int k = i;
        R pmin = d[i];
        for (int j = i + 1; j < n; ++j) if (d[j] < pmin) { k = j; pmin = d[j]; }
        if (k != i) {
            __syncwarp();
            if (lane == 0) { d[k] = d[i]; d[i] = pmin; }
            for (int row = lane; row < n; row += 32) {
                R* zr = Z + row * ldz;
                const R t = zr[i]; zr[i] = zr[k]; zr[k] = t;
            }
            __syncwarp();
        }
    }
    __syncwarp();
    if (lane == 0) for (int i = 0; i < n; ++i) d[i] *= anorm;
    __syncwarp();
    return unconverged;
}

// ============================================================================ QL, scalar chain only
// The same implicit QL as tridiag_ql, run by ONE thread for one pair, with d and
// e in shared memory interleaved over the CTA (element i of thread t at
// [i * stride + t]).  Instead of rotating Z, every rotation (c, s) is appended
// to a per-pair log in global memory: a sweep is a header entry
// (top = m - 1, count) followed by `count` rotations acting on column pairs
// (i, i+1), i = top, top-1, ..., top-count+1.  A header with count = 0 and
// top = -1 ends the log.  The eigenvalues are sorted ascending and perm[k]
// receives the pre-sort column index of eigenvalue k.
// Returns the number of unconverged off-diagonals, or -1 if the log capacity
// (cap entries) would be exceeded (the caller then falls back to tridiag_ql).  A T that is not finite
// gives n - 1, NaN in W and a log that turns Z to NaN.
// LOG = false: eigenvalues only (no log, no permutation; log, cap and perm are ignored).
template <typename R, bool LOG = true>
__device__ int ql_chain(int n, R* d, R* e, int stride, cplx<R>* log, int cap, int* perm, double* W) {
    using C = cplx<R>;
    const R eps = sizeof(R) == 8 ? R(1.1102230246251565e-16) : R(5.9604645e-08);
    const R eps2 = eps * eps;
    const R safmin = sizeof(R) == 8 ? R(2.2250738585072014e-308) : R(1.17549435e-38);
#define D(i) d[(i) * stride]
#define E(i) e[(i) * stride]
    R anorm = R(0);
    bool finite = true;
    for (int i = 0; i < n; ++i) { anorm = fmax(anorm, fabs(D(i))); finite = finite && isfinite(D(i)); }
    for (int i = 0; i + 1 < n; ++i) { anorm = fmax(anorm, fabs(E(i))); finite = finite && isfinite(E(i)); }
    if (!finite) {                                           // no sweep would converge: one of NaN instead
        const R nan = static_cast<R>(__longlong_as_double(0x7ff8000000000000ll));
        for (int k = 0; k < n; ++k) W[k] = nan;
        if constexpr (LOG) {
            if (n + 1 > cap) return -1;
            for (int k = 0; k < n; ++k) perm[k] = k;
            int pos = 0;
            if (n > 1) {
                log[pos++] = mk<R>(R(n - 2), R(n - 1));
                for (int k = 0; k + 1 < n; ++k) log[pos++] = mk<R>(nan, nan);
            }
            log[pos] = mk<R>(R(-1), R(0));
        }
        return n - 1;
    }
    anorm = pow2_norm(anorm);
    const R sc = R(1) / anorm;
    for (int i = 0; i < n; ++i) D(i) *= sc;
    for (int i = 0; i + 1 < n; ++i) E(i) *= sc;
    E(n - 1) = R(0);
    int pos = 0, unconverged = 0, iter = 0;
    const int maxit = 30 * n;                                // in all, as dsteqr
    for (int l = 0; l < n && unconverged == 0; ++l) {
        for (;;) {
            int m = l;
            for (; m < n - 1; ++m) {
                const R em = E(m);
                if (em * em <= (eps2 * fabs(D(m))) * fabs(D(m + 1)) + safmin) break;
            }
            if (m == l) break;
            if (iter == maxit) {
                for (int i = l; i + 1 < n; ++i) unconverged += E(i) != R(0) ? 1 : 0;
                break;
            }
            ++iter;
            int hdr = 0;
            if constexpr (LOG) {
                if (pos + (m - l) + 2 > cap) return -1;
                hdr = pos++;
            }
            const R el = E(l), dl = D(l);
            R g = (D(l + 1) - dl) / (R(2) * el);
            R r = sqrt(fma(g, g, R(1)));
            g = D(m) - dl + el / (g + copysign(r, g));
            R s = R(1), c = R(1), p = R(0);
            bool early = false;
            int i = m - 1;
            R ei = E(i), di = D(i);
            for (; i >= l; --i) {
                const R f = s * ei, b = c * ei;
                const R rr = fma(f, f, g * g);
                if (rr == R(0)) { D(i + 1) -= p; E(m) = R(0); early = true; break; }
                const R di1 = D(i + 1);
                const R ei_next = (i > l) ? E(i - 1) : R(0);     // prefetch: not written in this sweep
                const R di_next = (i > l) ? D(i - 1) : R(0);
                const R ri = rsqrt(rr);
                E(i + 1) = rr * ri;
                s = f * ri;
                c = g * ri;
                g = di1 - p;
                r = fma(di - g, s, R(2) * c * b);
                p = s * r;
                D(i + 1) = g + p;
                g = fma(c, r, -b);
                if constexpr (LOG) log[pos++] = mk<R>(c, s);
                ei = ei_next; di = di_next;
            }
            if constexpr (LOG) log[hdr] = mk<R>(R(m - 1), R(early ? (m - 1 - i) : (m - l)));
            if (early) continue;
            D(l) -= p; E(l) = g; E(m) = R(0);
        }
    }
    if constexpr (LOG) log[pos] = mk<R>(R(-1), R(0));
    // selection sort with the permutation recorded
    if constexpr (LOG) for (int k = 0; k < n; ++k) perm[k] = k;
    for (int k = 0; k + 1 < n; ++k) {
        int j = k;
        R pmin = D(k);
        for (int t = k + 1; t < n; ++t) if (D(t) < pmin) { j = t; pmin = D(t); }
        if (j != k) {
            D(j) = D(k); D(k) = pmin;
            if constexpr (LOG) { const int tp = perm[k]; perm[k] = perm[j]; perm[j] = tp; }
        }
    }
    for (int k = 0; k < n; ++k) W[k] = static_cast<double>(D(k) * anorm);
#undef D
#undef E
    return unconverged;
}

// ============================================================================ register-segment solvers
// Column (or row) work where the G lanes of a group share one column and lane g keeps
// the entries of rows i = g + G r, r < RM, in registers for the whole stage; only L
// or the reflectors are read from shared memory (the same address for every group:
// a broadcast).  Requires n <= G * RM and n <= (threads / G) columns per pass.

// Selects seg[r] for a runtime r (unrolled, so seg stays in registers).
template <int RM, typename C>
__device__ __forceinline__ C seg_get(const C (&seg)[RM], int r) {
    C v = seg[0];
#pragma unroll
    for (int q = 1; q < RM; ++q) if (q == r) v = seg[q];
    return v;
}
template <int RM, typename C>
__device__ __forceinline__ void seg_set(C (&seg)[RM], int r, C v) {
#pragma unroll
    for (int q = 0; q < RM; ++q) if (q == r) seg[q] = v;
}

// ============================================================================ QL log application
// Applies one pair's rotation log (ql_chain's format: a header (top, count), then count
// rotations (c, s) for columns top, top-1, ...; a header with top < 0 ends the log) to
// the row zrow of Z owned by this lane (own = false: the lane only helps stream the
// log).  The log is read 32 entries at a time with one coalesced load into the warp's
// stage buffer (64 entries, double-buffered) and read back by broadcast; within a sweep
// the rotation at column i loads z_i and carries z_{i+1} in a register.
template <typename R>
__device__ __forceinline__ void ql_log_apply_row(const cplx<R>* log, int cap, cplx<R>* stage, R* zrow, bool own) {
    using C = cplx<R>;
    const int lane = threadIdx.x & 31;
    int loaded = 0, buf = 0, remaining = 0, col = 0;
    C pre = log[lane];
    R carry = R(0);
    bool done = false;
    while (!done) {
        stage[buf * 32 + lane] = pre;
        __syncwarp();
        loaded += 32;
        if (loaded < cap) pre = log[min(loaded + lane, cap - 1)];
        const C* st = stage + buf * 32;
        int k = 0;
        while (k < 32) {
            if (remaining == 0) {
                const C h = st[k++];
                const int top = static_cast<int>(h.x);
                if (top < 0) { done = true; break; }
                remaining = static_cast<int>(h.y);
                col = top;
                if (own && remaining > 0) carry = zrow[col + 1];
                continue;
            }
            const int take = min(remaining, 32 - k);
            if (own) {
                for (int t = 0; t < take; ++t) {
                    const C cs = st[k + t];
                    const R zi = zrow[col - t];
                    zrow[col - t + 1] = fma(cs.y, zi, cs.x * carry);
                    carry = fma(cs.x, zi, -cs.y * carry);
                }
            }
            k += take;
            col -= take;
            remaining -= take;
            if (remaining == 0 && own) zrow[col + 1] = carry;
        }
        __syncwarp();
        buf ^= 1;
        if (!done && loaded >= cap) done = true;      // malformed log guard (never reached)
    }
}

// ============================================================================ packed lower triangle
// Column-major packed lower triangle: A(i, j), i >= j, at P[pk(j, n) + i - j].
__host__ __device__ __forceinline__ int pk(int j, int n) { return j * n - (j * (j - 1)) / 2; }

}  // namespace sbg
