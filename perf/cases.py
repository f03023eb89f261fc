"""The work that programs have this library do, as cases that can be timed and compared.

A case is a dict: ``call`` names the public entry point, ``kind`` the matrix pairs, ``n`` their
order (two bosonic modes per site: n = 2 N, odd only for general pairs), ``pairs`` the batch.

Calls
    dropin     ``sbg.geneig_full_n54_batched``: the fixed n = 54 launcher, device buffers in and out
    solver     ``sbg.Solver.launch``: the runtime-n handle, ``precision`` "fp64" or "mixed"
    queue      ``sbg.Queue.launch``: pairs of n in {12, 24, 32, 54, 96, 128} mixed in one launch
    spinwave   ``sbg.SpinWave.solve``: one magnetic cell swept over q, eigenvalues and intensities out
Kinds (A = diag(I, -I), B = [[P, Q], [conj Q, conj P]] + shift, except "general")
    qsweep     bond table of a random cell of N sites, 4 bonds per site, on a 64^3 q-grid; every B
               shifted to lambda_min = 1e-3 lambda_max
    random     Bogoliubov blocks with complex normal entries, lambda_min = 1e-2 lambda_max
    softmode   the same with one near-zero mode, lambda_min = 1e-6 lambda_max: q close to a
               Goldstone point.  (Milder than the 1e-8 of the near-Goldstone benchmark, where X is
               itself too ill-conditioned to be compared; the kernels that run and the shape of the
               spectrum are the same.)
    general    A Hermitian, B = I + G G^H / n, both full: pairs with no spin-wave structure

Eigenvectors are defined up to a phase, and the library, like LAPACK, does not choose it.  A
program that keeps or interpolates modes over q fixes it: every ``run`` that returns eigenvectors
turns each so that its overlap with one fixed vector is real and positive.  Intensities need no such
step.  Work is done on the current stream; nothing is synchronised.
"""
from __future__ import annotations

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "sunny-batched-geneig_b200"))

import sbg  # noqa: E402
from sbg import workloads  # noqa: E402

DEV = "cuda"
GRID = 64                               # q-points per axis of the sweeps
FRAC = {"qsweep": 1e-3, "random": 1e-2, "softmode": 1e-2}
SOFT_LEVEL = 1e-6


def listed():
    return [
        # The smallest call: one path segment of a few q-points through the drop-in launcher (the
        # reference's own fixtures hold 8 pairs).  Latency of the chain of stages.
        {"name": "n54 drop-in 8", "call": "dropin", "kind": "random", "n": 54, "pairs": 8},
        # The reference's own batched test: 1,024 pairs of general matrices.
        {"name": "n54 drop-in 1024", "call": "dropin", "kind": "general", "n": 54, "pairs": 1024},
        # The headline: a slab of the 64^3 q-sweep of a 27-site cell.
        {"name": "n54 q-sweep", "call": "solver", "precision": "fp64", "kind": "qsweep", "n": 54, "pairs": 32768},
        # The same sweep of a 16-site cell.
        {"name": "n32 q-sweep", "call": "solver", "precision": "fp64", "kind": "qsweep", "n": 32, "pairs": 65536},
        # An odd order and no spin-wave structure: a general batch of Hermitian-definite pairs.
        {"name": "n47 general", "call": "solver", "precision": "fp64", "kind": "general", "n": 47, "pairs": 8192},
        # Middle-sized cells.
        {"name": "n72", "call": "solver", "precision": "fp64", "kind": "random", "n": 72, "pairs": 4096},
        # 48-site cell near a Goldstone point.
        {"name": "n96 soft mode", "call": "solver", "precision": "fp64", "kind": "softmode", "n": 96, "pairs": 4096},
        {"name": "n128", "call": "solver", "precision": "fp64", "kind": "random", "n": 128, "pairs": 2048},
        # Large cell.
        {"name": "n192", "call": "solver", "precision": "fp64", "kind": "random", "n": 192, "pairs": 1024},
        # Cells of several sizes in one launch.
        {"name": "uneven queue", "call": "queue", "kind": "random", "pairs": 8192},
        # A whole intensity sweep: q in, eigenvalues and intensities out.
        {"name": "n54 spin-wave sweep", "call": "spinwave", "kind": "qsweep", "n": 54, "pairs": 16384},
        # The mixed-precision form at the headline order.
        {"name": "n54 mixed", "call": "solver", "precision": "mixed", "kind": "qsweep", "n": 54, "pairs": 8192},
    ]


def draw(rng):
    """Orders 8 to 256 and batches from a single pair to about 2e9 / n^3 (a sixth to a half of the
    largest listed case's time), both spread over their logarithm."""
    call = rng.choice(["solver"] * 7 + ["dropin", "queue", "spinwave"])
    if call == "queue":
        return {"call": call, "kind": "random", "pairs": int(round(2 ** rng.uniform(6.0, 12.0)))}
    n = 54 if call == "dropin" else int(round(2 ** rng.uniform(3.0, 8.0)))
    kind = "qsweep" if call == "spinwave" else rng.choice(["qsweep", "random", "softmode", "general"])
    if kind != "general":
        n += n & 1
    most = min(65536.0, 2e9 / n ** 3)
    pairs = max(1, int(round(math.exp(rng.uniform(0.0, math.log(most))))))
    case = {"call": call, "kind": kind, "n": n, "pairs": pairs}
    if call == "solver":
        case["precision"] = "mixed" if n <= 63 and rng.random() < 0.15 else "fp64"
    return case


# ------------------------------------------------------------------ inputs

def _cnormal(gen, shape, var=1.0):
    s = math.sqrt(var / 2.0)
    return torch.complex(torch.randn(shape, dtype=torch.float64, device=DEV, generator=gen) * s,
                         torch.randn(shape, dtype=torch.float64, device=DEV, generator=gen) * s)


def _top(M):
    """Largest eigenvalue of each positive semidefinite M, to about 1e-6: 24 squarings."""
    log = torch.zeros(M.shape[0], dtype=torch.float64, device=M.device)
    for k in range(24):
        f = torch.linalg.matrix_norm(M)
        log += torch.log(f) / 2.0 ** k
        M = M / f[:, None, None]
        M = M @ M
    return torch.exp(log + torch.log(torch.linalg.matrix_norm(M)) / 2.0 ** 24)


def _extremes(M):
    """(lambda_min, lambda_max) of each Hermitian M, to about 1e-6 of its norm."""
    lo, hi = [], []
    for P in M.split(8192):
        c = torch.linalg.matrix_norm(P)
        eye = torch.eye(P.shape[-1], dtype=P.dtype, device=P.device) * c[:, None, None]
        hi.append(_top(eye + P) - c)
        lo.append(c - _top(eye - P))
    return torch.cat(lo), torch.cat(hi)


def _shift(B, frac):
    """B + s I, in place, with lambda_min = frac * lambda_max."""
    lo, hi = _extremes(B)
    B.diagonal(dim1=1, dim2=2).add_(((frac * hi - lo) / (1.0 - frac)).to(B.dtype)[:, None])
    return B


def _metric(n, pairs):
    s = torch.ones(n, dtype=torch.complex128, device=DEV)
    s[n // 2:] = -1.0
    return torch.diag(s).expand(pairs, n, n)


def _blocks(P, Q):
    return torch.cat([torch.cat([P, Q], dim=2), torch.cat([Q.conj(), P.conj()], dim=2)], dim=1)


def _cell(N, seed):
    """A random cell: 4 bonds per site with 3 x 3 exchange, as (sites, coefficients, displacements,
    positions), the coefficients per bond Re a, Im a, Re b, Im b, c."""
    rng = np.random.default_rng(seed)
    u = np.array([1.0, 1.0j, 0.0]) / math.sqrt(2.0)
    sites, coef, disp = [], [], []
    for i in range(N):
        for _ in range(4):
            J = rng.normal(size=(3, 3))
            a, b = complex(u @ J @ u.conj()), complex(u @ J @ u)
            sites.append([i, int(rng.integers(N))])
            coef.append([a.real, a.imag, b.real, b.imag, J[2, 2]])
            disp.append(rng.uniform(-1.0, 1.0, 3))
    return np.array(sites), np.array(coef), np.array(disp), rng.uniform(0.0, 1.0, (N, 3))


def _q_points(pairs, seed):
    """Consecutive points of the grid from one that the seed picks."""
    start = np.random.default_rng(seed).integers(GRID ** 3)
    k = (torch.arange(pairs, device=DEV) + int(start)) % GRID ** 3
    k = torch.stack([k // GRID ** 2, (k // GRID) % GRID, k % GRID], dim=1)
    return (2.0 * math.pi / GRID) * k.to(torch.float64)


def _cell_B(N, cell, q):
    """B(q) of the cell without field: P_ij += a/2 e^{iqd}, P_ji += conj, Q_ij, Q_ji += b/2 e^{iqd},
    P_ii, P_jj -= c/2."""
    sites, coef, disp, _ = cell
    ph = torch.exp(1j * (q @ torch.as_tensor(disp, device=DEV).T))
    P = torch.zeros((q.shape[0], N, N), dtype=torch.complex128, device=DEV)
    Q = torch.zeros_like(P)
    for t, ((i, j), (ar, ai, br, bi, c)) in enumerate(zip(sites.tolist(), coef.tolist())):
        pa, pb = complex(ar, ai) / 2 * ph[:, t], complex(br, bi) / 2 * ph[:, t]
        P[:, i, j] += pa
        P[:, j, i] += pa.conj()
        Q[:, i, j] += pb
        Q[:, j, i] += pb
        P[:, i, i] -= c / 2
        P[:, j, j] -= c / 2
    return _blocks(P, Q)


def _pairs(kind, n, pairs, seed):
    """(A, B) as (pairs, n, n) tensors indexed [pair, row, column]."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    if kind == "general":
        G, H = _cnormal(gen, (pairs, n, n)), _cnormal(gen, (pairs, n, n))
        return (H + H.mH) / 2, torch.eye(n, dtype=H.dtype, device=DEV) + G @ G.mH / n
    N = n // 2
    if kind == "qsweep":
        B = _cell_B(N, _cell(N, seed), _q_points(pairs, seed))
    else:
        G, H = _cnormal(gen, (pairs, N, N), 1.0 / N), _cnormal(gen, (pairs, N, N), 1.0 / N)
        B = _blocks((G + G.mH) / math.sqrt(2.0), (H + H.mT) / math.sqrt(2.0))
    B = _shift(B, FRAC[kind])
    if kind == "softmode":
        norm = _extremes(B)[1]
        u = _cnormal(gen, (pairs, N, 1))
        v = torch.cat([u, u.conj()], dim=1)
        v = v / torch.linalg.vector_norm(v, dim=1, keepdim=True)
        B = B - v @ (v.mH @ B)
        B = B - (B @ v) @ v.mH
        B = B + (SOFT_LEVEL * norm)[:, None, None] * (v @ v.mH)
        B = (B + B.mH) / 2
    return _metric(n, pairs), B


def _flat(M):
    """[pair, row, column] to the library's layout: column-major, pairs contiguous."""
    return M.mT.reshape(M.shape[0], -1).contiguous()


def _reference_vector(n):
    """The vector every mode's overlap with is made real: fixed, with no zero and no symmetry."""
    k = torch.arange(n, dtype=torch.float64, device=DEV)
    return torch.polar(1.0 + 0.5 * torch.cos(1.7 * k), 0.9 * k * k)


@functools.lru_cache(maxsize=None)
def _solver(n, precision):
    """The handle a program keeps for all its batches of one order."""
    return sbg.Solver(n, precision=precision)


def _queue_inputs(pairs, seed):
    ns = workloads.uneven_sizes(pairs, seed=seed % (1 << 31))
    first = np.concatenate([[0], np.cumsum(ns.astype(np.int64) ** 2)])
    A = torch.empty(int(first[-1]), dtype=torch.complex128, device=DEV)
    B = torch.empty_like(A)
    at = {}
    for n in sorted({int(v) for v in ns}):
        start = torch.as_tensor(first[:-1][ns == n], device=DEV)
        at[n] = start[:, None] + torch.arange(n * n, device=DEV)
        a, b = _pairs("random", n, len(start), seed + n)
        A[at[n]] = _flat(a)
        B[at[n]] = _flat(b)
    return ns, at, A, B


def _sweep_inputs(case, seed):
    """(cell, field, q): one field for the sweep, which puts min lambda_min at 1e-3 max lambda_max."""
    N = case["n"] // 2
    cell, q = _cell(N, seed), _q_points(case["pairs"], seed)
    lo, hi = _extremes(_cell_B(N, cell, q))
    f = FRAC["qsweep"]
    return cell, float((f * hi.max() - lo.min()) / (1.0 - f)), q


def _outputs(pairs, n):
    return {"W": torch.empty((pairs, n), dtype=torch.float64, device=DEV),
            "X": torch.empty((pairs, n * n), dtype=torch.complex128, device=DEV),
            "info": torch.empty(pairs, dtype=torch.int32, device=DEV)}


def prepare(case, seed):
    call = case["call"]
    if call == "queue":
        ns, at, A, B = _queue_inputs(case["pairs"], seed)
        q = sbg.Queue(ns)
        return {"call": call, "queue": q, "A": A, "B": B, "at": at, "X": torch.empty_like(A),
                "W": torch.empty(int(ns.sum()), dtype=torch.float64, device=DEV),
                "info": torch.empty(len(ns), dtype=torch.int32, device=DEV),
                "ref": {n: _reference_vector(n) for n in at}}
    n, pairs = case["n"], case["pairs"]
    if call == "spinwave":
        (sites, coef, disp, pos), field, q = _sweep_inputs(case, seed)
        out = _outputs(pairs, n)
        del out["X"]
        return {"call": call, "model": sbg.SpinWave(n // 2, sites, coef, disp, pos, field), "q": q,
                "solver": _solver(n, "fp64"), "I": torch.empty_like(out["W"]), **out}
    A, B = _pairs(case["kind"], n, pairs, seed)
    s = {"call": call, "A": _flat(A), "B": _flat(B), "ref": _reference_vector(n), "n": n, **_outputs(pairs, n)}
    if call == "solver":
        s["solver"] = _solver(n, case["precision"])
    return s


# ------------------------------------------------------------------ one pass

def _fix_phase(V, ref):
    """V: one eigenvector per row; each turned so that its overlap with ref is real and positive."""
    z = V @ ref
    return V.mul_((z.conj() / z.abs())[:, None])


def run(s):
    if s["call"] == "spinwave":
        s["model"].solve(s["solver"], s["q"], s["W"], s["info"], I=s["I"])
        return {"W": s["W"], "I": s["I"], "info": s["info"]}
    if s["call"] == "queue":
        s["queue"].launch(s["A"], s["B"], s["W"], s["X"], s["info"])
        # the modes of each order, as the program goes on with them
        X = {str(n): _fix_phase(s["X"][at].view(-1, n), s["ref"][n]) for n, at in s["at"].items()}
        return {"W": s["W"], "X": X, "info": s["info"]}
    if s["call"] == "dropin":
        sbg.geneig_full_n54_batched(s["A"], s["B"], s["W"], s["X"], s["info"])
    else:
        s["solver"].launch(s["A"], s["B"], s["W"], s["X"], s["info"])
    _fix_phase(s["X"].view(-1, s["n"]), s["ref"])
    return {"W": s["W"], "X": s["X"], "info": s["info"]}


# ------------------------------------------------------------------ work and exact values

def _count(case):
    """(order, pairs of it) of the case."""
    if case["call"] != "queue":
        return [(case["n"], case["pairs"])]
    ns = workloads.uneven_sizes(case["pairs"])
    return [(int(n), int((ns == n).sum())) for n in np.unique(ns)]


def work(case):
    """LAPACK's counts for Cholesky (4/3 n^3), the two-sided reduction (4), the tridiagonalisation
    (16/3), Q Z (8) and the last triangular solve (4), real flops; the tridiagonal eigensolve is
    O(n^2).  Bytes: A in full, B's lower triangle, W, X, info; a sweep reads q and writes W and I."""
    flops = sum(68.0 / 3.0 * n ** 3 * p for n, p in _count(case))
    if case["call"] == "spinwave":
        return {"bytes": case["pairs"] * (24 + 16 * case["n"] + 4), "flops": flops}
    return {"bytes": sum(p * (16 * n * n + 8 * n * (n + 1) + 8 * n + 16 * n * n + 4) for n, p in _count(case)),
            "flops": flops}


def _exact_pairs(A, B):
    """(W, X) by Cholesky, triangular solves and eigh; X with one eigenvector per row."""
    L = torch.linalg.cholesky(B)
    C = torch.linalg.solve_triangular(L, A, upper=False)
    C = torch.linalg.solve_triangular(L, C.mH, upper=False)
    W, Y = torch.linalg.eigh((C + C.mH) / 2)
    return W, torch.linalg.solve_triangular(L.mH, Y, upper=True).mT


def _exact_modes(A, B):
    """W and the phase-fixed X, in pieces."""
    n = A.shape[-1]
    Ws, Xs = [], []
    for a, b in zip(A.split(2048), B.split(2048)):
        W, X = _exact_pairs(a, b)
        Ws.append(W)
        Xs.append(_fix_phase(X.reshape(-1, n).contiguous(), _reference_vector(n)))
    return torch.cat(Ws), torch.cat(Xs)


def exact(case, seed):
    if case["call"] == "queue":
        ns, at, A, B = _queue_inputs(case["pairs"], seed)
        first = np.concatenate([[0], np.cumsum(ns.astype(np.int64))])[:-1]
        Wall, X = torch.empty(int(ns.sum()), dtype=torch.float64, device=DEV), {}
        for n, i in at.items():
            W, X[str(n)] = _exact_modes(A[i].view(-1, n, n).mT, B[i].view(-1, n, n).mT)
            Wall[(torch.as_tensor(first[ns == n], device=DEV)[:, None] + torch.arange(n, device=DEV))] = W
        return {"W": Wall, "X": X, "info": None}
    n, pairs = case["n"], case["pairs"]
    if case["call"] == "spinwave":
        cell, field, q = _sweep_inputs(case, seed)
        B = _cell_B(n // 2, cell, q) + field * torch.eye(n, dtype=torch.complex128, device=DEV)
        W, X = _exact_modes(_metric(n, pairs), B)
        X = X.view(pairs, n, n)
        ph = torch.exp(-1j * (q @ torch.as_tensor(cell[3], device=DEV).T))
        F = ((X[:, :, :n // 2] + X[:, :, n // 2:]) @ ph[:, :, None]).squeeze(2)
        return {"W": W, "I": F.abs() ** 2 / (n // 2 * W.abs()), "info": None}
    W, X = _exact_modes(*_pairs(case["kind"], n, pairs, seed))
    return {"W": W, "X": X.view(pairs, n * n), "info": None}
