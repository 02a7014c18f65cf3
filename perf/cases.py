"""The workloads this package's speed is measured on.

Each case is one piece of work that a user has the package do through its
public entry points (`kernels`, `panelblas`, the panel matrices), on data that
is already where such a program keeps it: device matrices for the resident
calls, page-locked host panels for the range finders. `listed()` names the
sizes that stand for each kind of use, `draw(rng)` gives other sizes of the
same kinds, `prepare` makes a case's inputs from a seed, `run` is one pass,
`work` the bytes and operations a pass cannot do without, and `exact` the same
result from torch alone, in 64 bits.

Sizes follow the repository's own configurations: the 2^20 x 32 and 10^7 x 64
orthonormalizations, 128 columns, the uneven batch with N in [10^4, 2*10^6] and
k in {16, 32, 64}, the 215^3 and 342^3 grids, the band operator with 64
superdiagonals, panels of width 3 and 8, and the 4096 x 16 matrix of the smoke
run.
"""
import math
import random

import numpy as np
import torch

import __graft_entry__

fb = __graft_entry__.load()
K = fb.kernels
Z = torch.complex128

_backend = None


def backend():
    global _backend
    if _backend is None:
        _backend = fb.B200Backend(0)
    return _backend


def listed():
    return [
        # One small orthonormalization, as in the inner loop of a block solver:
        # all latency.
        {"name": "cholqr2_small", "kind": "cholqr2", "N": 4096, "k": 16, "kappa": 1.0},
        # A sketch of a million rows: a few passes over half a gigabyte.
        {"name": "cholqr2_2p20_k32", "kind": "cholqr2", "N": 1 << 20, "k": 32, "kappa": 1.0},
        # The headline orthonormalization: ill-conditioned, ten gigabytes.
        {"name": "cholqr2_1e7_k64", "kind": "cholqr2", "N": 10_000_000, "k": 64, "kappa": 1e6},
        # More columns than one tile holds, and a ragged last row block.
        {"name": "cholqr2_wide_k128", "kind": "cholqr2", "N": 2_500_003, "k": 128, "kappa": 1e4},
        # Many independent matrices of uneven size in one call.
        {"name": "cholqr2_batch", "kind": "batch", "count": 32, "low": 10_000, "high": 1_000_000, "shapes": 7},
        # The device half of a streamed pass: two row blocks (the second one
        # ragged), each solved against R and accumulated into the next Gram.
        {"name": "stream_pass", "kind": "stream", "rows": 1_875_079, "last": 1_234_567, "k": 64, "kappa": 1e6},
        # Q^H (G Q) for the 7-point Laplacian, everything resident.
        {"name": "project_215", "kind": "project", "nx": 215, "ny": 215, "nz": 215, "k": 64},
        # Forward pass and both pullbacks of a loss through cholqr2! and
        # project, G a Hermitian band.
        {"name": "adjoint_2p20", "kind": "adjoint", "N": 1 << 20, "k": 64, "kd": 64},
        # Y C with a square factor.
        {"name": "rightmul", "kind": "rightmul", "N": 2_500_003, "s": 64, "r": 64},
        # One panel of a randomized sketch: seeded Gaussian columns generated
        # on the device and the operator applied to them.
        {"name": "sketch_342_w3", "kind": "sketch", "nx": 342, "ny": 342, "nz": 342, "w": 3},
        # The whole range finder on page-locked host panels, Float64 storage
        # and ComplexF32 storage (with the shifted CholeskyQR3).
        {"name": "range_finder", "kind": "range", "nx": 96, "ny": 97, "nz": 95, "k": 32, "w": 8, "narrow": False},
        {"name": "range_finder_c64", "kind": "range", "nx": 64, "ny": 65, "nz": 63, "k": 48, "w": 12, "narrow": True},
    ]


def draw(rng):
    """One more case of the ranges above."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["cholqr2", "cholqr2", "cholqr2", "cholqr2", "batch", "stream", "project", "adjoint", "rightmul",
                       "sketch", "range"])
    if kind == "cholqr2":
        k = log(5, 160)
        N = log(max(1000, 4 * k), 10_000_000)
        # Never more arithmetic or memory than the largest listed case.
        N = min(N, int(4.0e10 / k ** 2), int(6.0e8 / k))
        return {"kind": kind, "N": N, "k": k, "kappa": rng.choice([1.0, 1e2, 1e4, 1e6])}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 32), "low": log(2_000, 20_000), "high": log(50_000, 1_000_000),
                "shapes": rng.randrange(1 << 30)}
    if kind == "stream":
        rows = log(20_000, 2_500_000)
        return {"kind": kind, "rows": rows, "last": rng.randint(rows // 8, rows), "k": log(8, 100),
                "kappa": rng.choice([1e2, 1e4, 1e6])}
    if kind == "project":
        return {"kind": kind, "nx": log(24, 215), "ny": log(24, 215), "nz": log(24, 215), "k": log(5, 64)}
    if kind == "adjoint":
        return {"kind": kind, "N": log(20_000, 1 << 20), "k": log(8, 64), "kd": rng.choice([3, 16, 40, 64])}
    if kind == "rightmul":
        return {"kind": kind, "N": log(5_000, 2_500_000), "s": log(4, 100), "r": log(4, 100)}
    if kind == "sketch":
        return {"kind": kind, "nx": log(24, 342), "ny": log(24, 342), "nz": log(24, 342), "w": log(1, 12)}
    k = rng.choice([16, 24, 32, 40, 48])
    nx, ny = log(24, 96), log(24, 96)
    return {"kind": kind, "nx": nx, "ny": ny, "nz": min(log(24, 96), int(2.8e7 / (k * nx * ny))), "k": k,
            "w": rng.choice([6, 8, 12]), "narrow": rng.random() < 0.4}


# ---- inputs ----------------------------------------------------------------

def _cuda():
    return torch.device("cuda", 0)


def _matrix(t):
    """The N x k column-major device matrix over a (k, N) tensor."""
    return fb.DeviceMatrix(t.data_ptr(), (t.shape[1], t.shape[0]), t.shape[1], np.dtype(np.complex128), t)


def _generator(seed):
    g = torch.Generator(device=_cuda())
    g.manual_seed(int(seed))
    return g


def _gaussian(g, k, N):
    return torch.randn((k, N), dtype=Z, device=_cuda(), generator=g)


def _conditioned(g, k, N, kappa):
    """Columns of an N x k Gaussian times diag(s) V^H, s log-spaced from 1 to
    1/kappa, V unitary: the (k, N) transpose of it."""
    x = _gaussian(g, k, N)
    if kappa <= 1.0 or k == 1:
        return x
    V = torch.linalg.qr(_gaussian(g, k, k))[0]
    s = torch.logspace(0, -math.log10(kappa), k, dtype=torch.float64, device=_cuda())
    C = s.to(Z)[:, None] * V.conj().T
    return torch.matmul(C.T, x)


def _empty(k, N):
    return torch.empty((k, N), dtype=Z, device=_cuda())


def _batch_shapes(case):
    rng = random.Random(case["shapes"])
    lo, hi = math.log(case["low"]), math.log(case["high"])
    return [(int(math.exp(rng.uniform(lo, hi))), rng.choice([16, 32, 64])) for _ in range(case["count"])]


def _split(flat, shapes):
    out, at = [], 0
    for N, k in shapes:
        out.append(flat[at:at + N * k].view(k, N))
        at += N * k
    return out


def _upper(Yt):
    """The R of Yt's matrix, upper triangular with a positive diagonal, as the
    (k, k) transpose of it."""
    G = torch.matmul(Yt.conj(), Yt.T)
    return torch.linalg.cholesky(0.5 * (G + G.conj().T)).conj().contiguous()


def _range_plan(case):
    N = case["nx"] * case["ny"] * case["nz"]
    return fb.ResidencyPlan(device_budget=8 * N * case["k"] * 16 + 2 * fb.GiB,
                            host_budget=4 * N * case["k"] * 16 + fb.GiB, backend=backend(),
                            host_eltype=np.complex64 if case["narrow"] else None)


def prepare(case, seed):
    b = backend()
    kind = case["kind"]
    if kind == "range":
        plan = _range_plan(case)
        N = case["nx"] * case["ny"] * case["nz"]
        X = fb.GhostPanels(np.complex128, N, case["k"], plan=plan, seed=int(seed), w=case["w"])
        Y = fb.PanelMatrix.undef(np.complex128, N, case["k"], plan=plan, w=case["w"])
        G = fb.Laplacian7((case["nx"], case["ny"], case["nz"]), 0.5 + 0.1j)
        return {"kind": kind, "X": X, "Y": Y, "G": G, "narrow": case["narrow"]}
    g = _generator(seed)
    if kind == "cholqr2":
        N, k = case["N"], case["k"]
        s = {"Y": _conditioned(g, k, N, case["kappa"]), "Q": _empty(k, N), "R": _empty(k, k)}
        s |= {"Qm": _matrix(s["Q"]), "Rm": _matrix(s["R"])}
    elif kind == "batch":
        shapes = _batch_shapes(case)
        total, small = sum(N * k for N, k in shapes), sum(k * k for _, k in shapes)
        s = {"Y": torch.randn(total, dtype=Z, device=_cuda(), generator=g),
             "Q": torch.empty(total, dtype=Z, device=_cuda()), "R": torch.empty(small, dtype=Z, device=_cuda())}
        s["Qms"] = [_matrix(t) for t in _split(s["Q"], shapes)]
        s["Rms"] = [_matrix(t) for t in _split(s["R"], [(k, k) for _, k in shapes])]
    elif kind == "stream":
        N, k = case["rows"] + case["last"], case["k"]
        Y = _conditioned(g, k, N, case["kappa"])
        s = {"Y": Y, "R": _upper(Y), "Q": _empty(k, N), "G": _empty(k, k)}
        s |= {"Qm": _matrix(s["Q"]), "Rm": _matrix(s["R"]), "Gm": _matrix(s["G"]),
              "blocks": [(0, case["rows"]), (case["rows"], N)]}
    elif kind == "project":
        grid = (case["nx"], case["ny"], case["nz"])
        N, k = grid[0] * grid[1] * grid[2], case["k"]
        s = {"Q": _gaussian(g, k, N), "GQ": _empty(k, N), "S": _empty(k, k)}
        s["Q"].mul_(1.0 / math.sqrt(N))
        s |= {"Qm": _matrix(s["Q"]), "GQm": _matrix(s["GQ"]), "Sm": _matrix(s["S"]),
              "G": fb.Laplacian7(grid, 0.5 + 0.1j)}
    elif kind == "adjoint":
        N, k, kd = case["N"], case["k"], case["kd"]
        s = {"Y": _gaussian(g, k, N), "W": _gaussian(g, k, N), "D": _gaussian(g, kd + 1, N)}
        s["D"].mul_(math.sqrt(N / ((2 * kd + 1) * k)))
        s |= {n: _empty(k, N) for n in ("Q", "GQ", "Qbar")} | {n: _empty(k, k) for n in ("R", "S", "T")}
        s |= {n + "m": _matrix(s[n]) for n in ("Y", "W", "Q", "GQ", "Qbar", "R", "S", "T")}
        s["G"] = fb.HermitianBand(b, _matrix(s["D"]))
    elif kind == "rightmul":
        N, m, r = case["N"], case["s"], case["r"]
        s = {"A": _gaussian(g, m, N), "C": _gaussian(g, r, m), "D": _empty(r, N)}
        s |= {n + "m": _matrix(s[n]) for n in ("A", "C", "D")}
    else:
        grid = (case["nx"], case["ny"], case["nz"])
        N, w = grid[0] * grid[1] * grid[2], case["w"]
        s = {"seed": int(seed), "X": _empty(w, N), "Y": _empty(w, N), "G": fb.Laplacian7(grid, 0.5 + 0.1j)}
        s |= {"Xm": _matrix(s["X"]), "Ym": _matrix(s["Y"])}
    s["kind"] = kind
    return s


# ---- one pass ----------------------------------------------------------------

def run(state):
    b, s = backend(), state
    kind = s["kind"]
    if kind == "cholqr2":
        # cholqr2! works in place, so a program that keeps Y copies it first.
        s["Q"].copy_(s["Y"])
        K.cholqr2_resident(b, s["Qm"], s["Rm"])
        return {"Q": s["Q"], "R": s["R"]}
    if kind == "batch":
        s["Q"].copy_(s["Y"])
        K.cholqr2_batched(b, s["Qms"], s["Rms"])
        return {"Q": s["Q"], "R": s["R"]}
    if kind == "stream":
        # The copy stands where the sweep's upload puts a row block.
        every = slice(None)
        for step, (r0, r1) in enumerate(s["blocks"]):
            block = s["Qm"].view(slice(r0, r1), every)
            s["Q"][:, r0:r1].copy_(s["Y"][:, r0:r1])
            K.rdiv_upper(b, block, s["Rm"])
            K.gram_accumulate(b, s["Gm"], block, block, 1.0, 0.0 if step == 0 else 1.0)
        return {"Q": s["Q"], "G": s["G"]}
    if kind == "project":
        s["G"].apply(b, s["GQm"], s["Qm"])
        K.gram_accumulate(b, s["Sm"], s["Qm"], s["GQm"], 1.0, 0.0)
        return {"GQ": s["GQ"], "S": s["S"]}
    if kind == "adjoint":
        # loss = Re tr(W^H Q) + ||Q^H G Q||_F^2 of (Q, R) = cholqr2!(Y).
        s["Q"].copy_(s["Y"])
        K.cholqr2_resident(b, s["Qm"], s["Rm"], wait=False)
        s["G"].apply(b, s["GQm"], s["Qm"])
        K.gram_accumulate(b, s["Sm"], s["Qm"], s["GQm"], 2.0, 0.0)
        K.gram_accumulate(b, s["Tm"], s["Wm"], s["Qm"], 1.0, 0.0)
        s["Qbar"].copy_(s["W"])
        K.project_adjoint(b, s["Qbarm"], s["GQm"], s["Sm"], None, accumulate=True)
        K.cholqr2_adjoint(b, s["Qbarm"], s["Ym"], s["Rm"], s["Qbarm"], None)
        return {"R": s["R"], "S": s["S"], "T": s["T"], "Ybar": s["Qbar"]}
    if kind == "rightmul":
        K.rightmul_gemm(b, s["Dm"], s["Am"], s["Cm"])
        return {"D": s["D"]}
    if kind == "sketch":
        K.ghost_fill(b, s["Xm"], 0, 0, s["seed"], np.complex128)
        s["G"].apply(b, s["Ym"], s["Xm"])
        return {"X": s["X"], "Y": s["Y"]}
    fb.panelmul(s["Y"], s["G"], s["X"])
    R = fb.cholqr3(s["Y"]) if s["narrow"] else fb.cholqr2(s["Y"])
    S = fb.project(s["Y"], s["G"])
    return {"Q": [p.storage() for p in s["Y"].panels], "R": R, "S": S}


# ---- what a pass cannot do without ---------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "cholqr2":
        N, k = case["N"], case["k"]
        return {"bytes": 32.0 * N * k + 16.0 * k * k, "flops": 16.0 * N * k * k}
    if kind == "batch":
        shapes = _batch_shapes(case)
        return {"bytes": sum(32.0 * N * k + 16.0 * k * k for N, k in shapes), "flops": sum(16.0 * N * k * k for N, k in shapes)}
    if kind == "stream":
        N, k = case["rows"] + case["last"], case["k"]
        return {"bytes": 32.0 * N * k + 32.0 * k * k, "flops": 8.0 * N * k * k}
    if kind == "project":
        N, k = case["nx"] * case["ny"] * case["nz"], case["k"]
        return {"bytes": 32.0 * N * k + 16.0 * k * k, "flops": 8.0 * N * k * k + 16.0 * N * k}
    if kind == "adjoint":
        N, k, kd = case["N"], case["k"], case["kd"]
        flops = 16.0 * N * k * k + 8.0 * N * k * (2 * kd + 1) + 16.0 * N * k * k + 8.0 * N * k * k + 20.0 * N * k * k
        return {"bytes": 16.0 * N * (3 * k + kd + 1) + 48.0 * k * k, "flops": flops}
    if kind == "rightmul":
        N, m, r = case["N"], case["s"], case["r"]
        return {"bytes": 16.0 * (N * (m + r) + m * r), "flops": 8.0 * N * m * r}
    if kind == "sketch":
        N, w = case["nx"] * case["ny"] * case["nz"], case["w"]
        return {"bytes": 32.0 * N * w, "flops": 80.0 * N * w}
    N, k = case["nx"] * case["ny"] * case["nz"], case["k"]
    return {"bytes": (8.0 if case["narrow"] else 16.0) * N * k + 32.0 * k * k,
            "flops": (24.0 if case["narrow"] else 16.0) * N * k * k + 8.0 * N * k * k + 112.0 * N * k}


# ---- the same results from torch ------------------------------------------------

def _qr(Yt):
    """(Q^T, R^T) of Yt's matrix, R with a positive diagonal."""
    Q, R = torch.linalg.qr(Yt.T)
    d = torch.diagonal(R)
    ph = d / d.abs()
    return (Q * ph).T, (R * ph.conj()[:, None]).T


def _laplace(xt, grid, shift):
    """(6 + shift) v minus the six neighbours, per row of xt."""
    nx, ny, nz = grid
    out = torch.empty_like(xt)
    for c in range(xt.shape[0]):
        v = xt[c].view(nz, ny, nx)
        o = v * (6.0 + shift)
        o[1:] -= v[:-1]
        o[:-1] -= v[1:]
        o[:, 1:] -= v[:, :-1]
        o[:, :-1] -= v[:, 1:]
        o[:, :, 1:] -= v[:, :, :-1]
        o[:, :, :-1] -= v[:, :, 1:]
        out[c] = o.reshape(-1)
    return out


def _philox_gaussian(seed, N, cols):
    """The complex normals of a ghost matrix: Philox4x32-10 with counter (row,
    column) and the seed as key, then Box and Muller."""
    out = _empty(cols, N)
    low = (1 << 32) - 1
    row = torch.arange(N, dtype=torch.int64, device=_cuda())
    for col in range(cols):
        c = [row & low, row >> 32, torch.full_like(row, col & low), torch.full_like(row, col >> 32)]
        k0, k1 = seed & low, (seed >> 32) & low
        for _ in range(10):
            p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
            c = [((p1 >> 32) & low) ^ c[1] ^ k0, p1 & low, ((p0 >> 32) & low) ^ c[3] ^ k1, p0 & low]
            k0, k1 = (k0 + 0x9E3779B9) & low, (k1 + 0xBB67AE85) & low
        n1 = ((c[0] << 21) | (c[1] >> 11)) + 1
        b2 = (c[2] << 21) | (c[3] >> 11)
        rad = torch.sqrt(-torch.log(n1.to(torch.float64) * 2.0 ** -53))
        ang = b2.to(torch.float64) * (2.0 ** -53 * 2.0 * math.pi)
        out[col] = torch.complex(rad * torch.cos(ang), rad * torch.sin(ang))
    return out


def _band(Dt, xt):
    """The Hermitian band stored by diagonals in the rows of Dt, on rows of xt."""
    N = xt.shape[1]
    y = xt * Dt[0].real
    for d in range(1, Dt.shape[0]):
        if d >= N:
            break
        e = Dt[d, :N - d]
        y[:, :N - d] += e * xt[:, d:]
        y[:, d:] += e.conj() * xt[:, :N - d]
    return y


def exact(case, seed):
    kind = case["kind"]
    if kind == "range":
        grid = (case["nx"], case["ny"], case["nz"])
        N, w, k = grid[0] * grid[1] * grid[2], case["w"], case["k"]
        X = _philox_gaussian(int(seed), N, k)
        q, r = _qr(_laplace(X, grid, 0.5 + 0.1j))
        S = torch.matmul(q.conj(), _laplace(q.contiguous(), grid, 0.5 + 0.1j).T)
        kept = np.complex64 if case["narrow"] else np.complex128
        Q = q.T.cpu().numpy().astype(kept)
        return {"Q": [np.asfortranarray(Q[:, j:j + w]) for j in range(0, k, w)],
                "R": np.asfortranarray(r.T.cpu().numpy()), "S": np.asfortranarray(S.cpu().numpy())}
    g = _generator(seed)
    if kind == "cholqr2":
        q, r = _qr(_conditioned(g, case["k"], case["N"], case["kappa"]))
        return {"Q": q, "R": r}
    if kind == "batch":
        shapes = _batch_shapes(case)
        Y = torch.randn(sum(N * k for N, k in shapes), dtype=Z, device=_cuda(), generator=g)
        pairs = [_qr(t) for t in _split(Y, shapes)]
        return {"Q": torch.cat([q.reshape(-1) for q, _ in pairs]), "R": torch.cat([r.reshape(-1) for _, r in pairs])}
    if kind == "stream":
        Y = _conditioned(g, case["k"], case["rows"] + case["last"], case["kappa"])
        Q = torch.linalg.solve_triangular(_upper(Y), Y, upper=False)
        return {"Q": Q, "G": torch.matmul(Q.conj(), Q.T).T}
    if kind == "project":
        grid = (case["nx"], case["ny"], case["nz"])
        N = grid[0] * grid[1] * grid[2]
        Q = _gaussian(g, case["k"], N).mul_(1.0 / math.sqrt(N))
        GQ = _laplace(Q, grid, 0.5 + 0.1j)
        return {"GQ": GQ, "S": torch.matmul(Q.conj(), GQ.T).T}
    if kind == "adjoint":
        N, k, kd = case["N"], case["k"], case["kd"]
        Y, W, D = _gaussian(g, k, N), _gaussian(g, k, N), _gaussian(g, kd + 1, N)
        D.mul_(math.sqrt(N / ((2 * kd + 1) * k)))
        q, r = _qr(Y)
        q = q.contiguous()
        GQ = _band(D, q)
        S = 2.0 * torch.matmul(q.conj(), GQ.T)
        T = torch.matmul(W.conj(), q.T)
        Qbar = W + torch.matmul((S + S.conj().T).T, GQ)
        M = -torch.matmul(Qbar.conj(), q.T)
        L = torch.tril(M, -1)
        H = L + L.conj().T + torch.diag(torch.diagonal(M).real.to(Z))
        B = Qbar + torch.matmul(H.T, q)
        # Ybar R^H = B, transposed: conj(R) Ybar^T = B^T.
        Ybar = torch.linalg.solve_triangular(r.T.conj(), B, upper=True)
        return {"R": r, "S": S.T, "T": T.T, "Ybar": Ybar}
    if kind == "rightmul":
        A, C = _gaussian(g, case["s"], case["N"]), _gaussian(g, case["r"], case["s"])
        return {"D": torch.matmul(C, A)}
    grid = (case["nx"], case["ny"], case["nz"])
    X = _philox_gaussian(int(seed), grid[0] * grid[1] * grid[2], case["w"])
    return {"X": X, "Y": _laplace(X, grid, 0.5 + 0.1j)}
