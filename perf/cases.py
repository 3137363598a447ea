"""The work that programs have this library do, as cases for measuring it.

A case names one public entry point (or the short sequence that a program runs) and its sizes:

  spmv      y = A x of a square operator                                  Mat.mult
  lanczos   the Lanczos run between two restarts, columns k..m            BV.matLanczos
  restart   the basis update V(:, 0:e) = V(:, 0:k) Q of a thick restart   BV.multInPlace
  solve     a whole eigensolve, eigenpairs left on the GPU                EPS.solve
  dot       the Gram matrix Y^T X of two blocks                           BV.dot
  combine   Y = X Q + Y, Ritz vectors from a block                        BV.mult
  orth      Cholesky orthogonalisation of a block                         BV.orthogonalize
  filter    Y = alpha (A X - shift X) - beta Z on row-major blocks        rowblock_spmm
  aij       y = A x and z = A^T w of a rectangular power-law matrix       Mat.mult, Mat.multTranspose
  batch     many small eigenproblems in one launch                        BatchEPS.solve
  neural    loss and gradients of the neural warm start                   NeuralOperator.lossGrad

`listed` has one or two of each, `draw` others from the ranges between and around them.
"""
import math

import numpy as np
import torch

import slepc_b200 as S
from slepc_b200 import learned as LN
from slepc_b200 import problems as P

F64 = torch.float64


def listed():
    return [
        # the operator of the library's headline eigenproblem, applied once per Lanczos step
        {"name": "spmv_lap3d_128", "kind": "spmv", "op": "lap3d", "a": 128, "b": 128, "c": 128},
        # a desktop-size eigenproblem (the 2-D Laplacian of the tutorials): every launch counts
        {"name": "lanczos_lap2d_100", "kind": "lanczos", "op": "lap2d", "a": 100, "b": 100, "c": 1, "k": 16, "m": 32},
        # one thick-restart cycle of the headline eigenproblem: ncv 80, half of the basis kept
        {"name": "lanczos_lap3d_128", "kind": "lanczos", "op": "lap3d", "a": 128, "b": 128, "c": 128, "k": 40, "m": 80},
        # the basis update at the end of that cycle
        {"name": "restart_128", "kind": "restart", "n": 2097152, "k": 80, "e": 56},
        # a whole small solve of a heterogeneous-medium operator, with the tutorial's grid
        {"name": "solve_diffusion_72", "kind": "solve", "a": 72, "b": 75, "nev": 4, "ncv": 20},
        # the projected matrices of a block step with blocks [X R P] of 16 on a 512 x 512 grid
        {"name": "dot_512_48", "kind": "dot", "n": 262144, "kx": 48, "ky": 48},
        # the block orthogonalisation of that step
        {"name": "orth_512_16", "kind": "orth", "n": 262144, "l": 0, "k": 16},
        # one degree of the Chebyshev filter of the mixed-precision form on the headline operator
        {"name": "filter_128_f32", "kind": "filter", "a": 128, "b": 128, "c": 128, "x32": True, "bp": 64},
        # both halves of one application of A^T A in the cross-product SVD, values stored in FP32
        {"name": "aij_f32_200k", "kind": "aij", "m": 200000, "n": 50000, "row": 20, "f32": True},
        # a batch of k-NN graph operators, eight pairs of each
        {"name": "batch_knn_192", "kind": "batch", "nprob": 192, "lo": 500, "hi": 4000, "nev": 8, "ncv": 24},
        # a training gradient of the warm-start network on coarse fields, and on full-size ones
        {"name": "neural_64", "kind": "neural", "N": 64, "B": 16},
        {"name": "neural_512", "kind": "neural", "N": 512, "B": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, op, lo, hi):
    """Grid edges, odd ones among them, with between lo and hi points."""
    n = _log(rng, lo, hi)
    if op == "lap3d":
        a = max(8, int(n ** (1 / 3) * rng.uniform(0.8, 1.2)))
        b = max(8, int(n ** (1 / 3) * rng.uniform(0.8, 1.2)))
        c = max(4, min(n // (a * b), hi // (a * b)))
        return a, b, c
    a = max(8, int(n ** 0.5 * rng.uniform(0.7, 1.4)))
    return a, max(8, min(n // a, hi // a)), 1


def draw(rng):
    kind = rng.choice(["spmv", "lanczos", "lanczos", "restart", "solve", "dot", "combine", "orth", "filter", "aij",
                       "batch", "neural"])
    if kind == "spmv":
        op = rng.choice(["lap2d", "lap3d", "diffusion", "knn"])
        if op == "knn":
            return {"kind": kind, "op": op, "a": _log(rng, 500, 20000), "b": 1, "c": 1}
        a, b, c = _grid(rng, op, 10000, 2000000)
        return {"kind": kind, "op": op, "a": a, "b": b, "c": c}
    if kind == "lanczos":
        op = rng.choice(["lap2d", "lap3d", "diffusion", "knn"])
        m = rng.randint(18, 80)
        k = rng.randint(0, m // 2)
        if op == "knn":
            return {"kind": kind, "op": op, "a": _log(rng, 1000, 20000), "b": 1, "c": 1, "k": k, "m": m}
        a, b, c = _grid(rng, op, 5000, 1200000)
        return {"kind": kind, "op": op, "a": a, "b": b, "c": c, "k": k, "m": m}
    if kind == "restart":
        k = rng.randint(16, 80)
        return {"kind": kind, "n": _log(rng, 20000, 2000000), "k": k, "e": rng.randint(k // 2, (3 * k) // 4)}
    if kind == "solve":
        nev = rng.randint(2, 6)
        return {"kind": kind, "a": rng.randint(48, 80), "b": rng.randint(48, 80), "nev": nev,
                "ncv": rng.randint(2 * nev + 12, 40)}
    if kind == "dot":
        return {"kind": kind, "n": _log(rng, 16000, 262144), "kx": rng.randint(8, 48), "ky": rng.randint(8, 48)}
    if kind == "combine":
        return {"kind": kind, "n": _log(rng, 16000, 262144), "kx": rng.randint(8, 48), "ky": rng.randint(4, 24)}
    if kind == "orth":
        l = rng.randint(0, 16)
        return {"kind": kind, "n": _log(rng, 16000, 262144), "l": l, "k": l + rng.randint(4, 24)}
    if kind == "filter":
        a, b, c = _grid(rng, "lap3d", 60000, 900000)
        return {"kind": kind, "a": a, "b": b, "c": c, "x32": rng.random() < 0.75, "bp": 64}
    if kind == "aij":
        m = _log(rng, 10000, 200000)
        return {"kind": kind, "m": m, "n": max(500, int(m * rng.uniform(0.1, 0.5))), "row": rng.randint(6, 20),
                "f32": rng.random() < 0.7}
    if kind == "batch":
        lo = rng.randint(300, 800)
        nev = rng.randint(4, 8)
        return {"kind": kind, "nprob": _log(rng, 24, 192), "lo": lo, "hi": rng.randint(lo + 500, 4000), "nev": nev,
                "ncv": rng.randint(2 * nev + 6, 24)}
    N = _log(rng, 32, 384)
    return {"kind": "neural", "N": N, "B": rng.randint(1, max(1, min(16, 400000 // (N * N))))}


# ------------------------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(seed, *shape, dtype=F64):
    return torch.randn(*shape, generator=_gen(seed), dtype=dtype, device="cuda")


def _field(seed, a, b, corr=0.1):
    """exp of a smooth Gaussian field on an a x b grid: the coefficient of a heterogeneous medium."""
    ky = torch.fft.fftfreq(2 * a, d=1.0 / a, device="cuda", dtype=F64)
    kx = torch.fft.fftfreq(2 * b, d=1.0 / b, device="cuda", dtype=F64)
    damp = torch.exp(-math.pi ** 2 * corr ** 2 * (ky[:, None] ** 2 + kx[None, :] ** 2))
    f = torch.fft.ifft2(torch.fft.fft2(_randn(seed, 2 * a, 2 * b)) * damp).real[:a, :b]
    f = f - f.mean()
    return torch.exp(f / f.std())


def _grid_csr(dims, kappa=None):
    """CSR of the grid Laplacian (dims slowest first, zero outside), or of -div(kappa grad u) with harmonic-mean
    faces; columns ascend within a row.  Everything is built on the GPU."""
    N = math.prod(dims)
    idx = torch.arange(N, device="cuda").view(dims)
    cell = torch.ones(dims, dtype=F64, device="cuda") if kappa is None else kappa
    diag = torch.zeros(dims, dtype=F64, device="cuda")
    minus, plus = [], []
    for ax, d in enumerate(dims):
        if d == 1 and len(dims) == 3 and kappa is not None:
            continue
        lo, hi = cell.narrow(ax, 0, d - 1), cell.narrow(ax, 1, d - 1)
        face = 2 * lo * hi / (lo + hi)
        wall = 1.0 if kappa is None else 2.0
        diag.narrow(ax, 0, d - 1).add_(face)
        diag.narrow(ax, 1, d - 1).add_(face)
        diag.narrow(ax, 0, 1).add_(wall * cell.narrow(ax, 0, 1))
        diag.narrow(ax, d - 1, 1).add_(wall * cell.narrow(ax, d - 1, 1))
        for lst, at, frm in ((minus, 1, 0), (plus, 0, 1)):
            c = torch.full(dims, -1, device="cuda")
            v = torch.zeros(dims, dtype=F64, device="cuda")
            c.narrow(ax, at, d - 1).copy_(idx.narrow(ax, frm, d - 1))
            v.narrow(ax, at, d - 1).copy_(-face)
            lst.append((c.reshape(-1), v.reshape(-1)))
    every = minus + [(idx.reshape(-1), diag.reshape(-1))] + plus[::-1]
    cols = torch.stack([c for c, _ in every], dim=1)
    vals = torch.stack([v for _, v in every], dim=1)
    mask = cols >= 0
    rowptr = torch.zeros(N + 1, dtype=torch.int32, device="cuda")
    rowptr[1:] = mask.sum(1).cumsum(0).to(torch.int32)
    return rowptr, cols[mask].to(torch.int32).contiguous(), vals[mask].contiguous()


def _operator(case, seed):
    """(rowptr, colind, vals) on the GPU of a square case's operator."""
    if case["op"] == "knn":
        return tuple(torch.from_numpy(v).cuda() for v in P.knn_operator(case["a"], 8, seed))
    dims = (case["c"], case["b"], case["a"]) if case["op"] == "lap3d" else (case["b"], case["a"])
    return _grid_csr(dims, _field(seed, *dims) if case["op"] == "diffusion" else None)


def _mat(csr):
    torch.cuda.synchronize()  # the library copies the arrays on its own stream
    rowptr, colind, vals = csr
    return S.Mat().createAIJDevice(rowptr.numel() - 1, colind.numel(), rowptr.data_ptr(), colind.data_ptr(),
                                   vals.data_ptr())


class _Device:
    """FP64 device memory of the library as a tensor."""

    def __init__(self, ptr, shape, strides=None):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f8", "version": 3,
                                         "strides": strides}


def _columns(bv, m):
    n, _, ld = bv.getSizes()
    return torch.as_tensor(_Device(bv.getArrayPointer(), (m, ld)), device="cuda")[:, :n]


def _basis(X):
    """A BV whose columns are the rows of X."""
    m, n = X.shape
    bv = S.BV().create(n, m)
    _columns(bv, m).copy_(X)
    bv.setActiveColumns(0, m)
    return bv


def _theta(seed, N):
    # every parameter is nonzero, as after the first training steps
    dims = _dims(N)
    theta = LN.init_params(*dims, seed=seed)
    rng = np.random.default_rng([seed, 1])
    return (theta + 0.02 * rng.standard_normal(theta.size)).astype(np.float32)


def _dims(N):
    d = LN.DEFAULT_DIMS
    return N, d["width"], min(d["modes"], N), d["layers"], d["hidden"], 16


def _neural_data(seed, N, B):
    c = (torch.arange(N, device="cuda", dtype=F64) + 0.5) / N
    yy, xx = torch.meshgrid(c, c, indexing="ij")
    feats, targets = [], []
    for b in range(B):
        kap = _field(1000 * seed + b, N, N, 0.05 + 0.15 * b / B)
        feats.append(torch.stack([kap.log(), xx, yy]))
        # smooth orthogonal modes bent by the medium, unit norm: what the eigenvectors look like
        t = torch.stack([torch.sin(math.pi * (1 + k % 4) * xx) * torch.sin(math.pi * (1 + k // 4) * yy) for k in range(16)])
        t = t / kap.sqrt()
        targets.append(t / t.flatten(1).norm(dim=1)[:, None, None])
    return (torch.stack(feats).reshape(B, 3, N * N).float().contiguous(),
            torch.stack(targets).reshape(B, 16, N * N).float().contiguous())


def _block_sizes(case):
    return (case["k"], case["k"]) if case["kind"] == "orth" else (case["kx"], case["ky"])


def _batch_of(case, seed):
    ns = P.batch_sizes(case["nprob"], seed, case["lo"], case["hi"])
    return P.knn_batch(ns, 8, seed)


def prepare(case, seed):
    kind, st = case["kind"], {"case": case}
    if kind == "spmv":
        st["A"] = _mat(_operator(case, seed))
        st["x"] = _randn(seed, st["A"].n)
        st["y"] = torch.empty_like(st["x"])
    elif kind == "lanczos":
        st["A"] = A = _mat(_operator(case, seed))
        k, m = case["k"], case["m"]
        st["V"] = V = S.BV().create(A.n, m + 1)
        st["cols"] = _columns(V, m + 1)
        st["cols"][0].copy_(_randn(seed, A.n))
        torch.cuda.synchronize()
        V.orthonormalizeColumn(0)
        if k:
            V.matLanczos(A, 0, k)
    elif kind == "restart":
        n, k, e = case["n"], case["k"], case["e"]
        st["V"] = _basis(_randn(seed, k, n) / math.sqrt(n))
        st["cols"] = _columns(st["V"], k)
        st["Q"] = np.asfortranarray(np.linalg.qr(np.random.default_rng(seed).standard_normal((k, k)))[0])
    elif kind == "solve":
        st["A"] = A = _mat(_operator({**case, "op": "diffusion"}, seed))
        st["E"] = E = S.EPS().create()
        E.setOperators(A)
        E.setProblemType(S.EPS.ProblemType.HEP)
        E.setDimensions(case["nev"], case["ncv"])
        E.setTolerances(1e-10, 1000)
        E.setWhichEigenpairs(S.LARGEST_REAL)
        v0 = _randn(seed + 7, A.n)
        E.setInitialSpace(v0.cpu().numpy())
        st["v0"] = v0
    elif kind in ("dot", "combine", "orth"):
        kx, ky = _block_sizes(case)
        n = case["n"]
        st["X"] = _basis(_randn(seed, kx, n))
        st["Y"] = _basis(_randn(seed + 1, ky, n))
        if kind == "combine":
            st["Q"] = np.asfortranarray(np.random.default_rng(seed).standard_normal((kx, ky)))
        if kind == "orth":
            cols = _columns(st["X"], kx)
            if case["l"]:
                cols[: case["l"]] = torch.linalg.qr(cols[: case["l"]].T)[0].T
            st["Y"].setActiveColumns(case["l"], case["k"])
            st["Y"].setOrthogonalizationBlock(S.BV.OrthogBlockType.CHOL)
        st["cols"] = _columns(st["Y"], ky)
    elif kind == "filter":
        dt = torch.float32 if case["x32"] else F64
        st["A"] = _mat(_grid_csr((case["c"], case["b"], case["a"])))
        st["X"], st["Z"] = (_randn(seed + q, st["A"].n, case["bp"], dtype=dt) for q in (0, 1))
        st["Y"] = torch.empty_like(st["X"])
    elif kind == "aij":
        dt = np.float32 if case["f32"] else np.float64
        st["csr"] = csr = P.powerlaw_rect(case["m"], case["n"], case["row"], 1.8, seed)
        st["A"] = S.Mat().createAIJ(csr, size=(case["m"], case["n"]), dtype=dt)
        st["x"], st["w"] = _randn(seed, case["n"]), _randn(seed + 1, case["m"])
        st["y"], st["z"] = torch.empty_like(st["w"]), torch.empty_like(st["x"])
    elif kind == "batch":
        b = _batch_of(case, seed)
        st["B"] = B = S.BatchEPS().create(b.ns, b.rowptr, b.colind, b.vals)
        B.setDimensions(case["nev"], case["ncv"])
        B.setTolerances(1e-8)
        B.setWhichEigenpairs(S.LARGEST_REAL)
        B.setInitialVectors(np.random.default_rng(seed).standard_normal(int(b.ns.sum())))
        B.setThreads(256)
    else:
        st["op"] = op = S.NeuralOperator().create(*_dims(case["N"]))
        op.setParams(_theta(seed, case["N"]))
        st["F"], st["T"] = _neural_data(seed, case["N"], case["B"])
    torch.cuda.synchronize()
    return st


# ------------------------------------------------------------------------------------ one pass

def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "spmv":
        st["A"].mult(st["x"].data_ptr(), st["y"].data_ptr())
        return st["y"]
    if kind == "lanczos":
        alpha, betav, _, beta, _ = st["V"].matLanczos(st["A"], case["k"], case["m"])
        return {"alpha": alpha, "beta": betav, "last": beta, "V": st["cols"]}
    if kind == "restart":
        st["V"].multInPlace(st["Q"], 0, case["e"])
        return st["cols"]
    if kind == "solve":
        E, nev, n = st["E"], case["nev"], st["A"].n
        E.solve()
        X = torch.stack([torch.as_tensor(_Device(E.getEigenvectorPointer(i), (n,)), device="cuda") for i in range(nev)])
        X *= torch.sign(X @ st["v0"])[:, None]  # an eigenvector has no sign of its own: a program fixes one
        return {"values": np.array([E.getEigenvalue(i) for i in range(nev)]), "vectors": X}
    if kind == "dot":
        return st["X"].dot(st["Y"])
    if kind == "combine":
        st["Y"].mult(1.0, 1.0, st["X"], st["Q"])
        return st["cols"]
    if kind == "orth":
        st["Y"].setActiveColumns(0, case["k"])
        st["X"].copy(st["Y"])  # the block comes from elsewhere at each step
        st["Y"].setActiveColumns(case["l"], case["k"])
        R = st["Y"].orthogonalize(case["k"])
        return {"R": R, "Q": st["cols"]}
    if kind == "filter":
        S.rowblock_spmm(st["A"], case["bp"], st["X"].data_ptr(), st["Y"].data_ptr(), st["Z"].data_ptr(), 0.31, 6.0, 0.92,
                        x32=case["x32"])
        return st["Y"]
    if kind == "aij":
        st["A"].mult(st["x"].data_ptr(), st["y"].data_ptr())
        st["A"].multTranspose(st["w"].data_ptr(), st["z"].data_ptr())
        return st["y"], st["z"]
    if kind == "batch":
        st["B"].solve()
        return st["B"].getAll()[0][:, : case["nev"]]
    loss, grads = st["op"].lossGrad(st["F"], st["T"])
    return {"loss": loss, "grads": grads}


# ------------------------------------------------------------------------------------ floors

def _shape(case):
    """(rows, nonzeros) of a square case's operator."""
    if case.get("op") == "knn":
        return case["a"], 11 * case["a"]  # about: the symmetrised graph and its diagonal
    dims = [d for d in (case["a"], case["b"], case.get("c", 1)) if d > 1]
    n = math.prod(dims)
    if case.get("c", 1) == 1:  # a 2-D operator
        return n, 5 * n - 2 * case["a"] - 2 * case["b"]
    return n, n + 2 * sum(n - n // d for d in dims)


def work(case):
    kind = case["kind"]
    if kind in ("spmv", "lanczos", "solve", "filter"):
        n, nnz = _shape(case)
        csr = 12 * nnz + 4 * (n + 1)
    if kind == "spmv":
        return {"bytes": csr + 16 * n, "flops": 2 * nnz}
    if kind == "lanczos":
        k, m = case["k"], case["m"]
        # two classical Gram-Schmidt passes (a dot and an update each) per column: 8 n flops a column visited
        return {"bytes": csr + 8 * n * (m + 1), "flops": sum(2 * nnz + 8 * n * (j + 1) for j in range(k, m))}
    if kind == "restart":
        return {"bytes": 8 * case["n"] * (case["k"] + case["e"]), "flops": 2 * case["n"] * case["k"] * case["e"]}
    if kind == "solve":
        # at least one run of ncv steps
        return {"bytes": csr + 8 * n * (1 + case["nev"]),
                "flops": sum(2 * nnz + 8 * n * (j + 1) for j in range(case["ncv"]))}
    if kind == "dot":
        kx, ky = _block_sizes(case)
        return {"bytes": 8 * case["n"] * (kx + ky), "flops": 2 * case["n"] * kx * ky}
    if kind == "combine":
        kx, ky = _block_sizes(case)
        return {"bytes": 8 * case["n"] * (kx + 2 * ky), "flops": 2 * case["n"] * kx * ky}
    if kind == "orth":
        l, nc = case["l"], case["k"] - case["l"]
        return {"bytes": 16 * case["n"] * case["k"], "flops": 2 * case["n"] * (2 * l * nc + 2 * nc * nc)}
    if kind == "filter":
        s = 4 if case["x32"] else 8
        return {"bytes": (s + 4) * nnz + 3 * s * n * case["bp"], "flops": 2 * case["bp"] * (nnz + 2 * n)}
    if kind == "aij":
        m, n, nnz = case["m"], case["n"], case["m"] * case["row"]
        return {"bytes": 2 * nnz * (8 if case["f32"] else 12) + 4 * (m + n + 2) + 16 * (m + n), "flops": 4 * nnz}
    if kind == "batch":
        rows = case["nprob"] * (case["lo"] + case["hi"]) // 2
        return {"bytes": rows * (11 * 12 + 4 + 8) + 8 * case["nprob"] * case["nev"],
                "flops": rows * sum(22 + 8 * (j + 1) for j in range(case["ncv"]))}
    N, W, M, L, H, K = _dims(case["N"])
    per = 2 * N * N * (3 * W + L * W * W + W * H + H * K) + L * W * 4 * (M * N * N + M * M * N) + L * 2 * W * W * M * M
    theta = 4 * W + L * (W * W * M * M + W * W + W) + H * W + H + K * H + K
    return {"bytes": 4 * (case["B"] * N * N * (3 + K) + 2 * theta), "flops": 3 * case["B"] * per}


# ------------------------------------------------------------------------------------ in 64 bits

def _sparse(csr, n):
    rowptr, colind, vals = csr
    return torch.sparse_csr_tensor(rowptr.long(), colind.long(), vals, size=(rowptr.numel() - 1, n))


def _exact_lanczos(case, seed):
    csr = _operator(case, seed)
    n = csr[0].numel() - 1
    A = _sparse(csr, n)
    k, m = case["k"], case["m"]
    V = torch.zeros(m + 1, n, dtype=F64, device="cuda")
    v = _randn(seed, n)
    V[0] = v / v.norm()
    alpha, beta = np.zeros(m + 1), np.zeros(m + 1)
    for j in range(m):
        w = A @ V[j]
        h = torch.zeros(j + 1, dtype=F64, device="cuda")
        for _ in range(2):
            c = V[: j + 1] @ w
            w = w - c @ V[: j + 1]
            h += c
        b = w.norm()
        V[j + 1] = w / b
        if j >= k:
            alpha[j], beta[j] = float(h[j]), float(b)
    return {"alpha": alpha, "beta": beta, "last": float(beta[m - 1]), "V": V}


def _exact_neural(case, seed):
    N, W, M, L, H, K = _dims(case["N"])
    theta = torch.from_numpy(_theta(seed, N).astype(np.float64)).cuda().requires_grad_(True)
    Fe, T = (t.double() for t in _neural_data(seed, N, case["B"]))
    at = 0

    def take(*shape):
        nonlocal at
        at += math.prod(shape)
        return theta[at - math.prod(shape):at].view(shape)

    k = torch.arange(1, M + 1, device="cuda", dtype=F64)
    i = torch.arange(1, N + 1, device="cuda", dtype=F64)
    Sb = math.sqrt(2 / (N + 1)) * torch.sin(math.pi * i[:, None] * k[None, :] / (N + 1))
    B = case["B"]
    v = torch.einsum("oi,bip->bop", take(W, 3), Fe) + take(W)[None, :, None]
    for l in range(L):
        R, Wl, bl = take(W, W, M * M), take(W, W), take(W)
        C = (Sb.T @ v.view(B, W, N, N) @ Sb).reshape(B, W, M * M)
        D = torch.einsum("ocq,bcq->boq", R, C).reshape(B, W, M, M)
        u = (Sb @ D @ Sb.T).reshape(B, W, N * N) + torch.einsum("oc,bcp->bop", Wl, v) + bl[None, :, None]
        v = torch.nn.functional.gelu(u) if l < L - 1 else u
    h = torch.nn.functional.gelu(torch.einsum("hc,bcp->bhp", take(H, W), v) + take(H)[None, :, None])
    y = torch.einsum("kh,bhp->bkp", take(K, H), h) + take(K)[None, :, None]
    loss = (1 - (y * T).sum(2) ** 2 / (y * y).sum(2)).mean()
    (g,) = torch.autograd.grad(loss, theta)
    return {"loss": float(loss.detach()), "grads": g.cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "spmv":
        csr = _operator(case, seed)
        n = csr[0].numel() - 1
        return _sparse(csr, n) @ _randn(seed, n)
    if kind == "lanczos":
        return _exact_lanczos(case, seed)
    if kind == "restart":
        n, k, e = case["n"], case["k"], case["e"]
        V = _randn(seed, k, n) / math.sqrt(n)
        Q = torch.from_numpy(np.linalg.qr(np.random.default_rng(seed).standard_normal((k, k)))[0]).cuda()
        return torch.cat([Q[:, :e].T @ V, V[e:]])
    if kind == "solve":
        csr = _operator({**case, "op": "diffusion"}, seed)
        n = csr[0].numel() - 1
        if n > 6500:
            return None
        w, X = torch.linalg.eigh(_sparse(csr, n).to_dense())
        nev = case["nev"]
        X = X[:, -nev:].flip(1).T
        return {"values": w[-nev:].flip(0).cpu().numpy(), "vectors": X * torch.sign(X @ _randn(seed + 7, n))[:, None]}
    if kind in ("dot", "combine", "orth"):
        kx, ky = _block_sizes(case)
        X, Y = _randn(seed, kx, case["n"]), _randn(seed + 1, ky, case["n"])
        if kind == "dot":
            return (Y @ X.T).cpu().numpy()
        if kind == "combine":
            return Y + torch.from_numpy(np.random.default_rng(seed).standard_normal((kx, ky))).cuda().T @ X
        l, k = case["l"], case["k"]
        if l:
            X[:l] = torch.linalg.qr(X[:l].T)[0].T
        R = torch.zeros(k, k, dtype=F64, device="cuda")
        C = X[:l] @ X[l:].T
        Z = X[l:] - C.T @ X[:l]
        R[:l, l:] = C
        U = torch.linalg.cholesky(Z @ Z.T, upper=True)
        R[l:, l:] = U
        X[l:] = torch.linalg.solve_triangular(U.T, Z, upper=False)
        return {"R": R.cpu().numpy(), "Q": X}
    if kind == "filter":
        csr = _grid_csr((case["c"], case["b"], case["a"]))
        n = csr[0].numel() - 1
        dt = torch.float32 if case["x32"] else F64
        X, Z = (_randn(seed + q, n, case["bp"], dtype=dt).double() for q in (0, 1))
        return 0.31 * (_sparse(csr, n) @ X - 6.0 * X) - 0.92 * Z
    if kind == "aij":
        rowptr, colind, vals = (torch.from_numpy(v).cuda() for v in
                                P.powerlaw_rect(case["m"], case["n"], case["row"], 1.8, seed))
        rows = torch.repeat_interleave(torch.arange(case["m"], device="cuda"), rowptr[1:] - rowptr[:-1])
        x, w, v = _randn(seed, case["n"]), _randn(seed + 1, case["m"]), vals.double()
        y = torch.zeros(case["m"], dtype=F64, device="cuda").index_add_(0, rows, v * x[colind.long()])
        z = torch.zeros(case["n"], dtype=F64, device="cuda").index_add_(0, colind.long(), v * w[rows])
        return y, z
    if kind == "neural":
        return _exact_neural(case, seed)
    b = _batch_of(case, seed)
    if sum(int(n) ** 3 for n in b.ns) > 3e11:  # the dense eigenvalues of so many problems take too long
        return None
    out = np.zeros((case["nprob"], case["nev"]))
    for p in range(case["nprob"]):
        rp, ci, va = (torch.from_numpy(v).cuda() for v in b.problem(p))
        out[p] = torch.linalg.eigvalsh(_sparse((rp, ci, va), rp.numel() - 1).to_dense())[-case["nev"]:].flip(0).cpu().numpy()
    return out
