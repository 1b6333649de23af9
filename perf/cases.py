"""Performance cases: what a program that uses this library has it do, through its
public entry points.

Every case is a seeded synthetic Gaussian-process problem, X ~ U[0,1]^(N x d) and
y = sin(sum_k x_k) + N(0, 0.1^2), on a packed lower-triangle kernel matrix of block
size `bsz` (128 is the command line's default, 256 the large configurations').  The
kinds are the library's user-level paths:

  direct   assemble K, factor it (FP64), solve for one right-hand side
  solve    one more right-hand side for a factor the program already holds
  cg       conjugate gradients to eps on a K the program already holds
  mixed    assemble K, mixed-precision factor + FP64 refinement to 1e-14
  nlml     negative log marginal likelihood and its gradient (one optimiser step)
  predict  predictive mean at new points from alpha = K^-1 y

`listed()` names the fixed cases, `draw(rng)` gives others of the same ranges.
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

DEV = "cuda:0"


def _load():
    """The package under its import name (its directory name is not an identifier)."""
    if "hs_b200" not in sys.modules:
        pkg = Path(__file__).resolve().parent.parent / "heterogeneous-solvers_b200"
        spec = importlib.util.spec_from_file_location("hs_b200", pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["hs_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["hs_b200"]


def listed():
    return [
        # a few hundred points, the reference's default block size: launches and
        # latency are all there is (interactive use, inner loops of other programs)
        dict(name="direct_n500", kind="direct", N=500, d=8, bsz=128, ell=0.5),
        # the configuration N=4096, d=8, l=0.5, bsz=128
        dict(name="direct_n4096", kind="direct", N=4096, d=8, bsz=128, ell=0.5),
        # an ordinary data set of no particular size: padding in the last block row
        dict(name="direct_n9973", kind="direct", N=9973, d=16, bsz=256, ell=1.0),
        # the large configuration's generator (d=16, l=1, bsz=256) at a size whose
        # factor still takes under a second
        dict(name="direct_n32768", kind="direct", N=32768, d=16, bsz=256, ell=1.0),
        # new targets for a factor at hand
        dict(name="solve_n16384", kind="solve", N=16384, d=16, bsz=256, ell=1.0),
        # the command line's default algorithm at the N=4096 configuration ...
        dict(name="cg_n4096", kind="cg", N=4096, d=8, bsz=128, ell=0.5),
        # ... and on a matrix larger than L2, ragged
        dict(name="cg_n15000", kind="cg", N=15000, d=16, bsz=256, ell=1.0),
        # mixed precision at a small ragged size and at a quarter of the large
        # configuration's N (the FP16 split, the form the benchmark reports)
        dict(name="mixed_n3000", kind="mixed", N=3000, d=8, bsz=128, ell=0.5, prec="f16x3"),
        dict(name="mixed_n32768", kind="mixed", N=32768, d=16, bsz=256, ell=1.0, prec="f16x3"),
        # hyperparameter fitting: one function and gradient evaluation of an ARD
        # kernel, at a small ragged size and at the production size N=16384
        dict(name="nlml_n2000", kind="nlml", N=2000, d=8, bsz=256),
        dict(name="nlml_n16384", kind="nlml", N=16384, d=8, bsz=256),
        # predictions from a fitted model
        dict(name="predict_n16384", kind="predict", N=16384, Nt=5000, d=16, bsz=256, ell=1.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["direct", "direct", "direct", "solve", "cg", "mixed", "mixed", "nlml", "nlml", "predict"])
    bsz = rng.choice([128, 256])
    d, ell = rng.choice([(8, 0.5), (16, 1.0)])
    case = dict(kind=kind, d=d, bsz=bsz, ell=ell)
    if kind == "direct":
        case["N"] = _log_int(rng, 300, 28000)
    elif kind == "solve":
        case["N"] = _log_int(rng, 1000, 28000)
    elif kind == "cg":
        case["N"] = _log_int(rng, 1000, 14000)
    elif kind == "mixed":
        case["N"] = _log_int(rng, 1000, 30000)
        case["prec"] = rng.choice(["f16x3", "f16x3", "tf32x3", "bf16x3"])
    elif kind == "nlml":
        case.pop("ell")
        case["d"] = 8
        case["N"] = _log_int(rng, 500, 14000)
    else:
        case["N"] = _log_int(rng, 1000, 30000)
        case["Nt"] = _log_int(rng, 100, 10000)
    return case


SF2, SN2 = 1.0, 1e-2


def _inputs(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    N, d = case["N"], case["d"]
    X = torch.rand((N, d), dtype=torch.float64, device=DEV, generator=g)
    y = torch.sin(X.sum(dim=1)) + 0.1 * torch.randn(N, dtype=torch.float64, device=DEV, generator=g)
    out = {"X": X, "y": y}
    if case["kind"] == "nlml":
        # log lengthscales around log 1, log sf2 = 0, log sn2 = log 1e-2
        r = np.random.default_rng(seed)
        out["theta"] = np.concatenate([r.uniform(math.log(0.5), math.log(2.0), d), [0.0, math.log(SN2)]])
    if case["kind"] == "predict":
        out["Xt"] = torch.rand((case["Nt"], d), dtype=torch.float64, device=DEV, generator=g)
        # weights of the size and sign pattern K^-1 y has: residuals over the noise
        out["alpha"] = torch.randn(N, dtype=torch.float64, device=DEV, generator=g) * (0.1 / SN2)
    return out


def prepare(case, seed):
    hs = _load()
    s = dict(case, hs=hs, **_inputs(case, seed))
    N, bsz, kind = case["N"], case["bsz"], case["kind"]
    s["ctx"] = ctx = hs.Context(device=0, N=N, matrixBlockSize=bsz)
    if kind in ("nlml", "predict"):
        return s
    s["A"] = hs.SymmetricMatrix(N, bsz, device=DEV)
    s["b"] = hs.RightHandSide(N, bsz, device=DEV)
    s["b"].rightHandSideData[:N] = s["y"]
    if kind in ("solve", "cg"):
        hs.MatrixGenerator.assemble(ctx, s["A"].matrixData, s["X"], case["ell"], SF2, SN2)
    if kind == "solve":
        s["chol"] = hs.Cholesky(s["A"], ctx).solve_heterogeneous()
    return s


def run(s):
    hs, ctx, N, kind = s["hs"], s["ctx"], s["N"], s["kind"]
    if kind == "nlml":
        nlml, grad, _ = hs.gp_nlml_grad(ctx, s["X"], s["y"], s["theta"])
        return {"nlml": nlml, "grad": grad}
    if kind == "predict":
        return hs.gp_predict(ctx, s["X"], s["Xt"], s["alpha"], s["ell"], SF2)
    A, b = s["A"], s["b"]
    if kind == "cg":
        return hs.CG(A, b, ctx).solveHeterogeneous(epsilon=1e-10, iMax=20000).x
    if kind in ("direct", "mixed"):
        hs.MatrixGenerator.assemble(ctx, A.matrixData, s["X"], s["ell"], SF2, SN2)
    if kind == "mixed":
        return hs.MixedPrecisionSolver(A, ctx, s["prec"]).solve(b)
    b.rightHandSideData[:N] = s["y"]  # the substitution works in place
    if kind == "direct":
        L = hs.Cholesky(A, ctx).solve_heterogeneous().A_gpu
        hs.TriangularSystemSolver(A, L, b, ctx).solve()
        return {"L": L, "x": b.rightHandSideData}
    hs.TriangularSystemSolver(A, s["chol"].A_gpu, b, ctx).solve()
    return b.rightHandSideData


def work(case):
    N, d, kind = case["N"], case["d"], case["kind"]
    tri = 8.0 * N * (N + 1) / 2  # one triangle of K or L
    vec = 8.0 * N
    assembly = 0.5 * N * N * (3 * d + 2)  # distance, exponent, scale of each entry
    if kind == "direct":
        return {"bytes": vec * (d + 2) + tri, "flops": assembly + N**3 / 3 + 2.0 * N * N}
    if kind == "solve":
        return {"bytes": tri + 2 * vec, "flops": 2.0 * N * N}
    if kind == "cg":
        # about a thousand iterations (917 at N=4096, d=8; 2022 at N=131072, d=16),
        # each of which needs the whole of K
        return {"bytes": 1000 * tri, "flops": 1000 * 2.0 * N * N}
    if kind == "mixed":
        return {"bytes": vec * (d + 2), "flops": assembly + N**3 / 3}
    if kind == "nlml":
        # factor N^3/3, reverse-mode factor 2N^3/3, assembly twice (K and dK/dtheta)
        return {"bytes": vec * (d + 1), "flops": 2 * assembly + 1.0 * N**3}
    Nt = case["Nt"]
    return {"bytes": 8.0 * (N * (d + 1) + Nt * (d + 1)), "flops": 1.0 * N * Nt * (3 * d + 4)}


# ------------------------------------------------------------ 64-bit values
def _sqdist(X, Z):
    """Squared distances, summed feature by feature (no cancellation)."""
    D = torch.zeros((X.shape[0], Z.shape[0]), dtype=torch.float64, device=X.device)
    for k in range(X.shape[1]):
        D += (X[:, k, None] - Z[None, :, k]).square_()
    return D


def _kernel(X, ell):
    K = _sqdist(X, X).mul_(-0.5 / (ell * ell)).exp_().mul_(SF2)
    K.diagonal().add_(SN2)
    return K


def _padded(v, bsz):
    n = -(-v.numel() // bsz) * bsz
    out = torch.zeros(n, dtype=v.dtype, device=v.device)
    out[: v.numel()] = v
    return out


def _solve(K, L, y):
    """K^-1 y with one step of refinement."""
    x = torch.cholesky_solve(y[:, None], L)
    return (x + torch.cholesky_solve(y[:, None] - K @ x, L))[:, 0]


def _packed(L, bsz):
    """Column-by-column blocks of a lower-triangular matrix, zero padding."""
    N = L.shape[0]
    n = -(-N // bsz) * bsz
    cols = []
    for c in range(0, n, bsz):
        col = torch.zeros((n - c, bsz), dtype=L.dtype, device=L.device)
        part = L[c:, c : c + bsz]
        col[: part.shape[0], : part.shape[1]] = part
        cols.append(col.reshape(-1))
    return torch.cat(cols)


def _nlml(X, y, theta):
    N, d = X.shape
    Xs = X / torch.from_numpy(np.exp(theta[:d])).to(X.device)
    sf2, sn2 = math.exp(theta[d]), math.exp(theta[d + 1])
    R = _sqdist(Xs, Xs).mul_(-0.5).exp_().mul_(sf2)  # noise-free kernel
    K = R.clone()
    K.diagonal().add_(sn2)
    L = torch.linalg.cholesky(K)
    alpha = _solve(K, L, y)
    del K
    value = 0.5 * (y @ alpha) + L.diagonal().log().sum() + 0.5 * N * math.log(2 * math.pi)
    W = torch.cholesky_inverse(L)
    del L
    W -= alpha[:, None] * alpha[None, :]
    trace = W.diagonal().sum()
    W *= R
    del R
    grad = [0.5 * (W * (Xs[:, k, None] - Xs[None, :, k]).square_()).sum().item() for k in range(d)]
    grad += [0.5 * W.sum().item(), 0.5 * sn2 * trace.item()]
    return {"nlml": value.item(), "grad": np.asarray(grad)}


def exact(case, seed):
    s = _inputs(case, seed)
    X, y, kind = s["X"], s["y"], case["kind"]
    if kind == "nlml":
        return _nlml(X, y, s["theta"])
    if kind == "predict":
        out = torch.empty(case["Nt"], dtype=torch.float64, device=DEV)
        for i in range(0, case["Nt"], 1024):
            D = _sqdist(s["Xt"][i : i + 1024], X).mul_(-0.5 / case["ell"] ** 2).exp_()
            out[i : i + 1024] = SF2 * (D @ s["alpha"])
        return out
    K = _kernel(X, case["ell"])
    L = torch.linalg.cholesky(K)
    x = _padded(_solve(K, L, y), case["bsz"])
    if kind == "direct":
        return {"L": _packed(L, case["bsz"]), "x": x}
    return x
