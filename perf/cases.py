"""Performance cases of the deflated minimal residual solver.

Every case is a whole call that a user's program makes: a solve, or a sequence of solves, from
zero initial guesses and an empty deflation space, through the binding's public entry points.
The state that `prepare` returns holds what such a program keeps (the operator resident in a
System, a plugin or a Server) and that call's right-hand sides, drawn from the seed.  The
outputs are the solutions.  Tolerances are tight enough that two correct solvers agree far
beyond them.

Families ("form" of a case):
  batch    gdmr_solve_batch on device buffers: right-hand sides sharing one deflation space
  stream   gdmr_solve_batch one right-hand side after another, the deflation space recycled
  solve    gdmr_solve on host buffers: the reference's algorithm in complex128 or double-float
  plugin   the reference's plugin interface (initLS / impCsrLS / solveLS) in complex64
  multi    gdmr_multi_solve: several variable-coefficient operators at once, host buffers
  serve    the server: requests of several operators submitted together, host buffers
"""
import math
import os
import sys
from collections import OrderedDict

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gdmr-solver_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import gdmr  # noqa: E402
import problems  # noqa: E402


def _case(form, shape, nrhs, kappa, damping, m, k, tol, precision="mixed", rhs="source", capacity=0, stencil=False,
          operators=1, name=None):
    c = {"form": form, "nx": shape[0], "ny": shape[1], "nz": shape[2] if len(shape) > 2 else 0, "nrhs": nrhs,
         "kappa": float(kappa), "damping": float(damping), "m": m, "k": k, "tol": float(tol), "precision": precision,
         "rhs": rhs, "capacity": capacity or nrhs, "stencil": bool(stencil), "operators": operators}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The batch that the benchmark stands for: 64 Gaussian sources on a 96^3 grid in one call.
        _case("batch", (96, 96, 96), 64, 4, 0.1, 48, 24, 1e-10, name="batch_96_64rhs"),
        # One operator's share of a serving box: 64^3 at kappa 16, damping 0.2, a quarter of the batch.
        _case("batch", (64, 64, 64), 16, 16, 0.2, 48, 24, 1e-10, name="batch_64_16rhs"),
        # An odd-sized box with more right-hand sides than slots: systems leave, others take their place.
        _case("batch", (61, 47, 35), 21, 8, 0.1, 40, 16, 1e-10, capacity=12, name="batch_odd_refill"),
        # The 64 x 64 operator of the reference-parity configuration, its eight right-hand sides as one batch.
        _case("batch", (64, 64), 8, 20, 0.05, 40, 10, 1e-11, rhs="gauss", name="batch_2d_8rhs"),
        # The matrix-free operator: a 96^3 batch of 16 without reading a matrix.
        _case("batch", (96, 96, 96), 16, 4, 0.1, 48, 24, 1e-10, stencil=True, name="batch_96_stencil"),
        # A sequence of right-hand sides one at a time on a 128^3 grid, m = 60 and k = 20, space recycled.
        _case("stream", (128, 128, 128), 2, 6, 0.1, 60, 20, 1e-11, name="stream_128_mixed"),
        # The reference's algorithm in double-float on the benchmark's grid, one right-hand side.
        _case("solve", (96, 96, 96), 1, 10, 0.1, 48, 24, 1e-11, precision="fp64e", name="solve_96_fp64e"),
        # The same algorithm in native complex128 on a 3D grid.
        _case("solve", (64, 64, 64), 1, 8, 0.1, 48, 24, 1e-11, precision="fp64", name="solve_64_fp64"),
        # The reference-parity configuration: 64 x 64, complex128, right-hand sides in sequence.
        _case("solve", (64, 64), 2, 20, 0.05, 40, 10, 1e-11, precision="fp64", rhs="gauss", name="solve_2d_fp64"),
        # A control program of the reference: the complex64 plugin with a sparse operator.
        _case("plugin", (16, 16, 16), 2, 15, 0.2, 30, 8, 2e-7, precision="c64", name="plugin_c64"),
        # Uneven variable-coefficient operators solved at once, four right-hand sides each.
        _case("multi", (28, 20, 24), 4, 4, 0.1, 40, 16, 1e-11, rhs="gauss", operators=14, name="multi_14ops"),
        # A burst of requests on a server with two resident operators.
        _case("serve", (48, 48, 48), 12, 6, 0.1, 48, 24, 1e-11, operators=2, capacity=6, name="serve_2ops"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _grid(rng, cells_lo, cells_hi, dims):
    """Edge lengths of a box of about log-uniform volume, aspect ratios up to two, odd ones among them."""
    edge = _log(rng, cells_lo, cells_hi) ** (1.0 / dims)
    top = int(cells_hi ** (1.0 / dims))
    return tuple(max(6, min(top, int(round(edge * 2 ** rng.uniform(-0.5, 0.5))))) for _ in range(dims))


def draw(rng):
    form = rng.choice(["batch", "batch", "batch", "batch2d", "stencil", "stream", "fp64e", "fp64", "fp64_2d", "plugin",
                       "multi", "serve"])
    damping = rng.choice([0.05, 0.1, 0.2])
    m, k = rng.choice([(48, 24), (40, 16), (60, 20)])      # the larger grids
    ms, ks = rng.choice([(40, 16), (40, 10), (30, 8)])     # the smaller ones
    if form in ("batch", "stencil"):
        nrhs = int(round(_log(rng, 2, 64)))
        shape = _grid(rng, 20 ** 3, min(96 ** 3, 30e6 / nrhs), 3)
        cap = nrhs if rng.random() < 0.7 else max(1, nrhs // 2)
        if math.prod(shape) < 40 ** 3:
            m, k = ms, ks
        return _case("batch", shape, nrhs, rng.uniform(2, 5), damping, m, k, 1e-10, capacity=cap,
                     stencil=form == "stencil")
    if form == "batch2d":
        return _case("batch", _grid(rng, 32 ** 2, 96 ** 2, 2), int(round(_log(rng, 2, 32))), rng.uniform(5, 15), damping,
                     ms, ks, 1e-11, rhs="gauss")
    if form == "stream":
        return _case("stream", _grid(rng, 40 ** 3, 120 ** 3, 3), rng.choice([1, 2]), rng.uniform(3, 6), damping, m, k,
                     1e-11)
    if form == "fp64e":
        return _case("solve", _grid(rng, 24 ** 3, 80 ** 3, 3), 1, rng.uniform(3, 8), damping, m, k, 1e-11,
                     precision="fp64e")
    if form == "fp64":
        return _case("solve", _grid(rng, 16 ** 3, 64 ** 3, 3), 1, rng.uniform(3, 8), damping, ms, ks, 1e-11,
                     precision="fp64")
    if form == "fp64_2d":
        return _case("solve", _grid(rng, 24 ** 2, 72 ** 2, 2), rng.choice([1, 2, 3]), rng.uniform(5, 15), damping,
                     ms, ks, 1e-11, precision=rng.choice(["fp64", "fp64e"]), rhs="gauss")
    if form == "plugin":
        return _case("plugin", _grid(rng, 12 ** 3, 17 ** 3, 3), rng.choice([1, 2]), rng.uniform(10, 15), 0.2, 30, 8,
                     2e-7, precision="c64")
    if form == "multi":
        return _case("multi", _grid(rng, 18 ** 3, 28 ** 3, 3), rng.choice([2, 3, 4]), rng.uniform(2, 4), damping, ms, ks,
                     1e-11, rhs="gauss", operators=rng.randint(4, 14))
    return _case("serve", _grid(rng, 20 ** 3, 48 ** 3, 3), rng.randint(4, 12), rng.uniform(3, 6), damping, ms, ks, 1e-11,
                 operators=rng.choice([1, 2]), capacity=rng.randint(3, 6))


# ------------------------------------------------------------------ operators
_matrices = OrderedDict()     # the last few CSR matrices (host), by their parameters


def _matrix(kind, shape, *args):
    key = (kind, shape) + args
    if key not in _matrices:
        while len(_matrices) >= 16:
            _matrices.popitem(last=False)
        _matrices[key] = problems.helmholtz(shape, *args) if kind == "helmholtz" else problems.variable_helmholtz(shape, *args)
    _matrices.move_to_end(key)
    return _matrices[key]


def _shape(case):
    s = (case["nx"], case["ny"], case["nz"])
    return s if s[2] else s[:2]


def _shapes(case):
    """The boxes of a case's operators: uneven ones, from half to one and a half times the stated edges."""
    if case["operators"] == 1:
        return [_shape(case)]
    if case["form"] == "serve":
        return [_shape(case)] * case["operators"]
    u = problems.uniform01(31, 3 * case["operators"])
    return [tuple(max(6, int(round(e * 0.5 * 3.0 ** u[3 * i + a]))) for a, e in enumerate(_shape(case)))
            for i in range(case["operators"])]


def _operators(case):
    if case["form"] == "multi":
        return [_matrix("variable", s, case["kappa"], case["damping"], 500 + i) for i, s in enumerate(_shapes(case))]
    return [_matrix("helmholtz", s, case["kappa"], case["damping"] * (1 + i)) for i, s in enumerate(_shapes(case))]


# ------------------------------------------------------------------ right-hand sides
def _rhs(case, seed):
    """One (nrhs, n) complex128 device tensor an operator: unit complex Gaussians, or unit Gaussian
    sources (sigma three cells) at uniform positions plus 1% complex Gaussian noise."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    out = []
    for shape in _shapes(case):
        e = torch.randn(case["nrhs"], math.prod(shape), dtype=torch.complex128, device="cuda", generator=g)
        e /= e.norm(dim=1, keepdim=True)
        if case["rhs"] == "source":
            centre = torch.rand(case["nrhs"], len(shape), dtype=torch.float64, device="cuda", generator=g)
            s = torch.ones(case["nrhs"], 1, dtype=torch.float64, device="cuda")
            for ax, edge in enumerate(shape):
                i = torch.arange(edge, dtype=torch.float64, device="cuda")
                f = torch.exp(-(i[None] - centre[:, ax:ax + 1] * (edge - 1)) ** 2 / 18.0)
                s = (f[:, :, None] * s[:, None, :]).reshape(case["nrhs"], -1)
            e = s / s.norm(dim=1, keepdim=True) + 0.01 * e
        out.append(e)
    return out


# ------------------------------------------------------------------ states
class _Plugin:
    """The process's plugin (one may be live at a time, as the reference's) with its operator."""
    live, key = None, None

    @classmethod
    def get(cls, case):
        key = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "tol", "nrhs", "rhs")))
        if cls.key != key:
            if cls.live is not None:
                cls.live.close()
            A = _operators(case)[0]
            cls.live, cls.key = gdmr.LinearSystem(A.n, case["m"], case["k"], precision="c64"), key
            cls.live.imp_csr(A)
        return cls.live


def prepare(case, seed):
    mats, B = _operators(case), _rhs(case, seed)
    state = {"case": case}
    form = case["form"]
    if form == "plugin":
        _Plugin.get(case)
        state["b"] = B[0].to(torch.complex64).cpu().numpy()
    elif form == "serve":
        srv = gdmr.Server(budget_bytes=32 << 30)
        state["ops"] = [srv.add_operator(A, case["m"], case["k"], capacity=case["capacity"]) for A in mats]
        srv.start()
        state["server"], state["b"] = srv, [b.cpu().numpy() for b in B]
    else:
        cap = {"batch": case["capacity"], "multi": case["nrhs"]}.get(form, 1)
        state["systems"] = [gdmr.System(A, case["m"], case["k"], capacity=cap, precision=case["precision"]) for A in mats]
        if case["stencil"]:
            shape = _shape(case)
            state["systems"][0].set_stencil(shape, *problems.helmholtz_stencil(shape, case["kappa"], case["damping"]))
        if form in ("batch", "stream"):
            state["b"], state["x"] = B[0], torch.empty_like(B[0])
        else:
            state["b"] = [b.cpu().numpy() for b in B]
    return state


def run(state):
    case = state["case"]
    form, tol, b = case["form"], case["tol"], state["b"]
    if form == "plugin":
        ls = _Plugin.get(case)
        out = []
        for i in range(case["nrhs"]):
            ls.imp_img(b[i])
            ls.imp_src(np.zeros(b.shape[1], np.complex64))
            ls.solve(min(i, 1), tol, 2000)
            out.append(ls.exp_src())
        return out
    if form == "serve":
        srv = state["server"]
        tickets = [srv.submit(op, b[o][i], tol=tol) for i in range(case["nrhs"]) for o, op in enumerate(state["ops"])]
        return [srv.wait(t)[0] for t in tickets]
    systems = state["systems"]
    for s in systems:
        s.drop_deflation()
    if form == "multi":
        return [x for x, _ in gdmr.multi_solve(systems, b, tol=tol)]
    if form == "solve":
        return [systems[0].solve(b[0][i], mode=min(i, 1), tol=tol)[0] for i in range(case["nrhs"])]
    x = state["x"]
    x.zero_()
    torch.cuda.current_stream().synchronize()      # the library solves on streams of its own
    if form == "batch":
        systems[0].solve_batch_device(b.data_ptr(), x.data_ptr(), case["nrhs"], tol)
    else:
        for i in range(case["nrhs"]):
            systems[0].solve_batch_device(b[i].data_ptr(), x[i].data_ptr(), 1, tol)
    return x


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Each operator read once (CSR: a value and a column index an entry, the row pointers), each
    right-hand side read and each solution written once; one operator product a right-hand side."""
    size = 8 if case["precision"] == "c64" else 16
    moved = flops = 0
    for shape in _shapes(case):
        n = math.prod(shape)
        nnz = n + sum(2 * (n - n // e) for e in shape)
        moved += (0 if case["stencil"] else nnz * (size + 4) + 4 * (n + 1)) + 2 * size * n * case["nrhs"]
        flops += 8 * nnz * case["nrhs"]
    return {"bytes": moved, "flops": flops}


# ------------------------------------------------------------------ exact solutions
def _sine_solve(shape, kappa, damping, b, scale=1.0):
    """(-scale Laplacian - kappa^2 (1 + i damping))^-1 b on a Dirichlet grid: sine transforms along
    each axis diagonalise the 5- and 7-point operators."""
    x = b.reshape((b.shape[0],) + tuple(shape[::-1]))
    lam, transforms = 0.0, []
    for ax, edge in enumerate(shape):
        j = torch.arange(1, edge + 1, dtype=torch.float64, device=b.device)
        s = torch.sin(math.pi * torch.outer(j, j) / (edge + 1)) * math.sqrt(2.0 / (edge + 1))
        d = len(shape) - ax
        transforms.append((d, s.to(b.dtype)))
        lam = lam + (scale * 4 * (edge + 1) ** 2 * torch.sin(math.pi * j / (2 * (edge + 1))) ** 2).reshape(
            [edge if a == d - 1 else 1 for a in range(len(shape))])

    def transform(v):
        for d, s in transforms:
            v = torch.movedim(torch.tensordot(v, s, dims=([d], [0])), -1, d)
        return v

    return transform(transform(x) / (lam - kappa ** 2 * (1 + 1j * damping))).reshape(b.shape)


def _variable_solve(A, shape, kappa, damping, b):
    """A^-1 b by full GMRES in complex128, right-preconditioned with the constant-coefficient
    operator of the mean coefficient, restarted once to polish."""
    S = torch.sparse_csr_tensor(torch.from_numpy(A.indptr.astype(np.int64)).cuda(),
                                torch.from_numpy(A.indices.astype(np.int64)).cuda(),
                                torch.from_numpy(A.data).cuda(), (A.n, A.n))
    mean = 2.5 + 0.1j
    out = torch.empty_like(b)
    for i in range(b.shape[0]):
        x = torch.zeros_like(b[i])
        for _ in range(3):
            r = b[i] - S @ x
            beta = r.norm()
            if beta <= 1e-14 * b[i].norm():
                break
            V, P, H = [r / beta], [], []
            for j in range(80):
                P.append(_sine_solve(shape, kappa, damping, V[j][None], mean)[0])
                w = S @ P[j]
                Q = torch.stack(V)
                h = torch.zeros(82, dtype=b.dtype, device=b.device)
                for _ in range(2):
                    c = Q.conj() @ w
                    w = w - c @ Q
                    h[:j + 1] += c
                h[j + 1] = w.norm()
                H.append(h)
                V.append(w / h[j + 1])
                if j % 10 == 9:
                    Hm = torch.stack(H, 1)[:j + 2].cpu().numpy()
                    g = np.zeros(j + 2, np.complex128)
                    g[0] = float(beta)
                    y, *_ = np.linalg.lstsq(Hm, g, rcond=None)
                    if np.linalg.norm(g - Hm @ y) <= 1e-14 * float(b[i].norm()):
                        break
            x = x + torch.from_numpy(y).cuda() @ torch.stack(P[:len(y)])
        out[i] = x
    return out


def exact(case, seed):
    B = _rhs(case, seed)
    if case["form"] == "multi":
        return [_variable_solve(A, s, case["kappa"], case["damping"], b).cpu().numpy()
                for A, s, b in zip(_operators(case), _shapes(case), B)]
    if case["form"] == "plugin":
        B = [b.to(torch.complex64).to(torch.complex128) for b in B]
    X = [_sine_solve(s, case["kappa"], case["damping"] * (1 + i), b) for i, (s, b) in enumerate(zip(_shapes(case), B))]
    if case["form"] in ("batch", "stream"):
        return X[0]
    if case["form"] == "serve":
        return [X[o][i].cpu().numpy() for i in range(case["nrhs"]) for o in range(case["operators"])]
    return [X[0][i].cpu().numpy() for i in range(case["nrhs"])]
