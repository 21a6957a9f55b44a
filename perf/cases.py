"""What a user of the solver has it do, as measurable cases.

Every case goes through the package's public entry points (``LSKernel``,
``FMM2DTree`` and, for buffers on the device, ``aifmm_solve`` of the C ABI).
The leaf tables are a user's precomputed input (the reference reads them from
files): they are made here once per geometry by plain quadrature and handed to
``tables_set``, except in the ``tables`` kind, which is the call that makes them.

kinds
  solve   createTree + assemble + factorise + solve: a new geometry, as the
          reference's driver runs it
  cached  right-hand sides against factors kept on the device
  refined GMRES against the compressed operator, FP64 factors kept
  mixed   refactoring a kept assembly in complex64 and refining to FP64
  matvec  the exact dense product (the find_error protocol's fixture)
  field   total field u_inc + G phi of a solution
  matrix  a block of matrix entries into host memory (residual sampling)
  tables  the leaf tables by adaptive quadrature
"""
import ctypes
import functools
import math

import numpy as np
import torch

import aifmm_ls_b200 as aifmm

SERIES = 60        # the far-field series runs over n = -60 .. 60
DEV = "cuda:0"


# ---------------------------------------------------------------- the cases
def _case(name, kind, depth, n_cheb, kappa, q, tol_pow, nrhs, **more):
    return dict(name=name, kind=kind, depth=depth, n_cheb=n_cheb, degree=min(n_cheb, 6), kappa=float(kappa), q=q,
                tol_pow=tol_pow, nrhs=nrhs, **more)


def listed():
    return [
        # the smallest whole call: the reference driver's argv physics, one wave, depth 3 (2,304 unknowns)
        _case("solve_d3_ref_1", "solve", 3, 6, 10, "gaussian160", 8, 1),
        # the largest whole call that fits a short pass: the same physics at depth 6 (147,456 unknowns)
        _case("solve_d6_ref_1", "solve", 6, 6, 10, "gaussian160", 8, 1),
        # the benchmark's physics (kappa 40, wide Gaussian, tolerance 1e-10), 8 right-hand sides
        _case("solve_d5_gauss_8", "solve", 5, 6, 40, "gauss_aw", 10, 8),
        # 8 x 8 nodes, a disk at kappa 80 with a loose tolerance, 32 waves: other block sizes
        _case("solve_d4_disk_32", "solve", 4, 8, 80, "disk", 6, 32),
        # one right-hand side against kept factors, launch by launch, host buffers
        _case("cached_d4_gauss_1", "cached", 4, 6, 40, "gauss_aw", 10, 1, graph=False, device=False),
        # 8 right-hand sides on the device, replayed as a CUDA graph: a serving engine's solve
        _case("cached_d6_gauss_8_graph", "cached", 6, 6, 40, "gauss_aw", 10, 8, graph=True, device=True),
        # refined solves of a kept factorisation
        _case("refined_d4_gauss_8", "refined", 4, 6, 40, "gauss_aw", 10, 8),
        # the mixed form on the depths where it preconditions
        _case("mixed_d3_gauss_8", "mixed", 3, 6, 40, "gauss_aw", 10, 8),
        # the find_error fixture of the reference's default run (depth 5, 36,864 unknowns)
        _case("matvec_d5_ref_1", "matvec", 5, 6, 10, "gaussian160", 8, 1),
        # the field of three solutions
        _case("field_d4_gauss_3", "field", 4, 6, 40, "gauss_aw", 10, 3),
        # 64 sampled rows of the depth-5 matrix, for a residual
        _case("matrix_d5_disk_64", "matrix", 5, 6, 20, "disk", 8, 1, rows=64),
        # the leaf tables of one geometry
        _case("tables_d5_6x6", "tables", 5, 6, 10, "gaussian160", 8, 1),
    ]


def draw(rng):
    """One more case of the same kinds: 4 x 4 to 8 x 8 nodes, wavenumbers 5 to 80,
    tolerances 1e-6 to 1e-10, 1 to 64 right-hand sides (8 for the dense products)."""
    kind = rng.choice(["solve", "solve", "solve", "cached", "cached", "refined", "mixed", "matvec", "field", "matrix",
                       "tables"])
    n = rng.randint(4, 8)
    q = rng.choice(["gaussian160", "gauss_aw", "disk"])
    kappa = round(math.exp(rng.uniform(math.log(5), math.log(80))), 2)
    tol = rng.randint(6, 10)
    nr = int(round(math.exp(rng.uniform(0, math.log(64)))))
    deep = 5 if n <= 6 else 4
    more = {}
    if kind == "solve":
        depth = rng.randint(2, deep)
    elif kind == "cached":
        depth = rng.randint(3, deep)
        more = dict(graph=rng.random() < 0.5, device=rng.random() < 0.5)
    elif kind == "refined":
        depth, nr = rng.randint(3, 4), min(nr, 16)
        kappa = min(kappa, 40.0)
    elif kind == "mixed":
        depth, nr = rng.randint(2, 3), min(nr, 16)
        kappa, q = min(kappa, 40.0), rng.choice(["gaussian160", "gauss_aw"])
    elif kind in ("matvec", "field"):
        depth, nr = rng.randint(2, 4), rng.randint(1, 8)
    elif kind == "matrix":
        depth, nr = rng.randint(3, deep), 1
        more = dict(rows=int(round(math.exp(rng.uniform(0, math.log(100))))))
    else:
        depth, nr = rng.randint(3, 6), 1
    c = _case("", kind, depth, n, kappa, q, tol, nr, **more)
    del c["name"]
    return c


# ---------------------------------------------------------------- geometry, as the solver numbers it
_AMP = {"gaussian160": 1.5, "gauss_aw": 1.5, "disk": 2.0}


def _kw(case, kappa=None):
    return dict(n_cheb=case["n_cheb"], kappa=case["kappa"] if kappa is None else kappa, degree=case["degree"], L=1.0,
                depth=case["depth"], tol_pow=case["tol_pow"], q_kind=case["q"], q_amp=_AMP[case["q"]], q_width=32.0,
                q_radius=0.5)


def _rank(case):
    return case["n_cheb"] ** 2


def _points(case):
    return 4 ** case["depth"] * _rank(case)


def _cheb(n):
    return -np.cos((np.arange(n) + 0.5) / n * np.pi)


def _leaf_xy(depth):
    """leaf grid coordinates in Morton order (children: SW, SE, NE, NW)"""
    k = np.arange(4 ** depth)
    ix, iy = np.zeros_like(k), np.zeros_like(k)
    for level in range(depth):
        c = (k >> (2 * (depth - 1 - level))) & 3
        ix = 2 * ix + ((c == 1) | (c == 2))
        iy = 2 * iy + (c >= 2)
    return ix, iy


def _grid(case):
    """(leaf coordinates, leaf centres, points, contrast)"""
    depth, n = case["depth"], case["n_cheb"]
    h = 1.0 / 2 ** depth
    ix, iy = _leaf_xy(depth)
    centre = np.stack([-1 + (2 * ix + 1) * h, -1 + (2 * iy + 1) * h], 1)
    ch = h * _cheb(n)
    off = np.stack([np.tile(ch, n), np.repeat(ch, n)], 1)
    pts = (centre[:, None, :] + off[None, :, :]).reshape(-1, 2)
    r2 = (pts ** 2).sum(1)
    amp = _AMP[case["q"]]
    q = (amp * np.exp(-160 * r2) if case["q"] == "gaussian160" else amp * np.exp(-32.0 * r2)
         if case["q"] == "gauss_aw" else np.where(np.sqrt(r2) < 0.5, amp, 0.0))
    return np.stack([ix, iy], 1), centre, pts, q


def _bessel(R, nmax):
    """J_0 .. J_nmax (first axis), Y_0 and Y_1: downward recurrence normalised with
    J_0 + 2 sum J_2k = 1, and the Neumann series of Y_0 and Y_1 in the same values"""
    big = max(nmax, float(R.max()))
    N = int(big + 40 + 12 * big ** (1 / 3))
    N += N & 1
    out = torch.empty((nmax + 1,) + R.shape, dtype=torch.float64, device=R.device)
    jp, jc = torch.zeros_like(R), torch.full_like(R, 1e-280)
    norm, s0, s1 = 2 * jc, torch.zeros_like(R), torch.zeros_like(R)
    for k in range(N, 0, -1):
        jp, jc = jc, (2.0 * k / R) * jc - jp
        m = k - 1
        if m <= nmax:
            out[m] = jc
        if m % 2 == 0:
            norm = norm + (2.0 if m else 1.0) * jc
            if m:
                s0 = s0 + (-1) ** (m // 2) / (m // 2) * jc
        else:
            a, b = (m + 1) // 2, (m - 1) // 2
            s1 = s1 + ((-1) ** a / a - ((-1) ** b / b if b else 0.0)) * jc
        if k % 2 == 0:
            f = torch.where(jc.abs() > 1e100, torch.full_like(jc, 1e-100), torch.ones_like(jc))
            jp, jc, norm, s0, s1 = jp * f, jc * f, norm * f, s0 * f, s1 * f
            if m <= nmax:
                out[m:] *= f
    j0, j1, s0, s1 = jc / norm, jp / norm, s0 / norm, s1 / norm
    lg = torch.log(0.5 * R) + 0.57721566490153286
    y0 = (2 / math.pi) * (lg * j0 - 2 * s0)
    y1 = -(2 / math.pi) / R * j0 + (2 / math.pi) * (lg * j1 + s1)
    return out / norm, y0, y1


def _gauss(panels, order=12):
    """composite Gauss-Legendre rule on [-1, 1]^2: points and weights"""
    x, w = np.polynomial.legendre.leggauss(order)
    c = -1 + (2 * np.arange(panels) + 1) / panels
    x = (c[:, None] + x[None, :] / panels).ravel()
    w = np.tile(w / panels, panels)
    X, Y = np.meshgrid(x, x, indexing="ij")
    return torch.tensor(X.ravel(), device=DEV), torch.tensor(Y.ravel(), device=DEV), torch.tensor(
        np.outer(w, w).ravel(), device=DEV)


_CENTRES = [(-2, -2), (0, -2), (2, -2), (2, 0), (2, 2), (0, 2), (-2, 2), (-2, 0), (0, 0)]


@functools.lru_cache(maxsize=32)
def _tables(n, degree, kappa, depth):
    """The leaf tables M (121 x rank) and near (9 x rank x rank) by plain composite
    quadrature: moments of J_n(kappa r |P|) e^{-i n theta} against the tensor
    Chebyshev basis, and of H_0 for the nine colleague positions, times the
    pseudo-inverse of the basis at the nodes."""
    r = 1.0 / 2 ** depth
    ab = [(a, d - a) for d in range(degree) for a in range(d + 1)]
    ch = _cheb(n)
    nx, ny = np.tile(ch, n), np.repeat(ch, n)
    T = lambda v, k: np.cos(k * np.arccos(np.clip(v, -1, 1)))  # noqa: E731
    Qp = torch.tensor(np.linalg.pinv(np.stack([T(nx, a) * T(ny, b) for a, b in ab], 1)), device=DEV)

    def basis(X, Y):
        ax, ay = torch.acos(X.clamp(-1, 1)), torch.acos(Y.clamp(-1, 1))
        return torch.stack([torch.cos(a * ax) * torch.cos(b * ay) for a, b in ab], 1)

    X, Y, W = _gauss(4)
    J = _bessel(kappa * r * torch.hypot(X, Y), SERIES)[0]
    th = torch.atan2(Y, X)
    k = torch.arange(-SERIES, SERIES + 1, device=DEV, dtype=torch.float64)
    sign = 1.0 - 2.0 * ((k < 0) & (k.abs() % 2 == 1)).to(k.dtype)
    F = (sign[:, None] * J[k.abs().long()]) * torch.exp(-1j * k[:, None] * th[None, :]) * W
    M = (r * r) * (F @ basis(X, Y).to(F.dtype)) @ Qp.to(F.dtype)
    # H_0 has a logarithmic singularity at the node: the square is split at the node
    # (or its nearest point) and graded towards it, t -> t^4, in both directions
    t, w = (torch.tensor(0.5 * v, device=DEV) for v in np.polynomial.legendre.leggauss(24))
    t = t + 0.5
    g, dg = t ** 4, 4 * t ** 3 * w
    near = []
    for cx, cy in _CENTRES:
        p = [torch.tensor(v, device=DEV)[:, None] for v in (nx - cx, ny - cy)]
        u, du = [], []
        for v in p:
            c = v.clamp(-1, 1)
            u.append(torch.cat([c + (1 - c) * g, c - (1 + c) * g], 1))
            du.append(torch.cat([(1 - c) * dg, (1 + c) * dg], 1))
        X = u[0][:, :, None].expand(-1, -1, u[1].shape[1]).flatten(1)
        Y = u[1][:, None, :].expand(-1, u[0].shape[1], -1).flatten(1)
        W = (du[0][:, :, None] * du[1][:, None, :]).flatten(1)
        J, y0, _ = _bessel(kappa * r * torch.hypot(p[0] - X, p[1] - Y).clamp(min=1e-18), 0)
        H = torch.complex(J[0], y0) * W
        B = basis(X.flatten(), Y.flatten()).reshape(X.shape + (len(ab),)).to(H.dtype)
        near.append((0.25j * r * r) * (H[:, None, :] @ B)[:, 0] @ Qp.to(H.dtype))
    return M.cpu().numpy(), torch.stack(near).cpu().numpy()


def _rng(case, seed):
    return np.random.default_rng([int(seed), case["depth"], case["n_cheb"], case["nrhs"]])


def _complex(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def _inputs(case, seed):
    """the case's inputs on the host, from the seed alone"""
    rng = _rng(case, seed)
    kind, N, nr = case["kind"], _points(case), case["nrhs"]
    if kind == "tables":
        return {"kappa": case["kappa"] * rng.uniform(0.9, 1.1)}
    if kind == "matvec":
        return {"x": _complex(rng, nr, N)}
    if kind == "field":
        return {"theta": rng.uniform(0, 2 * np.pi, nr), "phi": _complex(rng, nr, N)}
    if kind == "matrix":
        rows = np.sort(rng.choice(N, min(case["rows"], N), replace=False))
        return {"rows": rows.astype(np.int32), "cols": np.arange(N, dtype=np.int32)}
    theta = rng.uniform(0, 2 * np.pi, nr)
    _, _, pts, q = _grid(case)
    ph = case["kappa"] * (np.outer(np.cos(theta), pts[:, 0]) + np.outer(np.sin(theta), pts[:, 1]))
    return {"b": -case["kappa"] ** 2 * q[None, :] * np.exp(1j * ph)}


# ---------------------------------------------------------------- prepare and run
class State:
    """what a user's program holds: the handle, the tree and the inputs"""


def prepare(case, seed):
    s = State()
    s.case, kind = case, case["kind"]
    s.inp = _inputs(case, seed)
    s.K = aifmm.LSKernel(**_kw(case, s.inp.get("kappa")))
    if kind == "tables":
        return s
    s.K.tables_set(*_tables(case["n_cheb"], case["degree"], case["kappa"], case["depth"]))
    if kind in ("matvec", "field", "matrix"):
        return s
    s.T = aifmm.FMM2DTree(s.K)
    if kind == "solve":
        return s
    s.T.createTree()
    s.T.assemble()
    if kind == "cached":
        s.T.factorize()
        if case["device"]:
            s.b = torch.from_numpy(s.inp["b"]).to(DEV)
            s.x = torch.empty_like(s.b)
        if case["graph"]:
            run(s)  # the first graph solve records the graph, once per factorisation
    elif kind == "refined":
        s.T.factorize(keep_assembly=True)
    return s


def _solve_device(s):
    """aifmm_solve on device buffers, ordered after and before the work on torch's stream"""
    lib, N = aifmm.load(), s.K.N
    ptr = ctypes.POINTER(ctypes.c_double)
    flags = aifmm.PTR_DEVICE | (aifmm.SOLVE_GRAPH if s.case["graph"] else 0)
    s.K._ck(lib.aifmm_solve(s.K.h, s.case["nrhs"], ctypes.cast(s.b.data_ptr(), ptr), N,
                            ctypes.cast(s.x.data_ptr(), ptr), N,
                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), flags))
    return s.x


def run(s):
    c, inp = s.case, s.inp
    kind = c["kind"]
    if kind == "solve":
        s.T.createTree()
        s.T.assemble()
        return {"x": s.T.solve(inp["b"])}
    if kind == "cached":
        return {"x": _solve_device(s) if c["device"] else s.T.solve_factored(inp["b"], graph=c["graph"])}
    if kind == "refined":
        x, iterations, _ = s.T.solve_refined(inp["b"], rtol=1e-10, maxit=30)
        return {"x": x, "iterations": iterations}
    if kind == "mixed":
        s.T.factorize(keep_assembly=True, precision=aifmm.PRECISION_C64)
        x, iterations, _ = s.T.solve_refined(inp["b"], rtol=1e-10, maxit=30)
        return {"x": x, "iterations": iterations}
    if kind == "matvec":
        return {"y": s.K.dense_matvec(inp["x"])}
    if kind == "field":
        return {"u": s.K.total_field(inp["theta"], inp["phi"])}
    if kind == "matrix":
        return {"A": s.K.getMatrix(inp["rows"], inp["cols"])}
    s.K.tables_compute(round6=True)
    M, near = s.K.tables_get()
    return {"M": M, "near": near}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    N, r, nr, leaves = _points(case), _rank(case), case["nrhs"], 4 ** case["depth"]
    boxes = leaves * 4 / 3
    kind = case["kind"]
    geometry = 24.0 * N + 16.0 * (121 * r + 9 * r * r)
    if kind in ("solve", "mixed"):
        # per box: the solves and products of one elimination step (about 160 block products)
        return {"bytes": geometry + 32.0 * N * nr, "flops": boxes * (8.0 * 160 * r ** 3 + 8.0 * 30 * r * r * nr)}
    if kind in ("cached", "refined"):
        # every kept block of a box (about 30) read once for all right-hand sides
        return {"bytes": boxes * 16.0 * 30 * r * r + 32.0 * N * nr, "flops": boxes * 8.0 * 30 * r * r * nr}
    if kind in ("matvec", "field"):
        # one Hankel sequence per target and source leaf, and its product with the leaf's moments
        return {"bytes": geometry + 32.0 * N * nr, "flops": N * leaves * 121 * (12.0 + 8.0 * nr)}
    if kind == "matrix":
        return {"bytes": geometry + 16.0 * case["rows"] * N, "flops": case["rows"] * leaves * 121 * (12.0 + 8.0 * r)}
    nb = case["degree"] * (case["degree"] + 1) // 2
    return {"bytes": 16.0 * (121 * r + 9 * r * r), "flops": 500.0 * (121 + 9 * r) * nb * 30.0}


# ---------------------------------------------------------------- 64-bit values
def _rows_of(case, rows, green=False):
    """rows of the dense matrix (or of G, without kappa^2 q and the identity)"""
    n, depth, kappa, r = case["n_cheb"], case["depth"], case["kappa"], _rank(case)
    M, near = (torch.from_numpy(t).to(DEV) for t in _tables(n, case["degree"], kappa, depth))
    xy, centre, pts, q = _grid(case)
    rows = np.asarray(rows)
    d = torch.from_numpy(pts[rows][:, None, :] - centre[None, :, :]).to(DEV)
    R, th = kappa * torch.hypot(d[..., 0], d[..., 1]), torch.atan2(d[..., 1], d[..., 0])
    off = xy[None, :, :] - xy[rows // r][:, None, :]
    close = torch.from_numpy((np.abs(off) <= 1).all(2)).to(DEV)
    R = torch.where(close, torch.full_like(R, 3.0 * kappa / 2 ** depth), R)
    J, ym, yc = _bessel(R, SERIES)
    out = torch.complex(J[0], ym)[..., None] * M[SERIES]
    for k in range(1, SERIES + 1):
        h, e = torch.complex(J[k], yc), torch.exp(1j * k * th)
        out += (h * e)[..., None] * M[SERIES + k] + (h * e.conj() * (-1) ** k)[..., None] * M[SERIES - k]
        ym, yc = yc, (2.0 * k / R) * yc - ym
    out *= 0.25j
    slot = np.array([[0, 1, 2], [7, 8, 3], [6, 5, 4]])
    a, leaf = np.nonzero(close.cpu().numpy())
    which = slot[off[a, leaf, 1] + 1, off[a, leaf, 0] + 1]
    out[a, leaf] = near[which, rows[a] % r]
    out = out.reshape(len(rows), -1)
    if not green:
        out *= torch.from_numpy(kappa ** 2 * q[rows]).to(DEV)[:, None]
        out[torch.arange(len(rows)), torch.from_numpy(rows.astype(np.int64))] += 1.0
    return torch.where(out.abs() < 1e-16, torch.zeros_like(out), out)


def _chunks(case, green=False):
    N = _points(case)
    step = max(1, min(N, int(2.5e7 / N)))
    for i in range(0, N, step):
        rows = np.arange(i, min(N, i + step))
        yield i, _rows_of(case, rows, green)


def _product(case, x, green=False):
    x = torch.from_numpy(x).to(DEV).T.contiguous()
    return torch.cat([A @ x for _, A in _chunks(case, green)]).T.contiguous()


def exact(case, seed):
    kind, N = case["kind"], _points(case)
    inp = _inputs(case, seed)
    if kind == "matvec" and N <= 10000:
        return {"y": _product(case, inp["x"])}
    if kind == "field" and N <= 10000:
        _, _, pts, _ = _grid(case)
        th = inp["theta"]
        ph = case["kappa"] * (np.outer(np.cos(th), pts[:, 0]) + np.outer(np.sin(th), pts[:, 1]))
        return {"u": _product(case, inp["phi"], green=True) + torch.from_numpy(np.exp(1j * ph)).to(DEV)}
    if kind == "matrix" and len(inp["rows"]) * N <= 6e6:
        return {"A": torch.cat([_rows_of(case, inp["rows"][i:i + 64]) for i in range(0, len(inp["rows"]), 64)])}
    if kind in ("solve", "cached") and N <= 2500 and case["q"] != "disk":
        # the exact system's solution: the compression's own error is the solver's
        # accuracy (a disk's jump leaves it too large to say anything)
        A = torch.cat([a for _, a in _chunks(case)])
        return {"x": torch.linalg.solve(A, torch.from_numpy(inp["b"]).to(DEV).T).T.contiguous()}
    return None
