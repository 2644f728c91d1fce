"""The work this framework is used for, as cases that can be timed and checked.

Sizes are those of the repository's configurations (40^3, 64x64x48, the
serving grids), of its tests and of ragged grids between them; models are the
benchmark's layered models with a seeded random perturbation, frequencies the
benchmark's 0.5 .. 2 Hz.  Refinement goes to 1e-11, one decade beyond the job
protocol's target, so that wavefields of two builds can be compared.
"""
import math

import numpy as np
import torch

import wtomo3d_gb300 as wt
from wtomo3d_gb300 import model

TOL = 1e-11
MAXIT = 60


def listed():
    return [
        # one source on the smallest test grid with factors at hand: the latency of a call
        dict(name="solve1_14x12x13", kind="solve", nx=14, ny=12, nz=13, dx=20.0, freq=1.5, nrhs=1, adjoint=False),
        # the FP64 handle that results are verified with
        dict(name="fp64_16x15x14", kind="frequency", nx=16, ny=15, nz=14, dx=25.0, freq=1.0, nrhs=4, fp64=True),
        # a frequency of a small survey: assembly, factors, plane-wave sources, wavefields
        dict(name="frequency_24x22x20", kind="frequency", nx=24, ny=22, nz=20, dx=20.0, freq=2.0, nrhs=8, fp64=False),
        # a caller's own matrix (19-point discretisation, general ordering), a few sources from the host
        dict(name="csr_21x19x17", kind="csr", nx=21, ny=19, nz=17, dx=25.0, freq=3.0, nrhs=3),
        # what the job protocol does per frequency: complex64 values from the host, factor, one source
        dict(name="values1_29x27x25", kind="values", nx=29, ny=27, nz=25, dx=25.0, freq=2.0, nrhs=1),
        # conjugate-transpose solves of an inversion on an odd grid
        dict(name="adjoint16_33x31x29", kind="solve", nx=33, ny=31, nz=29, dx=20.0, freq=1.0, nrhs=16, adjoint=True),
        # a misfit gradient: forward and adjoint solves, contraction
        dict(name="gradient_32x32x24", kind="gradient", nx=32, ny=32, nz=24, dx=25.0, freq=1.0, nrhs=16, nrx=8, nry=5),
        # one source with factors at hand on the 40^3 configuration
        dict(name="solve1_40x40x40", kind="solve", nx=40, ny=40, nz=40, dx=25.0, freq=1.0, nrhs=1, adjoint=False),
        # a frequency of the 40^3 configuration
        dict(name="frequency_40x40x40", kind="frequency", nx=40, ny=40, nz=40, dx=25.0, freq=1.0, nrhs=32, fp64=False),
        # the serving loop's batch: 64 columns on resident factors
        dict(name="solve64_48x48x48", kind="solve", nx=48, ny=48, nz=48, dx=20.0, freq=1.5, nrhs=64, adjoint=False),
        # a line search's step: the operator of the current model and its products
        dict(name="operator_64x64x48", kind="operator", nx=64, ny=64, nz=48, dx=25.0, freq=1.0, nrhs=32),
        # a frequency of the inversion configuration
        dict(name="frequency_64x64x48", kind="frequency", nx=64, ny=64, nz=48, dx=25.0, freq=1.0, nrhs=32, fp64=False),
    ]


def draw(rng):
    kind = rng.choice(["solve", "solve", "frequency", "frequency", "values", "csr", "gradient", "operator"])
    # nodes of the grid, spread over the logarithm; sides within a factor of ~1.5 of each other
    lo, hi = {"solve": (1500, 125000), "frequency": (2500, 125000), "values": (2500, 30000), "csr": (1500, 9000),
              "gradient": (4000, 60000), "operator": (8000, 190000)}[kind]
    side = math.exp(rng.uniform(math.log(lo), math.log(hi))) ** (1.0 / 3.0)
    nx, ny = (max(8, round(side * math.exp(rng.uniform(-0.2, 0.2)))) for _ in range(2))
    nz = min(max(8, round(side ** 3 / (nx * ny))), hi // (nx * ny))
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, dx=rng.choice([20.0, 25.0]), freq=rng.choice([1.0, 1.5, 2.0]))
    if kind == "solve":
        c.update(nrhs=rng.choice([1, 1, 2, 5, 16, 31, 32, 48, 64]), adjoint=rng.random() < 0.4)
    elif kind == "frequency":
        fp64 = nx * ny * nz <= 4000 and rng.random() < 0.5
        c.update(nrhs=rng.choice([1, 4, 8, 16, 29, 32]), fp64=fp64)
    elif kind == "gradient":
        c.update(nrhs=rng.choice([4, 8, 16]), nrx=rng.randint(3, 8), nry=rng.randint(2, 6))
    elif kind == "operator":
        c.update(nrhs=rng.choice([1, 7, 16, 32]))
    else:
        c.update(nrhs=rng.choice([1, 1, 2, 3, 8]))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _grid(c):
    """The case's grid, absorbing layers of 10 nodes or a quarter of the smallest side."""
    return wt.Grid(c["nx"], c["ny"], c["nz"], c["dx"], pmld=_layers(c) * c["dx"], fst=1, usemin=1)


def _layers(c):
    return min(10, min(c["nx"], c["ny"], c["nz"]) // 4)


def _model(c, seed):
    return model.layered_random(c["nx"], c["ny"], c["nz"], c["dx"], seed=seed)


def _omega(c):
    return 2 * math.pi * c["freq"]


def _point_forces(c, rng, k):
    """Positions inside the absorbing layers, below the surface, and components."""
    pad = _layers(c) * c["dx"]
    hi = np.array([c["nx"] - 1, c["ny"] - 1, c["nz"] - 1]) * c["dx"]
    lo = np.array([pad, pad, c["dx"]])
    return rng.uniform(lo, np.maximum(hi - pad, lo + c["dx"]), size=(k, 3)), rng.integers(0, 3, k)


def _plane_waves(rng, k):
    """Incidence 0.05 .. 30 degrees, any back-azimuth, as the benchmark draws them."""
    return np.radians(np.maximum(rng.uniform(0.0, 30.0, k), 0.05)), np.radians(rng.uniform(0.0, 360.0, k))


def _device_blocks(c, k, count):
    n = 3 * c["nx"] * c["ny"] * c["nz"]
    return [torch.zeros((k, n), dtype=torch.complex128, device="cuda") for _ in range(count)]


class _Stencil:
    """A caller's elastic operator: centred second differences of the wave
    equation (19 points, 3 components) on a smooth random medium, with
    absorption growing towards the sides.  Node (iz, ix, iy) is
    iz + nz (ix + nx iy), its 3 rows adjacent, columns ascending."""

    def __init__(self, c, seed, full):
        nx, ny, nz, h = c["nx"], c["ny"], c["nz"], c["dx"]
        vp, vs, rho = (a.astype(np.float64).transpose(2, 1, 0) for a in _model(c, seed))   # (ny, nx, nz)
        mu = vs * vs * rho
        lam = vp * vp * rho - 2 * mu
        self.shape, om2 = (ny, nx, nz), _omega(c) ** 2
        axis_of = {0: 1, 1: 0, 2: 2}   # component u, v, w -> array axis of x, y, z
        offs = [(y, x, z) for y in (-1, 0, 1) for x in (-1, 0, 1) for z in (-1, 0, 1)]
        if not full:                   # the grid graph has all 27, the caller's own matrix the 19 used
            offs = [o for o in offs if sum(map(abs, o)) <= 2]
        self.offsets = offs
        shape = self.shape
        self.blocks = np.zeros((len(offs), 3, 3) + shape, np.complex128)
        self.inside = np.zeros((len(offs),) + shape, bool)
        side = np.zeros(shape)
        for ax, m in enumerate(shape):
            i = np.arange(m)
            d = np.maximum(0, _layers(c) - np.minimum(i, m - 1 - i)) / max(1, _layers(c))
            side = np.maximum(side, (d ** 2).reshape([-1 if a == ax else 1 for a in range(3)]))
        diag = np.zeros((3, 3) + shape, np.complex128)
        for q, o in enumerate(offs):
            dst, src = self._cut(o)
            self.inside[q][dst] = True
            if o == (0, 0, 0):
                continue
            la, mm = lam.copy(), mu.copy()
            la[dst], mm[dst] = 0.5 * (lam[dst] + lam[src]), 0.5 * (mu[dst] + mu[src])
            if sum(map(abs, o)) == 1:
                for a in range(3):
                    k = (la + 2 * mm if o[axis_of[a]] else mm) / h ** 2
                    self.blocks[q, a, a] = -k
                    diag[a, a] += k
            elif sum(map(abs, o)) == 2:
                a, b = (a for a in range(3) if o[axis_of[a]])
                self.blocks[q, a, b] = self.blocks[q, b, a] = -(la + mm) * (o[axis_of[a]] * o[axis_of[b]]) / (4 * h ** 2)
        for a in range(3):
            diag[a, a] += -om2 * rho * (1 + 0.02j) - 1j * 0.2 * side * mu / h ** 2
        self.blocks[offs.index((0, 0, 0))] = diag
        self.blocks *= self.inside[:, None, None]

    def _cut(self, o):
        """Slices (row node, column node) that have a neighbour at offset o."""
        dst = tuple(slice(max(0, -d), m - max(0, d)) for d, m in zip(o, self.shape))
        src = tuple(slice(max(0, d), m - max(0, -d)) for d, m in zip(o, self.shape))
        return dst, src

    def csr(self):
        ny, nx, nz = self.shape
        nn = ny * nx * nz
        q = len(self.offsets)
        node = np.arange(nn).reshape(self.shape)
        step = np.array([z + nz * (x + nx * y) for y, x, z in self.offsets])
        mask = np.broadcast_to(self.inside.reshape(q, nn).T[:, None, :, None], (nn, 3, q, 3))
        cols = np.broadcast_to(3 * (node.reshape(nn, 1, 1, 1) + step[:, None]) + np.arange(3), (nn, 3, q, 3))
        vals = self.blocks.reshape(q, 3, 3, nn).transpose(3, 1, 0, 2)
        indptr = np.zeros(3 * nn + 1, np.int32)
        np.cumsum(mask.reshape(3 * nn, -1).sum(1), out=indptr[1:])
        return indptr, cols[mask].astype(np.int32), vals[mask]

    def times(self, x):
        """A x for x of shape (k, ny, nx, nz, 3)."""
        y = np.zeros_like(x)
        for q, o in enumerate(self.offsets):
            dst, src = self._cut(o)
            y[(slice(None),) + dst] += np.einsum("abyxz,kyxzb->kyxza", self.blocks[q][(slice(None), slice(None)) + dst],
                                                 x[(slice(None),) + src], optimize=True)
        return y


def _wavefields(c, seed):
    """k band-limited wavefields that vanish towards the sides, (k, ny, nx, nz, 3)."""
    rng = np.random.default_rng([seed, 77])
    shape, k = (c["ny"], c["nx"], c["nz"]), c["nrhs"]
    at = np.meshgrid(*[np.arange(m) / m for m in shape], indexing="ij")
    window = np.prod([np.sin(np.pi * (a + 0.5 / m)) ** 2 for a, m in zip(at, shape)], axis=0)
    x = np.zeros((k,) + shape + (3,), np.complex128)
    for j in range(k):
        for a in range(3):
            for _ in range(3):
                w = rng.uniform(-4, 4, 3)
                f = rng.standard_normal() + 1j * rng.standard_normal()
                x[j, ..., a] += f * np.exp(2j * np.pi * sum(t * s for t, s in zip(w, at)))
    return x * window[..., None]


def _stencil(c, seed):
    s = _Stencil(c, seed, full=c["kind"] == "values")
    if c["kind"] == "values":   # the caller's values are complex64
        s.blocks = s.blocks.astype(np.complex64).astype(np.complex128)
    return s


def prepare(c, seed):
    rng = np.random.default_rng([seed, 5])
    kind, k = c["kind"], c["nrhs"]
    st = dict(case=c)
    if kind in ("values", "csr"):
        s = _stencil(c, seed)
        indptr, indices, vals = s.csr()
        st["B"] = np.ascontiguousarray(s.times(_wavefields(c, seed)).reshape(k, -1)).T   # (n, k), columns contiguous
        if kind == "csr":
            st["solver"], st["a"], st["dtype"] = wt.Solver.from_csr(indptr, indices), vals, np.complex128
        else:
            st["solver"], st["a"], st["dtype"] = wt.Solver(_grid(c)), vals.astype(np.complex64), np.complex64
        return st
    s = st["solver"] = wt.Solver(_grid(c), wt.PREC_FP64 if c.get("fp64") else wt.PREC_MIXED)
    s.set_model(*_model(c, seed))
    if kind == "frequency":
        s.set_background(*model.layered(c["nx"], c["ny"], c["nz"]))
        st["layers"] = wt.Layered1D(*model.layered1d(c["nz"], c["dx"]))
        st["waves"] = _plane_waves(rng, k)
        st["F"], st["X"] = _device_blocks(c, k, 2)
        return st
    s.factor(_omega(c))
    if kind == "operator":
        st["X"] = torch.view_as_complex(torch.from_numpy(rng.standard_normal((k, s.n, 2))).cuda())
        st["Y"] = _device_blocks(c, k, 1)[0]
        return st
    st["F"], st["X"] = _device_blocks(c, k, 2)
    xyz, comp = _point_forces(c, rng, k)
    s.rhs_sources(xyz, comp, st["F"].data_ptr())
    if kind == "gradient":
        st["rec"] = model.surface_receivers(c["nx"], c["ny"], c["nz"], _layers(c), c["nrx"], c["nry"])
        # observed data: the predicted ones at a perturbed amplitude
        s.solve_device(st["F"].data_ptr(), st["X"].data_ptr(), k, tol=TOL, maxit=MAXIT)
        u = st["X"].view(k, -1, 3)[:, torch.from_numpy(st["rec"]).cuda()].cpu().numpy()
        st["dobs"] = u * (1 + 0.3 * (rng.standard_normal(u.shape) + 1j * rng.standard_normal(u.shape)))
    return st


def run(st):
    c, s = st["case"], st["solver"]
    kind, k = c["kind"], c["nrhs"]
    if kind in ("values", "csr"):
        s.set_values(st["a"], st["dtype"])
        return s.solve(st["B"], tol=TOL, maxit=MAXIT)
    if kind == "operator":
        s.update_operator()
        s.apply_device(st["X"].data_ptr(), st["Y"].data_ptr(), k)
        return st["Y"]
    if kind == "gradient":
        chi, grad, dpred = s.misfit_gradient(st["F"].data_ptr(), None, k, st["rec"], st["dobs"], tol=TOL, maxit=MAXIT)
        return dict(chi=chi, grad=grad, dpred=dpred)
    if kind == "frequency":
        s.factor(_omega(c))
        s.rhs_planewave(st["layers"], *st["waves"], d_F=st["F"].data_ptr())
    s.solve_device(st["F"].data_ptr(), st["X"].data_ptr(), k, tol=TOL, maxit=MAXIT, adjoint=c.get("adjoint", False))
    return [st["F"], st["X"]] if kind == "frequency" else st["X"]


def exact(c, seed):
    """The wavefields that the right-hand sides of the caller's operators were made from."""
    if c["kind"] not in ("values", "csr"):
        return None
    return np.ascontiguousarray(_wavefields(c, seed).reshape(c["nrhs"], -1)).T


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _fill(dims, leaf=64):
    """(entries, flops) of the factors of a plane-separator nested dissection
    of the box, by recursion: every separator plane is a front whose border is
    the part of the box's sides that earlier separators cover."""
    def go(d, cut):
        m = 3 * d[0] * d[1] * d[2]
        faces = [d[1] * d[2], d[0] * d[2], d[0] * d[1]]
        border = 3 * sum(faces[a] * cut[a] for a in range(3))
        if d[0] * d[1] * d[2] <= leaf:
            p, kids = m, []
        else:
            a = max(range(3), key=lambda i: d[i])
            p = 3 * faces[a]
            half = [(d[a] - 1) // 2, d[a] - 1 - (d[a] - 1) // 2]
            left, right = cut[a] - cut[a] // 2, cut[a] // 2
            kids = [(tuple(half[0] if i == a else v for i, v in enumerate(d)),
                     tuple(left + 1 if i == a else v for i, v in enumerate(cut))),
                    (tuple(half[1] if i == a else v for i, v in enumerate(d)),
                     tuple(right + 1 if i == a else v for i, v in enumerate(cut)))]
        e, f = p * p + 2.0 * p * border, 8.0 * (p ** 3 / 3 + p * p * border + p * border * border)
        for q in kids:
            if min(q[0]) > 0:
                key = (q[0], tuple(min(2, v) for v in q[1]))
                if key not in memo:
                    memo[key] = go(*key)
                e, f = e + memo[key][0], f + memo[key][1]
        return e, f
    memo = {}
    return go(tuple(dims), (0, 0, 0))


def work(c):
    """What one pass cannot do without: the operator's values and the model
    read or written once, the factors written once by a factorisation and read
    once by a solve (one pass of substitutions per 32 sources and one residual
    at least), sources read and wavefields written."""
    nx, ny, nz, k = c["nx"], c["ny"], c["nz"], c["nrhs"]
    n = 3 * nx * ny * nz
    nnz = 9 * (3 * nx - 2) * (3 * ny - 2) * (3 * nz - 2)
    entries, flops = _fill((nx, ny, nz))
    size = 16 if c.get("fp64") else 8
    passes = -(-k // 32)
    solve_bytes = passes * (entries * size + nnz * 16) + 2 * 16.0 * n * k
    solve_flops = (8.0 * entries + 8.0 * nnz) * k
    kind = c["kind"]
    if kind == "operator":
        return {"bytes": 16.0 * nnz + 2 * 16.0 * n * k + 12.0 * n / 3, "flops": 8.0 * nnz * k}
    if kind == "solve":
        return {"bytes": solve_bytes, "flops": solve_flops}
    if kind == "gradient":
        return {"bytes": 2 * solve_bytes + 2 * 16.0 * n * k + 8.0 * n,
                "flops": 2 * solve_flops + 8.0 * 27 * 9 * (n / 3) * k}
    source = 2 * 16.0 * nnz if kind == "frequency" else 0.0   # the operator and its background
    return {"bytes": solve_bytes + entries * size + 16.0 * nnz + source,
            "flops": solve_flops + flops + (16.0 * nnz * k if kind == "frequency" else 0.0)}
