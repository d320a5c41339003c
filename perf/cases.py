"""The work that users of this framework have it do, as timed cases.

Point-cloud transfers at the sizes of the repository's own configurations
(10k, 1M, 2M and 8M points, batches of uneven problems) and in between: setup
with one apply in both forms, from device and from host memory, kNN and
radius neighbourhoods, applies of a kept operator (one field, several
components), the adjoint, batches, and the nearest-neighbour operator.
Neighbourhoods hold at least half as many points again as the basis has
functions, as a transfer in earnest does: fewer leave the moment matrix
near-singular, and then the result is decided by rounding.
"""
from __future__ import annotations

import math

import torch

import datatransferkit_gb300 as dtk

DEV = "cuda:0"
BASES = {"constant": (dtk.Constant, 1), "linear": (dtk.Linear, 4), "quadratic": (dtk.Quadratic, 10)}
# neighbours a target, from and to, for each basis
NEIGHBOURS = {"constant": (4, 16), "linear": (6, 32), "quadratic": (16, 32)}


def listed():
    return [
        # a small coupling interface: latency and launches
        dict(name="mls_fp64_1k", kind="transfer", n_src=1000, n_tgt=1000, basis="linear", rbf=0, k=8,
             precision="fp64", targets="uniform", layout="right"),
        # the plain transfer of the configurations (10k x 10k, k = 20); Kokkos' device layout (LayoutLeft)
        dict(name="mls_fp64_10k", kind="transfer", n_src=10000, n_tgt=10000, basis="quadratic", rbf=2, k=20,
             precision="fp64", targets="uniform", layout="left"),
        # an ordinary mesh-to-mesh transfer of odd sizes in the mixed form
        dict(name="mls_mixed_100k", kind="transfer", n_src=131071, n_tgt=99991, basis="quadratic", rbf=4, k=32,
             precision="mixed", targets="uniform", layout="right"),
        # the FP64 form at scale: 2M sources, a jittered 126^3 grid of targets
        dict(name="mls_fp64_2m", kind="transfer", n_src=2000000, n_tgt=126 ** 3, basis="quadratic", rbf=2, k=32,
             precision="fp64", targets="grid", layout="right"),
        # the headline workload: 8M to 8M points in the mixed form
        dict(name="mls_mixed_8m", kind="transfer", n_src=8000000, n_tgt=8000000, basis="quadratic", rbf=4, k=32,
             precision="mixed", targets="uniform", layout="right"),
        # a transfer whose points and values live in (pinned) host memory
        dict(name="host_mixed_1m", kind="host", n_src=1000003, n_tgt=1000003, basis="quadratic", rbf=4, k=32,
             precision="mixed"),
        # radius neighbourhoods instead of kNN rows (about 120 points each)
        dict(name="radius_fp64_200k", kind="radius", n_src=200000, n_tgt=200000, basis="quadratic", rbf=2,
             mean=120, precision="fp64"),
        # time stepping with a kept operator: one field a step
        dict(name="apply_fp64_2m", kind="apply", n_src=2000000, n_tgt=2000000, basis="linear", rbf=2, k=32,
             precision="fp64", comps=1),
        # a vector field of three components through a kept operator
        dict(name="apply3_mixed_1m", kind="apply", n_src=1000000, n_tgt=1000000, basis="quadratic", rbf=4, k=32,
             precision="mixed", comps=3),
        # forward and backward of a least-squares loss: gradients of the values and of the coordinates
        dict(name="adjoint_1m", kind="adjoint", n_src=1000000, n_tgt=1000000, basis="quadratic", rbf=2, k=32),
        # many uneven transfers set up and applied together (sizes log-uniform in 1e3..1e5)
        dict(name="batch_64", kind="batch", problems=64, lo=1000, hi=100000, k=24, sizes=5),
        # the nearest-neighbour operator
        dict(name="nearest_2m", kind="nearest", n_src=2000000, n_tgt=2000000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["transfer", "transfer", "transfer", "host", "radius", "apply", "adjoint", "batch", "nearest"])
    basis = rng.choice(["linear", "quadratic", "quadratic", "quadratic", "constant"])
    rbf = rng.choice([0, 2, 4])
    k = rng.randint(*NEIGHBOURS[basis])
    if kind == "transfer":
        precision = rng.choice(["fp64", "mixed"])
        hi = 2000000 if precision == "fp64" else 8000000
        return dict(kind=kind, n_src=_log_int(rng, 1000, hi), n_tgt=_log_int(rng, 1000, hi), basis=basis, rbf=rbf,
                    k=k, precision=precision, targets="uniform", layout=rng.choice(["right", "left"]))
    if kind == "host":
        return dict(kind=kind, n_src=_log_int(rng, 1000, 2000000), n_tgt=_log_int(rng, 1000, 2000000), basis=basis,
                    rbf=rbf, k=k, precision=rng.choice(["mixed", "mixed", "fp64"]))
    if kind == "radius":
        # (a corner's neighbourhood has an eighth of the mean)
        mean = rng.randint(*{"constant": (20, 100), "linear": (70, 150), "quadratic": (140, 200)}[basis])
        return dict(kind=kind, n_src=_log_int(rng, 5000, 200000), n_tgt=_log_int(rng, 1000, 200000), basis=basis,
                    rbf=rbf, mean=mean, precision="fp64")
    if kind == "apply":
        return dict(kind=kind, n_src=_log_int(rng, 10000, 4000000), n_tgt=_log_int(rng, 10000, 4000000), basis=basis,
                    rbf=rbf, k=k, precision=rng.choice(["fp64", "mixed"]), comps=rng.choice([1, 1, 2, 3, 5]))
    if kind == "adjoint":
        return dict(kind=kind, n_src=_log_int(rng, 10000, 1000000), n_tgt=_log_int(rng, 10000, 1000000),
                    basis="quadratic", rbf=2, k=rng.randint(20, 32))
    if kind == "batch":
        return dict(kind=kind, problems=rng.randint(2, 64), lo=1000, hi=_log_int(rng, 2000, 100000),
                    k=rng.randint(16, 32), sizes=rng.randint(1, 10 ** 6))
    return dict(kind="nearest", n_src=_log_int(rng, 1000, 4000000), n_tgt=_log_int(rng, 1000, 4000000))


# -- inputs ----------------------------------------------------------------------
def _rand(n, d, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    return torch.rand((n, d), dtype=torch.float64, device=DEV, generator=g)


def _jittered(m, seed):
    i = torch.arange(m, dtype=torch.float64, device=DEV)
    grid = torch.stack(torch.meshgrid(i, i, i, indexing="ij"), dim=-1).reshape(-1, 3)
    return (grid + 0.25 + 0.5 * _rand(m ** 3, 3, seed)) / m


def _field(p, comp=0):
    """sin(2 pi x) cos(2 pi y) + z^2, another phase for each component."""
    return (torch.sin(2 * math.pi * p[:, 0] + comp) * torch.cos(2 * math.pi * p[:, 1]) + p[:, 2] ** 2).contiguous()


def _clouds(case, seed):
    src = _rand(case["n_src"], 3, 10 * seed + 1)
    m = round(case["n_tgt"] ** (1 / 3))
    if case.get("targets") == "grid" and m ** 3 == case["n_tgt"]:
        tgt = _jittered(m, 10 * seed + 2)
    else:
        tgt = _rand(case["n_tgt"], 3, 10 * seed + 2)
    return src, tgt


def _batch_sizes(case):
    g = torch.Generator().manual_seed(int(case["sizes"]))
    u = torch.rand(case["problems"], generator=g, dtype=torch.float64)
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    return torch.exp(lo + u * (hi - lo)).long().tolist()


def _batch_clouds(case, seed):
    """(basis name, sources, targets) of each problem."""
    out = []
    for p, n in enumerate(_batch_sizes(case)):
        basis = "quadratic" if p % 2 else "linear"
        out.append((basis, _rand(n, 3, 1000 * seed + 2 * p + 1), _rand(n, 3, 1000 * seed + 2 * p + 2)))
    return out


def _radius(case):
    """The radius whose ball holds `mean` of the sources in the unit cube."""
    return (3 * case["mean"] / (4 * math.pi * case["n_src"])) ** (1 / 3)


def _basis(name):
    return dtk.MultivariatePolynomialBasis(BASES[name][0], 3)


def _laid(p, layout):
    return p.t().contiguous().t() if layout == "left" else p


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        clouds = _batch_clouds(case, seed)
        problems = [dict(source_points=s, target_points=t, rbf=dtk.Wendland(2), basis=_basis(b), k=case["k"])
                    for b, s, t in clouds]
        values = torch.cat([_field(s) for _, s, _ in clouds])
        return dict(kind=kind, problems=problems, values=values)
    src, tgt = _clouds(case, seed)
    state = dict(kind=kind, case=case)
    if kind == "host":
        for name, v in (("src", src), ("tgt", tgt), ("values", _field(src))):
            state[name] = v.cpu().pin_memory()
        state["out"] = torch.empty(case["n_tgt"], dtype=torch.float64).pin_memory()
        return state
    state["src"], state["tgt"] = _laid(src, case.get("layout")), _laid(tgt, case.get("layout"))
    state["values"] = _field(src)
    state["out"] = torch.empty(case["n_tgt"], dtype=torch.float64, device=DEV)
    if kind == "apply":
        state["op"] = dtk.MovingLeastSquaresOperator(None, src, tgt, dtk.Wendland(case["rbf"]), _basis(case["basis"]),
                                                     k=case["k"], precision=case["precision"])
        if case["comps"] > 1:
            state["values"] = torch.stack([_field(src, c) for c in range(case["comps"])], dim=1)
            state["out"] = torch.empty((case["n_tgt"], case["comps"]), dtype=torch.float64, device=DEV)
    if kind == "adjoint":
        state["op"] = dtk.MovingLeastSquaresOperator(None, src, tgt, dtk.Wendland(case["rbf"]), _basis(case["basis"]),
                                                     k=case["k"], keep_points=True)
        state["wanted"] = _field(tgt, 0.1)
    return state


# -- one pass ----------------------------------------------------------------------
def run(state):
    kind, out = state["kind"], state.get("out")
    if kind == "batch":
        batch = dtk.MovingLeastSquaresBatch(state["problems"])
        out = torch.empty(batch.target_offsets[-1], dtype=torch.float64, device=DEV)
        batch.apply(state["values"], out)
        return out
    if kind == "apply":
        state["op"].apply(state["values"], out)
        return out
    if kind == "adjoint":
        op = state["op"]
        op.apply(state["values"], out)
        residual = out - state["wanted"]
        grad_values, grad_coords = op.apply_adjoint(residual, state["values"], coords=True)
        return dict(values=out, grad_values=grad_values, grad_coords=grad_coords)
    if kind == "nearest":
        op = dtk.NearestNeighborOperator(None, state["src"], state["tgt"])
        op.apply(state["values"], out)
        return out
    case = state["case"]
    rbf, basis = dtk.Wendland(case["rbf"]), _basis(case["basis"])
    if kind == "host":
        dtk.MovingLeastSquaresOperator.transfer_host(None, state["src"], state["tgt"], state["values"], out, rbf,
                                                     basis, k=case["k"], precision=case["precision"])
        return out
    rows = dict(radius=_radius(case)) if kind == "radius" else dict(k=case["k"])
    op = dtk.MovingLeastSquaresOperator(None, state["src"], state["tgt"], rbf, basis, precision=case["precision"],
                                        **rows)
    op.apply(state["values"], out)
    return out


# -- what a pass cannot do without ---------------------------------------------------
def _setup_flops(n_tgt, k, m):
    """Distances, weights, moments, a Cholesky solve and the coefficients."""
    return n_tgt * (k * (8 + 12) + k * m * (m + 1) + m ** 3 / 3 + 4 * m * m + 2 * k * m + 2 * k)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = _batch_sizes(case)
        flops = sum(_setup_flops(s, case["k"], 10 if p % 2 else 4) for p, s in enumerate(n))
        return dict(bytes=sum(n) * (24 + 24 + 8 + 8), flops=flops)
    ns, nt = case["n_src"], case["n_tgt"]
    if kind == "nearest":
        return dict(bytes=ns * (24 + 8) + nt * (24 + 8), flops=8 * nt)
    m = BASES[case["basis"]][1]
    if kind == "apply":
        c = case["comps"]
        coeff = 4 if case["precision"] == "mixed" else 8
        nnz = nt * case["k"]
        return dict(bytes=nnz * (4 + coeff) + 8 * c * (ns + nt), flops=2 * c * nnz)
    if kind == "adjoint":
        nnz = nt * case["k"]
        flops = 4 * nnz + _setup_flops(nt, case["k"], m) + nnz * (10 * m + 40)
        return dict(bytes=nnz * (2 * (4 + 8) + 4) + ns * (24 + 8 + 8 + 24) + nt * (24 + 3 * 8), flops=flops)
    k = case["mean"] if kind == "radius" else case["k"]
    return dict(bytes=ns * (24 + 8) + nt * (24 + 8), flops=_setup_flops(nt, k, m))


# -- the same results in plain torch, 64 bits ----------------------------------------
CHUNK = 1 << 16


class _Grid:
    """The sources in cubic cells of at least the given edge."""

    def __init__(self, src, edge):
        self.lo = src.min(0).values
        extent = float((src.max(0).values - self.lo).max()) or 1.0
        self.g = int(max(1, min(400, extent / edge)))
        self.edge = extent / self.g
        cell = self.cell_of(src)
        key = (cell[:, 0] * self.g + cell[:, 1]) * self.g + cell[:, 2]
        key, self.perm = torch.sort(key)
        counts = torch.bincount(key, minlength=self.g ** 3)
        self.start = torch.cat([counts.new_zeros(1), counts.cumsum(0)])
        self.src = src[self.perm]

    def cell_of(self, p):
        return ((p - self.lo) / self.edge).long().clamp(0, self.g - 1)

    def candidates(self, tgt, reach):
        """(positions in the sorted sources, valid) of every source within `reach` cells."""
        c, g = self.cell_of(tgt), self.g
        z0, z1 = (c[:, 2] - reach).clamp(min=0), (c[:, 2] + reach).clamp(max=g - 1)
        pos, ok = [], []
        for dx in range(-reach, reach + 1):
            for dy in range(-reach, reach + 1):
                x, y = c[:, 0] + dx, c[:, 1] + dy
                inside = (x >= 0) & (x < g) & (y >= 0) & (y < g)
                row = (x.clamp(0, g - 1) * g + y.clamp(0, g - 1)) * g
                first, last = self.start[row + z0], self.start[row + z1 + 1]
                count = torch.where(inside, last - first, 0)
                i = torch.arange(int(count.max()), device=tgt.device)[None]
                pos.append(first[:, None] + i)
                ok.append(i < count[:, None])
        pos, ok = torch.cat(pos, 1), torch.cat(ok, 1)
        return torch.where(ok, pos, 0), ok

    def distances(self, tgt, pos, ok):
        s = self.src
        d2 = (s[:, 0][pos] - tgt[:, :1]).square_()
        for d in (1, 2):
            d2 += (s[:, d][pos] - tgt[:, d:d + 1]).square_()
        return d2.masked_fill_(~ok, math.inf)


def _knn(grid, tgt, k):
    """(indices, valid) of the k nearest sources of each target."""
    k = min(k, grid.src.shape[0])
    idx = torch.empty((tgt.shape[0], k), dtype=torch.int64, device=tgt.device)
    todo, reach = torch.arange(tgt.shape[0], device=tgt.device), 1
    while todo.numel():
        again = []
        for part in todo.split(CHUNK // (reach * reach)):
            t = tgt[part]
            pos, ok = grid.candidates(t, reach)
            if pos.shape[1] < k:
                again.append(part)
                continue
            d2, at = grid.distances(t, pos, ok).topk(k, dim=1, largest=False)
            # nothing nearer can lie in the cells left out
            sure = d2[:, -1] <= (reach * grid.edge) ** 2
            if 2 * reach + 1 >= 2 * grid.g:
                sure |= torch.isfinite(d2[:, -1])
            idx[part[sure]] = grid.perm[pos.gather(1, at)[sure]]
            again.append(part[~sure])
        todo, reach = torch.cat(again), reach + 1
    return idx, torch.ones_like(idx, dtype=torch.bool)


def _within(grid, tgt, radius):
    """(indices, valid) of the sources within the radius, padded."""
    pos, ok = grid.candidates(tgt, 1)
    d2 = grid.distances(tgt, pos, ok)
    ok = torch.sqrt(d2) <= radius
    most = int(ok.sum(1).max())
    d2, at = d2.masked_fill(~ok, math.inf).topk(most, dim=1, largest=False)
    return grid.perm[pos.gather(1, at)], torch.isfinite(d2)


def _weights(rbf, x):
    u = (1 - x).clamp(min=0)
    if rbf == 0:
        return u ** 2
    if rbf == 2:
        return u ** 4 * (4 * x + 1)
    return u ** 6 * (35 * x * x + 18 * x + 3)


def _coefficients(s, t, ok, basis, rbf):
    """Row 0 of the weighted least-squares fit at each target: (n, k)."""
    x = s - t[:, None]
    d2 = x.square().sum(-1).masked_fill(~ok, 0.0)
    dist = torch.where(d2 > 0, d2, 1.0).sqrt() * (d2 > 0)
    r = 1.1 * dist.max(1, keepdim=True).values.clamp(min=10 * 2.220446049250313e-16)
    phi = _weights(rbf, dist / r) * ok
    x = x / r[..., None]
    p = [torch.ones_like(dist)]
    if basis != "constant":
        p += [x[..., 0], x[..., 1], x[..., 2]]
    if basis == "quadratic":
        p += [x[..., i] * x[..., j] for i in range(3) for j in range(i, 3)]
    p = torch.stack(p, -1)
    moments = p.transpose(1, 2) @ (phi[..., None] * p)
    e0 = torch.zeros((p.shape[0], p.shape[2], 1), dtype=p.dtype, device=p.device)
    e0[:, 0] = 1
    a = torch.linalg.solve(moments, e0)
    return phi * (p @ a)[..., 0]


def _spacing(n, k):
    return (3 * k / (4 * math.pi * n)) ** (1 / 3)


def _transfer(src, tgt, values, basis, rbf, k=None, radius=None):
    grid = _Grid(src, radius if radius else 1.5 * _spacing(src.shape[0], k))
    out = []
    for t in tgt.split(CHUNK // 2):
        idx, ok = _within(grid, t, radius) if radius else _knn(grid, t, k)
        c = _coefficients(src[idx], t, ok, basis, rbf)
        v = values[idx]
        out.append((c[..., None] * v).sum(1) if v.dim() == 3 else (c * v).sum(1))
    return torch.cat(out)


def _adjoint(case, src, tgt, values, wanted):
    grid = _Grid(src, 1.5 * _spacing(src.shape[0], case["k"]))
    y = torch.empty(tgt.shape[0], dtype=torch.float64, device=tgt.device)
    grad_values, grad_coords = torch.zeros_like(values), torch.zeros_like(src)
    at = 0
    for t in tgt.split(CHUNK // 2):
        idx, ok = _knn(grid, t, case["k"])
        s = src[idx].requires_grad_(True)
        v = values[idx].requires_grad_(True)
        with torch.enable_grad():
            out = (_coefficients(s, t, ok, case["basis"], case["rbf"]) * v).sum(1)
        residual = out.detach() - wanted[at:at + t.shape[0]]
        gs, gv = torch.autograd.grad(out, (s, v), residual)
        y[at:at + t.shape[0]] = out.detach()
        grad_values.index_add_(0, idx.reshape(-1), gv.reshape(-1))
        grad_coords.index_add_(0, idx.reshape(-1), gs.reshape(-1, 3))
        at += t.shape[0]
    return dict(values=y, grad_values=grad_values, grad_coords=grad_coords)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return torch.cat([_transfer(s, t, _field(s), b, 2, k=case["k"]) for b, s, t in _batch_clouds(case, seed)])
    src, tgt = _clouds(case, seed)
    if kind == "nearest":
        idx, _ = _knn(_Grid(src, 1.5 * _spacing(src.shape[0], 2)), tgt, 1)
        return _field(src)[idx[:, 0]]
    if kind == "adjoint":
        return _adjoint(case, src, tgt, _field(src), _field(tgt, 0.1))
    values = _field(src)
    if kind == "apply" and case["comps"] > 1:
        values = torch.stack([_field(src, c) for c in range(case["comps"])], dim=1)
    rows = dict(radius=_radius(case)) if kind == "radius" else dict(k=case["k"])
    out = _transfer(src, tgt, values, case["basis"], case["rbf"], **rows)
    return out.cpu() if kind == "host" else out
