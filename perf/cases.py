"""The searches and reductions whose speed is followed, through the package's public entry points.

``listed()`` names twelve cases, ``draw(rng)`` makes more of the same ranges: single searches (one to
three dimensions, 1e3 to 1e6 points, every mode and periodicity, COO and CSR, float32 and
float64), multi-level searches of adaptive clouds (up to 2^22 points), queries against a kept
structure, searches of a fixed size replayed step by step, batches of uneven clouds, ``radius`` with
batch vectors, and the scatter reductions over a neighbour list's rows and columns, forward and
backward.

``prepare`` makes a case's inputs on the GPU from a seed, ``run`` is one call (or one simulation
step) on them, ``work`` the bytes and operations the call cannot do without, ``exact`` the float
outputs in 64 bits.  A case's points lie where its sizes put them; the seed gives the order in which
they come (and the values of the reductions), so every seed has other inputs, other indices in
every output, and outputs of the same sizes.
"""
import math

import torch

import torchcompactradius_b200 as tcr
from torchcompactradius_b200.graphs import StaticSearch

DEVICE = "cuda"
FLOATS = {"float16": torch.float16, "float32": torch.float32, "float64": torch.float64}


def listed():
    return [
        # one small scene of a demo or a unit simulation, 64 x 64 particles: latency and launches count
        dict(name="grid_2d_4k_coo", kind="search", dim=2, n=4096, periodic="xy", mode="gather", format="coo",
             neighbours=32, spread=0.0, layout="grid", dtype="float32", algorithm="compact"),
        # the headline search: one 3D scene of 2^20 particles, per-particle supports, once per time step
        dict(name="uniform_3d_1m_csr", kind="search", dim=3, n=1 << 20, periodic="", mode="symmetric", format="csr",
             neighbours=50, spread=0.1, layout="uniform", dtype="float32", algorithm="compact"),
        # an ordinary periodic SPH box of odd size, pairs inside either particle's support
        dict(name="periodic_3d_100k_csr", kind="search", dim=3, n=100003, periodic="xyz", mode="superSymmetric",
             format="csr", neighbours=50, spread=0.1, layout="uniform", dtype="float32", algorithm="compact"),
        # an ordinary 2D channel (periodic along the flow), supports of the neighbours, COO for a graph network
        dict(name="channel_2d_300k_coo", kind="search", dim=2, n=300007, periodic="x", mode="scatter", format="coo",
             neighbours=32, spread=0.2, layout="uniform", dtype="float32", algorithm="compact"),
        # the largest: adaptive resolution, 70% of the particles in dense blobs, supports up to 4x apart
        dict(name="adaptive_3d_4m_mlm_coo", kind="search", dim=3, n=1 << 22, periodic="x", mode="scatter",
             format="coo", neighbours=32, spread=0.0, layout="blobs", dtype="float32", algorithm="mlm"),
        # sampling a kept structure: probe points against a scene that was sorted before
        dict(name="probe_3d_131k_of_1m_coo", kind="existing", dim=3, n=131071, n_ref=1 << 20, periodic="",
             mode="gather", format="coo", neighbours=50, spread=0.1),
        # a double-precision simulation step
        dict(name="float64_3d_150k_csr", kind="search", dim=3, n=150001, periodic="xyz", mode="symmetric",
             format="csr", neighbours=50, spread=0.1, layout="uniform", dtype="float64", algorithm="compact"),
        # the next time step of a scene of fixed size: new positions in, one replayed search
        dict(name="step_3d_65k_csr", kind="static", dim=3, n=65537, periodic="xyz", mode="gather", format="csr",
             neighbours=50, spread=0.1),
        # many scenes of a training set or sweep in one call
        dict(name="batch_256_clouds_csr", kind="batch", clouds=256, smallest=1000, largest=200000, mode="gather",
             format="csr"),
        # the torch_cluster call of a graph network's loader: a mini-batch of clouds as one tensor
        dict(name="radius_batch_96", kind="radius", dim=3, clouds=96, smallest=1000, largest=5000, neighbours=32),
        # an SPH density or a message aggregation and its gradient: one value per pair onto the rows
        dict(name="sum_rows_1m_train", kind="scatter", reduce="sum", rows=1 << 20, neighbours=50, features=1,
             dtype="float32", sorted=True, backward=True),
        # the transposed aggregation: feature vectors of the pairs onto their columns, in no order
        dict(name="mean_columns_100k_f8", kind="scatter", reduce="mean", rows=100003, neighbours=32, features=8,
             dtype="float32", sorted=False, backward=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "search", "mlm", "existing", "static", "batch", "radius", "scatter",
                       "scatter"])
    dim = rng.choice([1, 2, 2, 3, 3, 3])
    periodic = "".join(d for d in "xyz"[:dim] if rng.random() < 0.5)
    mode = rng.choice(["gather", "scatter", "symmetric", "superSymmetric"])
    fmt = rng.choice(["coo", "csr"])
    k = {1: rng.randint(8, 24), 2: rng.randint(16, 40), 3: rng.randint(24, 60)}[dim]
    spread = rng.choice([0.0, 0.1, 0.2])
    if kind == "search":
        return dict(kind="search", dim=dim, n=_log_int(rng, 1000, 1 << 20), periodic=periodic, mode=mode, format=fmt,
                    neighbours=k, spread=spread, layout="uniform", dtype=rng.choice(["float32"] * 3 + ["float64"]),
                    algorithm="compact")
    if kind == "mlm":
        return dict(kind="search", dim=3, n=_log_int(rng, 60000, 1 << 22), periodic=rng.choice(["", "x"]),
                    mode=rng.choice(["gather", "scatter"]), format=fmt, neighbours=32, spread=0.0, layout="blobs",
                    dtype="float32", algorithm="mlm")
    if kind == "existing":
        n_ref = _log_int(rng, 4000, 1 << 20)
        return dict(kind="existing", dim=dim, n=max(500, int(n_ref * rng.uniform(0.05, 0.5))), n_ref=n_ref,
                    periodic=periodic, mode=mode, format=fmt, neighbours=k, spread=spread)
    if kind == "static":
        return dict(kind="static", dim=dim, n=_log_int(rng, 1000, 500000), periodic=periodic, mode=mode, format=fmt,
                    neighbours=k, spread=spread)
    if kind == "batch":
        smallest = _log_int(rng, 1000, 10000)
        return dict(kind="batch", clouds=rng.randint(8, 200), smallest=smallest, largest=smallest * rng.randint(2, 10),
                    mode=mode, format=fmt)
    if kind == "radius":
        smallest = rng.randint(300, 2000)
        return dict(kind="radius", dim=max(dim, 2), clouds=rng.randint(8, 200), smallest=smallest,
                    largest=smallest * rng.randint(2, 5), neighbours=k)
    reduce = rng.choice(["sum", "mean", "max", "min"])
    features = rng.choice([1, 1, 3, 8, 16])
    rows = _log_int(rng, 2000, (1 << 20) // features)
    return dict(kind="scatter", reduce=reduce, rows=rows, neighbours=rng.randint(16, 50), features=features,
                dtype=rng.choice(["float32", "float32", "float16", "float64"]), sorted=rng.random() < 0.6,
                backward=reduce in ("sum", "mean") and rng.random() < 0.5)


# -- inputs ------------------------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(DEVICE).manual_seed(seed)


def _places(case):
    """The generator of a case's point positions: the same for every seed."""
    return _generator(1000 + case.get("n", case.get("rows", case.get("largest", 0))))


def _order(g, *tensors):
    """The points in an order drawn from g."""
    p = torch.randperm(tensors[0].shape[0], generator=g, device=DEVICE)
    return tuple(t.index_select(0, p) for t in tensors)


def _domain(dim, periodic):
    return tcr.DomainDescription(torch.full((dim,), -1.0), torch.full((dim,), 1.0),
                                 torch.tensor([d in periodic for d in "xyz"[:dim]]), dim)


def _support(n, dim, neighbours, extent=2.0):
    """The radius whose ball holds `neighbours` points of n uniform ones in a box of edge `extent`."""
    volume = neighbours * extent ** dim / n
    return {1: volume / 2, 2: math.sqrt(volume / math.pi), 3: (3 * volume / (4 * math.pi)) ** (1 / 3)}[dim]


def _uniform(g, n, dim, neighbours, spread):
    x = torch.rand(n, dim, generator=g, device=DEVICE) * 2 - 1
    h = _support(n, dim, neighbours) * (1 + spread * (2 * torch.rand(n, generator=g, device=DEVICE) - 1))
    return x, h


def _grid(g, n, neighbours):
    """A square of cell centres in [-1, 1]^2, each jittered by a tenth of the spacing."""
    side = math.isqrt(n)
    dx = 2.0 / side
    c = -1 + dx * (torch.arange(side, device=DEVICE) + 0.5)
    x = torch.stack(torch.meshgrid(c, c, indexing="ij"), -1).reshape(-1, 2)
    x = x + (torch.rand(x.shape, generator=g, device=DEVICE) * 0.2 - 0.1) * dx
    return x, torch.full((x.shape[0],), math.sqrt(neighbours * dx * dx / math.pi), device=DEVICE)


def _blobs(g, n, neighbours):
    """70% of the points in eight Gaussian blobs, the rest uniform; supports from the mixture's own
    density, at most 4x apart."""
    sigma, nb = 0.1, int(0.7 * n)
    centres = torch.rand(8, 3, generator=g, device=DEVICE) * 1.6 - 0.8
    pick = torch.randint(0, 8, (nb,), generator=g, device=DEVICE)
    x = torch.cat([centres[pick] + sigma * torch.randn(nb, 3, generator=g, device=DEVICE),
                   torch.rand(n - nb, 3, generator=g, device=DEVICE) * 2 - 1])
    x[:, 0] = torch.remainder(x[:, 0] + 1, 2) - 1
    x = x.clamp(-1.0, 0.999999)
    rho = torch.full((n,), 0.3 * n / 8, device=DEVICE)
    for c in centres:
        d = x - c
        d[:, 0] = torch.remainder(d[:, 0] + 1, 2) - 1
        rho += 0.7 * n / 8 / (2 * math.pi * sigma * sigma) ** 1.5 * torch.exp(-(d * d).sum(1) / (2 * sigma * sigma))
    top = (3 * neighbours / (4 * math.pi * 0.3 * n / 8)) ** (1 / 3)
    return x.contiguous(), ((3 * neighbours / (4 * math.pi * rho)) ** (1 / 3)).clamp(top / 4, top)


def _sizes(g, case):
    u = torch.rand(case["clouds"], generator=g, device=DEVICE).cpu()
    lo, hi = math.log(case["smallest"]), math.log(case["largest"])
    return torch.exp(lo + (hi - lo) * u).long().tolist()


def _pairs(case, seed):
    """A neighbour list's rows (ascending) or columns (points in no order), the values of the pairs
    and the gradient of the reduced output."""
    g = _generator(seed)
    n = case["rows"]
    count = torch.poisson(torch.full((n,), float(case["neighbours"]), device=DEVICE), generator=_places(case)).long()
    count, = _order(g, count)
    index = torch.repeat_interleave(torch.arange(n, device=DEVICE), count)
    if not case["sorted"]:
        index = torch.randint(0, n, index.shape, generator=g, device=DEVICE)
    shape = (index.numel(),) if case["features"] == 1 else (index.numel(), case["features"])
    src = torch.randn(shape, generator=g, device=DEVICE, dtype=torch.float32).to(FLOATS[case["dtype"]])
    grad = torch.randn((n,) + shape[1:], generator=g, device=DEVICE, dtype=torch.float32).to(src.dtype)
    return index, src, grad


def prepare(case, seed):
    kind = case["kind"]
    if kind == "scatter":
        index, src, grad = _pairs(case, seed)
        return dict(case=case, index=index, src=src.requires_grad_(case["backward"]), grad=grad)
    g, places = _generator(seed), _places(case)
    if kind == "batch":
        clouds, domains = [], []
        for k, n in enumerate(_sizes(places, case)):
            dim = 2 + k % 2
            clouds.append(tcr.PointCloud(*_order(g, *_uniform(places, n, dim, 32 if dim == 2 else 50, 0.0))))
            domains.append(_domain(dim, ("", "x", "y", "xy", "xyz"[:dim])[(k // 2) % 5]))
        return dict(case=case, clouds=clouds, domains=domains)
    if kind == "radius":
        sizes = _sizes(places, case)
        n = sum(sizes)
        x = torch.rand(n, case["dim"], generator=places, device=DEVICE)
        x = torch.cat([_order(g, part)[0] for part in x.split(sizes)])
        batch = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes)).to(DEVICE)
        return dict(case=case, x=x, batch=batch, r=_support(n / len(sizes), case["dim"], case["neighbours"], 1.0))
    dim = case["dim"]
    state = dict(case=case, domain=_domain(dim, case["periodic"]))
    if kind == "existing":
        x, h = _uniform(places, case["n_ref"], dim, case["neighbours"], case["spread"])
        q = torch.rand(case["n"], dim, generator=places, device=DEVICE) * 2 - 1
        state["query"] = tcr.PointCloud(*_order(g, q, h[:case["n"]]))
        x, h = _order(g, x, h)
        _, state["structure"] = tcr.radiusSearch(tcr.PointCloud(x, h), mode="symmetric", domain=state["domain"],
                                                 algorithm="compact", format=case["format"], returnStructure=True)
        return state
    if case.get("layout") == "grid":
        x, h = _grid(places, case["n"], case["neighbours"])
    elif case.get("layout") == "blobs":
        x, h = _blobs(places, case["n"], case["neighbours"])
    else:
        x, h = _uniform(places, case["n"], dim, case["neighbours"], case["spread"])
    if kind == "static":
        x, h, move = _order(g, x, h, torch.randn(x.shape, generator=places, device=DEVICE) * 0.05 * h[:, None])
        state["plan"] = StaticSearch(tcr.PointCloud(x, h), state["domain"], mode=case["mode"], format=case["format"])
        state["x"], state["h"] = (x + move).clamp(-1.0, 0.999999), h
        return state
    x, h = _order(g, x, h)
    if case["dtype"] == "float64":
        x, h = x.double(), h.double()
        d = state["domain"]
        state["domain"] = tcr.DomainDescription(d.min.double(), d.max.double(), d.periodic, dim)
    state["cloud"] = tcr.PointCloud(x, h)
    return state


# -- one pass ----------------------------------------------------------------------------------


def _arrays(adj):
    if hasattr(adj, "indptr") and hasattr(adj, "indices"):
        return adj.indices, adj.indptr, adj.rowEntries
    return adj.row, adj.col


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "search":
        return _arrays(tcr.radiusSearch(state["cloud"], mode=case["mode"], domain=state["domain"],
                                        algorithm=case["algorithm"], format=case["format"]))
    if kind == "existing":
        return _arrays(tcr.neighborSearchExisting(state["query"], state["structure"], mode=case["mode"],
                                                  format=case["format"]))
    if kind == "static":
        state["plan"].update(state["x"], state["h"])
        return _arrays(state["plan"].run())
    if kind == "batch":
        adj = tcr.radiusSearchBatch(state["clouds"], mode=case["mode"], domain=state["domains"],
                                    format=case["format"])
        if case["format"] == "csr":
            return adj.col, adj.indptr, adj.rowEntries
        return adj.row, adj.col
    if kind == "radius":
        return tcr.radius(state["x"], None, state["r"], state["batch"])
    reduce = getattr(tcr, "scatter_" + case["reduce"])
    out = reduce(state["src"], state["index"], 0, None, case["rows"])
    if case["backward"]:
        grad, = torch.autograd.grad(out, state["src"], state["grad"])
        return out.detach(), grad
    return out


# -- what a pass cannot do without -------------------------------------------------------------


def work(case):
    """Inputs read once, outputs written once; one distance per pair found, one operation per element
    reduced.  Pair counts from the clouds' mean neighbour numbers."""
    kind = case["kind"]
    if kind == "scatter":
        pairs, size = case["rows"] * case["neighbours"], FLOATS[case["dtype"]].itemsize
        values, out = pairs * case["features"] * size, case["rows"] * case["features"] * size
        if case["reduce"] in ("max", "min"):
            out += case["rows"] * case["features"] * 8
        if case["backward"]:
            values, out = 2 * values, 2 * out
        return {"bytes": 8 * pairs + values + out, "flops": pairs * case["features"]}
    if kind in ("batch", "radius"):
        lo, hi = case["smallest"], case["largest"]
        points = case["clouds"] * (hi - lo) / math.log(hi / lo)  # mean of the log-uniform sizes
        dim = case.get("dim", 2.5)
        pairs = points * case.get("neighbours", 41)
        fmt = case.get("format", "coo")
        queries = points
    else:
        dim, queries = case["dim"], case["n"]
        points = case.get("n_ref", queries)
        pairs = queries * case["neighbours"] * (1.25 if case.get("layout") == "blobs" else 1)
        fmt = case["format"]
    size = 8 if case.get("dtype") == "float64" else 4
    inputs = points * (dim + 1) * size + (queries * (dim + 1) * size if kind == "existing" else 0)
    outputs = 16 * pairs if fmt == "coo" else 8 * pairs + 12 * queries
    return {"bytes": int(inputs + outputs), "flops": int(pairs * 3 * dim)}


def exact(case, seed):
    """The reductions in 64 bits; the searches return indices and counts only."""
    if case["kind"] != "scatter":
        return None
    index, src, grad = _pairs(case, seed)
    n, src = case["rows"], src.double()
    if case["reduce"] in ("max", "min"):
        at = index if src.dim() == 1 else index[:, None].expand_as(src)
        low = float("-inf") if case["reduce"] == "max" else float("inf")
        out = torch.full((n,) + src.shape[1:], low, dtype=torch.float64, device=DEVICE)
        out = out.scatter_reduce(0, at, src, "a" + case["reduce"])
        return out.masked_fill(out.isinf(), 0.0), None
    out = torch.zeros((n,) + src.shape[1:], dtype=torch.float64, device=DEVICE).index_add_(0, index, src)
    count = torch.bincount(index, minlength=n).clamp(min=1).double()
    count = count if src.dim() == 1 else count[:, None]
    mean = case["reduce"] == "mean"
    if mean:
        out = out / count
    if not case["backward"]:
        return out
    grad = grad.double()
    return out, (grad / count if mean else grad).index_select(0, index)
