"""The evaluations that the library's speed is judged on, through its public Python entry points.

A case is one evaluation of potential and forces as a program calls it:

  call "step"     time stepping with particles on the GPU: set_particles (tree), execute, results into device
                  tensors, synchronize.
  call "host"     the same from host arrays and back to host arrays (``results()``), as a CPU code calls it.
  call "charges"  an iterative solver: the tree stays, set_charges, execute, results into device tensors.
  call "batch"    ``Batch.run`` over independent problems of uneven size, host arrays in and out.

``kernel``, ``precision``, ``order``, ``height``, ``nrhs`` are the handle's; ``dist`` is the shape of the particle
cloud ("uniform" in the unit cube, a "plummer" sphere of scale radius 0.1 cut to the cube, points on the surface of
an "ellipsoid" with semi-axes 0.5, 0.3, 0.2); charges are uniform in [-1, 1], on the ellipsoid in [0, 1].
"""
import math

import numpy as np
import torch

import scalfmm_b200 as S

AXES = (0.5, 0.3, 0.2)
PLUMMER_RADIUS = 0.1


def _case(name, call, kernel, precision, order, height, dist, n, nrhs=1, problems=1, smallest=0):
    c = dict(call=call, kernel=kernel, precision=precision, order=order, height=height, dist=dist, n=n, nrhs=nrhs,
             problems=problems, smallest=smallest)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small cloud from a CPU code: launches and latency
        _case("small_host_mixed", "host", "cheb_sym", "mixed", 5, 4, "uniform", 2003),
        # the plain form at the size of a quick CPU-comparable run
        _case("plain_20k_p5", "step", "cheb_sym", "fp64", 5, 5, "uniform", 20000),
        # the reference's published table: 20,000 particles, order 7, height 5, called from the host
        _case("plain_20k_p7_host", "host", "cheb_sym", "fp64", 7, 5, "uniform", 20000),
        # dense operators without the symmetry compression, an odd size
        _case("dense_65k_p5", "step", "cheb_dense", "fp64", 5, 5, "uniform", 65537),
        # order 8, where the truncation error falls below 1e-6
        _case("plain_150k_p8", "step", "cheb_sym", "fp64", 8, 5, "uniform", 150001),
        # one matrix-vector product of an iterative solver
        _case("solver_200k_p6", "charges", "cheb_sym", "mixed", 6, 5, "uniform", 200003),
        # the headline: one million particles, order 7, height 6, in both forms
        _case("headline_mixed", "step", "cheb_sym", "mixed", 7, 6, "uniform", 1000000),
        _case("headline_plain", "step", "cheb_sym", "fp64", 7, 6, "uniform", 1000000),
        # many charge vectors on one tree
        _case("rhs16_mixed", "step", "cheb_sym", "mixed", 7, 5, "uniform", 250007, nrhs=16),
        # a surface: uneven leaves, most of the box empty, Lagrange interpolation
        _case("surface_mixed", "step", "lagrange", "mixed", 6, 7, "ellipsoid", 2000000),
        _case("surface_plain", "step", "lagrange", "fp64", 6, 7, "ellipsoid", 500009),
        # independent clustered problems of uneven size
        _case("batch_mixed", "batch", "cheb_sym", "mixed", 5, 0, "plummer", 300000, problems=12, smallest=10000),
    ]


def _near_sources(dist, n, height):
    """Mean number of sources within a particle's leaf and its neighbours."""
    side = 2.0 ** (height - 1)
    if dist == "uniform":
        return n / side ** 3 * (3.0 - 2.0 / side) ** 3
    if dist == "plummer":  # mean over particles of the density, 45 / (1024 a^3) n
        return min(float(n), 27.0 * (45.0 / 1024.0 / PLUMMER_RADIUS ** 3 * n / side ** 3 + 1.0))
    return min(float(n), 14.3 * (n / (1.9 * side ** 2) + 1.0))  # a surface meets about 14 of the 27 leaves


def _height(dist, n, per_leaf, lowest, highest):
    """Height at which a particle sees about per_leaf others in its own leaf."""
    cells = {"uniform": 27.0, "plummer": 27.0, "ellipsoid": 14.3}[dist]
    best = min(range(lowest, highest + 1), key=lambda h: abs(math.log(_near_sources(dist, n, h) / cells / per_leaf)))
    return best


def _sizes(case):
    """Particle counts of a batch: spread over the logarithm from smallest to n."""
    k, lo, hi = case["problems"], case["smallest"], case["n"]
    return [int(lo * (hi / lo) ** ((j + 0.5) / k)) | 1 for j in range(k)]


def _batch_shape(case, j, n):
    order = case["order"] + j % 3
    return order, _height("plummer", n, 30.0, 4, 7)


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    call = rng.choice(["step", "step", "step", "host", "charges", "batch"])
    if call == "batch":
        lo = size(5000, 20000)
        return _case(None, call, "cheb_sym", rng.choice(["mixed", "mixed", "fp64"]), rng.choice([4, 5]), 0, "plummer",
                     size(40000, 120000), problems=rng.randint(3, 12), smallest=lo)
    precision = rng.choice(["mixed", "mixed", "fp64"])
    kernel = rng.choice(["cheb_sym", "cheb_sym", "cheb_dense", "lagrange"])
    dist = rng.choice(["uniform", "uniform", "plummer", "ellipsoid"])
    order = rng.randint(3, 7 if precision == "mixed" else 8)
    nrhs = rng.choice([1, 1, 1, 1, rng.randint(2, 16)])
    if kernel == "cheb_sym":
        top = 1000000 if precision == "mixed" else 300000
    else:  # the dense operators' work grows with order^6
        top = 500000 if precision == "mixed" else int(60000 * min(1.0, 5.0 / order) ** 6)
    if call == "host":
        top = min(top, 300000)
    n = size(1000, max(2000, top // nrhs))
    height = _height(dist, n, rng.uniform(20.0, 80.0), 3, 6 if kernel != "cheb_sym" and precision == "fp64" else 7)
    return _case(None, call, kernel, precision, order, height, dist, n, nrhs=nrhs)


def _points(dist, n, gen):
    """[3, n] FP64 positions on the GPU."""
    dev = gen.device
    if dist == "uniform":
        return torch.rand(3, n, generator=gen, device=dev, dtype=torch.float64)
    got, have = [], 0
    while have < n:
        u = torch.randn(3, 2 * n, generator=gen, device=dev, dtype=torch.float64)
        u /= u.norm(dim=0)
        t = torch.rand(2 * n, generator=gen, device=dev, dtype=torch.float64)
        if dist == "ellipsoid":  # uniform in area: keep in proportion to the surface element
            a, b, c = AXES
            p = u * torch.tensor(AXES, device=dev, dtype=torch.float64)[:, None]
            area = ((b * c * u[0]) ** 2 + (a * c * u[1]) ** 2 + (a * b * u[2]) ** 2).sqrt()
            p = (p + 0.5)[:, t * max(b * c, a * c, a * b) < area].clamp(0.0, math.nextafter(1.0, 0.0))
        else:
            p = u * (PLUMMER_RADIUS / (t ** (-2.0 / 3.0) - 1.0).sqrt()) + 0.5
            p = p[:, ((p >= 0.0) & (p < 1.0)).all(dim=0)]
        got.append(p)
        have += p.shape[1]
    return torch.cat(got, dim=1)[:, :n].contiguous()


def _particles(dist, n, nrhs, seed):
    """Positions [3, n] and charges [nrhs, n] on the GPU, from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    p = _points(dist, n, gen)
    q = torch.rand(nrhs, n, generator=gen, device="cuda", dtype=torch.float64)
    return p, q if dist == "ellipsoid" else 2.0 * q - 1.0


def prepare(case, seed):
    if case["call"] == "batch":
        problems = []
        for j, n in enumerate(_sizes(case)):
            p, q = _particles(case["dist"], n, 1, seed * 1000 + j)
            order, height = _batch_shape(case, j, n)
            x, y, z = (a.cpu().numpy().copy() for a in p)
            problems.append(dict(x=x, y=y, z=z, q=q[0].cpu().numpy().copy(), order=order, height=height))
        return dict(call="batch", batch=S.Batch(case["kernel"], case["precision"]), problems=problems)
    p, q = _particles(case["dist"], case["n"], case["nrhs"], seed)
    f = S.FMM(case["kernel"], case["order"], case["height"], nrhs=case["nrhs"], precision=case["precision"])
    state = dict(call=case["call"], fmm=f)
    if case["call"] == "host":
        state["particles"] = tuple(a.cpu().numpy().copy() for a in (p[0], p[1], p[2], q.reshape(-1)))
        return state
    state["particles"] = (p[0].contiguous(), p[1].contiguous(), p[2].contiguous(), q.reshape(-1))
    state["out"] = tuple(torch.zeros(case["nrhs"], case["n"], device="cuda", dtype=torch.float64) for _ in range(4))
    torch.cuda.synchronize()  # the handle works on a stream of its own
    if case["call"] == "charges":
        f.set_particles(*state["particles"])
        f.synchronize()
    return state


def run(state):
    if state["call"] == "batch":
        return state["batch"].run(state["problems"])
    f = state["fmm"]
    if state["call"] == "host":
        f.set_particles(*state["particles"])
        f.execute()
        return f.results()
    if state["call"] == "charges":
        f.set_charges(state["particles"][3])
    else:
        f.set_particles(*state["particles"])
    f.execute()
    f.results_into(*state["out"])
    f.synchronize()  # the results are on the handle's stream: waited for before torch reads them
    return state["out"]


def _work_one(kernel, order, height, dist, n, nrhs, moved):
    """Bytes: particles in, results out.  Operations: 20 per ordered near pair and right-hand side; per cell and
    transfer vector the two products of a compressed operator of rank about order^2 / 2 (first product once per
    source cell); P2M and L2P."""
    nn = order ** 3
    rank = order * order / 2.0
    flops = 20.0 * n * _near_sources(dist, n, height)
    cells = 0.0
    for level in range(2, height):
        full = {"uniform": 8.0 ** level, "plummer": min(8.0 ** level, n / 5.0), "ellipsoid": 1.9 * 4.0 ** level}[dist]
        cells += min(full, float(n))
    vectors = 160.0 if dist == "uniform" else 100.0 if dist == "plummer" else 44.0
    flops += cells * vectors * 4.0 * nn * rank + n * 8.0 * nn
    return moved * n, flops * nrhs


def work(case):
    if case["call"] == "batch":
        b = f = 0.0
        for j, n in enumerate(_sizes(case)):
            order, height = _batch_shape(case, j, n)
            b1, f1 = _work_one(case["kernel"], order, height, case["dist"], n, 1, 64.0)
            b, f = b + b1, f + f1
        return {"bytes": b, "flops": f}
    r = case["nrhs"]
    moved = 8.0 * ((0 if case["call"] == "charges" else 3) + 5 * r)
    b, f = _work_one(case["kernel"], case["order"], case["height"], case["dist"], case["n"], r, moved)
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times the measured distance between two correct evaluations at the precision: FP64 with its M2L
    sums in another order (up to 2.2e-14, largest single value 2e-13 at 20,000 particles), MIXED against FP64 (up
    to 8e-7, largest single value 2e-5; equispaced nodes on clustered particles 1.4e-6, 6e-5)."""
    if case["precision"] == "fp64":
        return {"rel": 1e-13, "max": 4e-12}
    if case["kernel"] == "lagrange":
        return {"rel": 6e-6, "max": 2.4e-4}
    return {"rel": 3e-6, "max": 8e-5}


def _direct(p, q):
    """Direct sum in 64 bits: [nrhs, n] potential and forces."""
    nrhs, n = q.shape
    out = torch.zeros(4, nrhs, n, device=p.device, dtype=torch.float64)
    rows = max(1, min(n, 4000000 // n))
    qt = q.t().contiguous()
    for a in range(0, n, rows):
        b = min(n, a + rows)
        d = [p[k, a:b, None] - p[k, None, :] for k in range(3)]
        r2 = d[0] * d[0]
        r2.addcmul_(d[1], d[1]).addcmul_(d[2], d[2])
        own = torch.arange(a, b, device=p.device)
        r2[own - a, own] = math.inf
        inv = r2.rsqrt_()
        out[0, :, a:b] = (inv @ qt).t()
        inv3 = inv * inv * inv
        for k in range(3):
            out[1 + k, :, a:b] = -q[:, a:b] * (d[k].mul_(inv3) @ qt).t()
    return out


def exact(case, seed):
    if case["call"] == "batch":
        sizes = _sizes(case)
        if sum(float(n) * n for n in sizes) > 2e11:
            return None
        got = []
        for j, n in enumerate(sizes):
            p, q = _particles(case["dist"], n, 1, seed * 1000 + j)
            o = _direct(p, q)
            got.append({k: o[i, 0].cpu().numpy() for i, k in enumerate(("phi", "fx", "fy", "fz"))})
        return got
    n, r = case["n"], case["nrhs"]
    if float(n) * n * (1 + r / 4.0) > 3e11:
        return None
    o = _direct(*_particles(case["dist"], n, r, seed))
    if case["call"] == "host":
        shape = (r, n) if r > 1 else (n,)
        return {k: o[i].cpu().numpy().reshape(shape) for i, k in enumerate(("phi", "fx", "fy", "fz"))}
    return tuple(o[i] for i in range(4))
