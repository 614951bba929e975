"""Performance cases of the Wilson-flow engine: what its users have it do, by size, precision and entry point.

A case is a dict of plain values with a "kind":

  flow       links in (page-locked host memory in file order, or the engine's own generator), ``Lattice.flow``,
             E(t), Q(t) and their x0 profiles out, with the flowed links where the program saves them
  measure    ``Lattice.measure`` of a resident configuration (E, Q and their profiles)
  densities  ``Lattice.site_densities`` and ``Lattice.measure_flowed`` (the q-density and flowed-measurement workflows)
  noalloc    ``lgf_measure_noalloc`` on links that another allocator holds in device memory
  heatbath   ``Lattice.heatbath`` (Cabibbo-Marinari + overrelaxation sweeps), ``Lattice.plaquette`` and the new links
  batch      ``Context.batch_run`` of an ensemble of uneven volumes

Links are exp(i s H), H Gaussian traceless Hermitian per link (s = 0.5, the generator of the throughput configurations:
about as rough as beta = 6 configurations), made on the GPU from the seed.  Numbers of an FP32-mixed flow are
float32 numbers, so they come back as float32; the rest is float64.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from msc_project_b200 import FP32MIXED, FP64, Context
from msc_project_b200.lgf import Job

EPS = 0.01  # the flow step of every configuration of this repository


# --------------------------------------------------------------------- cases
def _flow(name, shape, prec, steps, every, source, links_out, t0=0.0, at_t0=True):
    c = {"name": name, "kind": "flow", "n0": shape[0], "n1": shape[1], "n2": shape[2], "n3": shape[3], "precision": prec,
         "steps": steps, "every": every, "reunit": 10 if prec == "fp32mixed" else 0, "t0": t0, "at_t0": at_t0,
         "source": source, "links_out": links_out}
    return c


def _lat(name, kind, shape, prec="fp64", **more):
    return {"name": name, "kind": kind, "n0": shape[0], "n1": shape[1], "n2": shape[2], "n3": shape[3], "precision": prec, **more}


def listed():
    return [
        # the smallest job, every extent different: launches and latency are all of it
        _flow("flow_4x6x8x10_fp64", (4, 6, 8, 10), "fp64", 20, 5, "host", True),
        # the parity workload as a user runs it: 8^4, t = 1, E and Q after every step, flowed links saved
        _flow("flow_8x8x8x8_fp64", (8, 8, 8, 8), "fp64", 100, 1, "host", True),
        # an ordinary lattice that fits L2: measured every 10 steps, flowed links saved
        _flow("flow_16x16x16x16_fp64", (16, 16, 16, 16), "fp64", 50, 10, "host", True),
        # the bench lattice: a saved configuration in, flowed, its links saved
        _flow("flow_48x24x24x24_fp64", (48, 24, 24, 24), "fp64", 40, 10, "host", True),
        # the largest lattice of the served stream, in double: generated on the device, observables out
        _flow("flow_48x48x48x48_fp64", (48, 48, 48, 48), "fp64", 6, 3, "device", False),
        # the FP32-mixed throughput lattice, reunitarised every 10 steps
        _flow("flow_32x32x32x32_fp32mixed", (32, 32, 32, 32), "fp32mixed", 50, 10, "device", False),
        # a resumed FP32-mixed flow on a ragged lattice (slices that are no multiple of 32 sites), measured often
        _flow("flow_6x10x14x18_fp32mixed", (6, 10, 14, 18), "fp32mixed", 40, 5, "host", True, t0=1.0, at_t0=False),
        # one measurement of a resident configuration of the bench lattice
        _lat("measure_48x24x24x24_fp64", "measure", (48, 24, 24, 24)),
        # topological-charge density and flowed observables of an analysis-sized configuration
        _lat("densities_32x16x16x16_fp64", "densities", (32, 16, 16, 16)),
        # the measurement for callers whose memory another allocator owns
        _lat("noalloc_32x16x16x16_fp64", "noalloc", (32, 16, 16, 16)),
        # two ensemble updates (heatbath + 5 overrelaxation sweeps each), the plaquette and the new configuration
        _lat("heatbath_32x16x16x16_fp64", "heatbath", (32, 16, 16, 16), iters=2, over=5, beta=6.0),
        # an ensemble of uneven volumes in one call, FP32-mixed, as the 64-configuration ensemble is made up
        {"name": "batch_uneven_fp32mixed", "kind": "batch", "precision": "fp32mixed", "steps": 40, "every": 10, "reunit": 10,
         "volumes": "8x8x8x8*4,12x12x12x12*4,16x16x16x16*4,32x16x16x16*2"},
    ]


def _extents(rng, least, most):
    """Four even extents whose volume is spread over the logarithm of [least, most]."""
    target = math.exp(rng.uniform(math.log(least), math.log(most)))
    side = target ** 0.25
    while True:
        n = [max(4, min(64, 2 * round(side * math.exp(rng.uniform(-0.5, 0.5)) / 2))) for _ in range(3)]
        last = max(4, min(96, 2 * round(target / (n[0] * n[1] * n[2]) / 2)))
        n.insert(rng.randrange(4), last)
        if least / 2 <= math.prod(n) <= most and max(n) <= 64:
            return tuple(n)


def draw(rng):
    kind = rng.choice(["flow", "flow", "flow", "flow", "measure", "densities", "noalloc", "heatbath", "batch"])
    if kind == "flow":
        prec = rng.choice(["fp64", "fp32mixed"])
        shape = _extents(rng, 500, 2.0e6)
        V = math.prod(shape)
        steps = max(3, min(60, int(rng.uniform(0.3, 1.0) * 2.0e7 / V)))
        every = rng.choice([1, 2, 5, 10]) if V < 100000 else rng.choice([5, 10, 10])
        host = V < 800000 and rng.random() < 0.7
        c = _flow("", shape, prec, steps, every, "host" if host else "device", host and (prec == "fp64" or V < 100000),
                  t0=rng.choice([0.0, 1.0]), at_t0=rng.random() < 0.7)
    elif kind == "batch":
        sides = [4, 6, 8, 10, 12, 14, 16]
        parts = ["%dx%dx%dx%d*%d" % (rng.choice(sides), rng.choice(sides), rng.choice(sides), rng.choice(sides), rng.randint(1, 5))
                 for _ in range(rng.randint(2, 5))]
        prec = rng.choice(["fp64", "fp32mixed"])
        c = {"kind": "batch", "precision": prec, "steps": rng.randint(10, 50), "every": rng.choice([2, 5, 10]),
             "reunit": 10 if prec == "fp32mixed" else 0, "volumes": ",".join(parts)}
    elif kind == "heatbath":
        c = _lat("", "heatbath", _extents(rng, 500, 4.0e5), rng.choice(["fp64", "fp64", "fp32mixed"]), iters=rng.randint(1, 2),
                 over=rng.randint(1, 5), beta=round(rng.uniform(5.6, 6.4), 2))
    else:
        most = {"measure": 2.0e6, "densities": 4.0e5, "noalloc": 7.0e5}[kind]
        c = _lat("", kind, _extents(rng, 500, most), rng.choice(["fp64", "fp32mixed"]) if kind == "measure" else "fp64")
    c.pop("name", None)
    return c


def _shape(case):
    return tuple(case["n%d" % d] for d in range(4))


def _volumes(case):
    out = []
    for part in case["volumes"].split(","):
        s, n = part.split("*")
        out += [tuple(int(x) for x in s.split("x"))] * int(n)
    return out


def _prec(case):
    return FP64 if case["precision"] == "fp64" else FP32MIXED


# -------------------------------------------------------------------- inputs
def _su3_exp(X):
    """exp(X) of a batch of small 3x3 matrices in 64 bits: scaling, a Taylor sum, squarings."""
    squarings = max(0, math.ceil(math.log2(max(1e-30, float(torch.linalg.matrix_norm(X).max()) / 0.125))))
    X = X / 2.0 ** squarings
    eye = torch.eye(3, dtype=X.dtype, device=X.device)
    E = eye + X / 12
    for k in range(11, 0, -1):  # |X| <= 1/8: the term after these is below 1e-20
        E = eye + (X @ E) / k
    for _ in range(squarings):
        E = E @ E
    return E


def _links(shape, seed, scale=0.5):
    """Links exp(i scale H), float64 in file order on the GPU: (V, 4, 3, 3) complex."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    V = math.prod(shape)
    out = torch.empty((V, 4, 3, 3), dtype=torch.complex128, device="cuda")
    for lo in range(0, V, 1 << 18):
        n = min(1 << 18, V - lo)
        h = scale * torch.randn((n, 4, 8), dtype=torch.float64, device="cuda", generator=g) / 2
        H = torch.zeros((n, 4, 3, 3), dtype=torch.complex128, device="cuda")
        for a, (i, j) in enumerate(((0, 1), (0, 2), (1, 2))):
            H[..., i, j] = torch.complex(h[..., 2 * a], -h[..., 2 * a + 1])
            H[..., j, i] = torch.complex(h[..., 2 * a], h[..., 2 * a + 1])
        d3, d8 = h[..., 6], h[..., 7] / math.sqrt(3.0)
        H[..., 0, 0] = (d3 + d8).to(H.dtype)
        H[..., 1, 1] = (d8 - d3).to(H.dtype)
        H[..., 2, 2] = (-2 * d8).to(H.dtype)
        out[lo:lo + n] = _su3_exp(1j * H)
    return out


def _pinned(links):
    """The links as a page-locked host array in file order (what a program that loads saved configurations holds)."""
    flat = torch.view_as_real(links).reshape(-1)
    host = torch.empty(flat.shape, dtype=torch.float64, pin_memory=True)
    host.copy_(flat)
    return host


_contexts = {}


def _context(name):
    """One context per GPU and use, kept by the program (batches tune their kernels' shapes in theirs)."""
    if name not in _contexts:
        _contexts[name] = Context(0)
    return _contexts[name]


class _State(dict):
    """A state whose lattice is given back with it."""

    def __del__(self):
        if self.get("lat") is not None:
            self["lat"].close()


def _dp(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def _to_file_order(lat, host):
    """lgf_download_links into page-locked memory."""
    lat.ctx.check(lat.lib.lgf_download_links(lat.h, _dp(host)))
    return host


def prepare(case, seed):
    s = _State(case=case, seed=seed)
    if case["kind"] == "batch":
        s["links"] = [_pinned(_links(v, seed * 64 + i)).numpy() for i, v in enumerate(_volumes(case))]
        s["ctx"] = _context("batch")
        return s
    shape = _shape(case)
    if case["kind"] == "noalloc":
        _context("flow")  # places the library's scratch on the device
        s["links"] = _links(shape, seed)
        s["out"] = torch.empty(2 + 2 * shape[0], dtype=torch.float64, device="cuda")
        return s
    s["lat"] = _context("flow").lattice(shape, _prec(case))
    if case["kind"] == "flow":
        if case["source"] == "host":
            s["links"] = _pinned(_links(shape, seed))
        if case["links_out"]:
            s["out"] = torch.empty(math.prod(shape) * 72, dtype=torch.float64, pin_memory=True)
        return s
    s["lat"].upload(_pinned(_links(shape, seed)).numpy())
    if case["kind"] == "heatbath":
        s["out"] = torch.empty(math.prod(shape) * 72, dtype=torch.float64, pin_memory=True)
    return s


# ----------------------------------------------------------------- one pass
def _numbers(case, r):
    """A flow's results in the precision of its arithmetic."""
    f = np.float64 if case["precision"] == "fp64" else np.float32
    out = {"t": r.t, "E": r.E.astype(f), "Q": r.Q.astype(f)}
    if r.E_slice is not None:
        out.update(E_slice=r.E_slice.astype(f), Q_slice=r.Q_slice.astype(f))
    return out


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "flow":
        lat = s["lat"]
        if case["source"] == "host":
            lat.upload(s["links"].numpy())
        else:
            lat.generate(s["seed"], 0.5)
        r = lat.flow(EPS, case["steps"], case["every"], t0=case["t0"], measure_at_t0=case["at_t0"], reunit_every=case["reunit"],
                     slices=True)
        out = _numbers(case, r)
        if case["links_out"]:
            links = _to_file_order(lat, s["out"])
            out["links"] = links if case["precision"] == "fp64" else links.to(torch.float32)
        return out
    if kind == "measure":
        E, Q, es, qs = s["lat"].measure(slices=True)
        f = np.float64 if case["precision"] == "fp64" else np.float32
        return {"E": f(E), "Q": f(Q), "E_slice": es.astype(f), "Q_slice": qs.astype(f)}
    if kind == "densities":
        e, q = s["lat"].site_densities()
        E, Q = s["lat"].measure_flowed()
        return {"e": e, "q": q, "E_improved": E, "Q_clover": Q}
    if kind == "noalloc":
        shape = (ctypes.c_int * 4)(*_shape(case))
        rc = _context("flow").lib.lgf_measure_noalloc(_dp(s["links"]), shape, _dp(s["out"]),
                                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError("lgf_measure_noalloc: %d" % rc)
        return s["out"]
    if kind == "heatbath":
        lat = s["lat"]
        rejected = lat.heatbath(case["beta"], case["iters"], case["over"], s["seed"])
        f = np.float64 if case["precision"] == "fp64" else np.float32
        links = _to_file_order(lat, s["out"])
        return {"rejected": rejected, "plaquette": f(lat.plaquette()), "links": links if f is np.float64 else links.to(torch.float32)}
    jobs = [Job(v, _prec(case), links=u, eps=EPS, nsteps=case["steps"], meas_every=case["every"], reunit_every=case["reunit"],
                slices=True, want_links=i < 2) for i, (v, u) in enumerate(zip(_volumes(case), s["links"]))]
    s["ctx"].batch_run(jobs)
    f = np.float64 if case["precision"] == "fp64" else np.float32
    out = {"%s_%s" % (k, n): np.concatenate([_numbers(case, j.result)[k].reshape(-1) for j in part])
           for n, part in (("first", jobs[:2]), ("rest", jobs[2:])) if part for k in ("E", "Q", "E_slice", "Q_slice")}
    out["links"] = [j.links_out.astype(f, copy=False) for j in jobs[:2]]
    return out


# ------------------------------------------------------------ what it needs
# A complex 3x3 product is 198 operations.  A flow stage takes, per site and link, six staples (12 products), the force,
# the exponential and the update: 14,296 per site (the reference's count).  A measurement takes, per site and plane, the
# six distinct rectangles (12 path products, 6 projections) and their sums over the four corners they touch: about
# 40,000 per site.  A sweep updates 4 links by a staple sum and three SU(2) steps: about 11,500 per site.
STAGE_FLOPS, MEASURE_FLOPS, SWEEP_FLOPS = 14296.0, 40000.0, 11500.0


def _flow_work(case, V, nmeas, links_in, links_out):
    link = 576.0 if case["precision"] == "fp64" else 288.0
    # each step reads and writes a lattice that is too large to stay in registers once: links in, links out
    moved = 2 * link * case["steps"] + link * nmeas + 576.0 * (links_in + links_out)
    return {"bytes": V * moved, "flops": V * (3 * STAGE_FLOPS * case["steps"] + MEASURE_FLOPS * nmeas)}


def work(case):
    if case["kind"] == "batch":
        V = float(sum(math.prod(v) for v in _volumes(case)))
        return _flow_work(case, V, 1 + case["steps"] // case["every"], 1, 0)
    V = float(math.prod(_shape(case)))
    if case["kind"] == "flow":
        return _flow_work(case, V, case["at_t0"] + case["steps"] // case["every"], case["source"] == "host", case["links_out"])
    if case["kind"] == "heatbath":
        sweeps = case["iters"] * (1 + case["over"])
        link = 576.0 if case["precision"] == "fp64" else 288.0
        return {"bytes": V * (2 * link * sweeps + 576.0), "flops": V * SWEEP_FLOPS * sweeps}
    link = 288.0 if case["precision"] == "fp32mixed" else 576.0
    return {"bytes": V * (link + (16.0 if case["kind"] == "densities" else 0.0)),
            "flops": V * MEASURE_FLOPS * (2 if case["kind"] == "densities" else 1)}


# ---------------------------------------------------------- 64-bit reference
PLANES = ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))


def _at(A, mu, k):
    """The field A at x + k mu."""
    return torch.roll(A, -k, dims=mu)


def _traceless(W):
    """W minus its trace's third."""
    return W - torch.eye(3, dtype=W.dtype, device=W.device) * (torch.diagonal(W, dim1=-2, dim2=-1).sum(-1) / 3)[..., None, None]


def _force(U, mu):
    S = torch.zeros_like(U[mu])
    for nu in range(4):
        if nu == mu:
            continue
        S += _at(U[nu], mu, 1) @ (U[nu] @ _at(U[mu], nu, 1)).mH
        S += _at((U[mu] @ _at(U[nu], mu, 1)).mH @ U[nu], nu, -1)
    W = U[mu] @ S
    return -0.5 * _traceless(W - W.mH)


def _step(U):
    def moved(U, X):
        return [_su3_exp(X[m]) @ U[m] for m in range(4)]

    Z0 = [_force(U, m) for m in range(4)]
    U = moved(U, [EPS / 4 * z for z in Z0])
    A = [8 / 9 * _force(U, m) - 17 / 36 * Z0[m] for m in range(4)]
    U = moved(U, [EPS * a for a in A])
    X = [EPS * (3 / 4 * _force(U, m) - A[m]) for m in range(4)]
    return moved(U, X)


def _path(U, steps):
    """The product of links along (direction, sign) steps from every site."""
    P, here = None, [0, 0, 0, 0]
    for d, sign in steps:
        at = list(here)
        if sign < 0:
            at[d] -= 1
        L = U[d]
        for k in range(4):
            if at[k]:
                L = _at(L, k, at[k])
        L = L if sign > 0 else L.mH
        P = L if P is None else P @ L
        here[d] += sign
    return P


def _fields(U):
    """The clover and the improved field strength of every plane, Hermitian and traceless."""
    clover, improved = [], []
    for mu, nu in PLANES:
        sums = {}
        for a, b in ((1, 1), (2, 2), (1, 2), (2, 1), (1, 3), (3, 1)):
            C = torch.zeros_like(U[0])
            for sm, sn in ((1, 1), (1, -1), (-1, 1), (-1, -1)):
                W = _path(U, [(nu, sn)] * b + [(mu, sm)] * a) @ _path(U, [(mu, sm)] * a + [(nu, sn)] * b).mH
                C += W if sm * sn > 0 else -W
            sums[a, b] = -0.5j * _traceless(C - C.mH)
        c11, c22 = sums[1, 1] / 4, sums[2, 2] / 4
        c12, c13 = (sums[1, 2] + sums[2, 1]) / 8, (sums[1, 3] + sums[3, 1]) / 8
        clover.append(c11)
        improved.append(19 / 9 * c11 + c22 / 36 - 32 / 45 * c12 + c13 / 15)
    return clover, improved


def _trace(A, B):
    return (A * B.transpose(-1, -2)).sum((-1, -2)).real


def _energy(F):
    return sum(_trace(f, f) for f in F)


def _charge(F):
    return -_trace(F[5], F[0]) + _trace(F[4], F[1]) - _trace(F[2], F[3])


def _observables(U):
    clover, improved = _fields(U)
    e, q = _energy(clover), _charge(improved) / (4 * math.pi ** 2)
    host = lambda v: v.cpu().numpy()  # noqa: E731
    return {"E": float(e.mean()), "Q": float(q.sum()), "E_slice": host(e.mean((1, 2, 3))), "Q_slice": host(q.sum((1, 2, 3)))}


def _field(shape, links):
    return [links[:, m].reshape(*shape, 3, 3) for m in range(4)]


def _exact_flow(shape, links, steps, every, t0, at_t0):
    U, t, found = _field(shape, links), t0, []
    if at_t0:
        found.append({"t": t, **_observables(U)})
    for k in range(1, steps + 1):
        U = _step(U)
        t += EPS
        if every and k % every == 0:
            found.append({"t": t, **_observables(U)})
    out = {k: np.array([f[k] for f in found]) for k in ("t", "E", "Q", "E_slice", "Q_slice")}
    return out, torch.view_as_real(torch.stack([u.reshape(-1, 3, 3) for u in U], 1)).reshape(-1).cpu()


def exact(case, seed):
    kind = case["kind"]
    if kind == "heatbath":
        return None  # its rejection steps draw from the engine's own random numbers
    if kind == "batch":
        vols = _volumes(case)[:2]
        if sum(math.prod(v) for v in vols) * case["steps"] > 1.5e6:
            return None
        runs = [_exact_flow(v, _links(v, seed * 64 + i), case["steps"], case["every"], 0.0, True) for i, v in enumerate(vols)]
        out = {k + "_first": np.concatenate([r[0][k].reshape(-1) for r in runs]) for k in ("E", "Q", "E_slice", "Q_slice")}
        out["links"] = [r[1] for r in runs]
        return out
    shape = _shape(case)
    V = math.prod(shape)
    if kind == "flow":
        if case["source"] == "device" or V * case["steps"] > 4e6:
            return None
        out, links = _exact_flow(shape, _links(shape, seed), case["steps"], case["every"], case["t0"], case["at_t0"])
        if case["links_out"]:
            out["links"] = links
        return out
    if V > 1.2e6:
        return None
    U = _field(shape, _links(shape, seed))
    if kind == "densities":
        clover, improved = _fields(U)
        return {"e": _energy(clover).reshape(-1).cpu(), "q": _charge(improved).reshape(-1).cpu(),
                "E_improved": float(_energy(improved).mean()), "Q_clover": float(_charge(clover).sum()) / (4 * math.pi ** 2)}
    o = _observables(U)
    if kind == "measure":
        return o
    return torch.from_numpy(np.concatenate([[o["E"], o["Q"]], o["E_slice"], o["Q_slice"]]))
