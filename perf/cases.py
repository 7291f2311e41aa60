"""Performance cases of libqphix_b200: the calls a lattice QCD program (MILC)
makes through the library's C ABI, over the range of lattices, precisions and
options it makes them with.

Every case drives the public entry points through ``milc_qphix_b200.capi``.
Handles that a program keeps between calls (links, gauge field, momenta) are
made by ``prepare``; colour vectors are created, solved and extracted inside
``run`` as MILC does for every solve.  Raw arrays that a call reads or writes
inside ``run`` are ordinary pageable host arrays, as MILC's are.

Kinds of cases (``kind``):
  dslash     `n` applications of the even-odd Dslash, one parity after the
             other, then the vector's extraction (eigensolvers, sources,
             fermion-force preparation)
  cg         create V, QPHIX_*_asqtad_invert, extract V, destroy V; `inner`
             chooses the precision of the inner solve of the D3 call
  call       the same with create_L_from_raw / destroy_L around it: the whole
             sequence of MILC's glue when the gauge field has just changed
  multi      QPHIX_*_asqtad_invert_multi (RHMC's rational functions)
  batch      QPHIX_B200_D3_batch_invert: many right-hand sides, one or more
             lattices, in one call
  force      QPHIX_B200_*_asqtad_force: link gradients from n solutions
  gforce     QPHIX_*_symanzik_1loop_gauge_force on both checkerboards, then
             the momenta's extraction
"""
import ctypes as C
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NAIK = -1.0 / 24.0


def _package():
    """The package directory ``milc-qphix_b200`` as ``milc_qphix_b200``."""
    name = "milc_qphix_b200"
    if name not in sys.modules:
        d = os.path.join(ROOT, "milc-qphix_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return importlib.import_module(name + ".capi"), sys.modules[name].LIB_PATH


_LIB = None


def _library(dims):
    """The library, initialised for the lattice ``dims`` (one at a time)."""
    global _LIB
    if _LIB is None:
        capi, path = _package()
        _LIB = capi.QphixLib(path)
        _LIB.dims = None
    if _LIB.dims != tuple(dims):
        if _LIB.dims is not None:
            _LIB.finalize()
        if _LIB.init(dims) != 0:
            raise RuntimeError("QPHIX_init: " + _LIB.last_error())
    return _LIB


def _check(ok):
    if not ok:
        raise RuntimeError(_LIB.last_error() or "the call failed")
    return ok


# --------------------------------------------------------------------- cases --
def listed():
    return [
        # the smallest call: one Dslash on each parity of the smallest
        # benchmark lattice, where launches and the extraction count
        {"name": "dslash d 8^4", "kind": "dslash", "prec": "D", "dims": "8,8,8,8", "n": 2},
        # a polynomial of the operator on a production lattice (Chebyshev
        # filter, eigensolver block) in single precision
        {"name": "dslash f 24^3x48", "kind": "dslash", "prec": "F", "dims": "24,24,24,48", "n": 32},
        # the FP64 solve of a test or small-volume run: latency bound
        {"name": "cg d 8^4", "kind": "cg", "prec": "D", "dims": "8,8,8,8", "inner": "double", "compress": False,
         "mass": 0.05, "parity": "even", "resid": 1e-20},
        # single-precision solve (MILC's F3 build), odd sites
        {"name": "cg f 12^3x24 odd", "kind": "cg", "prec": "F", "dims": "12,12,12,24", "inner": "single",
         "compress": False, "mass": 0.05, "parity": "odd", "resid": 1e-11},
        # mixed-precision propagator solve on a production lattice with
        # compressed Naik links (the headline benchmark)
        {"name": "cg mixed 24^3x48", "kind": "cg", "prec": "D", "dims": "24,24,24,48", "inner": "single",
         "compress": True, "mass": 0.01, "parity": "even", "resid": 1e-20},
        # the same with 16-bit links on an intermediate volume
        {"name": "cg half-links 20^3x40", "kind": "cg", "prec": "D", "dims": "20,20,20,40", "inner": "half-links",
         "compress": True, "mass": 0.02, "parity": "even", "resid": 1e-20},
        # MILC's whole sequence when the gauge field has just changed:
        # link upload, solve, extraction
        {"name": "call mixed 16^3x32", "kind": "call", "prec": "D", "dims": "16,16,16,32", "inner": "single",
         "compress": True, "mass": 0.02, "parity": "even", "resid": 1e-20},
        # RHMC's rational function in the reference's FP64 recurrence
        {"name": "multi d 12^3x24", "kind": "multi", "prec": "D", "dims": "12,12,12,24", "inner": "double",
         "compress": False, "mass": 0.02, "shifts": 8, "parity": "even", "resid": 1e-20},
        # the same, mixed precision, 12 shifts, production lattice
        {"name": "multi mixed 24^3x48", "kind": "multi", "prec": "D", "dims": "24,24,24,48", "inner": "single",
         "compress": True, "mass": 0.005, "shifts": 12, "parity": "even", "resid": 1e-20},
        # many sources on one gauge field beside lattices of other volumes
        {"name": "batch 24^3x48 and 8 more", "kind": "batch", "dims": "24,24,24,48", "nrhs": 16,
         "more": "8,8,8,8/8,8,8,8/12,12,12,12/12,12,12,12/16,16,16,32/16,16,16,32/20,20,20,40/20,20,20,40",
         "mass": 0.02, "parity": "even", "resid": 1e-20},
        # fermion force of a rational function's residues
        {"name": "force d 16^3x32", "kind": "force", "prec": "D", "dims": "16,16,16,32", "n": 8, "parity": "even"},
        # improved gauge force of one molecular-dynamics kick
        {"name": "gforce d 24^3x48", "kind": "gforce", "prec": "D", "dims": "24,24,24,48", "loops": 3},
    ]


def _draw_dims(rng, lo, hi):
    """Four extents, multiples of 4 (QPHIX_init's rule), ragged, with lo <= V
    <= hi and V spread over its logarithm."""
    while True:
        v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        d = [4 * rng.randint(1, 8) for _ in range(3)] + [4 * rng.randint(1, 16)]
        if lo <= d[0] * d[1] * d[2] * d[3] <= hi and abs(math.log(d[0] * d[1] * d[2] * d[3] / v)) < 0.2:
            return ",".join(map(str, d))


def draw(rng):
    kind = rng.choice(["dslash", "cg", "cg", "cg", "call", "multi", "multi", "batch", "force", "gforce", "gforce"])
    v8, v12, v16, v20, v24 = 8 ** 4, 12 ** 3 * 24, 16 ** 3 * 32, 20 ** 3 * 40, 24 ** 3 * 48
    parity = rng.choice(["even", "odd"])
    mass = lambda lo, hi: round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 4)  # noqa: E731
    if kind == "dslash":
        return {"kind": kind, "prec": rng.choice("FD"), "dims": _draw_dims(rng, 512, v24),
                "n": rng.randint(1, 24)}
    if kind in ("cg", "call"):
        prec = rng.choice("DDDF") if kind == "cg" else "D"
        inner = "single" if prec == "F" else rng.choice(["double", "single", "single", "half-links", "half"])
        mixed = prec == "D" and inner != "double"
        top = v20 if kind == "call" else v24 if mixed else v16
        return {"kind": kind, "prec": prec, "dims": _draw_dims(rng, 1024, top), "inner": inner,
                "compress": mixed and rng.random() < 0.6, "mass": mass(0.015 if mixed else 0.02, 0.2),
                "parity": parity, "resid": 1e-11 if prec == "F" else 1e-20}
    if kind == "multi":
        inner = rng.choice(["double", "single", "single"])
        return {"kind": kind, "prec": "D", "dims": _draw_dims(rng, 1024, v16 if inner == "double" else v20),
                "inner": inner, "compress": inner == "single" and rng.random() < 0.6, "mass": mass(0.005, 0.05),
                "shifts": rng.randint(3, 15), "parity": parity, "resid": 1e-20}
    if kind == "batch":
        more = "/".join(_draw_dims(rng, 512, v12) for _ in range(rng.randint(0, 4)))
        return {"kind": kind, "dims": _draw_dims(rng, v8, v20), "nrhs": rng.randint(2, 16), "more": more,
                "mass": mass(0.02, 0.2), "parity": parity, "resid": 1e-20}
    if kind == "force":
        return {"kind": kind, "prec": rng.choice("DDF"), "dims": _draw_dims(rng, 512, v20), "n": rng.randint(1, 12),
                "parity": parity}
    return {"kind": kind, "prec": rng.choice("DDF"), "dims": _draw_dims(rng, 512, v24), "loops": rng.choice([1, 2, 3, 3])}


def _dims(text):
    return tuple(int(v) for v in text.split(","))


def _volume(dims):
    return dims[0] * dims[1] * dims[2] * dims[3]


def _lattices(case):
    return [_dims(case["dims"])] + [_dims(t) for t in case.get("more", "").split("/") if t]


def _shift_masses(case):
    """sqrt(m^2 + sigma/4) for RHMC-style shifts sigma, log-spaced 1e-5 .. 1."""
    n = case["shifts"]
    return [math.sqrt(case["mass"] ** 2 + 10.0 ** (-5.0 + 5.0 * k / (n - 1)) / 4) for k in range(n)]


GF_COEFFS = {1: (1.0, 0.0, 0.0), 2: (1.0, -0.05, 0.0), 3: (1.0, -0.0545, -0.0123)}
GF_EPS = 0.02


# -------------------------------------------------------------------- inputs --
# Fields are made on the GPU in lexicographic order (T, Z, Y, X) and put into
# MILC's raw even-first order for the library.
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7fffffff)
    return g


def _sum_mm(a, b):
    return (a[..., :, :, None] * b[..., None, :, :]).sum(-2)


def _su3(n, eps, gen):
    """n random SU(3) matrices near exp(i eps H), H Gaussian traceless
    Hermitian: the exponential to second order, then Gram-Schmidt."""
    z = torch.randn(n, 3, 3, 2, dtype=torch.float64, device="cuda", generator=gen)
    z = torch.view_as_complex(z)
    h = 0.5j * eps * (z + z.mH)
    h = h - (torch.diagonal(h, dim1=-2, dim2=-1).sum(-1) / 3)[:, None, None] * torch.eye(3, dtype=h.dtype, device="cuda")
    u = torch.eye(3, dtype=h.dtype, device="cuda") + h + 0.5 * _sum_mm(h, h)
    r0 = u[:, 0] / torch.linalg.vector_norm(u[:, 0], dim=-1, keepdim=True)
    r1 = u[:, 1] - (r0.conj() * u[:, 1]).sum(-1, keepdim=True) * r0
    r1 = r1 / torch.linalg.vector_norm(r1, dim=-1, keepdim=True)
    r2 = torch.stack([(r0[:, (k + 1) % 3] * r1[:, (k + 2) % 3] - r0[:, (k + 2) % 3] * r1[:, (k + 1) % 3]).conj()
                      for k in range(3)], -1)
    return torch.stack([r0, r1, r2], 1)


def _coords(dims):
    ax = [torch.arange(d, device="cuda") for d in dims]
    t, z, y, x = torch.meshgrid(ax[3], ax[2], ax[1], ax[0], indexing="ij")
    return x, y, z, t


def _links(dims, seed):
    """Fat links 0.9 x SU(3) and Naik links -1/24 x SU(3), staggered phases
    folded in: two (T, Z, Y, X, 4, 3, 3) complex fields."""
    gen = _generator(2 * seed + 1)
    shape = (dims[3], dims[2], dims[1], dims[0], 4, 3, 3)
    x, y, z, t = _coords(dims)
    eta = torch.stack([1 - 2 * (t & 1), 1 - 2 * ((t + x) & 1), 1 - 2 * ((t + x + y) & 1), torch.ones_like(t)], -1)
    eta = eta.to(torch.float64)[..., None, None]
    n = 4 * _volume(dims)
    return (0.9 * eta * _su3(n, 0.3, gen).reshape(shape), NAIK * eta * _su3(n, 0.3, gen).reshape(shape))


def _raw_order(dims):
    """Lexicographic index of every raw site (even sites first)."""
    x, y, z, t = _coords(dims)
    return torch.argsort(((x + y + z + t) & 1).reshape(-1), stable=True)


def _to_raw(dims, field, real):
    """A lexicographic complex field as a raw real array (on the GPU)."""
    f = field.reshape(_volume(dims), -1)[_raw_order(dims)]
    return torch.view_as_real(f).reshape(-1).to(real)


def _real(prec):
    return torch.float32 if prec == "F" else torch.float64


def _host(t):
    return t.cpu().numpy()


def _shifted(u, hop):
    """The forward links of x - hop mu at x (MILC's backward links)."""
    return torch.stack([torch.roll(u[..., mu, :, :], hop, dims=3 - mu) for mu in range(4)], -3)


def _raw_links(dims, seed, prec):
    fat, lng = _links(dims, seed)
    return {k: _host(_to_raw(dims, v, _real(prec))) for k, v in
            (("fat", fat), ("lng", lng), ("fatback", _shifted(fat, 1)), ("lngback", _shifted(lng, 3)))}


def _source(dims, seed, parity, k=0):
    """Gaussian colour vector on the sites of one parity (or both)."""
    gen = _generator(7919 * (seed + 1) + k)
    v = torch.randn(dims[3], dims[2], dims[1], dims[0], 3, 2, dtype=torch.float64, device="cuda", generator=gen)
    v = torch.view_as_complex(v)
    if parity == "evenodd":
        return v
    x, y, z, t = _coords(dims)
    return v * (((x + y + z + t) & 1) == (1 if parity == "odd" else 0))[..., None]


def _gauge(dims, seed):
    gen = _generator(3 * seed + 2)
    shape = (dims[3], dims[2], dims[1], dims[0], 4, 3, 3)
    u = _su3(4 * _volume(dims), 0.5, gen).reshape(shape)
    a = torch.view_as_complex(torch.randn(*shape, 2, dtype=torch.float64, device="cuda", generator=gen))
    return u, _ta(a)


# ----------------------------------------------------------------- the state --
class _State:
    """What a program keeps between calls; destroys its handles at the end."""

    def __init__(self, case, lib):
        self.case, self.lib, self.dims = case, lib, lib.dims
        self.kept = []

    def keep(self, destroy, *handle):
        self.kept.append((destroy, handle))
        return _check(handle[-1])

    def __del__(self):
        if self.lib.dims == self.dims:
            for destroy, handle in reversed(self.kept):
                destroy(*handle)


def prepare(case, seed):
    kind = case["kind"]
    dims = _dims(case["dims"])
    lib = _library(dims)
    s = _State(case, lib)
    prec = case.get("prec", "D")
    if kind in ("cg", "call", "multi"):
        lib.set_inner_precision(case["inner"] if prec == "D" else "double")
        lib.set_link_compression(case["compress"])
    real = _real(prec)
    if kind == "dslash":
        s.L = s.keep(lib.destroy_L, prec, lib.create_L(prec, _raw_links(dims, seed, prec)))
        src = _host(_to_raw(dims, _source(dims, seed, "evenodd"), real))
        s.v = [s.keep(lib.destroy_V, prec, lib.create_V(prec, a)) for a in (src, src, src)]
        s.out = np.zeros_like(src)
    elif kind in ("cg", "call"):
        links = _raw_links(dims, seed, prec)
        if kind == "call":
            s.links = links
        else:
            s.L = s.keep(lib.destroy_L, prec, lib.create_L(prec, links))
        s.src = _host(_to_raw(dims, _source(dims, seed, case["parity"]), real))
        s.guess, s.out = np.zeros_like(s.src), np.zeros_like(s.src)
    elif kind == "multi":
        s.L = s.keep(lib.destroy_L, prec, lib.create_L(prec, _raw_links(dims, seed, prec)))
        s.src = _host(_to_raw(dims, _source(dims, seed, case["parity"]), real))
        s.guess = np.zeros_like(s.src)
        s.out = [np.zeros_like(s.src) for _ in range(case["shifts"])]
    elif kind == "batch":
        lats = _lattices(case)
        s.B = s.keep(lib.batch_destroy_L, lib.batch_create_L(
            [(d, _raw_links(d, seed + 101 * k, "D")) for k, d in enumerate(lats)]))
        s.systems = [(k, case["mass"], _host(_to_raw(d, _source(d, seed, case["parity"], 100 * k + r), real)))
                     for k, d in enumerate(lats) for r in range(case["nrhs"] if k == 0 else 1)]
        s.out = [np.zeros_like(v[2]) for v in s.systems]
    elif kind == "force":
        s.L = s.keep(lib.destroy_L, prec, lib.create_L(prec, _raw_links(dims, seed, prec)))
        s.x = [s.keep(lib.destroy_V, prec, lib.create_V(
            prec, _host(_to_raw(dims, _source(dims, seed, case["parity"], k), real)), case["parity"]))
            for k in range(case["n"])]
        s.grad = [np.zeros(72 * _volume(dims), np.float32 if prec == "F" else np.float64) for _ in range(2)]
    else:
        u, mom = _gauge(dims, seed)
        raw_u, raw_a = _host(_to_raw(dims, u, real)), _host(_to_raw(dims, mom, real))
        s.G = {p: s.keep(lib.destroy_G, prec, lib.create_G(prec, raw_u, p)) for p in ("even", "odd")}
        s.F = {p: s.keep(lib.destroy_F, prec, lib.create_F(prec, raw_a, p)) for p in ("even", "odd")}
        s.out = np.zeros_like(raw_a)
    return s


def _coefs(n):
    return [0.3 + 0.1 * k for k in range(n)]


def _solve(s, L):
    c, lib = s.case, s.lib
    prec, parity = c["prec"], c["parity"]
    b = _check(lib.create_V(prec, s.src, parity))
    x = _check(lib.create_V(prec, s.guess, parity))
    it, info, res = lib.invert(prec, L, x, b, c["mass"], parity=parity, max_iter=2000, nrestart=5, resid=c["resid"])
    _check(info.status == 0)
    lib.extract_V(prec, x, parity, out=s.out)
    lib.destroy_V(prec, x)
    lib.destroy_V(prec, b)
    return s.out


def run(s):
    c, lib = s.case, s.lib
    kind, prec = c["kind"], c.get("prec", "D")
    if kind == "dslash":
        src, other = s.v[0], 0
        for k in range(c["n"]):
            # half applications: even from odd, then odd from that, ...
            dst = s.v[1 + other]
            lib.dslash(prec, s.L, dst, src, "even" if k % 2 == 0 else "odd")
            src, other = dst, 1 - other
        return lib.extract_V(prec, src, out=s.out)
    if kind == "cg":
        return _solve(s, s.L)
    if kind == "call":
        L = _check(lib.create_L(prec, s.links))
        out = _solve(s, L)
        lib.destroy_L(prec, L)
        return out
    if kind == "multi":
        b = _check(lib.create_V(prec, s.src, c["parity"]))
        xs = [_check(lib.create_V(prec, s.guess, c["parity"])) for _ in s.out]
        it, info, res = lib.invert_multi(prec, s.L, xs, b, _shift_masses(c), parity=c["parity"], max_iter=2000,
                                         nrestart=5, resid=c["resid"])
        _check(info.status == 0)
        for x, o in zip(xs, s.out):
            lib.extract_V(prec, x, c["parity"], out=o)
        for h in xs + [b]:
            lib.destroy_V(prec, h)
        return s.out
    if kind == "batch":
        for o in s.out:
            o.fill(0.0)  # the initial guesses
        it, info, res, outs = lib.batch_invert(s.B, s.systems, parity=c["parity"], max_iter=2000, resid=c["resid"],
                                               outs=s.out)
        _check(info.status == 0)
        return outs
    if kind == "force":
        n, real = c["n"], C.c_float if prec == "F" else C.c_double
        coef = (real * n)(*_coefs(n))
        ptr = [g.ctypes.data_as(C.POINTER(real)) for g in s.grad]
        f = getattr(lib.lib, "QPHIX_B200_%s3_asqtad_force" % prec)
        _check(f(s.L, n, coef, (C.c_void_p * n)(*s.x), 2 if c["parity"] == "even" else 1, *ptr) == 0)
        return s.grad
    co = dict(zip(("plaquette", "rectangle", "parallelogram"), GF_COEFFS[c["loops"]]))
    real = C.c_float if prec == "F" else C.c_double
    out = s.out.ctypes.data_as(C.POINTER(real))
    extract = getattr(lib.lib, "QPHIX_%s3_extract_F_to_raw" % prec)
    for p, code in (("even", 2), ("odd", 1)):
        _check(lib.gauge_force(prec, s.G[p], s.F[p], co, GF_EPS).status == 0)
        extract(out, s.F[p], code)
    return s.out


# -------------------------------------------------------------------- work --
# reals read or written once per site of the whole lattice: links 4 dirs x 18
# x (fat, Naik) -- the backward arrays repeat them --, a colour vector 6
def _iterations(mass):
    """Typical CG iterations of these fields to |r|/|b| = 1e-10."""
    return 1000.0 / (1.0 + mass / 0.012)


def work(case):
    kind = case["kind"]
    dims = _dims(case["dims"])
    V = _volume(dims)
    r = 4 if case.get("prec") == "F" else 8
    links, dslash_flops = 144 * r * V, 573.0 * V
    if kind == "dslash":
        return {"bytes": links + 9 * r * V, "flops": case["n"] * dslash_flops}
    if kind in ("cg", "call"):
        it = _iterations(case["mass"]) * (0.55 if case["prec"] == "F" else 1.0)
        return {"bytes": links * (2 if kind == "call" else 1) + 9 * r * V, "flops": it * (2 * dslash_flops + 36 * V)}
    if kind == "multi":
        it = _iterations(_shift_masses(case)[0])
        return {"bytes": links + 3 * r * V * (1 + case["shifts"]),
                "flops": it * (2 * dslash_flops + (18 + 18 * case["shifts"]) * V)}
    if kind == "batch":
        lats = _lattices(case)
        it = _iterations(case["mass"])
        systems = [_volume(d) * (case["nrhs"] if k == 0 else 1) for k, d in enumerate(lats)]
        return {"bytes": sum(1152.0 * _volume(d) for d in lats) + sum(72.0 * v for v in systems),
                "flops": sum(it * (1146 + 36) * v for v in systems)}
    if kind == "force":
        return {"bytes": (144 + 3 * case["n"]) * r * V + links,
                "flops": case["n"] * (dslash_flops + 8 * 9 * 10 * V)}
    # gauge force: plaquette staples alone, or with the six-link loops
    n = 6 if case["loops"] == 1 else 24 if case["loops"] == 2 else 48
    return {"bytes": 3 * 72 * r * V, "flops": 4.0 * V * (198 * (2 * 6 + 2 * (n - 6)) + 36 * n + 252)}


def tolerance(case):
    """About four times the largest error against 64 bits that the listed and
    drawn cases show (sums in another order differ by less)."""
    kind, single = case["kind"], case.get("prec", "D") == "F"
    if kind in ("cg", "call", "multi", "batch"):
        # the solvers stop at |r|/|b| < 1e-10 (D3; errors of 2e-10 .. 1.5e-9,
        # up to 1e-8 at the lightest masses) or 3e-6 (F3; 7e-6 at m = 0.05),
        # which fixes the solution up to the operator's condition number
        return {"rel": 1e-4 if single else 4e-8}
    # one to some thirty sums of 48 products per value
    return {"rel": 1.5e-6 if single else 4e-15}


# ------------------------------------------------------------------- exact --
def _mv(u, v):
    return (u * v[..., None, :]).sum(-1)


class _Operator:
    """D in 64 bits on lexicographic fields."""

    def __init__(self, dims, seed):
        self.u = _links(dims, seed)
        self.adj = [u.mH.contiguous() for u in self.u]

    def __call__(self, v):
        out = torch.zeros_like(v)
        for hop, u, w in ((1, self.u[0], self.adj[0]), (3, self.u[1], self.adj[1])):
            for mu in range(4):
                out += _mv(u[..., mu, :, :], torch.roll(v, -hop, dims=3 - mu))
                out -= torch.roll(_mv(w[..., mu, :, :], v), hop, dims=3 - mu)
        return out


def _cg(D, b, mass, tol=1e-13, limit=6000):
    x, r = torch.zeros_like(b), b.clone()
    p, rr = r.clone(), float((r.conj() * r).real.sum())
    stop = tol * tol * rr
    for _ in range(limit):
        ap = 4 * mass * mass * p - D(D(p))
        a = rr / float((p.conj() * ap).real.sum())
        x += a * p
        r -= a * ap
        new = float((r.conj() * r).real.sum())
        if new < stop:
            break
        p = r + (new / rr) * p
        rr = new
    return x


def _ta(m):
    a = 0.5 * (m - m.mH)
    tr = torch.diagonal(a, dim1=-2, dim2=-1).sum(-1) / 3
    return a - tr[..., None, None] * torch.eye(3, dtype=m.dtype, device=m.device)


def _path(u, steps):
    """Product of links along (axis, sign) steps from every site."""
    off, m = [0, 0, 0, 0], None
    for a, s in steps:
        if s < 0:
            off[a] -= 1
        link = torch.roll(u[..., a, :, :], [-o for o in off], dims=[3, 2, 1, 0])
        if s > 0:
            off[a] += 1
        else:
            link = link.mH
        m = link if m is None else _sum_mm(m, link)
    return m


def _staples(u, mu, coeffs):
    """Weighted sum of the staples of every link U_mu: paths from x + mu to x."""
    p, others, out = coeffs, [d for d in range(4) if d != mu], 0
    for nu in others:
        for s in (1, -1):
            paths = [(p[0], [(nu, s), (mu, -1), (nu, -s)])]
            paths += [(p[1], q) for q in ([(mu, 1), (nu, s), (mu, -1), (mu, -1), (nu, -s)],
                                          [(nu, s), (mu, -1), (mu, -1), (nu, -s), (mu, 1)],
                                          [(nu, s), (nu, s), (mu, -1), (nu, -s), (nu, -s)])]
            for rho in others:
                if rho != nu:
                    paths += [(p[2], [(nu, s), (rho, r), (mu, -1), (nu, -s), (rho, -r)]) for r in (1, -1)]
            for c, q in paths:
                if c != 0.0:
                    out = out + c * _path(u, q)
    return torch.roll(out, -1, dims=3 - mu)


def exact(case, seed):
    kind = case["kind"]
    dims = _dims(case["dims"])
    raw = lambda v, d=dims: _to_raw(d, v, torch.float64)  # noqa: E731
    if kind == "gforce":
        u, mom = _gauge(dims, seed)
        f = torch.stack([_ta(_sum_mm(u[..., mu, :, :], _staples(u, mu, GF_COEFFS[case["loops"]]))) for mu in range(4)],
                        -3)
        return raw(mom + GF_EPS * f)
    D = _Operator(dims, seed)
    if kind == "dslash":
        # the vectors hold the source on the parity that has not been written
        src = _source(dims, seed, "evenodd")
        x, y, z, t = _coords(dims)
        odd = (((x + y + z + t) & 1) == 1)[..., None]
        v, bufs, other = src, [src, src], 0
        for k in range(case["n"]):
            bufs[other] = torch.where(odd, bufs[other], D(v)) if k % 2 == 0 else torch.where(odd, D(v), bufs[other])
            v, other = bufs[other], 1 - other
        return raw(v)
    if kind in ("cg", "call"):
        return raw(_cg(D, _source(dims, seed, case["parity"]), case["mass"]))
    if kind == "multi":
        # the lightest and the heaviest shift and one between them
        b, masses = _source(dims, seed, case["parity"]), _shift_masses(case)
        some = {0, len(masses) // 2, len(masses) - 1}
        return [raw(_cg(D, b, m)) if k in some else None for k, m in enumerate(masses)]
    if kind == "batch":
        out = []
        for k, d in enumerate(_lattices(case)):
            D = _Operator(d, seed + 101 * k)
            for r in range(case["nrhs"] if k == 0 else 1):
                out.append(raw(_cg(D, _source(d, seed, case["parity"], 100 * k + r), case["mass"]), d)
                           if r == 0 else None)
        return out
    # force: dS = 2 s Re tr[dU W(z + hop mu) W(z)^dag], W = x or D x by parity
    x, y, z, t = _coords(dims)
    mine = (((x + y + z + t) & 1) == (1 if case["parity"] == "odd" else 0))[..., None]
    grads = [0, 0]
    for k, coef in enumerate(_coefs(case["n"])):
        v = _source(dims, seed, case["parity"], k)
        w = torch.where(mine, v, D(v))
        sign = (4.0 * mine.to(torch.float64) - 2.0)[..., None, None]
        for h, hop in enumerate((1, 3)):
            m = torch.stack([w.conj()[..., :, None] * torch.roll(w, -hop, dims=3 - mu)[..., None, :]
                             for mu in range(4)], -3)
            grads[h] = grads[h] + coef * sign * m.conj()
    return [raw(g) for g in grads]
