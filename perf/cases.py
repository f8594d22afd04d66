"""Performance cases of the thin-wire method-of-moments solver.

Each case is one thing that a program using this package has it do, through
the package's public entry points: the NEC2++ C API (a context is created,
given its cards, run, read out and deleted, as a script or an optimiser does
for every candidate), the batched sweep, the adjoint gradient and the dense
complex solve of the device C-ABI.  Sizes follow the package's own workloads
and tests (dipole, Yagi-Uda antennas, wire meshes, helix arrays).

    listed()             the fixed cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  the inputs of one pass, made from the seed
    run(state)           one pass; its outputs
    work(case)           bytes and operations that the pass cannot do without
    exact(case, seed)    the outputs in 64-bit arithmetic, where they have such
                         a value that does not come from this package

The numbers of a structure (all kinds but "matrix") are those of NEC's own
discretisation: adaptive quadrature steps, interpolated ground tables and
truncated constants are part of their definition, so plain 64-bit arithmetic
gives no independent value for them and exact() has none.
"""
import ctypes as C
import math
import types

import numpy as np

import necpp_b200 as nb
from necpp_b200 import adjoint, batch
from necpp_b200 import workloads as W

API = types.SimpleNamespace(helix=nb.nec_helix, nec_error_message=nb.nec_error_message,
                            **{k: getattr(nb, k) for k in dir(nb) if k.startswith("nec_") and k != "nec_error_message"})

MIXED, FP64 = 1, 0
FREE, PERFECT, REFLECTION, SOMMERFELD = 0, 1, 2, 3
# GN cards of the ground types: type, radials, permittivity, conductivity
GN = {PERFECT: (1, 0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0), REFLECTION: (0, 0, 13.0, 0.005, 0.0, 0.0, 0.0, 0.0),
      SOMMERFELD: (2, 0, 13.0, 0.005, 0.0, 0.0, 0.0, 0.0)}


def listed():
    return [
        # the smallest call: one centre-fed dipole and its pattern, as a
        # script's first example or an optimiser's inner loop runs it; all latency
        {"name": "dipole", "kind": "dipole", "nseg": 51, "nth": 91, "nph": 72, "precision": MIXED},
        # a Yagi's band plot: one FR card over 16 frequencies, a pattern each
        {"name": "yagi_band", "kind": "yagi", "elements": 9, "nseg": 21, "nfreq": 16, "nth": 91, "nph": 72,
         "ground": FREE},
        # wires close above real (Sommerfeld) ground with the near field over
        # it at two frequencies: ground tables and near-ground integrals
        {"name": "near_ground", "kind": "near_ground", "nseg": 21, "nfreq": 2, "nx": 9, "ny": 5, "nz": 3},
        # near electric and magnetic fields around a Yagi over reflecting
        # ground (exposure maps): many points, few segments
        {"name": "near_fields", "kind": "fields", "elements": 5, "nseg": 21, "nx": 25, "ny": 17, "nz": 11,
         "ground": REFLECTION},
        # an optimiser's gradient step: 9-element Yagi over Sommerfeld ground,
        # 27 parameters, forward solve and adjoint
        {"name": "yagi_gradient", "kind": "gradient", "elements": 9, "nseg": 21},
        # scattering of a wire-mesh plate over incidence angles: one
        # factorisation, a solve and a bistatic cut per angle
        {"name": "mesh_incidence", "kind": "mesh", "nwires": 16, "angles": 13, "nth": 91, "nph": 1},
        # a small array at an odd size (N = 909)
        {"name": "helix_3x3", "kind": "helix", "k": 3, "nseg": 101, "nth": 91, "nph": 72, "precision": MIXED},
        # the same physics in plain complex128, the choice of a user who wants
        # the reference's pivoting (N = 2880)
        {"name": "helix_4x4_fp64", "kind": "helix", "k": 4, "nseg": 180, "nth": 91, "nph": 72, "precision": FP64},
        # the plate at full resolution (N = 3280, 4-way junctions), one
        # incidence, full bistatic pattern
        {"name": "mesh_41", "kind": "mesh", "nwires": 41, "angles": 1, "nth": 181, "nph": 72},
        # the largest: the 8 x 8 helix array, N = 11520, all 64 feeds
        {"name": "helix_8x8", "kind": "helix", "k": 8, "nseg": 180, "nth": 91, "nph": 72, "precision": MIXED},
        # a design population: Yagi variants x frequencies in one batched call
        {"name": "batch_sweep", "kind": "batch", "variants": 128, "nfreq": 8},
        # a caller's own dense complex system at a ragged size
        {"name": "matrix_1501", "kind": "matrix", "n": 1501, "precision": MIXED},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("dipole", "yagi", "near_ground", "fields", "gradient", "mesh", "mesh", "helix", "helix", "helix",
                       "batch", "matrix"))
    if kind == "dipole":
        return {"kind": kind, "nseg": 2 * rng.randint(5, 75) + 1, "nth": rng.randint(19, 181), "nph": rng.randint(1, 72),
                "precision": rng.choice((MIXED, FP64))}
    if kind == "yagi":
        return {"kind": kind, "elements": rng.randint(3, 15), "nseg": 2 * rng.randint(5, 20) + 1,
                "nfreq": rng.randint(1, 16), "nth": rng.randint(19, 91), "nph": rng.randint(1, 72),
                "ground": rng.choice((FREE, PERFECT, REFLECTION))}
    if kind == "near_ground":
        return {"kind": kind, "nseg": rng.randint(11, 31), "nfreq": rng.randint(1, 2), "nx": rng.randint(2, 12),
                "ny": rng.randint(1, 6), "nz": rng.randint(1, 4)}
    if kind == "fields":
        return {"kind": kind, "elements": rng.randint(3, 9), "nseg": 2 * rng.randint(5, 20) + 1,
                "nx": rng.randint(5, 30), "ny": rng.randint(5, 20), "nz": rng.randint(3, 15),
                "ground": rng.choice((FREE, PERFECT, REFLECTION))}
    if kind == "gradient":
        return {"kind": kind, "elements": rng.randint(3, 9), "nseg": 2 * rng.randint(5, 15) + 1}
    if kind == "mesh":
        nwires = _log_int(rng, 8, 41)
        return {"kind": kind, "nwires": nwires, "angles": rng.randint(1, 19), "nth": rng.randint(19, 181),
                "nph": rng.randint(1, 18)}
    if kind == "helix":
        precision = rng.choice((MIXED, MIXED, FP64))
        n = _log_int(rng, 120, 11000 if precision == MIXED else 2880)
        k = rng.choice([q for q in range(1, 9) if 60 <= n // (q * q) <= 180] or [1 if n < 180 else 8])
        return {"kind": kind, "k": k, "nseg": max(60, min(180, n // (k * k))), "nth": rng.randint(19, 91),
                "nph": rng.randint(1, 72), "precision": precision}
    if kind == "batch":
        return {"kind": kind, "variants": _log_int(rng, 4, 128), "nfreq": rng.randint(1, 8)}
    return {"kind": kind, "n": _log_int(rng, 100, 2500), "precision": rng.choice((MIXED, FP64))}


# ---------------------------------------------------------------- inputs

class _Engine:
    """A device engine of the C-ABI (include/necgpu.h), as a program that
    brings its own matrices holds one."""

    def __init__(self):
        self.lib = nb.lib
        self.lib.necgpu_create.argtypes = [C.POINTER(C.c_void_p), C.c_int]
        self.lib.necgpu_destroy.argtypes = [C.c_void_p]
        self.lib.necgpu_last_error.restype = C.c_char_p
        self.lib.necgpu_last_error.argtypes = [C.c_void_p]
        self.lib.necgpu_matrix_solve.argtypes = [C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p,
                                                 C.c_void_p]
        self.h = C.c_void_p()
        if self.lib.necgpu_create(C.byref(self.h), 0) != 0:
            raise RuntimeError("necgpu_create: %s" % self.lib.necgpu_last_error(self.h))

    def __del__(self):
        if self.h:
            self.lib.necgpu_destroy(self.h)
            self.h = C.c_void_p()


def _matrix(n, rng):
    """An impedance-like system: retarded 1/r coupling between points of a
    few wavelengths' box, self terms that dominate their row."""
    x = rng.uniform(0.0, 3.0, (n, 3))
    r = np.sqrt(np.maximum(((x[:, None, :] - x[None, :, :]) ** 2).sum(axis=2), 1e-4))
    z = np.exp(-2j * math.pi * r) / r
    z[np.arange(n), np.arange(n)] = rng.uniform(0.5, 1.0, n) * n * np.exp(1j * rng.uniform(-1.0, 1.0, n))
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    return np.ascontiguousarray(z), b


def _population(variants, nfreq, rng):
    """Yagi designs of 3-15 elements with 11-41 segments each at nfreq
    frequencies: the sizes go with the case, the dimensions with the seed."""
    sizes = np.random.default_rng(variants)
    problems = []
    for _ in range(variants):
        segs = 2 * sizes.integers(5, 21, size=int(sizes.integers(3, 16))) + 1
        half, xs, rad, _ = W.yagi_params(rng, n_elements=len(segs), nseg=1)
        ctx = nb.nec_create()
        try:
            for e in range(len(segs)):
                _ok(nb.nec_wire(ctx, e + 1, int(segs[e]), float(xs[e]), 0.0, -float(half[e]), float(xs[e]), 0.0,
                                float(half[e]), float(rad[e]), 1.0, 1.0), "wire")
            _ok(nb.nec_geometry_complete(ctx, 0), "geometry")
            feed = int(segs[1] + 1) // 2
            _ok(nb.nec_ex_card(ctx, 0, 2, feed, 0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0), "ex")
            for f in np.linspace(140.0, 160.0, nfreq):
                problems.append(batch.host_problem(ctx, float(f), int(segs[0]) + feed - 1))
        finally:
            nb.nec_delete(ctx)
    return problems


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    s = types.SimpleNamespace(**case)
    if s.kind == "dipole":
        s.length, s.radius, s.freq = rng.uniform(0.9, 1.1), rng.uniform(0.5e-3, 2e-3), rng.uniform(140.0, 160.0)
    elif s.kind in ("yagi", "fields"):
        s.params = W.yagi_params(rng, n_elements=s.elements, nseg=s.nseg)
        s.f0 = rng.uniform(140.0, 145.0)
    elif s.kind == "near_ground":
        s.height, s.tilt = rng.uniform(0.08, 0.12), rng.uniform(0.2, 0.4)
        s.eps, s.sigma, s.freq = rng.uniform(8.0, 14.0), rng.uniform(0.004, 0.012), rng.uniform(145.0, 155.0)
    elif s.kind == "gradient":
        half, xs, rad, _ = W.yagi_params(rng, n_elements=s.elements, nseg=s.nseg)
        s.p = np.concatenate([half, xs, rad])
    elif s.kind == "mesh":
        s.theta, s.phi, s.freq = rng.uniform(0.0, 10.0), rng.uniform(0.0, 90.0), rng.uniform(145.0, 155.0)
    elif s.kind == "helix":
        s.seed, s.freq = int(seed), rng.uniform(980.0, 1020.0)
    elif s.kind == "batch":
        s.problems = _population(s.variants, s.nfreq, rng)
        s.theta, s.phi = batch.pattern_grid()
    else:
        s.z, s.b = _matrix(s.n, rng)
        s.engine = _Engine()
    return s


# ---------------------------------------------------------------- passes

def _ok(r, what):
    if r != 0:
        raise RuntimeError("%s failed: %s" % (what, nb.nec_error_message()))


def _grid(s, low=0.0, high=180.0):
    return (0, s.nth, s.nph, 1, 0, 0, 0, low, 0.0, (high - low) / max(1, s.nth - 1), 360.0 / s.nph, 0.0, 0.0)


def _read(ctx, results, cells, feeds):
    """What a caller reads of each result: currents, far field, input impedances."""
    out = {"currents": np.stack([nb.currents(ctx, i) for i in range(results)])}
    if cells:
        out["fields"] = np.stack([np.stack(nb.pattern_fields(ctx, i, cells)) for i in range(results)])
        out["gain"] = np.array([[nb.nec_gain_max(ctx, i), nb.nec_gain_mean(ctx, i)] for i in range(results)])
    if feeds:
        out["zin"] = np.array([[complex(nb.nec_impedance_real_indexed(ctx, i, f), nb.nec_impedance_imag_indexed(ctx, i, f))
                                for f in range(feeds)] for i in range(results)])
    return out


def _run_dipole(s, ctx):
    _ok(nb.nec_set_precision(ctx, s.precision), "precision")
    _ok(nb.nec_wire(ctx, 1, s.nseg, 0.0, 0.0, -0.5 * s.length, 0.0, 0.0, 0.5 * s.length, s.radius, 1.0, 1.0), "wire")
    _ok(nb.nec_geometry_complete(ctx, 0), "geometry")
    _ok(nb.nec_fr_card(ctx, 0, 1, s.freq, 0.0), "fr")
    _ok(nb.nec_ex_card(ctx, 0, 1, (s.nseg + 1) // 2, 0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0), "ex")
    _ok(nb.nec_rp_card(ctx, *_grid(s)), "rp")
    return _read(ctx, 1, s.nth * s.nph, 1)


def _run_yagi(s, ctx):
    over = s.ground != FREE
    W.yagi(API, ctx, s.params, height=8.0 if over else 0.0, nfreq=s.nfreq, f0=s.f0, df=0.5,
           ground=GN[s.ground] if over else None, pattern=_grid(s, 0.0, 88.0 if over else 180.0))
    return _read(ctx, s.nfreq, s.nth * s.nph, 1)


def _run_near_ground(s, ctx):
    n2 = max(5, s.nseg // 2)
    _ok(nb.nec_wire(ctx, 1, s.nseg, -0.5, 0.0, s.height, 0.5, 0.0, s.height, 1e-3, 1.0, 1.0), "wire")
    _ok(nb.nec_wire(ctx, 2, n2, 0.6, 0.0, 0.05, 0.6, s.tilt, 0.4, 1e-3, 1.0, 1.0), "wire")
    _ok(nb.nec_geometry_complete(ctx, 1), "geometry")
    _ok(nb.nec_gn_card(ctx, 2, 0, s.eps, s.sigma, 0.0, 0.0, 0.0, 0.0), "gn")
    _ok(nb.nec_fr_card(ctx, 0, s.nfreq, s.freq, 10.0), "fr")
    _ok(nb.nec_ex_card(ctx, 0, 1, (s.nseg + 1) // 2, 0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0), "ex")
    _ok(nb.nec_ne_card(ctx, 0, s.nx, s.ny, s.nz, -0.6, 0.1, 0.02, 1.2 / s.nx, 0.1, 0.1), "ne")
    _ok(nb.nec_rp_card(ctx, 0, 10, 4, 1, 0, 0, 0, 0.0, 0.0, 9.0, 90.0, 0.0, 0.0), "rp")
    out = _read(ctx, s.nfreq, 40, 1)
    out["near"] = np.stack([f for _, _, f in nb.near_fields(ctx)])
    return out


def _run_fields(s, ctx):
    half, xs, rad, segs = s.params
    for e in range(len(half)):
        _ok(nb.nec_wire(ctx, e + 1, int(segs[e]), float(xs[e]), 0.0, 1.5 - float(half[e]), float(xs[e]), 0.0,
                        1.5 + float(half[e]), float(rad[e]), 1.0, 1.0), "wire")
    _ok(nb.nec_geometry_complete(ctx, 0 if s.ground == FREE else 1), "geometry")
    if s.ground != FREE:
        _ok(nb.nec_gn_card(ctx, *GN[s.ground]), "gn")
    _ok(nb.nec_fr_card(ctx, 0, 1, s.f0, 0.0), "fr")
    _ok(nb.nec_ex_card(ctx, 0, 2, (s.nseg + 1) // 2, 0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0), "ex")
    box = (s.nx, s.ny, s.nz, -1.0, 0.31, 0.2, 5.0 / s.nx, 0.2, 0.25)
    _ok(nb.nec_ne_card(ctx, 0, *box), "ne")
    _ok(nb.nec_nh_card(ctx, 0, *box), "nh")
    near = nb.near_fields(ctx)
    return {"electric": near[0][2], "magnetic": near[1][2], "currents": nb.currents(ctx, 0)}


def _run_mesh(s, ctx):
    """nwires + nwires wires of nwires - 1 segments on 5 cm pitch, joined at
    the crossings; plane waves along a cut of incidence angles."""
    w, pitch = s.nwires, 0.05
    h, n = 0.5 * pitch * (w - 1), w - 1
    for k in range(w):
        c = -h + pitch * k
        _ok(nb.nec_wire(ctx, k + 1, n, -h, c, 0.0, h, c, 0.0, 1e-3, 1.0, 1.0), "wire")
    for k in range(w):
        c = -h + pitch * k
        _ok(nb.nec_wire(ctx, w + k + 1, n, c, -h, 0.0, c, h, 0.0, 1e-3, 1.0, 1.0), "wire")
    _ok(nb.nec_geometry_complete(ctx, 0), "geometry")
    _ok(nb.nec_fr_card(ctx, 0, 1, s.freq, 0.0), "fr")
    _ok(nb.nec_ex_card(ctx, 1, s.angles, 1, 0, s.theta, s.phi, 0.0, 4.0, 0.0, 0.0), "ex")
    _ok(nb.nec_rp_card(ctx, *_grid(s)), "rp")
    return _read(ctx, s.angles, s.nth * s.nph, 0)


def _run_helix(s, ctx):
    _ok(nb.nec_set_precision(ctx, s.precision), "precision")
    W.helix_array(API, ctx, k=s.k, seed=s.seed, nseg=s.nseg, freq_mhz=s.freq, pattern=_grid(s))
    return _read(ctx, 1, s.nth * s.nph, s.k * s.k)


_RUN = {"dipole": _run_dipole, "yagi": _run_yagi, "near_ground": _run_near_ground, "fields": _run_fields,
        "mesh": _run_mesh, "helix": _run_helix}


def run(state):
    s = state
    if s.kind == "batch":
        r = batch.sweep(s.problems, s.theta, s.phi)
        return {"zin": r["zin"], "cur": r["cur"], "gain": r["gain"], "status": r["status"]}
    if s.kind == "gradient":
        # a step of 10 um: well below every radius, and far enough above
        # rounding for the differences of the perturbed structures
        value, jac = adjoint.gradient(lambda ctx, p: W.yagi_ground_cards(API, ctx, p, nseg=s.nseg), s.p, 145.0, 80.0,
                                      0.0, h=1e-5)
        return {"value": value, "jac": jac}
    if s.kind == "matrix":
        x = np.empty(s.n, dtype=np.complex128)
        if nb.lib.necgpu_matrix_solve(s.engine.h, s.n, s.z.ctypes.data, s.b.ctypes.data, s.precision, x.ctypes.data,
                                      None) != 0:
            raise RuntimeError("matrix_solve: %s" % nb.lib.necgpu_last_error(s.engine.h))
        return {"x": x}
    ctx = nb.nec_create()
    try:
        return _RUN[s.kind](s, ctx)
    finally:
        nb.nec_delete(ctx)


# ---------------------------------------------------------------- work and exact values

# operations of one field evaluation: distances, a square root, a sine and
# cosine, quotients and three complex components (the closed-form far pair;
# the image over ground doubles it)
_PAIR, _DIR = 120.0, 60.0


def _solve_flops(n, rhs=1):
    return 8.0 / 3.0 * n ** 3 + 8.0 * n * n * rhs


def work(case):
    c = types.SimpleNamespace(**case)
    seg = 8 * 8.0  # a segment's eight doubles in
    if c.kind == "matrix":
        return {"bytes": 16.0 * (c.n * c.n + 2 * c.n), "flops": _solve_flops(c.n)}
    if c.kind == "batch":
        n, m = 227.0, c.variants * c.nfreq  # mean size of the seeded Yagi population: 9 elements of 25 segments
        flops = m * (_PAIR * n * n + _solve_flops(n) + _DIR * n * 91 * 72)
        return {"bytes": m * (n * (seg + 32.0) + 4.0 * 91 * 72), "flops": flops}
    if c.kind == "gradient":
        n, npar = c.elements * c.nseg, 3 * c.elements
        return {"bytes": (2 * npar + 1) * n * seg + 8.0 * 3 * npar,
                "flops": (2 * npar + 1) * 2 * _PAIR * n * n + _solve_flops(n, 4)}
    image, freqs, solves, points, dirs = 1.0, 1, 1, 0, getattr(c, "nth", 0) * getattr(c, "nph", 0)
    if c.kind == "dipole":
        n = c.nseg
    elif c.kind == "yagi":
        n, freqs = c.elements * c.nseg, c.nfreq
    elif c.kind == "near_ground":
        n, freqs, points, dirs = c.nseg + max(5, c.nseg // 2), c.nfreq, c.nx * c.ny * c.nz, 40
    elif c.kind == "fields":
        n, points = c.elements * c.nseg, 2 * c.nx * c.ny * c.nz
    elif c.kind == "mesh":
        n, solves = 2 * c.nwires * (c.nwires - 1), c.angles
    else:
        n = c.k * c.k * c.nseg
    if getattr(c, "ground", FREE) != FREE or c.kind == "near_ground":
        image = 2.0
    flops = freqs * (image * _PAIR * n * n + _solve_flops(n, solves) + image * _DIR * n * dirs * solves
                     + image * _PAIR * n * points)
    return {"bytes": n * seg + freqs * (solves * (16.0 * n + 32.0 * dirs) + 48.0 * points), "flops": flops}


def exact(case, seed):
    if case["kind"] != "matrix":
        return None
    z, b = _matrix(case["n"], np.random.default_rng(seed))
    return {"x": np.linalg.solve(z, b)}
