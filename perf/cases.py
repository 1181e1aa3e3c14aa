"""The workloads this library is measured on: what a program does with it per
call, through the public entry points, from the smallest calls to the largest.

kinds (the "kind" of a case):

  blocks      the four block hooks of the reference's mobility_solver in their
              order, host arrays in and out
  grand       the grand mobility (all four blocks at once), host arrays in and
              out
  solve       compute_velocities of a free body, as one Broyden iteration runs
              it: positions, forces and the last solution up, segment
              velocities, blob forces and body velocity back
  steps       implicit time steps of one swimmer from a perturbed start
  prescribed  the prescribed-cilia solve at the next phase of the beat, warm
              started from the last one
  flow        the flow field of a swimmer at a set of points
  served      requests of several uneven swimmers to a step server

precision "fp64" is the default form, with float64 host arrays. "fp32c" (FP32
pair sums, compensated) is driven as a program built with Real = float drives
it (the reference's shipped configuration): float host arrays through the
*_f32 copies where the call has them, and results kept as floats.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from timfilsimmod_gb300.flow_field import FlowFieldEvaluator
from timfilsimmod_gb300.geometry import (elastic_swimmer, fibonacci_sphere, icosphere,
                                         prescribed_swimmer)
from timfilsimmod_gb300.mobility import RpyMobilitySolver
from timfilsimmod_gb300.prescribed import PrescribedCiliaSolver
from timfilsimmod_gb300.serving import StepServer
from timfilsimmod_gb300.stepper import ImplicitStepper

SEG_SEP = 2.2
DEFAULT_DT = 36.3833 / 300.0  # the reference's default time step
KB = 1800.0


def listed():
    return [
        # the smallest swimmer of the tests: launches and host calls are the time
        dict(name="blocks_tiny_fp64", kind="blocks", precision="fp64", nfil=3, nseg=14,
             nblob=162),
        # the benchmark's product (640 filaments x 20 segments, 2562 blobs)
        dict(name="grand_medium_fp32c", kind="grand", precision="fp32c", nfil=640, nseg=20,
             nblob=2562),
        # the same in the default, reference-matching precision
        dict(name="blocks_medium_fp64", kind="blocks", precision="fp64", nfil=640, nseg=20,
             nblob=2562),
        # the largest swimmer of the benchmark
        dict(name="grand_large_fp32c", kind="grand", precision="fp32c", nfil=4000, nseg=20,
             nblob=10242),
        # one Broyden iteration's solve; ragged sizes, default precision
        dict(name="solve_ragged_fp64", kind="solve", precision="fp64", nfil=211, nseg=17,
             nblob=1289),
        # the same solve in the production form at the benchmark's sizes
        dict(name="solve_medium_fp32c", kind="solve", precision="fp32c", nfil=640, nseg=20,
             nblob=2562),
        # a validation run of the small swimmer against the reference
        dict(name="steps_small_fp64", kind="steps", precision="fp64", nfil=32, nseg=20,
             steps=3, dt=1e-3),
        # production steps at the reference's default DT (every step iterates)
        dict(name="steps_medium_fp32c", kind="steps", precision="fp32c", nfil=640, nseg=20,
             steps=2, dt=DEFAULT_DT),
        # prescribed beats, ragged sizes, free body, default precision
        dict(name="prescribed_ragged_fp64", kind="prescribed", precision="fp64", flags=6,
             nfil=97, nseg=13, nblob=642),
        # the benchmark's prescribed-cilia solve
        dict(name="prescribed_medium_fp32c", kind="prescribed", precision="fp32c", flags=7,
             nfil=640, nseg=20, nblob=2562),
        # a field for visualisation around the medium swimmer, on a 63^3 grid
        dict(name="flow_medium_fp32c", kind="flow", precision="fp32c", nfil=640, nseg=20,
             nblob=2562, points=250047),
        # several small swimmers served at once (an orbit search, a sweep)
        dict(name="served_small_fp32c", kind="served", precision="fp32c", requests=6,
             min_fil=16, max_fil=96, nseg=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["blocks", "grand", "solve", "steps", "prescribed", "flow", "grand",
                       "solve", "flow", "served"])
    prec = rng.choice(["fp64", "fp32c"])
    nseg = rng.randint(5, 25)
    if kind in ("blocks", "grand"):
        # fp64 pair sums cost about 40 times fp32c's: sizes up to the medium swimmer's
        segs = _log(rng, 40, 12800 if prec == "fp64" else 60000)
        return dict(kind=kind, precision=prec, nfil=max(1, segs // nseg), nseg=nseg,
                    nblob=_log(rng, 100, 2562 if prec == "fp64" else 8000))
    if kind == "solve":
        segs = _log(rng, 40, 4000 if prec == "fp64" else 12800)
        return dict(kind=kind, precision=prec, nfil=max(1, segs // nseg), nseg=nseg,
                    nblob=_log(rng, 150, 1300 if prec == "fp64" else 2562))
    if kind == "steps":
        if prec == "fp64":
            return dict(kind=kind, precision=prec, nfil=rng.randint(4, 32),
                        nseg=rng.randint(10, 20), steps=rng.randint(1, 3), dt=1e-3)
        return dict(kind=kind, precision=prec, nfil=_log(rng, 8, 500), nseg=rng.randint(10, 20),
                    steps=rng.randint(1, 2), dt=rng.choice([1e-3, DEFAULT_DT]))
    if kind == "prescribed":
        segs = _log(rng, 100, 1300 if prec == "fp64" else 10000)
        return dict(kind=kind, precision=prec, flags=rng.choice([6, 7]),
                    nfil=max(2, segs // nseg), nseg=nseg,
                    nblob=_log(rng, 150, 642 if prec == "fp64" else 2562))
    if kind == "flow":
        segs = _log(rng, 100, 12800)
        return dict(kind=kind, precision=prec, nfil=max(1, segs // nseg), nseg=nseg,
                    nblob=rng.choice([0, _log(rng, 100, 2562)]),
                    points=_log(rng, 500, 6000 if prec == "fp64" else 240000))
    return dict(kind="served", precision="fp32c", requests=rng.randint(2, 6),
                min_fil=rng.randint(8, 16), max_fil=rng.randint(24, 90),
                nseg=rng.randint(12, 20))


# -- geometry ------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _sphere(subdivisions):
    return icosphere(subdivisions)


def _body(nblob, nfil):
    """Blob references and radius: the icospheres of the repository's
    configurations at their sizes, else a Fibonacci lattice of the same
    spacing as the 2562-blob sphere's; larger where the filaments' roots would
    be closer than two segment diameters."""
    known = {162: (2, 10.0), 642: (3, 20.0), 2562: (4, 60.0), 10242: (5, 150.0)}
    room = 4.0 * math.sqrt(nfil / (4.0 * math.pi))
    if nblob in known:
        k, radius = known[nblob]
        radius = max(radius, room)
        return radius * _sphere(k), radius
    radius = max(60.0 * math.sqrt(nblob / 2562.0), room)
    return radius * fibonacci_sphere(nblob), radius


def _swimmer(case, seed):
    """A sphere with beating filaments: blob references, positions and N(0,1)
    forces, as the reference's arrays."""
    rng = np.random.default_rng(seed)
    nfil, nseg, nblob = case["nfil"], case["nseg"], case["nblob"]
    refs, radius = _body(nblob, nfil) if nblob else (np.zeros((0, 3)), _body(642, nfil)[1])
    n = fibonacci_sphere(nfil)
    helper = np.where(np.abs(n[:, 2:3]) < 0.9, [[0.0, 0.0, 1.0]], [[1.0, 0.0, 0.0]])
    t = np.cross(n, helper)
    t /= np.linalg.norm(t, axis=1, keepdims=True)
    phase = rng.uniform(0.0, 2.0 * np.pi, size=(nfil, 1))
    frac = (np.arange(nseg) + 0.5) / nseg
    theta = 0.5 * np.sin(phase - 2.0 * frac) * frac
    tang = np.cos(theta)[..., None] * n[:, None] + np.sin(theta)[..., None] * t[:, None]
    steps = np.concatenate([np.zeros((nfil, 1, 3)), SEG_SEP * tang[:, :-1]], axis=1)
    base = (radius + 1.0 + 0.5 * SEG_SEP) * n
    x_segs = (base[:, None] + np.cumsum(steps, axis=1)).reshape(-1)
    if not nblob:  # the wall-bounded flow form: everything above z = 0
        x_segs[2::3] += 1.0 + radius + (nseg + 1) * SEG_SEP
    f_segs = rng.normal(size=6 * nfil * nseg)
    f_blobs = rng.normal(size=3 * nblob)
    return refs, radius, x_segs, f_segs, f_blobs


def _floats(a):
    """A page-locked float copy of an array, as a numpy view and its owner."""
    t = torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32).reshape(-1)).pin_memory()
    return t.numpy(), t


class _Arrays:
    """The host arrays of one solver: the solver's own float64 ones (fp64) or
    page-locked floats with the *_f32 copies (fp32c)."""

    def __init__(self, solver, refs, x_segs, f_segs, f_blobs):
        self.s = solver
        self.single = solver.precision == "fp32c"
        s = solver
        names = ("x_segs", "f_segs", "v_segs", "x_blobs", "f_blobs", "v_blobs")
        given = dict(x_segs=x_segs, f_segs=f_segs, x_blobs=refs.reshape(-1), f_blobs=f_blobs)
        self.keep, self.a = [], {}
        for k in names:
            host = getattr(s, k + "_host")
            if k in given:
                host[:] = given[k]
            if self.single:
                host, owner = _floats(host)
                self.keep.append(owner)
            self.a[k] = host

    def _copy(self, what, name):
        a = self.a[name]
        self.s._call("tfs_copy_" + what + ("_f32" if self.single else ""), a.ctypes.data)
        return a

    def up(self, blobs=True):
        self._copy("segment_positions_to_device", "x_segs")
        self._copy("segment_forces_to_device", "f_segs")
        if blobs:
            self._copy("blob_positions_to_device", "x_blobs")
        self._copy("blob_forces_to_device", "f_blobs")

    def v_segs(self):
        return self._copy("segment_velocities_to_host", "v_segs")

    def v_blobs(self):
        return self._copy("blob_velocities_to_host", "v_blobs")


def _end_force(nseg):
    return 220.0 * KB / (2.6 * 2.6 * nseg * nseg)


# -- blocks, grand ---------------------------------------------------------------
def _prepare_product(case, seed):
    refs, _, x, f, fb = _swimmer(case, seed)
    s = RpyMobilitySolver(1, case["nfil"], case["nseg"], case["nblob"], case["precision"])
    return dict(s=s, a=_Arrays(s, refs, x, f, fb))


def _run_blocks(st):
    s, a = st["s"], st["a"]
    a.up()
    s.evaluate_segment_segment_mobility()
    s.evaluate_segment_blob_mobility()
    v_segs = a.v_segs()
    s.evaluate_blob_blob_mobility()
    v_blobs = a.v_blobs()
    s.wait_for_device()
    from_blobs = v_blobs.copy()  # the next product's copy overwrites the array
    s.evaluate_blob_segment_mobility()
    v_blobs = a.v_blobs()
    s.wait_for_device()
    return {"v_segs": v_segs, "v_blobs_from_blobs": from_blobs, "v_blobs_from_segs": v_blobs}


def _run_grand(st):
    s, a = st["s"], st["a"]
    a.up()
    s.apply_grand_mobility()
    out = {"v_segs": a.v_segs(), "v_blobs": a.v_blobs()}
    s.wait_for_device()
    return out


# -- solve -----------------------------------------------------------------------
def _solve_inputs(case, seed):
    refs, _, x, f, _ = _swimmer(case, seed)
    rng = np.random.default_rng([seed, 1])
    swimmer_f = rng.normal(size=6) * math.sqrt(case["nfil"] * case["nseg"])
    last = f + 1e-2 * rng.normal(size=f.size)  # the forces of the last iteration
    return refs, x, f, last, swimmer_f


def _prepare_solve(case, seed):
    refs, x, f, last, swimmer_f = _solve_inputs(case, seed)
    s = RpyMobilitySolver(1, case["nfil"], case["nseg"], case["nblob"], case["precision"])
    s.set_blob_references(refs)
    s.set_body_pose(np.zeros(3), np.array([1.0, 0.0, 0.0, 0.0]))
    s.set_linear_solver(1e-8)
    s.make_body_reference_matrices()
    # the last iteration's solution is what this one starts from
    a = _Arrays(s, refs, x, last, np.zeros(refs.size))
    a.up(blobs=False)
    s.compute_velocities(swimmer_f)
    warm_f, warm_v = s.blob_forces(), s.body_velocities()
    a = _Arrays(s, refs, x, f, warm_f)
    blob_forces = np.empty_like(a.a["f_blobs"])
    if case["precision"] == "fp32c":
        blob_forces, owner = _floats(blob_forces)
        a.keep.append(owner)
    return dict(s=s, a=a, v=warm_v, sf=swimmer_f, fb=blob_forces)


def _run_solve(st):
    s, a = st["s"], st["a"]
    a.up(blobs=False)
    s.set_body_velocities(st["v"])
    s.compute_velocities(st["sf"])
    v = a.v_segs()
    fb = st["fb"]
    s._call("tfs_copy_blob_forces_to_host" + ("_f32" if a.single else ""), fb.ctypes.data)
    body = s.body_velocities()
    s.wait_for_device()
    return {"v_segs": v, "f_blobs": fb, "v_body": body.astype(v.dtype)}


# -- steps -----------------------------------------------------------------------
def _make_stepper(case, precision):
    nfil, nseg = case["nfil"], case["nseg"]
    blob_refs, fil_refs, fil_dirs, radius = elastic_swimmer(nfil, nseg, SEG_SEP)
    efm = _end_force(nseg)
    s = RpyMobilitySolver(1, nfil, nseg, len(blob_refs), precision, end_force_magnitude=int(efm))
    s.set_blob_references(blob_refs)
    s.set_linear_solver(1e-8)
    st = ImplicitStepper(s, nfil, nseg, fil_refs, fil_dirs, seg_sep=SEG_SEP, dt=case["dt"],
                         tol=1e-4, end_force_magnitude=efm, body_radius=radius)
    return s, st


def _rotations(n, seed):
    return 1e-4 * np.random.default_rng(seed).normal(size=3 * n)


def _prepare_steps(case, seed):
    s, st = _make_stepper(case, case["precision"])
    return dict(s=s, st=st, steps=case["steps"], single=case["precision"] == "fp32c",
                rot=_rotations(case["nfil"] * case["nseg"], seed))


def _run_steps(state):
    st = state["st"]
    st.reset(state["rot"])
    for nt in range(state["steps"]):
        st.step(nt)
    got = st.state()
    out = {k: got[k] for k in ("x", "q", "body_x", "body_q")}
    if state["single"]:
        return {k: v.astype(np.float32) for k, v in out.items()}
    return dict(out, lam=got["lam"], tether=got["tether"])


# -- prescribed cilia --------------------------------------------------------------
_TABLE = 2.0 * np.pi * np.arange(100) / 100
PHASE_FORCE, ANGLE_FORCE = 1.0 + 0.5 * np.sin(_TABLE), 0.2 * np.cos(_TABLE)


def _prescribed_inputs(case, seed):
    rng = np.random.default_rng(seed)
    refs, radius = _body(case["nblob"], case["nfil"])
    g = prescribed_swimmer(case["nfil"], case["nseg"], radius=radius, subdivisions=0,
                           seg_sep=2.6)
    g.blob_references = refs
    phase = rng.uniform(0.0, 2.0 * np.pi, g.nfil)
    omega = 2.0 * np.pi * (1.0 + 0.05 * rng.uniform(-1.0, 1.0, g.nfil))
    angle = rng.uniform(-0.1, 0.1, g.nfil)
    return g, phase, omega, angle


def _prepare_prescribed(case, seed):
    g, phase, omega, angle = _prescribed_inputs(case, seed)
    ps = PrescribedCiliaSolver(case["flags"], g.nfil, g.nseg, g.blob_references, g.seg_sep,
                               PHASE_FORCE, ANGLE_FORCE, tol=1e-10, precision=case["precision"])
    ps.set_solution(phase_dot=omega)
    last = phase - 1e-2 * omega  # the last time step's phases
    x, vp, va = g.kinematics(last, angle)
    ps.compute_velocities(x, vp, va, last, omega, angle, omega)
    warm = ps.solution()
    x, vp, va = g.kinematics(phase, angle)
    return dict(ps=ps, warm=warm, args=(x, vp, va, phase, omega, angle, omega),
                single=case["precision"] == "fp32c", free=not case["flags"] & 1)


def _run_prescribed(st):
    ps = st["ps"]
    ps.set_solution(**st["warm"])
    ps.compute_velocities(*st["args"])
    out = ps.solution()
    if not st["free"]:
        del out["v_body"]
    return {k: v.astype(np.float32) for k, v in out.items()} if st["single"] else out


# -- flow --------------------------------------------------------------------------
def _flow_inputs(case, seed):
    refs, _, x, f, fb = _swimmer(case, seed)
    xs = x.reshape(-1, 3)
    lo, hi = xs.min(0) - 10.0, xs.max(0) + 10.0
    n, rng = case["points"], np.random.default_rng([seed, 2])
    m = round(n ** (1.0 / 3.0))
    if m ** 3 == n:  # a grid of cell centres
        c = (np.arange(m) + 0.5) / m
        z, y, xx = np.meshgrid(c, c, c, indexing="ij")
        p = np.stack([xx.ravel(), y.ravel(), z.ravel()], axis=1)
    else:            # tracer particles
        p = rng.uniform(size=(n, 3))
    if not case["nblob"]:
        lo[2] = 0.0
    return refs, x, f, fb, lo + p * (hi - lo)


def _prepare_flow(case, seed):
    refs, x, f, fb, points = _flow_inputs(case, seed)
    ev = FlowFieldEvaluator(1, case["nfil"], case["nseg"], case["nblob"], case["points"],
                            precision=case["precision"])
    for name, val in (("x_flow", points), ("x_segs", x), ("f_segs", f), ("x_blobs", refs),
                      ("f_blobs", fb)):
        getattr(ev, name + "_host")[:] = val.reshape(-1)
    return dict(ev=ev, single=case["precision"] == "fp32c")


def _run_flow(st):
    ev = st["ev"]
    ev.read_positions_and_forces()
    v = ev.velocities()
    ev.wait()
    return {"v": v.astype(np.float32) if st["single"] else v}


# -- served requests ---------------------------------------------------------------
def _prepare_served(case, seed):
    rng = np.random.default_rng(seed)
    k, nseg = case["requests"], case["nseg"]
    # uneven sizes over the whole range, the same for every seed (a server
    # keeps its swimmers); the perturbed starts are the seed's
    sizes = [round(case["min_fil"] * (case["max_fil"] / case["min_fil"]) ** (i / max(1, k - 1)))
             for i in range(k)]
    sv = StepServer(num_workers=4, precision="fp32c", linear_tol=1e-8, dt=1e-3, tol=1e-4,
                    seg_sep=SEG_SEP, end_force_magnitude=_end_force(nseg))
    reqs = []
    for i, nf in enumerate(sizes):
        blob_refs, fil_refs, fil_dirs, radius = elastic_swimmer(nf, nseg, SEG_SEP)
        reqs.append((blob_refs, fil_refs, fil_dirs, nseg, 1,
                     1e-4 * rng.normal(size=3 * nf * nseg), radius))
    st = dict(sv=sv, reqs=reqs)
    _run_served(st)  # the server has these swimmers resident
    return st


def _run_served(st):
    sv = st["sv"]
    tickets = [sv.submit(*r) for r in st["reqs"]]
    out = []
    for t in tickets:
        r = sv.poll(t, wait=True)
        out.append({k: r[k].astype(np.float32) for k in ("x", "q", "body")})
    return out


_PREPARE = dict(blocks=_prepare_product, grand=_prepare_product, solve=_prepare_solve,
                steps=_prepare_steps, prescribed=_prepare_prescribed, flow=_prepare_flow,
                served=_prepare_served)
_RUN = dict(blocks=_run_blocks, grand=_run_grand, solve=_run_solve, steps=_run_steps,
            prescribed=_run_prescribed, flow=_run_flow, served=_run_served)


def prepare(case, seed):
    return case["kind"], _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state[0]](state[1])


# -- what a pass cannot do without ---------------------------------------------------
def work(case):
    """Canonical flops of the pair sums (93 for a 6x6 pair, 56 for 6x3 and 3x6,
    40 for 3x3; flow 44 per segment source and 28 per blob source, 87 for a
    segment source above the wall), one operator application per solve; bytes
    of the arrays in and out. Iterative calls need several times the flops."""
    size = 4 if case["precision"] == "fp32c" else 8
    if case["kind"] == "served":
        ns = case["requests"] * math.sqrt(case["min_fil"] * case["max_fil"]) * case["nseg"]
        one = ns / case["requests"]
        return {"bytes": 8 * 14.0 * ns,
                "flops": case["requests"] * (93.0 * one * one + 112 * one * 642 + 40 * 642 ** 2)}
    ns = case["nfil"] * case["nseg"]
    if case["kind"] == "steps":
        nb = 642 if case["nfil"] < 128 else 2562
        return {"bytes": 8.0 * (3 + 7) * ns,
                "flops": case["steps"] * (93.0 * ns * ns + 112.0 * ns * nb + 40.0 * nb * nb)}
    nb = case["nblob"]
    if case["kind"] == "flow":
        n = case["points"]
        return {"bytes": 8.0 * (6 * n + 9 * ns + 6 * nb),
                "flops": n * ((44.0 if nb else 87.0) * ns + 28.0 * nb)}
    if case["kind"] == "prescribed":
        return {"bytes": 8.0 * (12 * ns + 3 * nb), "flops": 40.0 * (ns + nb) ** 2}
    return {"bytes": float(size * (15 * ns + 9 * nb)),
            "flops": 93.0 * ns * ns + 112.0 * ns * nb + 40.0 * nb * nb}


# -- the same in 64 bits ---------------------------------------------------------------
def _t(a, cols):
    return torch.as_tensor(np.asarray(a, dtype=np.float64).reshape(-1, cols), device="cuda")


def _blocks_of(xt, xs):
    """Slices of the targets whose pair matrices hold about 2^24 entries."""
    step = max(1, (1 << 24) // max(1, len(xs)))
    return [slice(i, min(len(xt), i + step)) for i in range(0, len(xt), step)]


def _mobility(xt, xs, f, tau=None, rot=False):
    """RPY velocities (and angular velocities, rot) of unit spheres at xt from
    forces f (and torques tau) on unit spheres at xs, mu = 1 (Rotne & Prager
    1969; Yamakawa 1970; overlapping spheres by Wajnryb et al. 2013)."""
    out = torch.zeros(len(xt), 6 if rot else 3, dtype=torch.float64, device="cuda")
    cols = f if tau is None else torch.cat([f, tau], dim=1)
    for sl in _blocks_of(xt, xs):
        d = [xt[sl, k:k + 1] - xs[None, :, k] for k in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        r = torch.sqrt(r2)
        near = r2 <= 4.0
        ir = 1.0 / torch.where(r2 == 0.0, 1.0, r)
        ir2 = ir * ir
        A = torch.where(near, 4.0 / 3.0 - 0.375 * r, ir + (2.0 / 3.0) * ir * ir2)
        # coefficient of (d.F) d
        B = torch.where(near, 0.125 * ir, ir * ir2 - 2.0 * ir * ir2 * ir2)
        df = d[0] * f[:, 0] + d[1] * f[:, 1] + d[2] * f[:, 2]
        v = A @ f
        B *= df
        v += torch.stack([(B * d[k]).sum(1) for k in range(3)], dim=1)
        if tau is not None or rot:
            # coefficient of T x d and F x d
            E = torch.where(near, (8.0 - 3.0 * r) / 16.0, ir * ir2)
            G = [(E * d[k]) @ cols for k in range(3)]

            def cross(c):  # sum over sources of (column vector at c) x d E
                return torch.stack([G[2][:, c + 1] - G[1][:, c + 2],
                                    G[0][:, c + 2] - G[2][:, c],
                                    G[1][:, c] - G[0][:, c + 1]], dim=1)

            if tau is not None:
                v += cross(3)
            if rot:
                w = cross(0)
                if tau is not None:
                    A = torch.where(near, (5.0 * r * r2 - 54.0 * r + 64.0) / 64.0, -0.5 * ir * ir2)
                    B = torch.where(near, 3.0 * (6.0 - r2) * ir / 64.0, 1.5 * ir * ir2 * ir2)
                    B *= d[0] * tau[:, 0] + d[1] * tau[:, 1] + d[2] * tau[:, 2]
                    w += A @ tau + torch.stack([(B * d[k]).sum(1) for k in range(3)], dim=1)
                out[sl, 3:] = w
        out[sl, :3] = v
    return out / (8.0 * math.pi)


def _matrix(x):
    """The dense translational mobility matrix (3n, 3n) of unit spheres at x."""
    n = len(x)
    M = torch.empty(n, 3, n, 3, dtype=torch.float64, device="cuda")
    for sl in _blocks_of(x, x):
        d = [x[sl, k:k + 1] - x[None, :, k] for k in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        r = torch.sqrt(r2)
        near = r2 <= 4.0
        ir = 1.0 / torch.where(r2 == 0.0, 1.0, r)
        A = torch.where(near, 4.0 / 3.0 - 0.375 * r, ir + (2.0 / 3.0) * ir ** 3)
        B = torch.where(near, 0.125 * ir, ir ** 3 - 2.0 * ir ** 5)
        for i in range(3):
            for j in range(3):
                M[sl, i, :, j] = B * d[i] * d[j] + (A if i == j else 0.0)
    return M.reshape(3 * n, 3 * n) / (8.0 * math.pi)


def _repulsion(xt, xs, skip, magnitude):
    """The reference's barrier force on unit spheres at xt from those at xs;
    skip(i, j): the pairs that do not repel."""
    out = torch.zeros_like(xt)
    for sl in _blocks_of(xt, xs):
        d = [xt[sl, k:k + 1] - xs[None, :, k] for k in range(3)]
        r = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
        i = torch.arange(len(xt), device="cuda")[sl, None]
        j = torch.arange(len(xs), device="cuda")[None, :]
        act = (r < 2.2) & ~skip(i, j)
        fac = torch.clamp(1.0 - 5.0 * (r - 2.0), max=1.0)
        fac = torch.where(act, magnitude * fac ** 4 / torch.where(act, r, 1.0), 0.0)
        out[sl] = torch.stack([(fac * d[k]).sum(1) for k in range(3)], dim=1)
    return out


def _rigid(d):
    """K (3n, 6): the velocities of points at d from a body's (U, Omega)."""
    n = len(d)
    K = torch.zeros(n, 3, 6, dtype=torch.float64, device="cuda")
    for k in range(3):
        K[:, k, k] = 1.0
    K[:, 0, 4], K[:, 0, 5] = d[:, 2], -d[:, 1]
    K[:, 1, 3], K[:, 1, 5] = -d[:, 2], d[:, 0]
    K[:, 2, 3], K[:, 2, 4] = d[:, 1], -d[:, 0]
    return K.reshape(3 * n, 6)


def _host(**named):
    return {k: v.reshape(-1).cpu().numpy() for k, v in named.items()}


def _seen(case, *arrays):
    """The inputs as the call gets them (floats for fp32c)."""
    if case["precision"] == "fp32c":
        return [np.asarray(a, dtype=np.float32).astype(np.float64) for a in arrays]
    return arrays


def _exact_product(case, seed):
    refs, _, x, f, fb = _swimmer(case, seed)
    x, f, xb, fb = _seen(case, x, f, refs, fb)
    xs, f6, xb, fb = _t(x, 3), _t(f, 6), _t(xb, 3), _t(fb, 3)
    fs, ts = f6[:, :3].contiguous(), f6[:, 3:].contiguous()
    v = _mobility(xs, xs, fs, ts, rot=True) + _mobility(xs, xb, fb, rot=True)
    bb, bs = _mobility(xb, xb, fb), _mobility(xb, xs, fs, ts)
    if case["kind"] == "blocks":
        return _host(v_segs=v, v_blobs_from_blobs=bb, v_blobs_from_segs=bs)
    return _host(v_segs=v, v_blobs=bb + bs)


def _exact_solve(case, seed):
    refs, x, f, _, swimmer_f = _solve_inputs(case, seed)
    x, f = _seen(case, x, f)
    xs, f6, xb = _t(x, 3), _t(f, 6).clone(), _t(refs, 3)
    nseg = case["nseg"]
    mag = 2.0 * int(_end_force(nseg))

    def fil(i, j):  # itself and its neighbours on the same filament
        return (i // nseg == j // nseg) & ((i - j).abs() <= 1)

    def never(i, j):
        return (i < 0) & (j < 0)

    f6[:, :3] += _repulsion(xs, xs, fil, mag) + _repulsion(xs, xb, never, mag)
    rep = _repulsion(xb, xs, never, mag) + _repulsion(xb, xb, lambda i, j: i == j, mag)
    K = _rigid(xb)
    total = torch.as_tensor(swimmer_f, device="cuda") + K.T @ rep.reshape(-1)
    fs, ts = f6[:, :3].contiguous(), f6[:, 3:].contiguous()
    vb = _mobility(xb, xs, fs, ts).reshape(-1)
    n = len(vb)
    S = torch.zeros(n + 6, n + 6, dtype=torch.float64, device="cuda")
    S[:n, :n] = _matrix(xb)
    S[:n, n:] = -K
    S[n:, :n] = -K.T
    sol = torch.linalg.solve(S, torch.cat([-vb, -total]))
    lam = sol[:n].reshape(-1, 3).contiguous()
    v = _mobility(xs, xs, fs, ts, rot=True) + _mobility(xs, xb, lam, rot=True)
    return _host(v_segs=v, f_blobs=lam, v_body=sol[n:])


def _generalised(phase, table):
    """The reference's cyclic cubic Hermite interpolation of a table over one
    period (its slope at node 0 is one-sided)."""
    n = len(table)
    p = phase / (2.0 * np.pi)
    p = (p - np.floor(p)) * n
    lo = np.minimum(p.astype(int), n - 1)
    hi = (lo + 1) % n
    slope = 0.5 * (np.roll(table, -1) - np.roll(table, 1))
    at_lo = np.where(lo == 0, table[1] - table[0], slope[lo])
    at_hi = np.where(hi == 0, table[0] - table[n - 1], slope[hi])
    t = p - lo
    return (table[lo] * (2 * t ** 3 - 3 * t ** 2 + 1) + at_lo * (t ** 3 - 2 * t ** 2 + t)
            + table[hi] * (3 * t ** 2 - 2 * t ** 3) + at_hi * (t ** 3 - t ** 2))


def _exact_prescribed(case, seed):
    nfil, nseg = case["nfil"], case["nseg"]
    ns, nb = nfil * nseg, case["nblob"]
    if ns + nb > 4500:  # a dense solve of 3 (ns + nb) unknowns
        return None
    g, phase, omega, angle = _prescribed_inputs(case, seed)
    x, vp, va = g.kinematics(phase, angle)
    xs, xb = _t(x, 3), _t(g.blob_references, 3)
    pts = torch.cat([xs, xb])
    n, free = 3 * (ns + nb), not case["flags"] & 1
    cols = [_rigid(pts)] if free else []
    row = torch.arange(3 * ns, device="cuda")
    for k in (vp, va):
        K = torch.zeros(n, nfil, dtype=torch.float64, device="cuda")
        K[row, row // (3 * nseg)] = _t(k, 1)[:, 0]
        cols.append(K)
    C = torch.cat(cols, dim=1)
    m = C.shape[1]
    S = torch.zeros(n + m, n + m, dtype=torch.float64, device="cuda")
    S[:n, :n] = _matrix(pts)
    S[:n, n:] = -C
    S[n:, :n] = -C.T
    length = g.seg_sep * (nseg - 1)
    qp = _generalised(phase, PHASE_FORCE) * 0.5 * omega / np.pi
    qa = _generalised(phase, ANGLE_FORCE) * 0.5 * omega / np.pi - 2.0 * omega * length ** 3 * angle
    rhs = np.concatenate([np.zeros(n + m - 2 * nfil), -qp, -qa])
    sol = torch.linalg.solve(S, torch.as_tensor(rhs, device="cuda")).cpu().numpy()
    out = dict(f_segs=sol[:3 * ns].reshape(-1, 3), f_blobs=sol[3 * ns:n].reshape(-1, 3),
               phase_dot=sol[n + m - 2 * nfil:n + m - nfil], angle_dot=sol[n + m - nfil:])
    if free:
        out["v_body"] = sol[n:n + 6]
    return out


def _exact_flow(case, seed):
    refs, x, f, fb, points = _flow_inputs(case, seed)
    p, xs, f6, xb, fb = _t(points, 3), _t(x, 3), _t(f, 6), _t(refs, 3), _t(fb, 3)
    out = torch.zeros_like(p)
    fs = f6[:, :3].contiguous()

    def stokeslet(d, src, sign=1.0):
        ir = torch.rsqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
        w = (d[0] * src[:, 0] + d[1] * src[:, 1] + d[2] * src[:, 2]) * ir ** 3
        v = ir @ src + torch.stack([(w * d[k]).sum(1) for k in range(3)], dim=1)
        return sign * v, ir

    for sl in _blocks_of(p, xs):
        d = [p[sl, k:k + 1] - xs[None, :, k] for k in range(3)]
        v, ir = stokeslet(d, fs)
        ir3 = ir ** 3
        G = [(ir3 * d[k]) @ f6[:, 3:] for k in range(3)]
        v += torch.stack([G[2][:, 1] - G[1][:, 2], G[0][:, 2] - G[2][:, 0],
                          G[1][:, 0] - G[0][:, 1]], dim=1)
        if not case["nblob"]:  # the image system of a no-slip wall at z = 0 (Blake 1971)
            z, h = p[sl, 2:3], xs[None, :, 2]
            X, Y, Z = d[0], d[1], z + h
            v += stokeslet([X, Y, Z], fs, -1.0)[0]
            R2 = X * X + Y * Y + Z * Z
            D = 2.0 * h * torch.rsqrt(R2) ** 5
            v[:, 0] += (D * ((3 * X * X - R2) * z * fs[:, 0] + 3 * X * Y * z * fs[:, 1]
                             + (R2 - 3 * Z * z) * X * fs[:, 2])).sum(1)
            v[:, 1] += (D * (3 * X * Y * z * fs[:, 0] + (3 * Y * Y - R2) * z * fs[:, 1]
                             + (R2 - 3 * Z * z) * Y * fs[:, 2])).sum(1)
            v[:, 2] += (D * ((3 * Z * z + R2) * X * fs[:, 0] + (3 * Z * z + R2) * Y * fs[:, 1]
                             + (R2 - 3 * Z * Z) * z * fs[:, 2])).sum(1)
        else:
            d = [p[sl, k:k + 1] - xb[None, :, k] for k in range(3)]
            v += stokeslet(d, fb)[0]
        out[sl] = v
    return {"v": (out / (8.0 * math.pi)).cpu().numpy()}


def exact(case, seed):
    if case["kind"] in ("blocks", "grand"):
        return _exact_product(case, seed)
    if case["kind"] == "solve":
        return _exact_solve(case, seed)
    if case["kind"] == "prescribed":
        return _exact_prescribed(case, seed)
    if case["kind"] == "flow":
        return _exact_flow(case, seed)
    return None  # hundreds of nested solves: far over 20 seconds
