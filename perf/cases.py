"""The solves that this framework is timed on, and what they answer in 64 bits.

A case is one call of a user's program, host arrays in and host arrays out:

  sweep   a mesh that is already on the GPU (``CudaEngine.prepare``) solved over a
          sweep of frequencies (``CudaEngine.solve``)
  jobs    several uploaded small meshes solved in one call (``Context.solve_jobs``)
  system  one physical-system request from its mesh file to its results
          (``Gb300SystemBackend``), the mesh upload included
  field   the exterior field of retained boundary traces (``evaluate_bem_field``)

The mixed form's answers are single precision wherever a result leaves the
framework (``FrequencyResult``, the physical system's float32 quantities and the
float32 field are complex64), so the sweeps and jobs of that form hand them on as
complex64 too; the FP64 form's stay complex128.  Every frequency's pressure and
field is an output of its own.
"""

from __future__ import annotations

import functools
import importlib
import math
import os
import random
import shutil
import tempfile

import numpy as np
import torch

SOUND_SPEED = 343.0
RHO = 1.205


def _pkg(name: str):
    return importlib.import_module("boundary-lab_gb300." + name)


# ------------------------------------------------------------------- cases --


def _case(kind, mesh, faces, form, n_freq, f_lo, f_hi, n_points, n_rhs=1, symmetry="off", n_jobs=1):
    return dict(kind=kind, mesh=mesh, faces=faces, form=form, n_freq=n_freq, f_lo=f_lo, f_hi=f_hi, n_points=n_points,
                n_rhs=n_rhs, symmetry=symmetry, n_jobs=n_jobs)


def listed() -> list[dict]:
    cases = [
        # one frequency of a small enclosure: a designer moving a slider, latency counts
        ("one_1k", _case("sweep", "box", 1000, "mixed", 1, 1000.0, 1000.0, 146)),
        # the small job of the serving stream: 16 frequencies, polar arcs and a sphere
        ("sweep_1k", _case("sweep", "box", 1000, "mixed", 16, 100.0, 8000.0, 1146)),
        # four queued small jobs of similar size sharing their launches
        ("jobs_4x1k", _case("jobs", "box", 1100, "mixed", 8, 100.0, 8000.0, 1146, n_jobs=4)),
        # half model of a symmetric cabinet with two driven channels
        ("sweep_half_2k5", _case("sweep", "box", 2500, "mixed", 12, 100.0, 9000.0, 1000, n_rhs=2, symmetry="x")),
        # the batched sweep's box
        ("sweep_5k", _case("sweep", "box", 5000, "mixed", 32, 50.0, 10000.0, 2000)),
        # the headline box: one interactive frequency, and a call of the sweep (two lanes of 15)
        ("one_10k", _case("sweep", "box", 10000, "mixed", 1, 3000.0, 3000.0, 2146)),
        ("sweep_10k", _case("sweep", "box", 10000, "mixed", 30, 200.0, 12000.0, 2146)),
        # the large model: a horn in a box, a quarter of its 32-frequency sweep
        ("sweep_horn_20k", _case("sweep", "horn", 22300, "mixed", 8, 500.0, 16000.0, 5000)),
        # the plain FP64 form: the small sphere's sweep, and two frequencies of a cabinet
        ("fp64_sphere_1k", _case("sweep", "sphere", 1280, "fp64", 16, 100.0, 3000.0, 1000)),
        ("fp64_4k", _case("sweep", "box", 4000, "fp64", 2, 500.0, 2000.0, 1000)),
        # a whole request as the program's front end sends it, mesh file to results
        ("system_2k", _case("system", "box", 2000, "mixed", 16, 100.0, 8000.0, 1146)),
        # a balloon plot of a retained solution
        ("field_10k", _case("field", "box", 10000, "mixed", 1, 3000.0, 3000.0, 5000)),
    ]
    return [dict(name=name, **c) for name, c in cases]


def _log_int(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _seconds(case: dict) -> float:
    """A rough pass time, to keep drawn cases within the listed ones' cost."""
    return work(case)["flops"] / (1.2e11 if case["form"] == "fp64" else 5.0e13) + 2e-3


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["sweep", "sweep", "sweep", "sweep", "fp64", "jobs", "system", "field"])
    while True:
        form = "mixed"
        n_rhs = rng.choice([1, 1, 1, 2, 3, 4])
        symmetry = rng.choice(["off", "off", "off", "x", "xy"])
        n_points = _log_int(rng, 5, 5000)
        f_hi = rng.uniform(1500.0, 14000.0)
        f_lo = f_hi / rng.uniform(1.5, 60.0)
        n_jobs = 1
        mesh = "box"
        if kind == "sweep":
            mesh = rng.choice(["box", "box", "box", "sphere", "horn"])
            faces, n_freq = _log_int(rng, 150, 20000), _log_int(rng, 1, 32)
        elif kind == "fp64":
            form, faces, n_freq = "fp64", _log_int(rng, 150, 4500), _log_int(rng, 1, 16)
        elif kind == "jobs":
            n_jobs = rng.randint(2, 5)
            faces, n_freq, symmetry = _log_int(rng, 200, 3000), rng.randint(1, 6), "off"
        elif kind == "system":
            form = rng.choice(["mixed", "mixed", "mixed", "fp64"])
            faces, n_freq, n_rhs = _log_int(rng, 200, 1500 if form == "fp64" else 8000), _log_int(rng, 1, 24), 1
        else:
            form = rng.choice(["mixed", "mixed", "fp64"])
            faces, n_freq, n_rhs = _log_int(rng, 200, 20000), 1, 1
        if mesh != "box":
            symmetry = "off"
        if mesh == "horn":
            faces = max(faces, 2000)
        if mesh == "sphere":
            faces = min(faces, 6000)
        # at least four elements a wavelength, as a user's mesh has
        f_hi = min(f_hi, 343.0 / (4.0 * math.sqrt(2.0 * _AREA[mesh] / faces)) * (2.0 if symmetry == "off" else 1.0))
        f_lo = min(f_lo, f_hi / 1.2)
        if n_freq == 1:
            f_lo = f_hi
        case = _case("sweep" if kind == "fp64" else kind, mesh, faces, form, n_freq, round(f_lo, 2), round(f_hi, 2),
                     n_points, n_rhs, symmetry, n_jobs)
        limit = 0.45 if form == "fp64" else 0.25
        while _seconds(case) > limit and case["n_freq"] > 1:
            case["n_freq"] -= 1
            if case["n_freq"] == 1:
                case["f_lo"] = case["f_hi"]
        if _seconds(case) <= limit:
            return case


_AREA = {"box": 0.37, "sphere": 0.13, "horn": 1.45}  # m^2


# ------------------------------------------------------------------- inputs --


@functools.lru_cache(maxsize=32)
def _base_mesh(mesh: str, faces: int, symmetry: str):
    """(vertices, faces, radiating faces) of a case before the seed stretches it."""
    meshes = _pkg("meshes")
    if mesh == "sphere":
        if faces != 1280:
            v, f = meshes.cube_sphere(0.1, max(3, round(math.sqrt(faces / 12.0))))
            c = v[f].mean(axis=1)
            return v, f, c[:, 2] / np.linalg.norm(c, axis=1) > math.cos(math.radians(30.0))
        m = meshes.sphere_with_cap(0.1, 3, 30.0)
    elif mesh == "horn":
        m = meshes.horn_in_box(target_faces=faces)
    elif symmetry == "off":
        m = meshes.box_with_piston((0.3, 0.2, 0.25), faces, 0.05, "+z")
    else:
        # the part of the box at x >= 0 (and y >= 0), open on the symmetry planes
        half = np.array([0.15, 0.1 if symmetry == "xy" else 0.2, 0.25])
        m = meshes.box_with_piston(half, faces, 0.05, "+z")
        v = m.vertices + np.array([half[0] / 2, half[1] / 2 if symmetry == "xy" else 0.0, 0.0])
        v[np.abs(v) < 1e-12] = 0.0
        drop = (v[m.faces][:, :, 0] == 0.0).all(axis=1)
        if symmetry == "xy":
            drop |= (v[m.faces][:, :, 1] == 0.0).all(axis=1)
        f = m.faces[~drop]
        c = v[f].mean(axis=1)
        rad = (c[:, 2] > 0.125 - 1e-9) & (np.hypot(c[:, 0], c[:, 1]) < 0.05)
        used = np.unique(f)
        at = np.full(len(v), -1)
        at[used] = np.arange(len(used))
        return v[used], at[f].astype(np.int32), rad
    return m.vertices, m.faces, m.tags == meshes.RADIATOR_TAG


def _fibonacci(n: int, radius: float) -> np.ndarray:
    i = np.arange(n) + 0.5
    z = 1.0 - 2.0 * i / n
    a = math.pi * (1.0 + math.sqrt(5.0)) * i
    r = np.sqrt(1.0 - z * z)
    return radius * np.stack([r * np.cos(a), r * np.sin(a), z], axis=1)


def _inputs(case: dict, seed: int, job: int = 0) -> dict:
    """One job's arrays: the case's mesh stretched by a few per cent, unit drives, points, frequencies."""
    rng = np.random.default_rng([seed, job])
    faces = case["faces"] if case["n_jobs"] == 1 else int(case["faces"] * (0.85 + 0.1 * job))
    v, f, rad = _base_mesh(case["mesh"], faces, case["symmetry"])
    v = v * (1.0 + 0.03 * rng.uniform(-1.0, 1.0, 3))
    if case["kind"] == "system":  # a mesh file's and a float32 request's decimals
        v = np.round(v, 9)
    drives = np.zeros((case["n_rhs"], len(f)), np.complex128)
    drives[0, rad] = 1.0 if case["kind"] == "system" else complex(*rng.normal(size=2))
    c = v[f].mean(axis=1)
    for r in range(1, case["n_rhs"]):  # further channels: drivers elsewhere on the surface
        at = c[rng.integers(len(f))]
        drives[r, np.linalg.norm(c - at, axis=1) < 0.04] = complex(*rng.normal(size=2))
    freqs = np.geomspace(case["f_lo"], case["f_hi"], case["n_freq"]) * (1.0 + 0.01 * rng.uniform(-1.0, 1.0))
    if case["form"] == "mixed" and case["kind"] == "system":
        freqs = freqs.astype(np.float32).astype(np.float64)
    points = _fibonacci(case["n_points"], 2.0 + 0.1 * rng.uniform())
    return dict(vertices=v, faces=f, drives=drives, points=points, freqs=freqs)


def _traces(case: dict, seed: int, n_vertices: int, n_faces: int):
    """Boundary traces of a retained solution: smooth over the surface's numbering, single or double precision."""
    rng = np.random.default_rng([seed, 77])
    dtype = np.complex64 if case["form"] == "mixed" else np.complex128
    p = rng.normal(size=n_vertices) + 1j * rng.normal(size=n_vertices)
    q = 20.0 * (rng.normal(size=n_faces) + 1j * rng.normal(size=n_faces))
    return p.astype(dtype), q.astype(dtype)


# ------------------------------------------------------------------- states --


class _Sweep:
    def __init__(self, case, seed):
        x = _inputs(case, seed)
        self.dtype = np.complex64 if case["form"] == "mixed" else np.complex128
        self.freqs = x["freqs"]
        self.engine = _pkg("engine").CudaEngine(precision=case["form"])
        self.engine.prepare(x["vertices"], x["faces"], x["drives"], x["points"], symmetry=case["symmetry"])

    def run(self):
        r = self.engine.solve(self.freqs, SOUND_SPEED, RHO)
        p, u = r.pressure.astype(self.dtype, copy=False), r.field.astype(self.dtype, copy=False)
        return {"pressure": list(p), "field": list(u)}

    def __del__(self):
        if getattr(self, "engine", None) is not None:
            self.engine.close()


class _Jobs:
    def __init__(self, case, seed):
        native = _pkg("native")
        self.dtype = np.complex64 if case["form"] == "mixed" else np.complex128
        self.precision = native.BEM_PRECISION_MIXED if case["form"] == "mixed" else native.BEM_PRECISION_FP64
        self.ctx, _ = _pkg("engine").shared_context(0)
        self.jobs = []
        for j in range(case["n_jobs"]):
            x = _inputs(case, seed, j)
            m = self.ctx.upload_mesh(x["vertices"], x["faces"])
            m.set_excitation(x["drives"])
            m.set_observation_points(x["points"])
            self.jobs.append((m, x["freqs"]))

    def run(self):
        out, _ = self.ctx.solve_jobs(self.jobs, precision=self.precision, sound_speed=SOUND_SPEED, rho=RHO)
        return {"pressure": [list(p.astype(self.dtype, copy=False)) for p, _ in out],
                "field": [list(u.astype(self.dtype, copy=False)) for _, u in out]}

    def __del__(self):
        for m, _ in getattr(self, "jobs", []):
            m.release()


class _System:
    def __init__(self, case, seed):
        x = _inputs(case, seed)
        self.dir = tempfile.mkdtemp(prefix="bem_case_")
        path = os.path.join(self.dir, "mesh.msh")
        tags = np.where(x["drives"][0] != 0, 2, 1).astype(np.int32)
        _pkg("meshes").write_gmsh22(path, x["vertices"], x["faces"], tags)
        boundaries = [{"id": f"b:{name}", "name": name, "region_id": "air", "kind": "moving" if tag == 2 else "rigid",
                       "group": {"mesh_id": "m", "dimension": 2, "tag": tag, "name": None}, "parameters": {}}
                      for name, tag in (("wall", 1), ("driver", 2))]
        system = {
            "id": "s", "name": "cabinet", "contract_version": 1, "interfaces": [], "assumptions": [],
            "meshes": [{"id": "m", "name": "m", "file": path, "purpose": "bem_surface", "scale_to_m": 1.0,
                        "translation_m": [0.0, 0.0, 0.0]}],
            "regions": [{"id": "air", "name": "air", "kind": "unbounded_air", "mesh_ids": ["m"], "loss_model": {},
                         "sound_speed_m_per_s": SOUND_SPEED, "density_kg_per_m3": RHO}],
            "boundaries": boundaries,
            "components": [{"id": "c", "name": "driver", "kind": "ideal_velocity_source", "boundary_ids": ["b:driver"],
                            "parameters": {"boundary_motion_weights": {"b:driver": 1.0}}}],
            "excitation_ports": [{"id": "p", "name": "driver", "component_id": "c", "kind": "normal_velocity"}]}
        self.request = {
            "schema_version": 1, "compiled_system": system, "frequencies_hz": x["freqs"].tolist(),
            "excitation_port_ids": ["p"],
            "outputs": [{"id": "far", "quantity": "exterior_pressure", "options": {"points_m": x["points"].tolist()}},
                        {"id": "bem", "quantity": "bem_boundary_pressure"}],
            "solver_options": {"symmetry": case["symmetry"]}}
        self.backend = _pkg("system_exterior").Gb300SystemBackend(
            precision="float32" if case["form"] == "mixed" else "float64")

    def run(self):
        session = self.backend.create_system_session(self.request)
        out = {"pressure": [], "field": []}
        for result in session.solve_stream():
            values = {q.id: q.values for q in result.quantities}
            out["pressure"].append(values["bem"])
            out["field"].append(values["far"])
        return out

    def __del__(self):
        if getattr(self, "dir", None):
            shutil.rmtree(self.dir, ignore_errors=True)


class _Field:
    count = 0

    def __init__(self, case, seed):
        cf = _pkg("coupled_field")
        x = _inputs(case, seed)
        p, q = _traces(case, seed, len(x["vertices"]), len(x["faces"]))
        _Field.count += 1
        self.request = cf.BemFieldEvaluationRequest(
            domain_key=f"solution {_Field.count}", points_m=x["points"].astype(np.float32),
            boundary_points_m=x["vertices"].astype(np.float32), boundary_triangles=x["faces"].astype(np.int64),
            boundary_pressure=p, boundary_normal_derivative=q, frequency_hz=float(x["freqs"][0]),
            sound_speed_m_per_s=SOUND_SPEED, symmetry=case["symmetry"])
        self.evaluator = cf.FieldEvaluator()
        self.evaluate = cf.evaluate_bem_field
        self.run()  # the domain's upload, as the first request on a solution does

    def run(self):
        return {"field": self.evaluate(self.request, evaluator=self.evaluator)}

    def __del__(self):
        if getattr(self, "evaluator", None) is not None:
            self.evaluator.release()


def prepare(case: dict, seed: int):
    return {"sweep": _Sweep, "jobs": _Jobs, "system": _System, "field": _Field}[case["kind"]](case, seed)


def run(state):
    return state.run()


def work(case: dict) -> dict:
    """One Green's function and its weighting (20 flop) per quadrature pair, the LU and its
    solves, and one per source and point; inputs read once, answers written once."""
    n_bytes = flops = 0.0
    esz = 8 if case["form"] == "mixed" else 16
    for j in range(case["n_jobs"]):
        faces = case["faces"] if case["n_jobs"] == 1 else int(case["faces"] * (0.85 + 0.1 * j))
        v, f, _ = _base_mesh(case["mesh"], faces, case["symmetry"])
        nv, nf = float(len(v)), float(len(f))
        images = {"off": 1, "x": 2, "xy": 4}[case["symmetry"]]
        n_out = case["n_points"] * case["n_rhs"] * case["n_freq"]
        if case["kind"] == "field":
            flops += 20.0 * 3 * nf * images * case["n_points"]
            n_bytes += 12 * (nv + nf + case["n_points"]) + esz * (nv + nf + n_out)
            continue
        flops += case["n_freq"] * (20.0 * 36 * nf * nf * images + 8.0 / 3.0 * nv**3 + 8.0 * nv * nv * case["n_rhs"]
                                   + 20.0 * 6 * nf * images * case["n_points"] * case["n_rhs"])
        n_bytes += 24 * nv + 12 * nf + 24 * case["n_points"] + 16 * case["n_rhs"] * nf
        n_bytes += esz * (n_out + nv * case["n_rhs"] * case["n_freq"])
    return {"bytes": n_bytes, "flops": flops}


# ---------------------------------------------------------- 64-bit answers --
# The Galerkin P1 / DP0 Burton-Miller discretisation (six-point or three-point rule on
# pairs that share no vertex, Duffy rules of order 4 on those that do) in torch float64:
# (M/2 - D + (i/k) H) p = -(S + (i/k)(K' + M10/2)) q, then u = D p - S q off the surface.

_RULES = {
    6: ([[0.4459484909159651, 0.4459484909159651], [0.0915762135097710, 0.0915762135097700],
         [0.1081030181680700, 0.4459484909159651], [0.4459484909159651, 0.1081030181680700],
         [0.8168475729804590, 0.0915762135097700], [0.0915762135097710, 0.8168475729804580]],
        [0.5 * w for w in (0.2233815896780110, 0.1099517436553220, 0.2233815896780110, 0.2233815896780110,
                           0.1099517436553220, 0.1099517436553220)]),
    3: ([[1 / 6, 1 / 6], [2 / 3, 1 / 6], [1 / 6, 2 / 3]], [1 / 6, 1 / 6, 1 / 6]),
}


def _basis(p: np.ndarray) -> np.ndarray:
    return np.stack([1.0 - p[:, 0] - p[:, 1], p[:, 0], p[:, 1]], axis=1)


def _duffy(kind: int, order: int = 4):
    """(test points, trial points, weights) for coincident (1), edge (2) and vertex (3) pairs."""
    x, w = np.polynomial.legendre.leggauss(order)
    x, w = 0.5 * (x + 1.0), 0.5 * w
    # (xsi, eta1) from the test rule, (eta2, eta3) from the trial rule
    e1, s, e3, e2 = (g.ravel() for g in np.meshgrid(x, x, x, x, indexing="ij"))
    ww = np.einsum("i,j,k,l->ijkl", w, w, w, w).ravel()
    if kind == 1:
        base = ww * s**3 * e1**2 * e2
        maps = [(s, s * (1 - e1 + e1 * e2), s * (1 - e1 * e2 * e3), s * (1 - e1), 1),
                (s * (1 - e1 * e2 * e3), s * (1 - e1), s, s * (1 - e1 + e1 * e2), 1),
                (s, s * (e1 - e1 * e2 + e1 * e2 * e3), s * (1 - e1 * e2), s * (e1 - e1 * e2), 1),
                (s * (1 - e1 * e2), s * (e1 - e1 * e2), s, s * (e1 - e1 * e2 + e1 * e2 * e3), 1),
                (s * (1 - e1 * e2 * e3), s * (e1 - e1 * e2 * e3), s, s * (e1 - e1 * e2), 1),
                (s, s * (e1 - e1 * e2), s * (1 - e1 * e2 * e3), s * (e1 - e1 * e2 * e3), 1)]
    elif kind == 2:
        base = ww * s**3 * e1**2
        maps = [(s, s * e1 * e3, s * (1 - e1 * e2), s * e1 * (1 - e2), 1),
                (s, s * e1, s * (1 - e1 * e2 * e3), s * e1 * e2 * (1 - e3), e2),
                (s * (1 - e1 * e2), s * e1 * (1 - e2), s, s * e1 * e2 * e3, e2),
                (s * (1 - e1 * e2 * e3), s * e1 * e2 * (1 - e3), s, s * e1, e2),
                (s * (1 - e1 * e2 * e3), s * e1 * (1 - e2 * e3), s, s * e1 * e2, e2)]
    else:
        base = ww * s**3 * e2
        maps = [(s, s * e1, s * e2, s * e2 * e3, 1), (s * e2, s * e2 * e3, s, s * e1, 1)]
    test = np.concatenate([np.stack([a - b, b], axis=1) for a, b, _, _, _ in maps])
    trial = np.concatenate([np.stack([c - d, d], axis=1) for _, _, c, d, _ in maps])
    return test, trial, np.concatenate([base * m for *_, m in maps])


def _remap(p: np.ndarray, kind: int, a: int, b: int) -> np.ndarray:
    """A Duffy rule's points turned so that its singular vertex (edge) is local vertex a (edge a-b)."""
    if kind == 3:
        third = 1.0 - p[:, 0] - p[:, 1]
        return {0: p, 1: np.stack([third, p[:, 1]], 1), 2: np.stack([p[:, 0], third], 1)}[a]
    if kind == 2:
        ref = np.array([[0.0, 0.0], [1.0, 0.0], [0.0, 1.0]])
        v0, v1, v2 = ref[a], ref[b], ref[3 - a - b]
        return v0 + p[:, :1] * (v1 - v0) + p[:, 1:] * (v2 - v0)
    return p


class _Exact:
    IMAGES = {"off": [(1, 1)], "x": [(1, 1), (-1, 1)], "xy": [(1, 1), (-1, 1), (1, -1), (-1, -1)]}

    def __init__(self, x: dict, symmetry: str, points_per_face: int):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.f_np = np.asarray(x["faces"], np.int64)
        self.v_np = np.asarray(x["vertices"], np.float64)
        self.sym = symmetry
        t = self.t
        self.v, self.f = t(self.v_np), torch.as_tensor(self.f_np, device=self.dev)
        self.nv, self.nf = len(self.v_np), len(self.f_np)
        pts, w = _RULES[points_per_face]
        self.phi, self.w = t(_basis(np.array(pts))), t(np.array(w))  # [Q, 3], [Q]
        tri = self.v[self.f]
        e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
        n = torch.linalg.cross(e1, e2)
        self.area2 = torch.linalg.norm(n, dim=1)
        self.n = n / self.area2[:, None]
        # surface curls n x grad phi_a: the opposite edges over twice the area
        opp = torch.stack([tri[:, 2] - tri[:, 1], tri[:, 0] - tri[:, 2], tri[:, 1] - tri[:, 0]], dim=1)
        self.curl = opp / self.area2[:, None, None]
        self.tri = tri
        self.q_pts = torch.einsum("qa,fad->fqd", self.phi, tri)  # [nf, Q, 3]
        self.points = t(x["points"])

    def t(self, a):
        return torch.as_tensor(np.asarray(a, np.float64), device=self.dev)

    def _image(self, s):
        """Trial data of the image (sx, sy): signs, normals, curls, quadrature points, vertices on its planes."""
        sx, sy = s
        d = self.t([sx, sy, 1.0])
        on = np.ones(self.nv, bool)
        if sx < 0:
            on &= self.v_np[:, 0] == 0.0
        if sy < 0:
            on &= self.v_np[:, 1] == 0.0
        return d, self.n * d, self.curl * d * (sx * sy), self.q_pts * d, on

    @staticmethod
    def _green(r2, k):
        rinv = torch.rsqrt(r2)
        z = k * r2 * rinv
        g = rinv / (4.0 * math.pi)
        return torch.complex(torch.cos(z) * g, torch.sin(z) * g), rinv

    def _touching(self, on):
        """(test, trial, local test vertices, local trial vertices) of the pairs that share a vertex in `on`."""
        by_vertex = [[] for _ in range(self.nv)]
        for g, face in enumerate(self.f_np):
            for b, v in enumerate(face):
                if on[v]:
                    by_vertex[v].append((g, b))
        groups: dict = {}
        for i, face in enumerate(self.f_np):
            shared: dict = {}
            for a, v in enumerate(face):
                for g, b in by_vertex[v]:
                    shared.setdefault(g, []).append((a, b))
            for g, ab in shared.items():
                if len(ab) == 3:
                    key = (1, 0, 0, 0, 0)
                elif len(ab) == 2:
                    (a0, b0), (a1, b1) = sorted(ab, key=lambda p: p[1])
                    key = (2, a0, a1, b0, b1)
                else:
                    key = (3, ab[0][0], 0, ab[0][1], 0)
                groups.setdefault(key, []).append((i, g))
        return {k: torch.as_tensor(np.array(v), device=self.dev) for k, v in groups.items()}

    def solve(self, k: float, q: np.ndarray):
        """(pressure [n_rhs, nv], field [n_rhs, n_points]) for Neumann data q [n_rhs, nf]."""
        c128 = torch.complex128
        qd = torch.as_tensor(q, device=self.dev, dtype=c128)
        driven = torch.nonzero((qd != 0).any(dim=0)).ravel()
        Q, nv, nf = len(self.w), self.nv, self.nf
        A = torch.zeros((nv, nv), dtype=c128, device=self.dev)
        b = torch.zeros((nv, qd.shape[0]), dtype=c128, device=self.dev)
        eta = 1j / k
        mass = torch.einsum("q,qa,qb->ab", self.w, self.phi, self.phi)
        m10 = torch.einsum("q,qa->a", self.w, self.phi)
        local = 0.5 * self.area2[:, None, None] * mass
        A.view(-1).index_add_(0, (self.f[:, :, None] * nv + self.f[:, None, :]).reshape(-1), local.reshape(-1).to(c128))
        lb = -eta * 0.5 * torch.einsum("f,a,rf->far", self.area2.to(c128), m10.to(c128), qd)
        b.index_add_(0, self.f.reshape(-1), lb.reshape(-1, qd.shape[0]))
        cw = (self.phi * self.w[:, None]).to(c128)  # [Q, 3]
        step = max(1, int(2.5e7 // (nf * Q)))
        for s in self.IMAGES[self.sym]:
            d, ng, cg, yq, on = self._image(s)
            live = torch.as_tensor(on, device=self.dev)
            for f0 in range(0, nf, step):
                fs = slice(f0, min(nf, f0 + step))
                ff = self.f[fs]
                far = torch.ones((len(ff), nf), dtype=torch.bool, device=self.dev)
                for a in range(3):
                    for c in range(3):
                        far &= ~((ff[:, a, None] == self.f[None, :, c]) & live[ff[:, a], None])
                jac = self.area2[fs, None] * self.area2[None, :] * far
                nn = self.n[fs] @ ng.T
                L = torch.zeros((len(ff), 3, nf, 3), dtype=c128, device=self.dev)
                S0 = torch.zeros((len(ff), nf), dtype=c128, device=self.dev)
                for m in range(Q):
                    x = self.q_pts[fs, m]
                    r2 = rn = 0.0
                    for dim in range(3):
                        dr = yq[None, :, :, dim] - x[:, None, None, dim]
                        r2 = r2 + dr * dr
                        rn = rn + dr * ng[None, :, None, dim]
                    r2 = torch.where(far[:, :, None], r2, torch.ones_like(r2))
                    g, rinv = self._green(r2, k)
                    S0 += self.w[m] * (g @ self.w.to(c128))
                    # -(dG/dn_y) - i k (n_x . n_y) G
                    e = -g * torch.complex(-rn * rinv * rinv, k * (rn * rinv + nn[:, :, None]))
                    hs = e @ cw  # [c, nf, 3]
                    for a in range(3):
                        L[:, a] += cw[m, a] * hs
                    del g, e, hs, r2, rn, rinv
                cc = torch.einsum("cad,gbd->cagb", self.curl[fs], cg)
                L = jac[:, None, :, None] * (L + eta * cc * S0[:, None, :, None])
                rows = torch.zeros((len(ff) * 3, nv), dtype=c128, device=self.dev)
                rows.index_add_(1, self.f.reshape(-1), L.reshape(len(ff) * 3, nf * 3))
                A.index_add_(0, ff.reshape(-1), rows)
                del L, rows, cc, S0
                # right-hand side, driven faces only
                dr = yq[driven][None, None] - self.q_pts[fs][:, :, None, None]  # [c, Q, g, Q, 3]
                r2 = torch.where(far[:, driven][:, None, :, None], (dr * dr).sum(-1), torch.ones(1, device=self.dev,
                                                                                                 dtype=torch.float64))
                g, rinv = self._green(r2, k)
                tx = -(dr * self.n[fs][:, None, None, None]).sum(-1) * rinv
                op = g * (1.0 + eta * torch.complex(-rinv, torch.full_like(rinv, k)) * tx)
                op = torch.einsum("cmgn,n,ma->cag", op, self.w.to(c128), cw) * jac[:, None, driven]
                lb = -torch.einsum("cag,rg->car", op, qd[:, driven])
                b.index_add_(0, ff.reshape(-1), lb.reshape(-1, qd.shape[0]))
                del dr, r2, g, rinv, tx, op
            for (kind, a0, a1, b0, b1), pairs in self._touching(on).items():
                test, trial, w = _duffy(kind)
                pt = self.t(_basis(_remap(test, kind, a0, a1)))
                pr = self.t(_basis(_remap(trial, kind, b0, b1)))
                w = self.t(w)
                for p0 in range(0, len(pairs), max(1, 6000000 // len(w))):
                    pp = pairs[p0:p0 + max(1, 6000000 // len(w))]
                    ti, gi = pp[:, 0], pp[:, 1]
                    dr = torch.einsum("qa,pad->pqd", pr, self.tri[gi] * d) - torch.einsum("qa,pad->pqd", pt, self.tri[ti])
                    g, rinv = self._green((dr * dr).sum(-1), k)
                    g = g * w * (self.area2[ti] * self.area2[gi])[:, None]
                    ty = torch.einsum("pqd,pd->pq", dr, ng[gi]) * rinv
                    tx = -torch.einsum("pqd,pd->pq", dr, self.n[ti]) * rinv
                    nn = (self.n[ti] * ng[gi]).sum(-1)
                    e = -g * torch.complex(-ty * rinv, k * (ty + nn[:, None]))
                    cc = torch.einsum("pad,pbd->pab", self.curl[ti], cg[gi])
                    loc = torch.einsum("pq,qa,qb->pab", e, pt.to(c128), pr.to(c128)) + eta * cc * g.sum(1)[:, None, None]
                    A.view(-1).index_add_(0, (self.f[ti][:, :, None] * nv + self.f[gi][:, None, :]).reshape(-1),
                                          loc.reshape(-1))
                    op = g * (1.0 + eta * torch.complex(-rinv, torch.full_like(rinv, k)) * tx)
                    lb = -torch.einsum("pq,qa,rp->par", op, pt.to(c128), qd[:, gi])
                    b.index_add_(0, self.f[ti].reshape(-1), lb.reshape(-1, qd.shape[0]))
        p = torch.linalg.solve(A, b).T.contiguous()
        return p, self.field(k, p, qd)

    def field(self, k: float, p, qd):
        c128 = torch.complex128
        Q = len(self.w)
        pq = torch.einsum("qa,rfa->rfq", self.phi.to(c128), p[:, self.f])  # boundary pressure at the sources
        weight = (self.area2[:, None] * self.w).to(c128)
        out = torch.zeros((p.shape[0], len(self.points)), dtype=c128, device=self.dev)
        step = max(1, int(3e7 // (self.nf * Q)))
        for s in self.IMAGES[self.sym]:
            _, ng, _, yq, _ = self._image(s)
            for i in range(0, len(self.points), step):
                dr = yq[None] - self.points[i:i + step, None, None]
                g, rinv = self._green((dr * dr).sum(-1), k)
                t = (dr * ng[None, :, None]).sum(-1) * rinv
                dn = g * torch.complex(-t * rinv, k * t)
                out[:, i:i + step] += (torch.einsum("pfq,rfq->rp", dn, pq * weight)
                                       - torch.einsum("pfq,rfq->rp", g, qd[:, :, None] * weight))
        return out


def exact(case: dict, seed: int):
    """64-bit answers of as many of the case's frequencies as stay within some seconds."""
    if case["kind"] == "field":
        x = _inputs(case, seed)
        p, q = _traces(case, seed, len(x["vertices"]), len(x["faces"]))
        real = np.float32 if case["form"] == "mixed" else np.float64
        k = float(real(2 * np.pi) * real(x["freqs"][0]) / real(SOUND_SPEED))  # the request's own precision
        x["vertices"], x["points"] = x["vertices"].astype(np.float32), x["points"].astype(np.float32)
        ex = _Exact(x, case["symmetry"], 3)
        u = ex.field(k, torch.as_tensor(p.astype(np.complex128), device=ex.dev)[None],
                     torch.as_tensor(q.astype(np.complex128), device=ex.dev)[None])
        return {"field": u[0].cpu().numpy()}
    out = []
    images = {"off": 1, "x": 2, "xy": 4}[case["symmetry"]]
    for j in range(case["n_jobs"]):
        x = _inputs(case, seed, j)
        n = case["n_freq"]
        some = max(1, min(n, int(4e8 / (images * len(x["faces"]) ** 2 * case["n_jobs"]))))
        at = set(np.linspace(0, n - 1, some).round().astype(int).tolist()) if some > 1 else {n // 2}
        rho, c = RHO, SOUND_SPEED
        if case["kind"] == "system" and case["form"] == "mixed":
            rho, c = float(np.float32(rho)), float(np.float32(c))
        ex = _Exact(x, case["symmetry"], 6)
        pressure, field = [None] * n, [None] * n
        for i in sorted(at):
            omega = 2.0 * np.pi * x["freqs"][i]
            p, u = ex.solve(omega / c, 1j * rho * omega * x["drives"])
            pressure[i], field[i] = p.cpu().numpy(), u.cpu().numpy()
        out.append((pressure, field))
    if case["kind"] == "jobs":
        return {"pressure": [p for p, _ in out], "field": [u for _, u in out]}
    return {"pressure": out[0][0], "field": out[0][1]}
