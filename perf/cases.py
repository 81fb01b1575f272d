"""Performance cases of the dense Helmholtz BEM path: what a program that uses this package has the GPU do.

Every case goes through a public entry point: the batched session call that ``solve`` makes
(``NativeSession.assemble_solve_evaluate_standard_neumann_batch``, ``coupled_ib_batch``), the graph-captured
batches of many meshes (``BatchedSweeps``) and the shape gradients (``boundary_field``).  The meshes are the
package's generators: pulsating spheres and round exponential horns as quarter (yz+xz planes), half (yz plane)
or full surfaces.

A case's ``edge`` (metres, or the icosphere ``level``) sets the mesh size, ``shape`` its flare and lip.  The
``seed`` of :func:`prepare` scales the geometry, shifts the frequency grid and draws the velocity of every
driven face, so another seed is another problem on the same mesh topology.

:func:`exact` restates the discretisation in 64 bits with torch: six-point triangle rule, mirror images,
Duffy rules for touching triangles, dense solve, exterior field.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import hornlab_metal_bem_b200 as hb
from hornlab_metal_bem_b200 import generators
from hornlab_metal_bem_b200.adjoint import ShapeProblem, boundary_field, directivity_points
from hornlab_metal_bem_b200.batch import BatchedSweeps, SweepCase
from hornlab_metal_bem_b200.geometry import build_geometry_buffers
from hornlab_metal_bem_b200.mesh import make_pure_function_spaces, mesh_from_arrays
from hornlab_metal_bem_b200.native import NativeSession

SPEED_OF_SOUND = 343.0
AIR_DENSITY = 1.2041
THROAT, WALL, APERTURE = 2, 1, 12
PLANES = {"quarter": "yz+xz", "half": "yz", "full": None, "sphere": None, "baffled": None}
IMAGES = {"quarter": 4, "half": 2, "full": 1, "sphere": 1, "baffled": 1}


def listed():
    base = {"kind": "sweep", "shape": 0, "f_lo": 500.0, "f_hi": 20000.0, "points": 111, "sources": 1,
            "precision": "plain", "dense": "float32", "robin": False, "complex_k": False}
    return [
        # one frequency on a small closed body: the least a caller can ask for (latency and launches)
        dict(base, name="sphere162_1f", mesh="sphere", level=2, freqs=1, f_lo=1000.0, f_hi=1000.0, points=37),
        # the pulsating sphere that validates a set-up: 642 dofs, a short sweep
        dict(base, name="sphere642_8f", mesh="sphere", level=3, freqs=8, f_lo=200.0, f_hi=5000.0, points=37),
        # a streaming sweep of a production-size quarter horn hands over one frequency per call
        dict(base, name="quarter1043_1f", mesh="quarter", edge=0.007, freqs=1, f_lo=8000.0, f_hi=8000.0),
        # the headline sweep: quarter horn, 40 frequencies, three planes of 37 angles
        dict(base, name="quarter1043_40f", mesh="quarter", edge=0.007, freqs=40),
        # four drivers (velocity sources) sharing each frequency's matrix
        dict(base, name="quarter_4sources", mesh="quarter", edge=0.009, freqs=24, sources=4, shape=1),
        # lossy walls at complex wavenumbers on an odd-sized small mesh
        dict(base, name="quarter_robin_complexk", mesh="quarter", edge=0.0111, freqs=13, shape=2, f_hi=12000.0,
             robin=True, complex_k=True),
        # a balloon: few frequencies, thousands of observation points
        dict(base, name="half_balloon", mesh="half", edge=0.011, freqs=9, shape=3, f_hi=10000.0, points=2562),
        # the larger half horns of a design study, full band
        dict(base, name="half2k_40f", mesh="half", edge=0.0071, freqs=40, shape=4),
        # a full horn without symmetry in mixed precision
        dict(base, name="full4k_mixed", mesh="full", edge=0.0068, freqs=6, shape=5, f_lo=1000.0, precision="mixed"),
        # horn in an infinite baffle: coupled interior and half-space system
        dict(base, name="baffled_coupled", kind="coupled", mesh="baffled", edge=0.0085, freqs=6, shape=0, f_lo=1000.0,
             f_hi=10000.0),
        # one step of a shape optimisation: field and its gradient with respect to every vertex
        dict(base, name="shape_gradient", kind="gradient", mesh="full", edge=0.0095, freqs=20, f_lo=2000.0,
             f_hi=16000.0, points=13),
        # several variants of one design, captured once and swept concurrently
        dict(base, name="batch4_half", kind="batch", mesh="half", edge=0.0095, freqs=20, shape=7, meshes=4),
    ]


def draw(rng):
    base = {"shape": rng.randrange(1000), "sources": 1, "precision": "plain", "dense": "float32", "robin": False,
            "complex_k": False}
    kind = rng.choices(["sweep", "coupled", "gradient", "batch"], [8, 1, 1, 1])[0]
    f_lo = rng.uniform(200.0, 2000.0)
    case = dict(base, kind=kind, f_lo=f_lo, f_hi=rng.uniform(4000.0, 20000.0), points=rng.choice([37, 73, 111, 185]))
    if kind == "sweep":
        mesh = rng.choices(["sphere", "quarter", "half", "full"], [1, 4, 3, 2])[0]
        case["mesh"] = mesh
        if mesh == "sphere":
            case["level"] = rng.choice([1, 2, 3])
            case["f_hi"] = rng.uniform(2500.0, 6000.0)
        else:
            case["edge"] = {"quarter": 0.0060, "half": 0.0071, "full": 0.0075}[mesh] * math.exp(rng.uniform(0.0, 0.9))
        option = rng.choices(["none", "sources", "lossy", "mixed", "float64", "balloon"], [6, 1, 1, 1, 1, 1])[0]
        if option == "sources":
            case["sources"] = rng.randint(2, 6)
        elif option == "lossy":
            case["robin"], case["complex_k"] = rng.random() < 0.7, rng.random() < 0.7
        elif option == "mixed":
            case["precision"] = "mixed"
        elif option == "float64":
            case["dense"] = "float64"
        elif option == "balloon":
            case["points"] = rng.randint(500, 3000)
        case["freqs"] = int(round(math.exp(rng.uniform(0.0, math.log(40.99)))))
        if option == "float64":
            case["freqs"] = min(case["freqs"], 3)
            if mesh != "sphere":
                case["edge"] = max(case["edge"], {"quarter": 0.009, "half": 0.0125, "full": 0.016}[mesh])
        if mesh == "full":
            case["freqs"] = min(case["freqs"], 12)
    elif kind == "coupled":
        case.update(mesh="baffled", edge=rng.uniform(0.0088, 0.016), freqs=rng.randint(1, 6),
                    f_hi=rng.uniform(4000.0, 10000.0))
    elif kind == "gradient":
        case.update(mesh="full", edge=rng.uniform(0.0098, 0.018), freqs=rng.randint(3, 20), points=13)
    else:
        case.update(mesh="half", edge=rng.uniform(0.0098, 0.016), freqs=rng.randint(4, 20),
                    meshes=rng.randint(2, 4))
    if case["freqs"] == 1:
        case["f_lo"] = case["f_hi"]
    return case


# --------------------------------------------------------------------------- inputs
def _mesh(case, rng, shape):
    if case["mesh"] == "sphere":
        mesh = generators.icosphere(case["level"], 0.1)
    else:
        spec = generators.horn_spec_from_seed(shape, edge=case["edge"])
        mesh = (generators.baffled_horn(spec, aperture_tag=APERTURE) if case["mesh"] == "baffled" else
                generators.horn(spec, quarter=case["mesh"] == "quarter", half=case["mesh"] == "half"))
    v = np.asarray(mesh.grid.vertices, dtype=np.float64).T * rng.uniform(0.97, 1.03)
    return mesh_from_arrays(v, np.asarray(mesh.grid.elements).T, np.asarray(mesh.physical_tags))


def _points(case, mesh, rng):
    """Observation points (3, N): arcs about the mouth, or a Fibonacci balloon for large counts."""
    n = case["points"]
    z0 = float(np.max(np.asarray(mesh.grid.vertices)[2])) if case["mesh"] != "sphere" else 0.0
    r = rng.uniform(1.9, 2.1)
    if n > 300:
        i = np.arange(n) + 0.5
        th, ph = np.arccos(1.0 - 2.0 * i / n), np.pi * (1.0 + 5.0 ** 0.5) * i
    else:
        per = 37 if n % 37 == 0 else n
        planes = max(1, n // per)
        top = 0.5 * np.pi if case["mesh"] == "baffled" else np.pi
        th = np.tile(np.linspace(0.0, top, per), planes)
        ph = np.repeat(np.arange(planes) * np.pi / 4.0, per)
    p = np.stack([r * np.sin(th) * np.cos(ph), r * np.sin(th) * np.sin(ph), z0 + r * np.cos(th)])
    return np.ascontiguousarray(p, dtype=np.float32)


def _inputs(case, seed, member=0):
    rng = np.random.default_rng([int(seed), member])
    mesh = _mesh(case, rng, case["shape"] + member)
    p1, dp0 = make_pure_function_spaces(mesh.grid)
    buf = build_geometry_buffers(mesh.grid, mesh.physical_tags, p1, dp0)
    freqs = np.geomspace(case["f_lo"], case["f_hi"], case["freqs"]) * rng.uniform(0.98, 1.02)
    k = (2.0 * np.pi * freqs / SPEED_OF_SOUND).astype(np.float32)
    k_im = (0.01 * k).astype(np.float32) if case["complex_k"] else np.zeros_like(k)
    tags = np.asarray(buf.physical_tags_i32)
    driven = np.flatnonzero(tags == THROAT)
    q = np.zeros((case["sources"], len(k), buf.n_triangles), np.complex64)
    for s in range(case["sources"]):
        # a diaphragm in motion: mean velocity one, some breakup from face to face
        v = 1.0 + 0.2 * (rng.standard_normal(driven.size) + 1j * rng.standard_normal(driven.size))
        q[s][:, driven] = (1j * 2.0 * np.pi * freqs * AIR_DENSITY)[:, None] * v[None, :]
    beta = {WALL: complex(rng.uniform(0.02, 0.08), rng.uniform(-0.05, 0.05))} if case["robin"] else None
    obs = _points(case, mesh, rng) if case["kind"] != "gradient" else directivity_points(
        float(np.max(np.asarray(mesh.grid.vertices)[2])), np.linspace(10.0, 60.0, (case["points"] - 1) // 2)
    ).astype(np.float32)
    weights = None
    if case["kind"] == "gradient":
        shape = (len(k), obs.shape[1])
        weights = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    return {"mesh": mesh, "buf": buf, "freqs": freqs, "k": k, "k_im": k_im, "q": q, "beta": beta, "obs": obs,
            "weights": weights}


def prepare(case, seed):
    plane = PLANES[case["mesh"]]
    state = {"case": case}
    if case["kind"] == "batch":
        members = [_inputs(case, seed, m) for m in range(case["meshes"])]
        state["batch"] = BatchedSweeps(
            [SweepCase(i["buf"], i["k"], i["q"][0], i["obs"], [THROAT], plane) for i in members], n_streams=4,
            tuning=None, write_surface_pressure=True)
        return state
    i = _inputs(case, seed)
    state.update(i)
    if case["kind"] == "gradient":
        state["problem"] = ShapeProblem(i["buf"], i["k"], i["q"][0], i["obs"])
        v = np.asarray(i["buf"].vertices_3xn_f32, dtype=np.float64).T.copy()
        state["vertices"] = torch.from_numpy(v)
        state["weights"] = torch.from_numpy(i["weights"]).cuda()
    elif case["kind"] == "coupled":
        state["session"] = NativeSession(i["buf"], aperture_tag=APERTURE, velocity_source_tags=[THROAT])
    else:
        state["session"] = NativeSession(i["buf"], symmetry_plane=plane, check_open_edges=False)
    return state


# --------------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].run()
        return [{"field": o.field, "surface": o.surface_pressure, "impedance": o.tag_average.astype(np.complex64)}
                for o in state["batch"].outputs()]
    if case["kind"] == "gradient":
        v = state["vertices"].clone().requires_grad_(True)
        field = boundary_field(v, state["problem"])
        field.backward(state["weights"])
        # double accumulation of single-precision terms: a single-precision result
        return {"field": field.detach(), "gradient": v.grad.float()}
    kw = dict(k_imag_f32=state["k_im"], source_tags=[THROAT], impedance_source_tag=THROAT,
              write_surface_pressure=True, precision=case["precision"])
    if case["kind"] == "coupled":
        res = state["session"].coupled_ib_batch(state["freqs"], state["k"], state["q"][0], state["obs"], **kw)
        out = _stacked(res)
        out["aperture"] = np.stack([r.diagnostics["aperture_neumann"] for r in res])
        return out
    if state["beta"] is not None:
        kw["impedance_sources"] = state["beta"]
    if case["sources"] > 1:
        kw.update(extra_neumann_dp0=state["q"][1:], extra_impedance_source_tags=[THROAT] * (case["sources"] - 1))
    res = state["session"].assemble_solve_evaluate_standard_neumann_batch(
        state["freqs"], state["k"], state["q"][0], state["obs"], dense_solve_dtype=case["dense"], **kw)
    out = _stacked(res)
    if case["sources"] > 1:
        out["extra"] = [_stacked([r.extra_sources[s] for r in res]) for s in range(case["sources"] - 1)]
    return out


def _stacked(results):
    return {"field": np.stack([r.field for r in results]), "surface": np.stack([r.surface_pressure for r in results]),
            "impedance": np.array([r.impedance for r in results], np.complex64)}


def work(case):
    """Unavoidable work of one pass.  Assembly: 30 flops a kernel sample, each unordered pair of points once;
    LU 8/3 n^3; field 40 flops a sample (the gradient twice all of it).  Bytes: inputs, and the outputs."""
    total = {"bytes": 0.0, "flops": 0.0}
    for m in range(case.get("meshes", 1)):
        rng = np.random.default_rng(0)
        mesh = _mesh(case, rng, case["shape"] + m)
        n, T = np.asarray(mesh.grid.vertices).shape[1], np.asarray(mesh.grid.elements).shape[1]
        F, S, N, M = case["freqs"], case["sources"], case["points"], IMAGES[case["mesh"]]
        ap = int(np.sum(np.asarray(mesh.physical_tags) == APERTURE)) if case["mesh"] == "baffled" else 0
        order = n + ap
        lu = 8.0 / 3.0 * order ** 3 + 8.0 * order * order * S
        flops = F * (30.0 * 18.0 * T * T * M + lu + 40.0 * 6.0 * T * M * N * S)
        total["flops"] += (2.0 if case["kind"] == "gradient" else 1.0) * flops
        total["bytes"] += 12.0 * n + 24.0 * T + F * S * (8.0 * T + 8.0 * n + 8.0 * N) + 12.0 * N
    return total


# --------------------------------------------------------------------------- the discretisation in 64 bits
_X = np.array([0.4459484909159651, 0.0915762135097710, 0.1081030181680700,
               0.4459484909159651, 0.8168475729804590, 0.0915762135097710])
_Y = np.array([0.4459484909159651, 0.0915762135097700, 0.4459484909159651,
               0.1081030181680700, 0.0915762135097700, 0.8168475729804580])
_W = 0.5 * np.array([0.2233815896780110, 0.1099517436553220, 0.2233815896780110,
                     0.2233815896780110, 0.1099517436553220, 0.1099517436553220])
MASKS = {"quarter": [0, 1, 2, 3], "half": [0, 1], "full": [0], "sphere": [0], "baffled": [0]}


def _sign(mask, dev):
    return torch.tensor([-1.0 if mask >> c & 1 else 1.0 for c in range(3)], dtype=torch.float64, device=dev)


def _kernels(d, n, k, ki):
    """G and dG/dn_y of differences d = y - x (..., 3), both without the factor 1/(4 pi), zero at r = 0."""
    r2 = (d * d).sum(-1)
    inv = torch.where(r2 > 0, r2.clamp_min(1e-300).rsqrt(), torch.zeros_like(r2))
    r = r2 * inv
    G = torch.polar(torch.exp(-ki * r) * inv, k * r)
    D = G * torch.complex(-inv - ki, torch.full_like(inv, k)) * ((d * n).sum(-1) * inv)
    return G, D


def _duffy_rule(kind):
    x, w = np.polynomial.legendre.leggauss(4)
    x, w = 0.5 * (x + 1.0), 0.5 * w
    e1, xi, e2, e3 = (a.reshape(-1) for a in np.meshgrid(x, x, x, x, indexing="ij"))
    base = np.prod([a.reshape(-1) for a in np.meshgrid(w, w, w, w, indexing="ij")], axis=0) * xi ** 3
    e12, e123 = e1 * e2, e1 * e2 * e3
    if kind == 1:
        w = base * e1 ** 2 * e2
        parts = [(xi, xi * (1 - e1 + e12), xi * (1 - e123), xi * (1 - e1), w),
                 (xi * (1 - e123), xi * (1 - e1), xi, xi * (1 - e1 + e12), w),
                 (xi, xi * (e1 - e12 + e123), xi * (1 - e12), xi * (e1 - e12), w),
                 (xi * (1 - e12), xi * (e1 - e12), xi, xi * (e1 - e12 + e123), w),
                 (xi * (1 - e123), xi * (e1 - e123), xi, xi * (e1 - e12), w),
                 (xi, xi * (e1 - e12), xi * (1 - e123), xi * (e1 - e123), w)]
    elif kind == 2:
        w = base * e1 ** 2
        parts = [(xi, xi * e1 * e3, xi * (1 - e12), xi * e1 * (1 - e2), w),
                 (xi, xi * e1, xi * (1 - e123), xi * e12 * (1 - e3), w * e2),
                 (xi * (1 - e12), xi * e1 * (1 - e2), xi, xi * e123, w * e2),
                 (xi * (1 - e123), xi * e12 * (1 - e3), xi, xi * e1, w * e2),
                 (xi * (1 - e123), xi * e1 * (1 - e2 * e3), xi, xi * e12, w * e2)]
    else:
        w = base * e2
        parts = [(xi, xi * e1, xi * e2, xi * e2 * e3, w), (xi * e2, xi * e2 * e3, xi, xi * e1, w)]
    t1, t2, s1, s2, w = (np.concatenate(c) for c in zip(*parts))
    return t1 - t2, t2, s1 - s2, s2, w


def _onto(l1, l2, kind, x, y):
    """Points (x, y) of a Duffy rule moved onto the shared edge (l1, l2) or vertex l1 of each pair (P, R)."""
    x, y = x[None, :], y[None, :]
    one = lambda c: c.to(x.dtype)[:, None]  # noqa: E731
    if kind == 1:
        return x.expand(len(l1), -1), y.expand(len(l1), -1)
    if kind == 2:
        lc = 3 - l1 - l2
        (ax, ay), (bx, by), (cx, cy) = ((one(v == 1), one(v == 2)) for v in (l1, l2, lc))
        return ax + x * (bx - ax) + y * (cx - ax), ay + x * (by - ay) + y * (cy - ay)
    return torch.where(l1[:, None] == 1, 1 - x - y, x), torch.where(l1[:, None] == 2, 1 - x - y, y)


class _Exact:
    """Matrices of one mesh in 64 bits."""

    def __init__(self, case, buf):
        self.dev = dev = torch.device("cuda")
        as64 = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev)  # noqa: E731
        self.masks = MASKS[case["mesh"]]
        self.v = as64(buf.vertices_3xn_f32).T.contiguous()
        self.tri = torch.as_tensor(np.asarray(buf.triangles_3xm_i32, dtype=np.int64).T.copy(), device=dev)
        self.dof = torch.as_tensor(np.asarray(buf.p1_local2global_i32, dtype=np.int64), device=dev)
        self.area, self.nrm = as64(buf.triangle_areas_f32), as64(buf.triangle_normals_3xm_f32).T.contiguous()
        self.n, self.T = int(buf.p1_dof_count), len(self.tri)
        self.rw = float(len(self.masks))
        X, Y, W = as64(_X), as64(_Y), as64(_W)
        self.bas = torch.stack([1 - X - Y, X, Y])                             # (3, 6)
        self.pts = torch.einsum("iq,tic->tqc", self.bas, self.v[self.tri]).reshape(-1, 3)
        self.w = (W[None, :] * 2 * self.area[:, None]).reshape(-1)
        self.pn = self.nrm.repeat_interleave(6, 0)
        rows = torch.arange(6 * self.T, device=dev)
        self.phi = torch.zeros(6 * self.T, self.n, dtype=torch.float64, device=dev)   # weighted basis at the points
        for i in range(3):
            self.phi.index_put_((rows, self.dof[:, i].repeat_interleave(6)), self.w * self.bas[i].repeat(self.T),
                                accumulate=True)
        self.mean = torch.zeros(self.T, self.n, dtype=torch.float64, device=dev)      # P1 mean of each triangle
        for i in range(3):
            self.mean.index_put_((torch.arange(self.T, device=dev), self.dof[:, i]),
                                 torch.full((self.T,), 1 / 3, dtype=torch.float64, device=dev), accumulate=True)
        self.pairs = self._pairs()

    def _pairs(self):
        """Touching image pairs: (kind, test, trial, test mask, trial mask, l1, l2 of each side)."""
        out = {1: [], 2: [], 3: []}
        if len(self.masks) == 1:
            ids = {0: torch.arange(len(self.v), device=self.dev)}
        else:
            keys = [torch.round(self.v * _sign(m, self.dev) / 1e-6).long() for m in self.masks]
            inv = torch.unique(torch.cat(keys), dim=0, return_inverse=True)[1].reshape(len(self.masks), -1)
            ids = dict(zip(self.masks, inv))
        local = {m: ids[m][self.tri[:, [0, 2, 1] if bin(m).count("1") % 2 else [0, 1, 2]]] for m in self.masks}
        for tm in self.masks:
            for sm in self.masks:
                for t0 in range(0, self.T, 1000):
                    eq = (local[tm][t0:t0 + 1000, None, :, None] == local[sm][None, :, None, :]).flatten(2)
                    cnt = eq.sum(2)
                    for kind, c in ((1, 3), (2, 2), (3, 1)):
                        t, s = torch.nonzero(cnt == c, as_tuple=True)
                        if len(t) == 0:
                            continue
                        e = eq[t, s].to(torch.int8)
                        first, last = e.argmax(1), 8 - e.flip(1).argmax(1)
                        if kind == 1:
                            first, last = torch.zeros_like(first), torch.full_like(last, 4)
                        out[kind].append((t + t0, s, tm, sm, first // 3, last // 3, first % 3, last % 3))
        return out

    def _side(self, tris, mask, t1, t2):
        """Points and barycentrics of image-local (t1, t2) on image triangles."""
        if bin(mask).count("1") % 2:
            t1, t2 = t2, t1
        v = self.v[self.tri[tris]]
        p = v[:, None, 0] + t1[..., None] * (v[:, 1] - v[:, 0])[:, None] + t2[..., None] * (v[:, 2] - v[:, 0])[:, None]
        return p * _sign(mask, self.dev), torch.stack([1 - t1 - t2, t1, t2], -1)

    def duffy(self, waves):
        """Per group of touching pairs: (test, trial, test mask, per wavenumber (SLP (P, 3), DLP (P, 3, 3)) of
        singular minus regular)."""
        a = lambda z: torch.as_tensor(z, device=self.dev)  # noqa: E731
        rx, ry = a(np.repeat(_X, 6)), a(np.repeat(_Y, 6))
        sx, sy, rw = a(np.tile(_X, 6)), a(np.tile(_Y, 6)), a(np.outer(_W, _W).reshape(-1))
        for kind, groups in self.pairs.items():
            t1, t2, s1, s2, w = (a(z) for z in _duffy_rule(kind))
            w = torch.cat([w, -rw])
            for test, trial, tm, sm, tl1, tl2, sl1, sl2 in groups:
                step = max(1, 3_000_000 // len(w))
                for c in range(0, len(test), step):
                    te, tr = test[c:c + step], trial[c:c + step]
                    sides = []
                    for tris, mask, l1, l2, x, y, gx, gy in ((te, tm, tl1, tl2, t1, t2, rx, ry),
                                                            (tr, sm, sl1, sl2, s1, s2, sx, sy)):
                        x, y = _onto(l1[c:c + step], l2[c:c + step], kind, x, y)
                        x = torch.cat([x, gx.expand(len(tris), -1)], 1)
                        y = torch.cat([y, gy.expand(len(tris), -1)], 1)
                        sides.append(self._side(tris, mask, x, y))
                    (px, tb), (py, sb) = sides
                    d, nn = py - px, (self.nrm[tr] * _sign(sm, self.dev))[:, None]
                    same = (te == tr) & (tm == sm)
                    # the regular rule leaves the coincident point of a triangle with itself out
                    hole = torch.zeros_like(w, dtype=torch.bool)
                    hole[len(w) - 36::7] = True
                    ww = torch.where(same[:, None] & hole[None, :], torch.zeros_like(w), w[None, :].expand(len(te), -1))
                    ww = ww * (4 * self.area[te] * self.area[tr])[:, None] / (4 * math.pi)
                    blocks = []
                    for k, ki in waves:
                        G, D = _kernels(d, nn, k, ki)
                        blocks.append(((G * ww).unsqueeze(1).matmul(tb.to(G.dtype)).squeeze(1),
                                       (tb.to(D.dtype) * (D * ww)[..., None]).transpose(1, 2).matmul(sb.to(D.dtype))))
                    yield te, tr, tm, blocks

    def regular(self, k, ki, right_d, right_g):
        """phi^T D right_d and phi^T G right_g of the regular rule (images of the trial side summed)."""
        dev, P = self.dev, len(self.pts)
        out_d = torch.zeros(self.n, right_d.shape[1], dtype=torch.complex128, device=dev)
        out_g = torch.zeros(self.n, right_g.shape[1], dtype=torch.complex128, device=dev)
        step = max(6, 30_000_000 // P)
        times = lambda M, R: (torch.complex(M.real @ R, M.imag @ R) if not R.is_complex() else M @ R)  # noqa: E731
        for r in range(0, P, step):
            G = D = 0
            for m in self.masks:
                g, dd = _kernels(self.pts * _sign(m, dev) - self.pts[r:r + step, None], self.pn * _sign(m, dev), k, ki)
                G, D = G + g, D + dd
            left = self.phi[r:r + step].T.contiguous()
            for K, R, out in ((D, right_d, out_d), (G, right_g, out_g)):
                if R.shape[1]:
                    KR = times(K, R)
                    out += torch.complex(left @ KR.real, left @ KR.imag) / (4 * math.pi)
        return out_d, out_g

    def field(self, k, p, q, obs):
        p_pt = torch.einsum("iq,ti->tq", self.bas.to(p.dtype), p[self.dof]).reshape(-1) * self.w
        q_pt = q.repeat_interleave(6) * self.w
        out = []
        for o in range(0, len(obs), 200):
            acc = 0
            for m in self.masks:
                s = _sign(m, self.dev)
                G, D = _kernels(self.pts * s - obs[o:o + 200, None], self.pn * s, k, 0.0)
                acc = acc + D @ p_pt - G @ q_pt
            out.append(acc / (4 * math.pi))
        return torch.cat(out)

    def average(self, p, tags, tag):
        sel = torch.as_tensor(tags == tag, device=self.dev)
        a = self.area * sel
        return (p[self.dof].mean(1) * a).sum() / a.sum()


def _exact_one(case, i):
    ex = _Exact(case, i["buf"])
    dev, n, T = ex.dev, ex.n, ex.T
    tags = np.asarray(i["buf"].physical_tags_i32)
    q = torch.as_tensor(i["q"].astype(np.complex128), device=dev)             # (S, F, T)
    obs = torch.as_tensor(i["obs"].astype(np.float64), device=dev).T.contiguous()
    beta = torch.zeros(T, dtype=torch.complex128, device=dev)
    for tag, b in (i["beta"] or {}).items():
        beta[torch.as_tensor(tags == tag, device=dev)] = complex(np.complex64(b))
    ap = torch.as_tensor(np.flatnonzero(tags == APERTURE) if case["mesh"] == "baffled" else np.zeros(0, np.int64),
                         device=dev)
    m = len(ap)
    waves = [(float(k), float(ki)) for k, ki in zip(i["k"], i["k_im"])]
    S = q.shape[0]
    driven = torch.as_tensor(np.flatnonzero(tags == THROAT), device=dev)
    # columns of G that are needed: driven, lossy and aperture triangles
    need = torch.unique(torch.cat([driven, torch.nonzero(beta).reshape(-1), ap]))
    col = torch.full((T,), -1, dtype=torch.long, device=dev)
    col[need] = torch.arange(len(need), device=dev)
    dp0 = torch.zeros(6 * T, len(need), dtype=torch.float64, device=dev)
    pt = (need[:, None] * 6 + torch.arange(6, device=dev)).reshape(-1)
    dp0[pt, torch.arange(len(need), device=dev).repeat_interleave(6)] = ex.w[pt]
    mass = torch.zeros(n, n, dtype=torch.float64, device=dev)
    for a in range(3):
        for b in range(3):
            mass.index_put_((ex.dof[:, a], ex.dof[:, b]), ex.area * (1 / 6 if a == b else 1 / 12), accumulate=True)
    DLP = [torch.zeros(n, n, dtype=torch.complex128, device=dev) for _ in waves]
    SLP = [torch.zeros(n, len(need), dtype=torch.complex128, device=dev) for _ in waves]
    SAA = [torch.zeros(m, m, dtype=torch.complex128, device=dev) for _ in waves]
    where = torch.full((T,), -1, dtype=torch.long, device=dev)
    where[ap] = torch.arange(m, device=dev)
    for te, tr, tm, blocks in ex.duffy(waves):
        live = col[tr] >= 0
        both = (where[te] >= 0) & (where[tr] >= 0) if tm == 0 else torch.zeros_like(live)
        for f, (g, dd) in enumerate(blocks):
            DLP[f].index_put_((ex.dof[te][:, :, None].expand(-1, 3, 3), ex.dof[tr][:, None, :].expand(-1, 3, 3)), dd,
                              accumulate=True)
            SLP[f].index_put_((ex.dof[te][live], col[tr][live][:, None].expand(-1, 3)), g[live], accumulate=True)
            SAA[f].index_put_((where[te][both], where[tr][both]), g[both].sum(1) / ex.area[te][both], accumulate=True)
    fields, surfaces, imps, apertures = [[] for _ in range(S)], [[] for _ in range(S)], [[] for _ in range(S)], []
    for f, (k, ki) in enumerate(waves):
        d, g = ex.regular(k, ki, ex.phi, dp0)
        A = DLP[f] + ex.rw * d - 0.5 * ex.rw * mass
        slp = SLP[f] + ex.rw * g
        ik = complex(-ki, k)
        A -= ik * (slp * beta[need]) @ ex.mean[need].to(A.dtype)
        rhs = slp @ q[:, f, need].T                                           # (n, S)
        if m:
            x_ap = ex.pts.reshape(T, 6, 3)[ap].reshape(-1, 3)
            w_ap = torch.zeros(6 * m, m, dtype=torch.complex128, device=dev)
            w_ap[torch.arange(6 * m, device=dev), torch.arange(m, device=dev).repeat_interleave(6)] = \
                ex.w.reshape(T, 6)[ap].reshape(-1).to(w_ap.dtype)
            saa = SAA[f]
            for r in range(0, 6 * m, 600):
                G, _ = _kernels(x_ap - x_ap[r:r + 600, None], x_ap, k, 0.0)
                saa = saa + (w_ap[r:r + 600].T @ (G @ w_ap)) / (4 * math.pi) / ex.area[ap][:, None]
            K = torch.zeros(n + m, n + m, dtype=torch.complex128, device=dev)
            K[:n, :n], K[:n, n:], K[n:, :n], K[n:, n:] = A, -slp[:, col[ap]], ex.mean[ap], -2 * saa
            x = torch.linalg.solve(K, torch.cat([rhs, torch.zeros(m, S, dtype=rhs.dtype, device=dev)]))
            p, qa = x[:n], x[n:, 0]
            apertures.append(qa)
            e = obs.clone()
            e[:, 2].clamp_min_(0.0)
            G = torch.cat([_kernels(x_ap - e[o:o + 200, None], x_ap, k, 0.0)[0] for o in range(0, len(e), 200)])
            out = -2 * (G @ (w_ap @ qa)) / (4 * math.pi) * (obs[:, 2] >= -1e-5)
            fields[0].append(out)
        else:
            p = torch.linalg.solve(A, rhs)
        for s in range(S):
            ps = p[:, s].contiguous()
            if not m:
                fields[s].append(ex.field(k, ps, q[s, f] + ik * beta * ps[ex.dof].mean(1), obs))
            surfaces[s].append(ps)
            imps[s].append(ex.average(ps, tags, THROAT))
    host = lambda z: torch.stack(z).cpu().numpy()  # noqa: E731
    outs = [{"field": host(fields[s]), "surface": host(surfaces[s]), "impedance": host(imps[s])} for s in range(S)]
    if m:
        outs[0]["aperture"] = host(apertures)
    return outs


def exact(case, seed):
    if case["kind"] == "batch":
        outs = [_exact_one(case, _inputs(case, seed, m))[0] for m in range(case["meshes"])]
        return [dict(o, impedance=o["impedance"][:, None]) for o in outs]
    outs = _exact_one(case, _inputs(case, seed))
    if case["kind"] == "gradient":
        return {"field": outs[0]["field"], "gradient": None}
    out = dict(outs[0])
    if case["sources"] > 1:
        out["extra"] = outs[1:]
    return out
