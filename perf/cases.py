"""Performance cases: what a user of this library has it compute, over the sizes, precisions and physics it is used with.

A pass advances a domain (or a batch of shots) by a number of time steps through the public Python interface and reads
the results back, as a driver does between two outputs: ``Domain.run``, ``Domain.fields`` into a pinned host array,
``Domain.seismograms``; a gradient is one ``waveform_misfit`` forward and backward.  FP32 domains' results are kept in
float32, the precision they were computed in.  The steps per pass are far fewer than a run's (500 to 2000), and enough
that reading the fields back stays a minor part of the pass.

``exact`` advances the same inputs with plain torch in 64 bits: dense difference matrices along each axis and the
equations written over whole arrays.
"""
import math

import numpy as np
import torch

from waveqlab3d_q_gpu_b200 import _lib, anelastic, configs, shots
from waveqlab3d_q_gpu_b200.adjoint import AdjointSolver, waveform_misfit
from waveqlab3d_q_gpu_b200.domain import Domain
from waveqlab3d_q_gpu_b200.problem import AnelasticParams, Block, InterfaceParams, Problem, Source


# ------------------------------------------------------------------------------------------------------------- cases

def listed():
    return [
        # the smallest call: the 41^3 regression input of the test programs, where launches and latency count
        {"name": "cart41_f64", "kind": "cart", "nq": 41, "nr": 41, "ns": 41, "response": "elastic", "npml": 0,
         "prec": "fp64", "steps": 24},
        # plain Cartesian block of 101^3 points at CFL 0.5 with a surface array, the first benchmark configuration
        {"name": "cart101_f64", "kind": "cart", "nq": 101, "nr": 101, "ns": 101, "response": "elastic", "npml": 0,
         "prec": "fp64", "steps": 60},
        # a ragged attenuating basin block with absorbing layers on a Cartesian mesh
        {"name": "cart_q4_pml_f64", "kind": "cart", "nq": 93, "nr": 118, "ns": 75, "response": "anelastic-Q4", "npml": 12,
         "prec": "fp64", "steps": 30},
        # planar rupture in a random medium with frequency-dependent Q (two Cartesian blocks), both precisions
        {"name": "planar_fq8_f64", "kind": "planar", "nq": 224, "nr": 176, "ns": 112, "prec": "fp64", "steps": 12},
        {"name": "planar_fq8_f32", "kind": "planar", "nq": 192, "nr": 160, "ns": 128, "prec": "fp32", "steps": 24},
        # topography, Q8, absorbing layers, locked interface: the production wave propagation run, full size in FP64
        {"name": "hill201_q8_f64", "kind": "hill", "n": 201, "npml": 20, "prec": "fp64", "steps": 16},
        # the same at a lower resolution in FP32 (parameter sweeps)
        {"name": "hill145_q8_f32", "kind": "hill", "n": 145, "npml": 15, "prec": "fp32", "steps": 40},
        # elastic curvilinear block of ragged size with characteristic boundaries only
        {"name": "curv_el_f64", "kind": "curv", "nq": 83, "nr": 121, "ns": 67, "response": "elastic", "prec": "fp64",
         "steps": 30},
        # many independent shots of uneven size in one batch, FP32, elastic and Q4 in turn
        {"name": "shots_f32", "kind": "shots", "sizes": "64,83,97,110,128,72,101,90", "prec": "fp32", "steps": 24},
        # waveform-misfit gradient with respect to material and moment tensor (full-waveform inversion step)
        {"name": "gradient_f64", "kind": "gradient", "nq": 81, "nr": 97, "ns": 65, "prec": "fp64", "steps": 40},
        # the upwind operator pair of the published Q8 regression inputs
        {"name": "upwind4_q8_f64", "kind": "cart", "nq": 61, "nr": 61, "ns": 61, "response": "anelastic-Q8", "npml": 0,
         "prec": "fp64", "steps": 16, "fd": "upwind4"},
        # spontaneous rupture on a small two-block elastic problem, fault outputs read with the fields
        {"name": "rupture_f64", "kind": "rupture", "nq": 51, "nr": 81, "ns": 61, "prec": "fp64", "steps": 40},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["cart", "cart", "planar", "hill", "curv", "shots", "gradient", "upwind", "rupture"])
    prec = rng.choice(["fp64", "fp32"])
    if kind in ("cart", "upwind"):
        c = {"kind": "cart", "nq": size(30, 160), "nr": size(30, 160), "ns": size(30, 160),
             "response": rng.choice(["elastic", "anelastic-Q4", "anelastic-Q8"]), "npml": rng.choice([0, 0, 8, 12]),
             "prec": prec, "steps": 2 * rng.randint(6, 20)}
        if kind == "upwind":
            c.update(nq=size(30, 90), nr=size(30, 90), ns=size(30, 90), fd="upwind4", npml=0)
        return c
    if kind == "planar":
        return {"kind": kind, "nq": 2 * size(24, 110), "nr": size(40, 180), "ns": size(40, 130), "prec": prec,
                "steps": 2 * rng.randint(5, 10)}
    if kind == "hill":
        return {"kind": kind, "n": 2 * size(30, 84) + 1, "npml": rng.choice([8, 10, 15]), "prec": prec,
                "steps": 2 * rng.randint(6, 14)}
    if kind == "curv":
        return {"kind": kind, "nq": size(30, 130), "nr": size(30, 130), "ns": size(30, 130),
                "response": rng.choice(["elastic", "anelastic-Q4", "anelastic-Q8"]), "prec": prec,
                "steps": 2 * rng.randint(6, 16)}
    if kind == "shots":
        return {"kind": kind, "sizes": ",".join(str(size(40, 120)) for _ in range(rng.randint(3, 9))), "prec": prec,
                "steps": 2 * rng.randint(8, 16)}
    if kind == "gradient":
        return {"kind": kind, "nq": size(40, 90), "nr": size(40, 90), "ns": size(40, 70), "prec": "fp64",
                "steps": rng.randint(16, 36)}
    return {"kind": kind, "nq": size(25, 80), "nr": size(40, 110), "ns": size(40, 90), "prec": prec,
            "steps": 2 * rng.randint(8, 24)}


def work(case):
    """Bytes and operations of a pass.  Per point and RK stage: fields and rates read and written (36 words), material
    (3), metric and Jacobian of curvilinear meshes (10), 24 words per relaxation mechanism and two quality factors, 36
    words per point of an absorbing layer; a reverse sweep moves the same arrays twice again (recomputation and
    adjoint).  Operations: six taps per derivative."""
    size = 8 if case["prec"] == "fp64" else 4
    words = ops = 0
    for n, resp, curv, npml_faces, npml in _blocks_of(case):
        pts = n[0] * n[1] * n[2]
        nm = {"elastic": 0, "anelastic-Q4": 4, "anelastic-Q8": 8, "anelastic-fQ8": 8}[resp]
        words += pts * (39 + (10 if curv else 0) + 24 * nm + (2 if nm and resp != "anelastic-fQ8" else 0))
        for ax in npml_faces:
            words += 36 * npml * pts // n[ax]
        ops += pts * ((540 if curv else 210) + 40 * nm)
    scale = 5 * case["steps"] * (3 if case["kind"] == "gradient" else 1)
    return {"bytes": size * words * scale, "flops": ops * scale}


def _blocks_of(case):
    """(points per axis, response, curvilinear, axes of the absorbing layers, their width) of every block."""
    k = case["kind"]
    if k == "cart":
        return [((case["nq"], case["nr"], case["ns"]), case["response"], False,
                 [0, 1, 1, 2, 2] if case["npml"] else [], case["npml"])]
    if k == "planar":
        return [((case["nq"] // 2, case["nr"], case["ns"]), "anelastic-fQ8", False, [], 0)] * 2
    if k == "hill":
        n = case["n"]
        b = (((n + 1) // 2, n, n), "anelastic-Q8", True)
        return [b + ([1, 1, 2, 2], case["npml"]), b + ([0, 1, 1, 2, 2], case["npml"])]
    if k == "curv":
        return [((case["nq"], case["nr"], case["ns"]), case["response"], True, [], 0)]
    if k == "gradient":
        return [((case["nq"], case["nr"], case["ns"]), "elastic", True, [], 0)]
    if k == "shots":
        return [((s, s, s), "anelastic-Q4" if i % 2 else "elastic", False, [], 0)
                for i, s in enumerate(int(v) for v in case["sizes"].split(","))]
    return [((case["nq"], case["nr"], case["ns"]), "elastic", False, [], 0)] * 2


# ------------------------------------------------------------------------------------------------------------ inputs

_Q = dict(Qs0=60.0, Qp0=120.0, fref=1.0, fmin=0.05, fmax=20.0)


def _node(block, i, j, k):
    """Physical coordinates of the 0-based grid node (i, j, k)."""
    if block.coords is not None:
        return [float(v) for v in block.coords[:, k, j, i]]
    return [block.aqrs[a] + (block.bqrs[a] - block.aqrs[a]) / (block.nqrs[a] - 1) * m for a, m in enumerate((i, j, k))]


def _put_sources(block, nodes, rng, f0=3.0):
    block.sources = [Source("ricker", f0, 1.2 / f0, *(float(v) for v in rng.uniform(-1.0, 1.0, 6)), *_node(block, *n))
                     for n in nodes]


def _put_receivers(block, count):
    """A line of stations along r on the q-min face; their nodes are in ``_receiver_nodes``."""
    block.receivers = np.array([_node(block, *n) for n in _receiver_nodes(block, count)])


def _receiver_nodes(block, count=12):
    nq, nr, ns = block.nqrs
    return [(0, (j * (nr - 1)) // count + 3, ns // 2) for j in range(count) if (j * (nr - 1)) // count + 3 < nr]


def _layered(depth, rng):
    """Vs growing with depth (fraction 0..1) through a few seeded layers: lambda, mu, rho in the units of the solver."""
    tops = np.sort(rng.uniform(0.0, 1.0, 3))
    vs = (2.0 + 0.9 * depth + 0.2 * np.searchsorted(tops, depth.ravel()).reshape(depth.shape))
    rho = 1.7 + 0.2 * math.sqrt(3.0) * vs
    mu = rho * vs * vs
    return np.stack([mu, mu, rho])   # Vp = sqrt(3) Vs: lambda = mu


def _problem(case, seed):
    """The problems of a case (one, or one per shot), sources and stations on grid nodes."""
    rng = np.random.default_rng(1000003 * (seed % 100003) + 17)
    k = case["kind"]
    if k == "shots":
        out = []
        for i, s in enumerate(int(v) for v in case["sizes"].split(",")):
            p = shots.random_shot(7 * seed + i, nmin=s, nmax=s, steps=case["steps"],
                                  response="anelastic-Q4" if i % 2 else "elastic")
            b = p.blocks[0]
            _put_sources(b, [(s // 2, s // 3, s // 2)], rng)
            _put_receivers(b, 12)
            out.append(p)
        return out
    if k == "hill":
        p = configs.hill_two_block_q8(n=case["n"], h=10.0 / (case["n"] - 1), npml=case["npml"], seed=seed % 1000003)
        b = p.blocks[0]
        _put_sources(b, [(b.nqrs[0] // 2, b.nqrs[1] // 2, b.nqrs[2] // 2)], rng)
        _put_receivers(b, 12)
    elif k == "planar":
        p = configs.planar_fault_fq8(nq=case["nq"], nr=case["nr"], ns=case["ns"], seed=seed % 1000003)
        _put_receivers(p.blocks[0], 12)
        p.blocks[1].receivers = None
        a = p.anelastic    # the fit of the attenuation law is part of the input
        a.tau, a.strength_s, a.strength_p = anelastic.coefficients(p.response, a)
    elif k == "rupture":
        nq, nr, ns, h = case["nq"], case["nr"], case["ns"], 0.1
        L = [h * (n - 1) for n in (nq, nr, ns)]
        y, z = np.meshgrid(np.linspace(-1, 1, nr), np.linspace(-1, 1, ns))
        tl = 70.0 + 3.0 * np.sin(4 * y + rng.uniform(0, 6)) * np.cos(3 * z + rng.uniform(0, 6))
        tl[(np.abs(y) < 0.35) & (np.abs(z) < 0.35)] = 84.0
        blocks = []
        for side in range(2):
            blocks.append(Block(nqrs=(nq, nr, ns), aqrs=(side * L[0], 0.0, 0.0), bqrs=((1 + side) * L[0], L[1], L[2]),
                                rho_s_p=(2.67, 3.464, 6.0), lqrs=(1 - side, 2, 1), rqrs=(side, 1, 1)))
            _put_receivers(blocks[-1], 12)
        blocks[1].receivers = None
        ip = InterfaceParams(coupling="slip-weakening_friction", fs=0.677, fd=0.525, Dc=0.4, tau0_n=np.full((ns, nr), -120.0),
                             tau0_m=np.zeros((ns, nr)), tau0_l=tl, fs_map=np.full((ns, nr), 0.677))
        p = Problem(blocks=blocks, type_of_mesh="cartesian", CFL=0.5, source_order=4, interface=ip)
    elif k in ("curv", "gradient"):
        p = configs.adjoint_block(nq=case["nq"], nr=case["nr"], ns=case["ns"], seed=seed % 1000003)
        b = p.blocks[0]
        p.response = case.get("response", "elastic")
        p.anelastic = AnelasticParams(**_Q)
        nq, nr, ns = b.nqrs
        if k == "gradient":   # shallow and short enough that the waves meet the stations within the steps
            _put_sources(b, [(8, nr // 2, ns // 2)], rng, f0=8.0)
        else:
            _put_sources(b, [(nq // 2, nr // 2, ns // 2), (nq // 2, nr // 3, ns // 2)], rng)
        _put_receivers(b, 12)
    else:
        nq, nr, ns, h, npml = case["nq"], case["nr"], case["ns"], 0.1, case["npml"]
        b = Block(nqrs=(nq, nr, ns), bqrs=tuple(h * (n - 1) for n in (nq, nr, ns)), rho_s_p=(2.7, 3.5, 6.06),
                  lqrs=(2, 1, 1), rqrs=(1, 1, 1))
        b.material = _layered(np.broadcast_to(np.linspace(0.0, 1.0, nq), (ns, nr, nq)), rng)
        if npml:
            b.npml, b.pml_lqrs, b.pml_rqrs = npml, (False, True, True), (True, True, True)
        _put_sources(b, [(nq // 2, nr // 2, ns // 2)], rng)
        _put_receivers(b, 12)
        p = Problem(blocks=[b], response=case["response"], type_of_mesh="cartesian", CFL=0.5, source_order=4,
                    anelastic=AnelasticParams(**_Q))
        if case.get("fd") == "upwind4":
            p.fd_type, p.order = "upwind", 4
    p.w_stride = 1
    return [p]


def _start_fields(shape, seed):
    """A wavefield in the middle of a run: smooth random velocities of some cm/s (in the solver's units) and the
    stresses that go with them, from noise a few grid points long."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device="cpu").manual_seed(int(seed))
    coarse = torch.randn((1, 9) + tuple(max(4, n // 6) for n in shape), generator=g, dtype=torch.float64).to(dev)
    F = torch.nn.functional.interpolate(coarse, size=shape, mode="trilinear", align_corners=True)[0]
    F[:3] *= 0.05
    F[3:] *= 0.05 * 9.0
    return F.cpu().numpy()


def _starts(problems, seed):
    return [[_start_fields(tuple(reversed(b.nqrs)), 31 * seed + 1000 * i + j) for j, b in enumerate(p.blocks)]
            for i, p in enumerate(problems)]


def _observed(case, nrec, seed):
    """Recorded station velocities (steps, stations, 3): a pulse arriving along the line of stations."""
    rng = np.random.default_rng(seed % 1000003)
    t = np.arange(case["steps"])[:, None, None] / case["steps"]
    return 0.02 * rng.standard_normal((1, nrec, 3)) * np.exp(-((t - rng.uniform(0.3, 0.9, (1, nrec, 1))) / 0.15) ** 2)


def prepare(case, seed):
    problems = _problem(case, seed)
    if case["kind"] == "gradient":
        p = problems[0]
        s = p.blocks[0].sources
        moment = torch.tensor([[v.mxx, v.myy, v.mzz, v.mxy, v.mxz, v.myz] for v in s], dtype=torch.float64)
        return {"kind": "gradient", "solver": AdjointSolver(p, case["steps"]),
                "material": torch.from_numpy(p.blocks[0].material.copy()).requires_grad_(True),
                "moment": moment.requires_grad_(True), "observed": _observed(case, len(p.blocks[0].receivers), seed)}
    state = {"kind": case["kind"], "steps": case["steps"], "f32": case["prec"] == "fp32"}
    if case["kind"] == "shots":
        state["batch"] = shots.ShotBatch(problems, precision=case["prec"], nsteps_hint=case["steps"])
        domains = state["batch"].domains
    else:
        domains = [Domain(problems[0], precision=case["prec"], nsteps_hint=case["steps"])]
    state["domains"] = domains
    pin = torch.cuda.is_available()
    state["host"] = []
    for d, fs in zip(domains, _starts(problems, seed)):
        for b, F in enumerate(fs):
            d.set_fields(F, b)
        state["host"].append([torch.empty(F.shape, dtype=torch.float64, pin_memory=pin) for F in fs])
    if state["f32"]:
        state["single"] = [[torch.empty(h.shape, dtype=torch.float32) for h in hs] for hs in state["host"]]
    return state


def run(state):
    if state["kind"] == "gradient":
        state["material"].grad = state["moment"].grad = None
        chi = waveform_misfit(state["material"], state["moment"], state["solver"], state["observed"])
        chi.backward()
        return {"misfit": chi.detach(), "material": state["material"].grad, "moment": state["moment"].grad}
    for d in state["domains"]:   # the stations of this pass only
        _lib.check(_lib.load().wql3d_reset_samples(d.handle), "wql3d_reset_samples")
    if "batch" in state:
        state["batch"].run(state["steps"])
        state["batch"].synchronize()
    else:
        state["domains"][0].run(state["steps"])
    out = {"fields": [], "stations": []}
    for i, d in enumerate(state["domains"]):
        for b, h in enumerate(state["host"][i]):
            d.fields(b, out=h.numpy())
            out["fields"].append(state["single"][i][b].copy_(h) if state["f32"] else h)
        seis = d.seismograms(0)
        out["stations"].append(seis.astype(np.float32) if state["f32"] else seis)
    if state["kind"] in ("rupture", "planar"):
        out["slip"] = state["domains"][0].fault("S")
        if state["f32"]:
            out["slip"] = out["slip"].astype(np.float32)
    return out


# ---------------------------------------------------------------------------------------------- the same in plain torch

_RK_A = (0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0,
         -3550918686646.0 / 2091501179385.0, -1275806237668.0 / 842570457699.0)
_RK_B = (1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0, 1720146321549.0 / 2090206949498.0,
         3134564353537.0 / 4481467310338.0, 2277821191437.0 / 14882151754819.0)
_RK_C = (0.0, 1432997174477.0 / 9575080441755.0, 2526269341429.0 / 6820363962896.0,
         2006345519317.0 / 3224310063776.0, 2802321613138.0 / 2924317926251.0, 1.0)
# boundary rows of the sixth-order summation-by-parts difference (points 1, 2, ... from the boundary)
_SBP6 = ((-1.582533518939116, 2.033378678700676, -0.141512858744873, -0.450398306578272, 0.104488069284042, 0.036577936277544),
         (-0.462059195631158, 0.0, 0.287258622978251, 0.258816087376832, -0.069112065532624, -0.014903449191300),
         (0.071247104721830, -0.636451095137907, 0.0, 0.606235523609147, -0.022902190275815, -0.018129342917256),
         (0.114713313798970, -0.290087484386815, -0.306681191361148, 0.0, 0.520262285050482, -0.051642265516119,
          0.013435342414630),
         (-0.036210680656541, 0.105400944933782, 0.015764336127392, -0.707905442575989, 0.0, 0.769199413962647,
          -0.164529643265203, 0.018281071473911),
         (-0.011398193015050, 0.020437334208704, 0.011220896474665, 0.063183694641876, -0.691649024426814, 0.0,
          0.739709139060752, -0.147941827812150, 0.016437980868017))
# fourth-order upwind pair: interior row and boundary rows of the forward (P) and backward (M) operators
_UP4_P = ((-1.530612244897959, 2.091836734693878, -0.591836734693878, 0.030612244897959),
          (-0.461748633879781, -0.180327868852459, 0.811475409836066, -0.234972677595628, 0.065573770491803),
          (0.089430894308943, -0.475609756097561, -0.707317073170732, 1.581300813008130, -0.585365853658537,
           0.097560975609756),
          (0.030201342281879, -0.073825503355705, -0.218120805369128, -0.785234899328859, 1.449664429530201,
           -0.483221476510067, 0.080536912751678))
_UP4_M = ((-1.408163265306122, 1.724489795918367, -0.224489795918367, -0.091836734693878),
          (-0.560109289617486, 0.180327868852459, 0.319672131147541, 0.060109289617486),
          (0.235772357723577, -1.207317073170732, 0.707317073170732, 0.264227642276423),
          (-0.010067114093960, 0.288590604026846, -1.305369127516778, 0.785234899328859, 0.241610738255034))
_SYM = ((3, 6, 7), (6, 4, 8), (7, 8, 5))   # stress components of the symmetric tensor


def _matrix(n, left, right, inner, first):
    D = np.zeros((n, n))
    for i in range(n):
        for k, c in enumerate(inner):
            if 0 <= i + first + k < n:
                D[i, i + first + k] = c
    for r, row in enumerate(left):
        D[r] = 0.0
        D[r, :len(row)] = row
    for r, row in enumerate(right):
        D[n - 1 - r] = 0.0
        D[n - 1 - r, n - len(row):] = [-c for c in reversed(row)]
    return D * (n - 1)


def _sbp(n):
    return _matrix(n, _SBP6, _SBP6, (-1 / 60, 0.15, -0.75, 0.0, 0.75, -0.15, 1 / 60), -3)


def _along(D, T, a):
    """D applied along axis a (0: q, the last dimension; 1: r; 2: s, the third last)."""
    if a == 0:
        return T @ D.T
    if a == 1:
        return D @ T
    return (D @ T.reshape(T.shape[0], T.shape[1], -1)).reshape(T.shape)


def _face(T, f):
    """The face f (q-min, q-max, r-min, ...) of an array whose last three dimensions are s, r, q."""
    return T.select(-1 - (f >> 1), -1 if f & 1 else 0)


class _Exact:
    """One block in plain torch, 64 bits."""

    def __init__(self, p, b, dev, material=None):
        t = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=dev)  # noqa: E731
        self.p, self.b, self.dev = p, b, dev
        n = self.n = b.nqrs
        self.shape = tuple(reversed(n))
        metric = [t(_sbp(m)) for m in n]
        if p.fd_type == "upwind":
            inP, inM = (-1 / 4, -5 / 6, 3 / 2, -1 / 2, 1 / 12), (-1 / 12, 1 / 2, -3 / 2, 5 / 6, 1 / 4)
            self.Dv = [t(_matrix(m, _UP4_P, _UP4_M, inP, -1)) for m in n]
            self.Ds = [t(_matrix(m, _UP4_M, _UP4_P, inM, -3)) for m in n]
        else:
            self.Dv = self.Ds = metric
        self.pen = [(144.0 / 49.0 if p.fd_type == "upwind" else 1.0 / 0.315949074074074) * (m - 1) for m in n]
        self.curv = p.type_of_mesh == "curvilinear"
        if self.curv:
            X = t(b.coords)
            g = torch.stack([torch.stack([_along(metric[a], X[c:c + 1], a)[0] for a in range(3)]) for c in range(3)])
            cof = torch.stack([torch.stack([g[(c + 1) % 3, (a + 1) % 3] * g[(c + 2) % 3, (a + 2) % 3] -
                                            g[(c + 1) % 3, (a + 2) % 3] * g[(c + 2) % 3, (a + 1) % 3]
                                            for a in range(3)]) for c in range(3)])
            self.J = (g[0] * cof[0]).sum(0)
            self.X = cof / self.J     # X[r, a] = d(axis a) / d(coordinate r)
        else:
            self.J = None
            self.X = [1.0 / (b.bqrs[a] - b.aqrs[a]) for a in range(3)]
        self.nm = {"elastic": 0, "anelastic-Q4": 4, "anelastic-Q8": 8, "anelastic-fQ8": 8}[p.response]
        if material is None:
            if b.material is not None:
                m = t(b.material)
            else:
                rho, cs, cp = b.rho_s_p
                m = torch.stack([torch.full(self.shape, v, dtype=torch.float64, device=dev)
                                 for v in (rho * (cp * cp - 2 * cs * cs), rho * cs * cs, rho)])
            material = self._unrelaxed(m, t) if self.nm else m
        self.M = material
        z = lambda *s: torch.zeros(s + self.shape, dtype=torch.float64, device=dev)  # noqa: E731
        self.F, self.DF = z(9), z(9)
        if self.nm:
            self.eta, self.deta = z(6, self.nm), z(6, self.nm)
        self.slab, self.Q, self.DQ = {}, {}, {}
        for f, on in enumerate(b.pml()):
            if not (on and b.npml):
                continue
            a, w = f >> 1, b.npml
            sl = [slice(None)] * 3
            sl[2 - a] = slice(n[a] - w, n[a]) if f & 1 else slice(0, w)
            i = torch.arange(1, n[a] + 1, dtype=torch.float64, device=dev)
            dist = (i - w) if f == 4 else (i - (n[a] - w)) if f & 1 else (i - (1 + w))
            d = 3.0 * math.log(1.0e3) * (dist / w).abs()
            view = [1, 1, 1]
            view[2 - a] = -1
            self.slab[f] = (tuple(sl), d[sl[2 - a]].view(view))
            self.Q[f] = torch.zeros_like(self.F[(slice(None),) + tuple(sl)])
            self.DQ[f] = torch.zeros_like(self.Q[f])
        self.srcs = [self._source(s) for s in b.sources]

    def _unrelaxed(self, m, t):
        """Unrelaxed moduli from the moduli at the reference frequency."""
        p, b = self.p, self.b
        a = p.anelastic
        w2 = (2 * math.pi * a.fref) ** 2
        if p.response == "anelastic-fQ8":
            self.tau, self.ss, self.ps = (list(map(float, v)) for v in (a.tau, a.strength_s, a.strength_p))
            vs = sum(c / (w2 * x * x + 1) for c, x in zip(self.ss, self.tau))
            vp = sum(c / (w2 * x * x + 1) for c, x in zip(self.ps, self.tau))
        else:
            N = self.nm
            lo, hi = 1 / (2 * math.pi * a.fmax), 1 / (2 * math.pi * a.fmin)
            self.tau = [math.exp(math.log(lo) + (2 * k - 1) / (2 * N) * math.log(hi / lo)) for k in range(1, N + 1)]
            w = ((1.549360, 0.804277, 0.887718, 1.464160) if N == 4 else
                 (1.50589707, 0.0, 0.52793567, 0.53065494, 0.32862132, 0.64375916, 0.0, 1.32751442))
            self.qs = t(b.qs_inv) if b.qs_inv is not None else torch.full_like(m[0], 1.0 / a.Qs0)
            self.qp = t(b.qp_inv) if b.qp_inv is not None else torch.full_like(m[0], 1.0 / a.Qp0)
            self.w = w
            s = sum(c / (w2 * x * x + 1) for c, x in zip(w, self.tau))
            vs, vp = s * self.qs, s * self.qp
        mu, l2m = m[1] / (1 - vs), (m[0] + 2 * m[1]) / (1 - vp)
        return torch.stack([l2m - 2 * mu, mu, m[2]])

    def _source(self, s):
        """(tensor components, support weights as a full array, time function) of a source on a grid node."""
        b = self.b
        if b.coords is not None:
            d = sum((b.coords[c] - v) ** 2 for c, v in enumerate((s.x, s.y, s.z)))
            k, j, i = np.unravel_index(np.argmin(d), d.shape)
        else:
            i, j, k = (int(round((v - b.aqrs[a]) / (b.bqrs[a] - b.aqrs[a]) * (self.n[a] - 1)))
                       for a, v in enumerate((s.x, s.y, s.z)))
        w9 = (-0.01171875, -0.03125, 0.046875, 0.28125, 0.4296875, 0.28125, 0.046875, -0.03125, -0.01171875)
        full = torch.ones(self.shape, dtype=torch.float64, device=self.dev)
        for a, c in enumerate((i, j, k)):
            line = torch.zeros(self.n[a], dtype=torch.float64, device=self.dev)
            for o in range(-4, 5):
                if 0 <= c + o < self.n[a]:
                    line[c + o] = w9[o + 4]
            view = [1, 1, 1]
            view[2 - a] = -1
            full = full * line.view(view) * (self.X[a, a] if self.curv else self.X[a]) * (self.n[a] - 1)
        M = torch.tensor([s.mxx, s.myy, s.mzz, s.mxy, s.mxz, s.myz], dtype=torch.float64, device=self.dev)

        def ricker(t):
            x = (math.pi * s.duration * (t - s.t_init)) ** 2
            return (1 - 2 * x) * math.exp(-x)
        return [M, full, ricker]

    def terms(self, F):
        """Velocity gradients U[r][c] = d v_c / d x_r and, per row r, the stress fluxes d sigma_rc / d x_r."""
        dv = [_along(self.Dv[a], F[:3], a) for a in range(3)]
        if not self.curv:
            U = [self.X[r] * dv[r] for r in range(3)]
            S = [self.X[r] * _along(self.Ds[r], F[list(_SYM[r])], r) for r in range(3)]
            return U, S
        U, S = [], []
        for r in range(3):
            U.append(sum(self.X[r, a] * dv[a] for a in range(3)))
            S.append(sum(_along(self.Ds[a], self.J * self.X[r, a] * F[list(_SYM[r])], a) for a in range(3)) / self.J)
        return U, S

    def boundary(self, F, f):
        """Characteristic boundary term of face f: what is subtracted from the rates, and from the layer's fields."""
        b, a, plus = self.b, f >> 1, f & 1
        sg = 1.0 if plus else -1.0
        u = _face(F, f)
        lam, mu, rho = _face(self.M, f)
        Zp, Zs = torch.sqrt(rho * (lam + 2 * mu)), torch.sqrt(rho * mu)
        r = {1: 0.0, 2: 1.0, 3: -1.0}[b.bc()[f]]
        if self.curv:
            q = torch.stack([_face(self.X[c, a], f) for c in range(3)])
            norm = torch.sqrt((q * q).sum(0))
            n = q / norm
        else:
            norm, n = self.X[a], torch.zeros_like(u[:3])
            n[a] = 1.0
        T = torch.stack([sum(n[j] * u[_SYM[i][j]] for j in range(3)) for i in range(3)])
        vn, Tn = n * (n * u[:3]).sum(0), n * (n * T).sum(0)
        vt, Tt = u[:3] - vn, T - Tn
        P = 0.5 * ((1 - r) * (Zp * vn + Zs * vt) + sg * (1 + r) * T)
        R = 0.5 * ((1 - r) * u[:3] + sg * (1 + r) * (Tn / Zp + Tt / Zs))
        g = torch.cat([norm * P, sg * norm * torch.stack(
            [n[0] * R[0], n[1] * R[1], n[2] * R[2], n[1] * R[0] + n[0] * R[1], n[2] * R[0] + n[0] * R[2],
             n[2] * R[1] + n[1] * R[2]])])
        tr = g[3] + g[4] + g[5]
        s = torch.cat([g[:3] / rho, 2 * mu * g[3:6] + lam * tr, mu * g[6:9]])
        return self.pen[a] * s, self.pen[a] * g

    def stage(self, k, t, dt, jump):
        """One Runge-Kutta stage; jump: {face: interface term already times its penalty}."""
        A, Bdt, F = _RK_A[k], _RK_B[k] * dt, self.F
        lam, mu, rho = self.M
        U, S = self.terms(F)
        e = [U[0][0], U[1][1], U[2][2], U[1][0] + U[0][1], U[2][0] + U[0][2], U[2][1] + U[1][2]]
        tr = e[0] + e[1] + e[2]
        l2m = lam + 2 * mu
        R = torch.cat([(S[0] + S[1] + S[2]) / rho, torch.stack([2 * mu * e[c] + lam * tr for c in range(3)]),
                       torch.stack([mu * e[c] for c in range(3, 6)])])
        for f, (sl, d) in self.slab.items():
            Q, s9 = self.Q[f], (slice(None),) + sl
            a, ls, ms, rs = f >> 1, lam[sl], mu[sl], rho[sl]
            qt = Q[3] + Q[4] + Q[5]
            R[s9] -= d * torch.cat([Q[:3] / rs, 2 * ms * Q[3:6] + ls * qt, ms * Q[6:9]])
            src = torch.zeros_like(Q)
            src[:3] = S[a][s9]
            for c in range(3):
                src[_SYM[a][c]] = U[a][c][sl]
            self.DQ[f] = A * self.DQ[f] + src - (d + 1.0) * Q
        if self.nm:
            if self.slab:
                e = [x.clone() for x in e]
                for f, (sl, d) in self.slab.items():
                    for c in range(3):
                        e[_SYM[f >> 1][c] - 3][sl] -= d * self.Q[f][_SYM[f >> 1][c]]
                tr = e[0] + e[1] + e[2]
            R[3:] -= self.eta.sum(1)
            for c in range(6):
                for i in range(self.nm):
                    if self.p.response == "anelastic-fQ8":
                        g = (self.ss[i] * 2 * mu * e[c] + (l2m * self.ps[i] - 2 * mu * self.ss[i]) * tr) if c < 3 else \
                            self.ss[i] * mu * e[c]
                    else:
                        g = self.w[i] * ((2 * mu * self.qs * e[c] + (l2m * self.qp - 2 * mu * self.qs) * tr) if c < 3
                                         else mu * self.qs * e[c])
                    self.deta[c, i] = A * self.deta[c, i] + (g - self.eta[c, i]) / self.tau[i]
            self.eta += Bdt * self.deta
        ts = t + _RK_C[k] * dt
        for M, w, fn in self.srcs:
            R = torch.cat([R[:3], R[3:] - fn(ts) * M.view(6, 1, 1, 1) * w])
        for f in range(6):
            if self.b.bc()[f] > 0:
                s, g = self.boundary(F, f)
                R = self._minus(R, f, s)
                if f in self.slab:
                    _face(self.DQ[f], f).sub_(g)
        for f, s in jump.items():
            R = self._minus(R, f, s)
        self.DF = A * self.DF + R
        self.F = F + Bdt * self.DF
        for f in self.slab:
            self.Q[f] = self.Q[f] + Bdt * self.DQ[f]

    @staticmethod
    def _minus(R, f, s):
        if R.requires_grad:
            pad = torch.zeros_like(R)
            _face(pad, f).copy_(s)
            return R - pad
        _face(R, f).sub_(s)
        return R


def _interface(p, L, R, I, k, dt):
    """Interface terms {block: {face: term}} of the plane q-max of L / q-min of R (normal along x), and the slip state."""
    u, v = _face(L.F, 1), _face(R.F, 0)
    Z = []
    for blk, f in ((L, 1), (R, 0)):
        lam, mu, rho = _face(blk.M, f)
        Zp, Zs = torch.sqrt(rho * (lam + 2 * mu)), torch.sqrt(rho * mu)
        Z.append(torch.stack([Zp, Zs, Zs]))
    tr = [3, 6, 7]
    pch, qch = Z[0] * u[:3] - u[tr], Z[1] * v[:3] + v[tr]
    eta = 1.0 / (1.0 / Z[0] + 1.0 / Z[1])
    phi = eta * (qch / Z[1] - pch / Z[0])
    T, V = phi.clone(), torch.zeros_like(phi)
    if p.interface.coupling != "locked":
        ip = p.interface
        t0 = torch.as_tensor(np.stack([ip.tau0_n, ip.tau0_m, ip.tau0_l]), dtype=torch.float64, device=u.device)
        fs = torch.as_tensor(ip.fs_map, dtype=torch.float64, device=u.device)
        full = t0 + phi
        sn = (-full[0]).clamp(min=0.0)
        strength = sn * (fs - (fs - ip.fd) * I["S"][3].clamp(max=ip.Dc) / ip.Dc)
        load = torch.sqrt(full[1] ** 2 + full[2] ** 2)
        slip = load > strength
        Vs = torch.where(slip, (load - strength) / eta[1], torch.ones_like(load))
        den = eta[1] + strength / Vs
        for c in (1, 2):
            V[c] = torch.where(slip, full[c] / den, torch.zeros_like(load))
            T[c] = phi[c] - eta[1] * V[c]
    hatR, hatL = (pch + T) / Z[0] + V, (qch - T) / Z[1] - V
    I["DS"] = _RK_A[k] * I["DS"]
    I["DS"][:3] += hatR - hatL
    dv = (hatR - hatL)[1:]
    I["DS"][3] += torch.sqrt((dv * dv).sum(0))
    out = []
    for blk, f, g, hat, z, sg in ((L, 1, u, hatL, Z[0], 1.0), (R, 0, v, hatR, Z[1], -1.0)):
        lam, mu, rho = _face(blk.M, f)
        norm = _face(blk.X[0, 0], f) if blk.curv else blk.X[0]
        d = 0.5 * (z * (g[:3] - hat) + sg * (g[tr] - T))
        r = d / z
        s = torch.stack([norm * d[0] / rho, norm * d[1] / rho, norm * d[2] / rho, sg * (lam + 2 * mu) * norm * r[0],
                         sg * lam * norm * r[0], sg * lam * norm * r[0], sg * mu * norm * r[1], sg * mu * norm * r[2],
                         torch.zeros_like(r[0])])
        out.append({f: blk.pen[0] * s})
    return out


def _advance(p, blocks, steps, dt, sample):
    I = None
    if len(blocks) == 2:
        face = blocks[0].shape[:2]
        I = {k: torch.zeros((4,) + face, dtype=torch.float64, device=blocks[0].dev) for k in ("S", "DS")}
    t = 0.0
    for _ in range(steps):
        sample(t, blocks[0].F)
        for k in range(5):
            jumps = _interface(p, *blocks, I, k, dt) if I else [{}]
            for blk, j in zip(blocks, jumps):
                blk.stage(k, t, dt, j)
            if I:
                I["S"] = I["S"] + _RK_B[k] * dt * I["DS"]
        t += dt
    return I


def _time_step(p):
    return min(p.CFL * min((b.bqrs[i] - b.aqrs[i]) / (b.nqrs[i] - 1) for i in range(3)) /
               math.sqrt(b.rho_s_p[1] ** 2 + b.rho_s_p[2] ** 2) for b in p.blocks)


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    problems = _problem(case, seed)
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed, problems[0], dev)
    out = {"fields": [], "stations": []}
    with torch.no_grad():
        for p, starts in zip(problems, _starts(problems, seed)):
            blocks = [_Exact(p, b, dev) for b in p.blocks]
            for blk, F in zip(blocks, starts):
                blk.F = torch.as_tensor(F, device=dev)
            dt = _time_step(p)
            if p.response != "elastic":
                dt = min(dt, 2.0 * min(blocks[0].tau))
            nodes = _receiver_nodes(p.blocks[0])
            i, j, k = (torch.tensor([n[a] for n in nodes], device=dev) for a in range(3))
            rows = []

            def sample(t, F):
                v = F[:3, k, j, i].T
                rows.append(torch.cat([torch.full_like(v[:, :1], t), v], 1))
            I = _advance(p, blocks, case["steps"], dt, sample)
            out["fields"] += [blk.F for blk in blocks]
            out["stations"].append(torch.stack(rows))
            if case["kind"] in ("rupture", "planar"):
                out["slip"] = I["S"]
    return out


def _exact_gradient(case, seed, p, dev):
    """The gradient by reverse-mode differentiation of the plain steps, a step at a time."""
    b = p.blocks[0]
    m = torch.as_tensor(b.material, device=dev).requires_grad_(True)
    s = b.sources
    M = torch.tensor([[v.mxx, v.myy, v.mzz, v.mxy, v.mxz, v.myz] for v in s], dtype=torch.float64, device=dev,
                     requires_grad=True)
    blk = _Exact(p, b, dev)
    obs = torch.as_tensor(_observed(case, len(b.receivers), seed), device=dev)
    dt = _time_step(p)
    i, j, k = (torch.tensor([n[a] for n in _receiver_nodes(b)], device=dev) for a in range(3))

    def step(F, m, M, n):
        blk.F, blk.M, blk.DF = F, m, torch.zeros_like(F)
        for q in range(len(s)):
            blk.srcs[q][0] = M[q]
        for q in range(5):
            blk.stage(q, n * dt, dt, {})
        return blk.F
    states = [torch.zeros((9,) + blk.shape, dtype=torch.float64, device=dev)]
    with torch.no_grad():
        for n in range(case["steps"]):
            states.append(step(states[-1], m, M, n))
    res = [F[:3, k, j, i].T - obs[n] for n, F in enumerate(states[:-1])]
    chi = 0.5 * sum((r * r).sum() for r in res)
    bar = torch.zeros_like(states[0])
    gm, gM = torch.zeros_like(m), torch.zeros_like(M)
    for n in reversed(range(case["steps"])):
        F = states[n].clone().requires_grad_(True)
        with torch.enable_grad():
            a, c, d = torch.autograd.grad(step(F, m, M, n), (F, m, M), bar, allow_unused=True)
        bar = a.clone()
        for c_ in range(3):
            bar[c_].index_put_((k, j, i), res[n][:, c_], accumulate=True)
        gm += c
        gM += d
    return {"misfit": chi.detach(), "material": gm, "moment": gM}
