"""The work that programs on this framework give it, as measurable cases.

A case is one of these kinds:

``frame``     A running simulation: ``Model.Step`` advances one frame (its
              force bins reset, the substeps, the copy of the state to the
              host) and the program goes on with the next frame.
``study``     A parameter study: a stored state is uploaded, advanced by a
              short run and copied back, then the next member of the study
              follows. The run packs the particles afresh each time.
``members``   A program written against the member functions of
              GPU_Implementation5 that drives every substep itself, kernel by
              kernel.
``ensemble``  Several indentation cases advanced together.
``train``     The learned projection fitted to labelled pairs.
``infer``     The learned projection evaluated on a batch of states.

Simulated blocks are the seeded lattices of ``icempm_b200.make_block`` with
the material of ``icempm_b200.configs``. ``crushed`` puts a crushed zone in
front of the indenter, as it is found late in a frame: crushed particles with
a spread of Jp_inv in sheared, compressed ice.

A simulation's outputs are the fields that a program on the GPU reads from
the device SoA (``SimParams.pts_array``) after the frame, each in the type in
which the form holds it: FP64 forms give float64; the FP32 forms hold
velocity, Bp, P, Q, the strain Fe - I and Jp_inv - 1 in float32 and the
position in fixed point, which float64 represents.
"""
from __future__ import annotations

import json
import math

import numpy as np
import torch

import icempm_b200 as im
from icempm_b200 import configs
from icempm_b200 import surrogate as sg
from icempm_b200.ensemble import Ensemble

FORMS = {"fp32": im.FORM_FP32, "fp64": im.FORM_FP64, "stepwise": im.FORM_FP64_STEPWISE}


def listed():
    return [
        # the benchmark's workload of 999,424 particles in the FP32 form: frames of a long run
        dict(name="frame_fp32_1m", kind="frame", form="fp32", gx=2048, gy=512, cx=1024, cy=244, h=4 / 2048,
             substeps=1000, crushed=False),
        # the 69,632-particle workload: a coarse run, about one tile per two SMs
        dict(name="frame_fp32_70k", kind="frame", form="fp32", gx=512, gy=128, cx=256, cy=68, h=4 / 512,
             substeps=1000, crushed=False),
        # a quick look at a small block on a grid that no tile divides: launches and latency
        dict(name="frame_fp32_14k_odd", kind="frame", form="fp32", gx=333, gy=101, cx=97, cy=37, h=4 / 512,
             substeps=500, crushed=False),
        # the 249,856-particle workload with its crushed zone, member after member of a study
        dict(name="study_fp32_250k_crushed", kind="study", form="fp32", gx=1024, gy=256, cx=512, cy=122, h=4 / 1024,
             substeps=300, crushed=True),
        # the 999,424-particle workload where double precision is wanted
        dict(name="frame_fp64_1m", kind="frame", form="fp64", gx=2048, gy=512, cx=1024, cy=244, h=4 / 2048,
             substeps=400, crushed=False),
        # double precision on an odd grid with a crushed zone
        dict(name="study_fp64_100k_odd", kind="study", form="fp64", gx=611, gy=203, cx=301, cy=83, h=4 / 512,
             substeps=300, crushed=True),
        # the form that a context has until another is asked for: the reference's three kernels
        dict(name="frame_stepwise_70k", kind="frame", form="stepwise", gx=512, gy=128, cx=256, cy=68, h=4 / 512,
             substeps=500, crushed=False),
        dict(name="frame_stepwise_1m", kind="frame", form="stepwise", gx=2048, gy=512, cx=1024, cy=244, h=4 / 2048,
             substeps=200, crushed=False),
        # a program that calls the member functions itself, as the reference's own Model::Step does
        dict(name="members_250k", kind="members", form="stepwise", gx=1024, gy=256, cx=512, cy=122, h=4 / 1024,
             substeps=100, crushed=False),
        # eight cases of the ensemble workload (20,000 to 500,000 particles each)
        dict(name="ensemble_fp32_8", kind="ensemble", form="fp32", cases=8, n_min=20000, n_max=500000, substeps=400),
        # the learned projection: the default batch of its trainer, and an evaluation on held-out states
        dict(name="train_64_tiles", kind="train", pairs=200000, tiles=64, steps=300),
        dict(name="infer_500k", kind="infer", rows=500000, warp=False),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the ranges above: blocks of 2,000 to 1,000,000
    particles of any aspect on grids of any size, each form; ensembles of 2
    to 8; batches of 4 to 296 tiles; batches of 1,000 to 500,000 rows."""
    kind = rng.choice(["frame", "frame", "study", "study", "frame", "members", "ensemble", "train", "infer"])
    if kind == "train":
        return dict(kind=kind, pairs=int(_log(rng, 1e4, 3e5)), tiles=int(_log(rng, 4, 296)), steps=rng.randint(100, 400))
    if kind == "infer":
        return dict(kind=kind, rows=int(_log(rng, 1e3, 5e5)), warp=rng.random() < 0.3)
    if kind == "ensemble":
        n_min = int(_log(rng, 1e4, 5e4))
        return dict(kind=kind, form=rng.choice(["fp32", "fp32", "fp64"]), cases=rng.randint(2, 8), n_min=n_min,
                    n_max=n_min * rng.randint(2, 8), substeps=rng.randint(150, 400))
    form = "stepwise" if kind == "members" else rng.choice(["fp32", "fp32", "fp64", "stepwise"])
    cells = _log(rng, 500, 250000)
    aspect = _log(rng, 1.5, 5.0)
    cy = max(12, int(round(math.sqrt(cells / aspect))))
    cx = max(16, int(round(cells / cy)))
    n = 4 * cx * cy
    most = {"fp32": 1000, "fp64": 400, "stepwise": 200}[form]
    substeps = max(40, min(most, int({"fp32": 1e9, "fp64": 4e8, "stepwise": 2e8}[form] / n)))
    if kind != "frame":
        substeps = min(substeps, 300 if kind == "study" else 100)
    return dict(kind=kind, form=form, gx=cx + rng.randint(60, 160) + cx // 2, gy=cy + rng.randint(30, 80) + cy // 4,
                cx=cx, cy=cy, h=4 / rng.choice([512, 768, 1024, 1536, 2048]), substeps=substeps,
                crushed=kind == "study" and rng.random() < 0.7)


# ------------------------------------------------------------------ scenes

def _particles(c):
    if c["kind"] == "ensemble":
        return sum(4 * x[1] * x[2] for x in _members(c))
    return 4 * c["cx"] * c["cy"]


def _members(c, seed=12345):
    return configs.c4_cases(c["cases"], seed, c["n_min"], c["n_max"])


def _block(c):
    """Indenter radius and height for a block: the workloads' 0.15 m at
    0.2 m, smaller for a block that is lower than theirs."""
    high = c["cy"] * c["h"]
    return min(0.15, 0.3 * high), min(0.2, 0.45 * high)


def _params(c):
    p = im.SimParams()
    p.Reset()
    r, _ = _block(c)
    # the workloads' time step is 2.56e-4 s per metre of cell size
    p.ParseString(json.dumps(dict(configs.MATERIAL, GridX=c["gx"], GridY=c["gy"], GridXDimension=c["gx"] * c["h"],
                                  InitialTimeStep=2.56e-4 * c["h"], IndDiameter=2 * r)))
    p.UpdateEveryNthStep = c["substeps"]
    return p


def _scene(c, seed):
    """(params, particle SoA in host pitches) of a case's block."""
    p = _params(c)
    soa = im.make_block(p, c["cx"], c["cy"], ind_y_above_floor=_block(c)[1], grain_size=0.05, seed=seed)
    p.nPtsPitch = im.pitch_elems(p.nPts)
    p.nGridPitch = im.pitch_elems(p.GridTotal)
    if c["crushed"]:
        S = im.SoA(soa, p.nPtsPitch, p.nPts)
        rng = np.random.default_rng(seed)
        # the zone: within 8 cells of the indenter's surface, thinning out
        d = np.hypot(S.pos[0] - p.indenter_x, S.pos[1] - p.indenter_y) - p.IndDiameter / 2
        near = np.exp(-np.maximum(d, 0) / (4 * p.cellsize))
        hit = rng.random(p.nPts) < 0.8 * near
        S.crushed[:] = hit
        S.Jp_inv[:] += hit * 0.01 * rng.standard_normal(p.nPts)
        S.Fe[0] -= 1e-3 * near
        S.Fe[:] += 3e-4 * near * rng.standard_normal((4, p.nPts))
        S.vel[0] = p.IndVelocity * near
    return p, soa


def _load(p, soa, form):
    m = im.Model()
    m.prms = p.copy()
    m.gpu.model = m
    m.gpu.cuda_allocate_arrays(p.GridTotal, p.nPts)
    m.gpu.tmp_transfer_buffer[: soa.size] = soa
    m.gpu.transfer_ponts_to_device()
    m.Prepare()
    m.gpu.set_form(FORMS[form])
    return m


class _Device:
    """A device array of the library as torch sees it."""

    def __init__(self, pointer, shape, kind):
        self.__cuda_array_interface__ = dict(data=(int(pointer), False), shape=shape, typestr=kind, version=3)


class _Fields:
    """A model's fields on the GPU, read on the model's own stream."""

    def __init__(self, m, form, bp=True, pq=True):
        p, self.fp32 = m.prms, form == "fp32"
        n, pitch = int(p.nPts), int(p.nPtsPitch)
        rows = torch.as_tensor(_Device(p.pts_array, (im.N_PTS_ARRAYS, pitch), "<f8"), device="cuda")
        self.stream = torch.cuda.ExternalStream(m.gpu.stream_handle())
        self.view = {"pos": rows[im.IDX_POSX: im.IDX_POSX + 2, :n], "vel": rows[im.IDX_VELX: im.IDX_VELX + 2, :n],
                     "Fe": rows[im.IDX_FE00: im.IDX_FE00 + 4, :n], "Jp": rows[im.IDX_JP_INV, :n],
                     "bins": torch.as_tensor(_Device(p.indenter_force_accumulator, (2 * p.n_indenter_subdivisions,),
                                                     "<f8"), device="cuda")}
        if bp:
            self.view["Bp"] = rows[im.IDX_BP00: im.IDX_BP00 + 4, :n]
        if pq:
            self.view["PQ"] = rows[im.IDX_P: im.IDX_Q + 1, :n]
        self.one = {"Fe": torch.tensor([1.0, 0.0, 0.0, 1.0], dtype=torch.float64, device="cuda")[:, None],
                    "Jp": torch.ones((), dtype=torch.float64, device="cuda")}
        self.wide = {k: torch.empty_like(self.view[k], memory_format=torch.contiguous_format) for k in self.one}
        self.out = {k: torch.empty(v.shape, dtype=torch.float32 if self.fp32 and k != "pos" else torch.float64,
                                   device="cuda") for k, v in self.view.items()}
        self.view["crushed"] = torch.as_tensor(_Device(p.pts_array, (n,), "|u1"), device="cuda")
        self.out["crushed"] = torch.empty(n, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

    def read(self):
        with torch.cuda.stream(self.stream):
            for k, v in self.view.items():
                if self.fp32 and k in self.one:
                    v = torch.sub(v, self.one[k], out=self.wide[k])
                self.out[k].copy_(v)
        return self.out


def _pairs(rows, seed):
    """Features and targets of the learned projection: trial states of
    crushed ice and what the projection changes in them (a smooth function of
    the features of the size met in the simulations)."""
    rng = np.random.default_rng(seed)
    x = np.empty((rows, sg.N_IN), dtype=np.float32)
    x[:, 0] = rng.normal(0.2, 1.0, rows)
    x[:, 1] = x[:, 0] - np.abs(rng.normal(0.0, 1.5, rows))
    x[:, 2] = rng.normal(0.1, 0.5, rows)
    x[:, 3] = rng.uniform(0.8, 2.5, rows)
    x[:, 4] = rng.uniform(1.0, 2.7, rows)
    x[:, 5] = 0.45
    gap = x[:, 0] - x[:, 1]
    keep = np.tanh(gap * x[:, 4]) / (1.0 + np.abs(x[:, 2]))
    y = np.stack([-0.5 * (gap - keep), 0.5 * (gap - keep), 0.05 * x[:, 3] * x[:, 2]], axis=1).astype(np.float32)
    return x, y


# ----------------------------------------------------------------- prepare

def prepare(case, seed):
    c = case
    if c["kind"] == "train":
        x, y = _pairs(c["pairs"], seed)
        net = sg.init_net(seed)
        sg.normalise(net, x, y)
        return dict(case=c, x=x, y=y, net=net, seed=seed & 0x7fffffff)
    if c["kind"] == "infer":
        x, y = _pairs(c["rows"], seed)
        net = sg.init_net(seed)
        sg.normalise(net, x, y)
        return dict(case=c, x=x, net=net)
    if c["kind"] == "ensemble":
        models = [configs.c4_model(x, seed=seed + k) for k, x in enumerate(_members(c))]
        e = Ensemble(FORMS[c["form"]])
        for m in models:
            m.prms.UpdateEveryNthStep = c["substeps"]
            e.add(m)
        return dict(case=c, models=models, ensemble=e,
                    fields=[_Fields(m, c["form"], bp=False, pq=False) for m in models])
    p, soa = _scene(c, seed)
    m = _load(p, soa, c["form"])
    s = dict(case=c, model=m, fields=_Fields(m, c["form"]))
    if c["kind"] == "study":
        # the stored state stays in one pinned buffer, frames arrive in another
        s["start"], s["prms"] = m.gpu.tmp_transfer_buffer, m.prms.copy()
        s["frame"] = torch.zeros(s["start"].size, dtype=torch.float64, pin_memory=True).numpy()
    return s


# --------------------------------------------------------------------- run

def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "train":
        net = state["net"].copy()
        loss = sg.train(net, state["x"], state["y"], steps=c["steps"], batch_tiles=c["tiles"], seed=state["seed"])
        return dict(net=net, loss=loss)
    if kind == "infer":
        return sg.infer(state["net"], state["x"], warp_form=c["warp"])
    if kind == "ensemble":
        for m in state["models"]:
            m.gpu.cuda_reset_indenter_force_accumulator()
        state["ensemble"].run(c["substeps"])
        for m in state["models"]:
            m.gpu.cuda_transfer_from_device()
        return [f.read() for f in state["fields"]]
    m = state["model"]
    g = m.gpu
    if kind == "frame":
        m.Step()
    elif kind == "study":
        m.prms.SimulationStep, m.prms.SimulationTime = 0, 0.0
        m.prms.indenter_x = state["prms"].indenter_x
        g.tmp_transfer_buffer = state["start"]
        g.transfer_ponts_to_device()
        g.tmp_transfer_buffer = state["frame"]
        m.Prepare()
        g.cuda_reset_indenter_force_accumulator()
        g.run_substeps(m.prms, c["substeps"])
        g.cuda_transfer_from_device()
    else:
        p = m.prms
        g.cuda_reset_indenter_force_accumulator()
        for k in range(c["substeps"]):
            p.SimulationTime += p.InitialTimeStep
            p.indenter_x = p.indenter_x_initial + p.SimulationTime * p.IndVelocity
            g.cuda_reset_grid()
            g.cuda_p2g()
            g.cuda_update_nodes(p.indenter_x, p.indenter_y)
            g.cuda_g2p(k == c["substeps"] - 1)
        p.SimulationStep += c["substeps"]
        g.cuda_transfer_from_device()
    return state["fields"].read()


# -------------------------------------------------------------------- work

def _stencil_nodes(cx, cy):
    return (cx + 2) * (cy + 2)


def work(case):
    """What a pass cannot do without. A substep reads and writes each
    particle's state once (FP32 form 36 bytes: position, strain, Jp_inv and
    flags; FP64 100 bytes; the step-wise form also velocity and Bp, which its
    kernels hand on through memory: 192 bytes) and each node that a particle
    reaches once (mass and momentum). About 330 operations per particle and
    substep: both transfers over 9 nodes, the strain update and the stress. A
    frame also copies the 128-byte record of each particle to the host, and a
    study uploads it."""
    c = case
    mlp = 2.0 * (sg.N_IN * sg.N_HID + sg.N_HID * sg.N_HID + sg.N_HID * sg.N_OUT)
    if c["kind"] == "train":
        rows = 128.0 * c["tiles"] * c["steps"]
        return dict(bytes=4.0 * (sg.N_IN + sg.N_OUT) * (c["pairs"] + rows), flops=3 * mlp * rows)
    if c["kind"] == "infer":
        return dict(bytes=4.0 * (sg.N_IN + sg.N_OUT) * c["rows"], flops=mlp * c["rows"])
    n = _particles(c)
    nodes = (sum(_stencil_nodes(x[1], x[2]) for x in _members(c)) if c["kind"] == "ensemble"
             else _stencil_nodes(c["cx"], c["cy"]))
    particle, node = {"fp32": (36, 12), "fp64": (100, 24), "stepwise": (192, 24)}[c["form"]]
    copies = 128.0 * n * (2 if c["kind"] == "study" else 1)
    return dict(bytes=c["substeps"] * (2.0 * particle * n + 2.0 * node * nodes) + copies, flops=330.0 * n * c["substeps"])


# ------------------------------------------------------------------- exact

def _project(P, F, Jp, on):
    """The Drucker-Prager map of the particles `on`: F_new = U diag(r) U^T F
    with U the eigenvectors of F F^T."""
    b00, b11 = F[0] * F[0] + F[1] * F[1], F[2] * F[2] + F[3] * F[3]
    b01, hd = F[0] * F[2] + F[1] * F[3], 0.5 * (F[0] * F[0] + F[1] * F[1] - F[2] * F[2] - F[3] * F[3])
    J = F[0] * F[3] - F[1] * F[2]
    rho, mean = torch.sqrt(hd * hd + b01 * b01), 0.5 * (b00 + b11)
    p = -0.5 * P.kappa * (J * J - 1)
    q = 2 * P.mu / J * rho
    hydro = (p < -P.DP_threshold_p) | (Jp < 1)
    je = math.sqrt(2 * P.DP_threshold_p / P.kappa + 1)
    qn = torch.where(p > P.IceCompressiveStrength, torch.zeros_like(p),
                     torch.clamp((p + P.DP_threshold_p) * P.DP_tan_phi, max=P.IceShearStrength))
    cone = ~hydro & (q >= qn)
    new_rho = torch.where(cone, qn * J / (2 * P.mu), rho)
    s0, s1 = mean + rho, mean - rho  # squared singular values
    r0 = torch.where(hydro, torch.sqrt(je / s0), torch.sqrt((mean + new_rho) / s0))
    r1 = torch.where(hydro, torch.sqrt(je / s1), torch.sqrt((mean - new_rho) / s1))
    a, d = 0.5 * (r0 + r1), 0.5 * (r0 - r1)
    d = torch.where(rho > 0, d / torch.where(rho > 0, rho, torch.ones_like(rho)), torch.zeros_like(rho))
    m00, m01, m11 = a + d * hd, d * b01, a - d * hd
    new = torch.stack([m00 * F[0] + m01 * F[2], m00 * F[1] + m01 * F[3], m01 * F[0] + m11 * F[2],
                       m01 * F[1] + m11 * F[3]])
    on = on & (hydro | cone)
    return torch.where(on, new, F), torch.where(on & hydro, Jp * (je / J), Jp)


def _outside(P, g, p, q):
    """The failure surfaces of the grains (residues g), before crushing."""
    pmax = P.IceCompressiveStrength * (1 + P.GrainVariability * 0.05 * (-10 + g[0]))
    pmin = -P.IceTensileStrength * (1 + P.GrainVariability * 0.033 * (-15 + g[1]))
    qmax = P.IceShearStrength * (1 + P.GrainVariability * 0.1 * (-10 + g[2]))
    beta = -pmin / pmax
    msq = 4 * qmax * qmax * (1 + 2 * beta) / (pmax * (1 + beta)) ** 2
    tension = (p < -3e6) | (q > 2 * torch.sqrt(-pmax * pmin) * qmax / (pmax - pmin) * (p + 3e6) / 3e6)
    return torch.where(p < 0, tension, (1 + 2 * beta) * q * q + msq * (p + beta * pmax) * (p - pmax) > 0)


def _simulate(P, soa, n):
    """n substeps of the reference's method in float64 with plain torch."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    S = im.SoA(soa, int(P.nPtsPitch), int(P.nPts))
    up = lambda a: torch.from_numpy(np.array(a)).to(dev)  # noqa: E731
    x, v, F, B, Jp, crushed = up(S.pos), up(S.vel), up(S.Fe), up(S.Bp), up(S.Jp_inv), up(S.crushed) != 0
    grain = up(S.grain).to(torch.int64)
    res = [(grain % 21).double(), ((grain + 3) % 30).double(), ((grain + 4) % 11).double()]
    GX, GY, h, dt, m = P.GridX, P.GridY, P.cellsize, P.InitialTimeStep, P.ParticleMass
    gx = (torch.arange(GX * GY, device=dev) % GX).double()
    gy = (torch.arange(GX * GY, device=dev) // GX).double()
    nsub = P.n_indenter_subdivisions
    bins = torch.zeros(2 * nsub, dtype=torch.float64, device=dev)
    reach = (gy * h - P.indenter_y) ** 2 < P.IndRSq
    rows = torch.nonzero(reach).reshape(-1)  # nodes in the indenter's band
    cols = gx[rows], gy[rows]
    floor, top = gy <= 2, gy >= GY - 3
    left, right = gx <= 2, gx >= GX - 3
    t, PQ = P.SimulationTime, None
    for _ in range(n):
        t += dt
        ind_x = P.indenter_x_initial + t * P.IndVelocity
        X = x / h
        base = torch.trunc(X - 0.5)
        f = X - base
        w = [0.5 * (1.5 - f) ** 2, 0.75 - (f - 1) ** 2, 0.5 * (f - 0.5) ** 2]
        node = base[1].long() * GX + base[0].long()
        J = F[0] * F[3] - F[1] * F[2]
        b00, b11, b01 = F[0] * F[0] + F[1] * F[1], F[2] * F[2] + F[3] * F[3], F[0] * F[2] + F[1] * F[3]
        s1, s2, half = P.mu / J, P.kappa * (J * J - 1), 0.5 * (b00 + b11)
        k = dt * P.ParticleVolume * P.Dp_inv
        A = [m * B[0] - k * (s1 * (b00 - half) + s2), m * B[1] - k * s1 * b01,
             m * B[2] - k * s1 * b01, m * B[3] - k * (s1 * (b11 - half) + s2)]
        mass, mom = torch.zeros(GX * GY, dtype=torch.float64, device=dev), None
        mx, my = torch.zeros_like(mass), torch.zeros_like(mass)
        for i in range(3):
            d0 = (i - f[0]) * h
            u0, u1 = m * v[0] + A[0] * d0, m * v[1] + A[2] * d0
            for j in range(3):
                W, d1 = w[i][0] * w[j][1], (j - f[1]) * h
                at = node + (j * GX + i)
                mass.index_add_(0, at, W * m)
                mx.index_add_(0, at, W * (u0 + A[1] * d1))
                my.index_add_(0, at, W * (u1 + A[3] * d1))
        some = mass > 0
        safe = torch.where(some, mass, torch.ones_like(mass))
        vx, vy = mx / safe, torch.where(some, my / safe - dt * P.Gravity, torch.zeros_like(my))
        vmax, speed = 0.5 * h / dt, torch.sqrt(vx * vx + vy * vy)
        fast = torch.where(speed > vmax, vmax / torch.where(speed > 0, speed, torch.ones_like(speed)),
                           torch.ones_like(speed))
        vx, vy = vx * fast, vy * fast
        # contact with the indenter
        n0, n1 = cols[0] * h - ind_x, cols[1] * h - P.indenter_y
        z = n0 * n0 + n1 * n1
        inside = (z < P.IndRSq) & some[rows]
        z = torch.where(z > 0, torch.sqrt(z), torch.ones_like(z))
        n0, n1 = n0 / z, n1 / z
        a, b = vx[rows], vy[rows]
        vn = (a - P.IndVelocity) * n0 + b * n1
        hit = inside & (vn < 0)
        na, nb = torch.where(hit, a - n0 * vn, a), torch.where(hit, b - n1 * vn, b)
        at = ((torch.atan2(n0, n1) + math.pi) * (nsub / (2 * math.pi))).long().clamp(0, nsub - 1)
        force = torch.stack([(a - na) * mass[rows] / dt, (b - nb) * mass[rows] / dt], dim=1) * hit[:, None]
        bins.view(nsub, 2).index_add_(0, at, force)
        vx[rows], vy[rows] = na, nb
        vx[floor] = 0
        vy[floor] = 0
        vy = torch.where(top & (vy > 0), torch.zeros_like(vy), vy)
        vx = torch.where((left & (vx < 0)) | (right & (vx > 0)), torch.zeros_like(vx), vx)
        v, B = torch.zeros_like(v), torch.zeros_like(B)
        for i in range(3):
            for j in range(3):
                W, at = w[i][0] * w[j][1], node + (j * GX + i)
                a, b = W * vx[at], W * vy[at]
                v[0] += a
                v[1] += b
                d0, d1 = (i - f[0]) * (4 / h), (j - f[1]) * (4 / h)
                B[0] += a * d0
                B[1] += a * d1
                B[2] += b * d0
                B[3] += b * d1
        x = x + dt * v
        F = torch.stack([F[0] + dt * (B[0] * F[0] + B[1] * F[2]), F[1] + dt * (B[0] * F[1] + B[1] * F[3]),
                         F[2] + dt * (B[2] * F[0] + B[3] * F[2]), F[3] + dt * (B[2] * F[1] + B[3] * F[3])])
        J = F[0] * F[3] - F[1] * F[2]
        hd, b01 = 0.5 * (F[0] * F[0] + F[1] * F[1] - F[2] * F[2] - F[3] * F[3]), F[0] * F[2] + F[1] * F[3]
        p, q = -0.5 * P.kappa * (J * J - 1), 2 * P.mu / J * torch.sqrt(hd * hd + b01 * b01)
        PQ = torch.stack([p, q])
        crushed = crushed | _outside(P, res, p, q)
        F, Jp = _project(P, F, Jp, crushed)
    return dict(pos=x, vel=v, Fe=F, Bp=B, Jp=Jp, PQ=PQ, bins=bins, crushed=crushed.to(torch.uint8))


def _as_form(out, form, keep=None):
    if form == "fp32":  # the strain and Jp_inv - 1, as the form holds them
        out["Fe"] = out["Fe"] - torch.tensor([1.0, 0.0, 0.0, 1.0], dtype=torch.float64, device=out["Fe"].device)[:, None]
        out["Jp"] = out["Jp"] - 1
    # whether a particle at its failure surface is crushed by now is no computed number
    return {k: (None if k == "crushed" else v) for k, v in out.items() if keep is None or k in keep}


def _sampled(seed, step, rows, n):
    """The trainer's batch: a 32-bit mix of the seed, the step and the row."""
    u = np.uint32
    with np.errstate(over="ignore"):
        h = u(seed) ^ (u(step) * u(0x9E3779B9)) ^ (np.arange(rows, dtype=u) * u(0x85EBCA6B))
        h ^= h >> u(16)
        h *= u(0x7feb352d)
        h ^= h >> u(15)
        h *= u(0x846ca68b)
        h ^= h >> u(16)
    return (h % u(n)).astype(np.int64)


def exact(case, seed):
    c = case
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if c["kind"] in ("train", "infer"):
        rows = c["pairs"] if c["kind"] == "train" else c["rows"]
        x, y = _pairs(rows, seed)
        net = sg.init_net(seed)
        sg.normalise(net, x, y)
        w = {k: torch.from_numpy(v.astype(np.float64)).to(dev) for k, v in sg.views(net).items()}
        X = (torch.from_numpy(x).to(dev).double() - w["x_mu"]) / w["x_sd"]
        names = ["W1", "b1", "W2", "b2", "W3", "b3"]
        gelu = lambda z: torch.nn.functional.gelu(z, approximate="tanh")  # noqa: E731
        net_of = lambda a: gelu(gelu(a @ w["W1"].T + w["b1"]) @ w["W2"].T + w["b2"]) @ w["W3"].T + w["b3"]  # noqa: E731
        if c["kind"] == "infer":
            return net_of(X) * w["y_sd"] + w["y_mu"]
        Y = (torch.from_numpy(y).to(dev).double() - w["y_mu"]) / w["y_sd"]
        for k in names:
            w[k].requires_grad_(True)
        m, v = {k: torch.zeros_like(w[k]) for k in names}, {k: torch.zeros_like(w[k]) for k in names}
        loss = []
        for s in range(c["steps"]):
            at = torch.from_numpy(_sampled(seed & 0x7fffffff, s, 128 * c["tiles"], rows)).to(dev)
            e = ((net_of(X[at]) - Y[at]) ** 2).mean()
            loss.append(e.detach())
            grads = torch.autograd.grad(e, [w[k] for k in names])
            frac = s / (c["steps"] - 1) if c["steps"] > 1 else 0.0
            lr = 2e-3 * (0.05 + 0.475 * (1 + math.cos(math.pi * frac)))
            with torch.no_grad():
                for k, g in zip(names, grads):
                    m[k] = 0.9 * m[k] + 0.1 * g
                    v[k] = 0.999 * v[k] + 0.001 * g * g
                    w[k] -= lr * (m[k] / (1 - 0.9 ** (s + 1))) / (torch.sqrt(v[k] / (1 - 0.999 ** (s + 1))) + 1e-8)
        flat = [w[k].detach().reshape(-1) for k in names + ["x_mu", "x_sd", "y_mu", "y_sd"]]
        return dict(net=torch.cat(flat), loss=torch.stack(loss))
    if c["kind"] == "ensemble":
        got = []
        for k, (over, cx, cy, ind_y) in enumerate(_members(c)):
            gx, gy = configs.C4["grid"]
            p = im.SimParams()
            p.Reset()
            p.ParseString(json.dumps(dict(configs.MATERIAL, GridX=gx, GridY=gy, GridXDimension=configs.C4["dim"],
                                          InitialTimeStep=configs.C4["dt"], **over)))
            soa = im.make_block(p, cx, cy, ind_y_above_floor=ind_y, grain_size=0.05, seed=seed + k)
            p.nPtsPitch = im.pitch_elems(p.nPts)
            got.append(_as_form(_simulate(p, soa, c["substeps"]), c["form"],
                                ("pos", "vel", "Fe", "Jp", "bins", "crushed")))
        return got
    p, soa = _scene(c, seed)
    return _as_form(_simulate(p, soa, c["substeps"]), c["form"])
