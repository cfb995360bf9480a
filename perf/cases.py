"""Cases that time the reactive-transport library through its public binding (clb.py).

A case is a program's unit of work between two looks at its fields: a number of steps on one
domain (or on an ensemble of domains) and the fields read back to pinned host memory. The kinds:

  flow       D3Q19 steps of a sphere pack at a fixed pressure drop, then the velocity
  solve      the flow of a sphere pack from rest to the settled-energy criterion, then the velocity
  transport  D3Q7 steps of 1 to 8 species with a rate law (decay, Monod, dual Monod with two
             biofilm microbes), then every concentration and biomass field
  coupled    an update interval of the coupled run: transport, dual-Monod kinetics, the biofilm
             automaton every iteration, the flow re-solved at its end
  chemistry  transport of the 5-component 12-species tableau in a rough fracture with equilibrium
             speciation of every voxel (Newton-Raphson, or the trained surrogate) and a growing
             mineral, then the sealing update
  ensemble   steps of many small uneven domains advanced as one batch

Sizes follow the repository's own configurations (workloads.py: packs of 64x32x32, 256x128x128 and
256^3, the 192^3 fracture, 96 uneven domains) and lie around them. Every input is made from the
seed: grains, diffusivities, rate constants, biomass.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "complab3d-gems_b200"))

import clb  # noqa: E402
import workloads  # noqa: E402

PRECISION = {"f64": clb.F64, "f32": clb.F32, "f16s": clb.F16S}
STORED = {"f64": 8, "f32": 4, "f16s": 2}
LAWS = {"none": clb.LAW_NONE, "decay": clb.LAW_DECAY, "monod": clb.LAW_MONOD, "dual": clb.LAW_DUAL_MONOD}
DELTA_P = 1e-4
FLOW_BEFORE = 100   # flow steps from rest before a transport case takes its velocity
WALL, PORE, ROCK = 1, 2, 0


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one small domain of a parameter sweep, stepped by itself: a step is a few microseconds
        # of work, so launches and latency count
        dict(name="flow_small_f32", kind="flow", nx=48, ny=24, nz=24, porosity=0.40, rmin=2.0, rmax=4.0, tau=0.8,
             precision="f32", steps=200),
        # the smallest configuration's flow, in the reference's FP64, from rest to the criterion
        dict(name="solve_64x32x32_f64", kind="solve", nx=64, ny=32, nz=32, porosity=0.40, rmin=4.0, rmax=4.0,
             tau=0.8, precision="f64", eps=1e-6),
        # the flow-only configuration (permeability of a tight pack)
        dict(name="flow_256x128x128_f32", kind="flow", nx=256, ny=128, nz=128, porosity=0.35, rmin=3.0, rmax=8.0,
             tau=0.7, precision="f32", steps=100),
        # an odd-sized scan in the compressed storage
        dict(name="flow_odd_f16s", kind="flow", nx=197, ny=143, nz=131, porosity=0.38, rmin=3.0, rmax=7.0, tau=0.9,
             precision="f16s", steps=100),
        # a large scan, far beyond the L2 cache
        dict(name="flow_384x256x256_f32", kind="flow", nx=384, ny=256, nz=256, porosity=0.35, rmin=3.0, rmax=8.0,
             tau=0.7, precision="f32", steps=100),
        # the smallest configuration's transport: one decaying solute, FP64
        dict(name="transport_64x32x32_f64", kind="transport", nx=64, ny=32, nz=32, porosity=0.40, rmin=4.0, rmax=4.0,
             tau=0.8, species=1, law="decay", precision="f64", steps=400),
        # ordinary multi-species transport on an odd-sized pack
        dict(name="transport_odd_3_f32", kind="transport", nx=129, ny=97, nz=113, porosity=0.42, rmin=3.0, rmax=6.0,
             tau=0.8, species=3, law="monod", precision="f32", steps=100),
        # the largest configuration's transport: 8 species, two biofilm microbes
        dict(name="transport_256cube_8_f32", kind="transport", nx=256, ny=256, nz=256, porosity=0.40, rmin=3.0,
             rmax=8.0, tau=0.8, species=8, law="dual", precision="f32", steps=100),
        # an update interval of the coupled run at half the configuration's edge, biofilm spreading
        dict(name="coupled_128cube_8_f32", kind="coupled", nx=128, ny=128, nz=128, porosity=0.40, rmin=3.0, rmax=8.0,
             tau=0.8, species=8, precision="f32", steps=100),
        # precipitation with equilibrium chemistry, solved exactly and by the learned surrogate
        dict(name="chemistry_newton", kind="chemistry", nx=128, ny=128, nz=96, aperture=12.0, solver="newton",
             steps=20),
        dict(name="chemistry_surrogate", kind="chemistry", nx=96, ny=96, nz=64, aperture=12.0, solver="surrogate",
             steps=20),
        # the parameter sweep: 96 uneven domains as one batch
        dict(name="ensemble_96", kind="ensemble", domains=96, steps=100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flow", "flow", "solve", "transport", "transport", "transport", "coupled", "chemistry", "ensemble"])
    rmin = rng.choice([2.0, 3.0, 4.0])
    pack = dict(porosity=round(rng.uniform(0.32, 0.50), 3), rmin=rmin, rmax=rmin + rng.choice([0.0, 2.0, 4.0]),
                tau=round(rng.uniform(0.6, 1.0), 3))
    if kind == "flow":
        return dict(kind=kind, nx=_log(rng, 32, 320), ny=_log(rng, 24, 200), nz=_log(rng, 24, 200), **pack,
                    precision=rng.choice(["f32", "f32", "f64", "f16s"]), steps=100)
    if kind == "solve":
        return dict(kind=kind, nx=_log(rng, 32, 96), ny=_log(rng, 24, 64), nz=_log(rng, 24, 64), **pack,
                    precision=rng.choice(["f32", "f64"]), eps=1e-6)
    if kind == "transport":
        return dict(kind=kind, nx=_log(rng, 32, 224), ny=_log(rng, 24, 160), nz=_log(rng, 24, 160), **pack,
                    species=rng.choice([1, 2, 3, 4, 5, 8]), law=rng.choice(["none", "decay", "monod", "dual", "dual"]),
                    precision=rng.choice(["f32", "f32", "f64", "f16s"]), steps=100)
    if kind == "coupled":
        return dict(kind=kind, nx=_log(rng, 64, 144), ny=_log(rng, 48, 128), nz=_log(rng, 48, 128), **pack,
                    species=rng.choice([3, 4, 8]), precision="f32", steps=100)
    if kind == "chemistry":
        return dict(kind=kind, nx=_log(rng, 48, 128), ny=_log(rng, 48, 112), nz=_log(rng, 40, 96),
                    aperture=round(rng.uniform(8.0, 16.0), 1), solver=rng.choice(["newton", "surrogate"]), steps=20)
    return dict(kind=kind, domains=_log(rng, 8, 96), steps=100)


# ------------------------------------------------------------------ inputs from the seed
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _rng(seed, salt):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, salt])


def _ghosts(inner):
    """The two ghost x-planes a run adds to a geometry: copies of the first and last plane."""
    return np.concatenate([inner[:1], inner, inner[-1:]]).astype(np.int8)


def _sphere_pack(rng, nx, ny, nz, porosity, rmin, rmax):
    """Overlapping spheres of radius U[rmin, rmax] at uniform centres, as many as leave `porosity`
    open on average, confining walls on the four side faces; [nx + 2][ny][nz]."""
    mean = 4.0 / 3.0 * math.pi * float(np.mean(np.linspace(rmin, rmax, 65) ** 3))
    m = rmax  # centres reach one radius outside, so the faces are as dense as the inside
    volume = (nx + 2 * m) * (ny + 2 * m) * (nz + 2 * m)
    n = max(1, int(round(-math.log(porosity) * volume / mean)))
    dev = _device()
    c = torch.from_numpy(rng.uniform(0.0, 1.0, (n, 3)) * np.array([nx + 2 * m, ny + 2 * m, nz + 2 * m]) - m).to(dev)
    r2 = torch.from_numpy(rng.uniform(rmin, rmax, n) ** 2).to(dev)
    base = torch.round(c).long()
    grain = torch.zeros(nx * ny * nz, dtype=torch.bool, device=dev)
    R = int(math.ceil(rmax)) + 1
    ax = torch.arange(-R, R + 1, device=dev)
    off = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    off = off[(off * off).sum(1) <= (rmax + 1.0) ** 2]
    chunk = max(1, (1 << 22) // n)
    for k in range(0, off.shape[0], chunk):
        p = base[:, None, :] + off[None, k:k + chunk, :]
        d = p - c[:, None, :]
        ok = (d * d).sum(-1) <= r2[:, None]
        for a, s in enumerate((nx, ny, nz)):
            ok &= (p[..., a] >= 0) & (p[..., a] < s)
        q = p[ok]
        grain[(q[:, 0] * ny + q[:, 1]) * nz + q[:, 2]] = True
    mat = torch.where(grain, WALL, PORE).to(torch.int8).reshape(nx, ny, nz)
    mat[:, 0], mat[:, -1], mat[:, :, 0], mat[:, :, -1] = WALL, WALL, WALL, WALL
    return _ghosts(mat.cpu().numpy())


def _fracture(rng, nx, ny, nz, aperture):
    """A rough fracture across z: two rock surfaces `aperture` apart around a smooth random mid-plane."""
    kx, ky = np.meshgrid(np.fft.fftfreq(nx) * nx, np.fft.fftfreq(ny) * ny, indexing="ij")
    k = np.sqrt(kx * kx + ky * ky)
    amp = np.where(k > 0, np.maximum(k, 1.0) ** -1.8, 0.0)
    h = np.fft.ifft2(amp * np.exp(2j * np.pi * rng.uniform(size=(nx, ny)))).real
    mid = nz / 2 + h / max(1e-12, np.abs(h).max()) * 0.25 * nz
    z = np.arange(nz)
    inner = np.where(np.abs(z[None, None, :] - mid[:, :, None]) <= 0.5 * aperture, PORE, ROCK)
    return _ghosts(inner)


def _species(rng, n):
    out = []
    for k in range(n):
        d = float(rng.uniform(0.02, 0.2))
        fed = k < 3
        out.append(dict(omega_pore=workloads.omega_from_d(d), omega_biofilm=workloads.omega_from_d(0.5 * d), mobile=1,
                        left_type=clb.DIRICHLET if fed else clb.NEUMANN, right_type=clb.NEUMANN,
                        left_bc=float(rng.uniform(0.5, 1.0)) if fed else 0.0, c0=float(rng.uniform(0.05, 0.2))))
    return out


def _law(rng, law, n):
    if law == "decay":
        return list(rng.uniform(5e-4, 2e-3, n))
    if law == "monod":
        return list(10.0 ** rng.uniform(-6, -3, n)) + [0.1] * n
    return [1e-4, 0.1, 0.4, 1e-6] if law == "dual" else []


def _inputs(case, seed):
    """Everything of a pack case that the seed decides."""
    rng = _rng(seed, 1)
    mat = _sphere_pack(rng, case["nx"], case["ny"], case["nz"], case["porosity"], case["rmin"], case["rmax"])
    x = dict(mat=mat, shape=mat.shape, bio_codes=(), perm_ratio=(), biomass=None)
    law = "dual" if case["kind"] == "coupled" else case.get("law", "none")
    if law == "dual":
        flat = mat.reshape(-1)
        pore = np.flatnonzero(flat == PORE)
        free = pore
        if case["kind"] == "coupled":  # colonies that can spread (see workloads.pack256cube_8species)
            free = np.flatnonzero(workloads.percolating_pores(flat, mat.shape))
        seeded = rng.choice(free, size=max(2, min(free.size, int(0.02 * pore.size))), replace=False)
        half = seeded.size // 2
        flat[seeded[:half]], flat[seeded[half:]] = 3, 4
        bio = np.zeros((2, flat.size))
        full = rng.uniform(50.0, 100.0, flat.size) if case["kind"] == "coupled" else np.full(flat.size, 50.0)
        for m in range(2):
            bio[m, flat == 3 + m] = full[flat == 3 + m]
        x.update(bio_codes=(3, 4), perm_ratio=(0.1, 0.1), biomass=bio)
    if "species" in case:
        x.update(species=_species(rng, case["species"]), law=law, params=_law(rng, law, case["species"]))
    return x


def _chemistry_inputs(case, seed):
    rng = _rng(seed, 2)
    mat = _fracture(rng, case["nx"], case["ny"], case["nz"], case["aperture"])
    S, logK, comp = workloads.tableau_5x12(1004)
    ns = S.shape[0]
    sp = [dict(omega_pore=1 / 0.9, omega_biofilm=1 / 0.9, mobile=1, left_type=clb.DIRICHLET, right_type=clb.NEUMANN,
               left_bc=float(10 ** rng.uniform(-5, -3.5)), c0=float(10 ** rng.uniform(-6, -4))) for _ in range(ns)]
    sp[0].update(c0=3e-3, left_bc=2e-3)
    for s in (1, 2):
        sp[s].update(c0=2e-3, left_bc=2e-3)
    sp.append(dict(omega_pore=1.0, omega_biofilm=1.0, mobile=0, left_type=clb.NEUMANN, right_type=clb.NEUMANN, left_bc=0.0,
                   c0=0.0))
    nu = [0.0] * (ns + 1)
    nu[1] = nu[2] = 1.0
    deposit = rng.uniform(0.0, 1e-3, mat.size) * (mat.reshape(-1) == PORE)
    return dict(mat=mat, shape=mat.shape, S=S, logK=logK, comp=comp, species=sp, mineral=[2e-6, -6.0, ns] + nu, ns=ns,
                full=1e-3, deposit=deposit, tau=0.8)


def _ensemble_inputs(case, seed):
    rng, sizes = _rng(seed, 3), _rng(case["domains"], 4)  # the sizes belong to the case, not to the seed
    doms = []
    for _ in range(case["domains"]):
        nx, nyz = int(sizes.choice([32, 48, 64, 96])), int(sizes.choice([24, 32, 48]))
        mat = _sphere_pack(rng, nx, nyz, nyz, float(rng.uniform(0.3, 0.5)), 2.0, 4.0)
        species = []
        for _ in range(3):
            d = float(rng.uniform(0.05, 0.2))
            species.append(dict(omega_pore=workloads.omega_from_d(d), omega_biofilm=workloads.omega_from_d(0.5 * d),
                                mobile=1, left_type=clb.DIRICHLET, right_type=clb.NEUMANN, left_bc=1.0, c0=0.0))
        doms.append(dict(mat=mat, shape=mat.shape, tau=float(rng.uniform(0.6, 1.0)), species=species,
                         params=list(10.0 ** rng.uniform(-6, -3, 3)) + [0.1] * 3))
    return doms


# ------------------------------------------------------------------ the program
def _pinned(shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def _domain(x, tau, precision):
    nx, ny, nz = x["shape"]
    return clb.Domain(x["mat"].reshape(-1), nx, ny, nz, tau, flow_precision=PRECISION[precision],
                      ade_precision=PRECISION[precision], bio_codes=x.get("bio_codes", ()),
                      perm_ratio=x.get("perm_ratio", ()))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "chemistry":
        x = _chemistry_inputs(case, seed)
        D = _domain(x, x["tau"], "f32")
        D.flow_init(DELTA_P)
        D.flow_step(FLOW_BEFORE)
        D.ade_init(x["species"])
        D.couple_velocity()
        D.speciation_setup(x["S"], x["logK"], x["comp"], tol=1e-10)
        D.set_speciation_mode(clb.SPEC_NR)
        D.set_abiotic_kinetics(clb.LAW_MINERAL, x["mineral"], 0)
        D.set_concentration(x["ns"], x["deposit"])
        D.precip_setup(x["ns"], x["full"])
        if case["solver"] == "surrogate":
            D.surrogate_train([-6.0] * x["ns"], [-2.5] * x["ns"], n_samples=100000, epochs=6, seed=1 + int(seed) % 1000,
                              from_domain=True, jitter=0.6)
            D.surrogate_set_check(0.02, 2, 1e-6)
            D.set_speciation_mode(clb.SPEC_MLP_NR)
        D.sync()
        return dict(case=case, D=D, out=_pinned((x["ns"] + 1, D.N)))
    if kind == "ensemble":
        doms = _ensemble_inputs(case, seed)
        Ds = []
        for x in doms:
            D = _domain(x, x["tau"], "f32")
            D.flow_init(DELTA_P)
            D.flow_step(20)
            D.ade_init(x["species"])
            D.couple_velocity()
            D.set_kinetics(clb.LAW_MONOD, x["params"], 1.0)
            D.sync()
            Ds.append(D)
        B = clb.Batch(Ds)
        B.schedule(persistent=False, staged_flow=True)
        n = sum(D.N for D in Ds)
        return dict(case=case, Ds=Ds, B=B, u=_pinned(3 * n, torch.float32), out=_pinned((3, n)))
    x = _inputs(case, seed)
    D = _domain(x, case["tau"], case["precision"])
    D.flow_init(DELTA_P)
    if kind in ("flow", "solve"):
        D.sync()
        return dict(case=case, D=D, u=_pinned(3 * D.N, torch.float64 if case["precision"] == "f64" else torch.float32))
    if kind == "coupled":
        D.flow_solve(20000, 1e-6, allow_unconverged=True)
    else:
        D.flow_step(FLOW_BEFORE)
    D.ade_init(x["species"])
    D.couple_velocity()
    M = 0
    if x["biomass"] is not None:
        D.set_biomass(x["biomass"])
        M = 2
    D.set_kinetics(LAWS[x["law"]], x["params"], 1.0)
    if kind == "coupled":
        D.ca_setup(100.0, 0.1, 1 + int(seed) % 1000)
    D.sync()
    return dict(case=case, D=D, M=M, out=_pinned((case["species"] + M, D.N)))


def _fields(D, out, species, microbes=0):
    """Every concentration, then every biomass field, into the rows of a pinned array."""
    L = clb.lib()
    for s in range(species):
        D._check(L.clb_get_field(D.h, clb.FIELD_CONCENTRATION, s, clb.C.c_void_p(out[s].data_ptr()), 0))
    for m in range(microbes):
        D._check(L.clb_get_field(D.h, clb.FIELD_BIOMASS, m, clb.C.c_void_p(out[species + m].data_ptr()), 0))
    return out


def _velocity(D, u):
    a = u.numpy()
    D.velocity(dtype=a.dtype, out=a)
    return u


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "flow":
        state["D"].flow_step(case["steps"])
        return _velocity(state["D"], state["u"])
    if kind == "solve":
        state["D"].flow_init(DELTA_P)
        state["D"].flow_solve(200000, case["eps"])
        return _velocity(state["D"], state["u"])
    if kind == "transport":
        state["D"].ade_step(case["steps"])
        return _fields(state["D"], state["out"], case["species"], state["M"])
    if kind == "coupled":
        D = state["D"]
        D.run(case["steps"], ca=True, ade_update_interval=1, resolve_every=case["steps"], flow_max_iterations=20000,
              flow_eps=1e-6)
        # single precision, as the lattices hold them
        return dict(fields=_fields(D, state["out"], case["species"], 2).float(), material=D.material())
    if kind == "chemistry":
        D = state["D"]
        D.ade_step(case["steps"])
        D.geometry_update()
        return _fields(D, state["out"], state["out"].shape[0]).float()
    state["B"].step(case["steps"])
    at = 0
    for D in state["Ds"]:
        _velocity(D, state["u"][3 * at:3 * (at + D.N)])
        _fields(D, state["out"][:, at:at + D.N], 3)
        at += D.N
    return dict(u=state["u"], c=state["out"])


# ------------------------------------------------------------------ what a pass cannot do without
def _open(case):
    inner = max(1, case["ny"] - 2) * max(1, case["nz"] - 2)
    return (case["nx"] + 2) * inner * case["porosity"]


def work(case):
    """Every population of every step read and written once, the per-node inputs of a step (velocity,
    material) read once, and the fields written once. Operations: about 250 per flow node, 40 per
    species node, and 40 Newton-Raphson iterations of 1000 operations per speciated voxel."""
    kind = case["kind"]
    if kind == "ensemble":
        n = case["domains"] * 62 * (24.0 ** 2 + 32.0 ** 2 + 48.0 ** 2) / 3
        k = 0.35 * n
        per = 2 * 19 * 4 + 3 * 2 * 7 * 4 + 13
        return dict(bytes=case["steps"] * k * per + n * (12 + 24), flops=case["steps"] * k * (250 + 3 * 40))
    if kind == "chemistry":
        n = (case["nx"] + 2) * case["ny"] * case["nz"]
        k = (case["nx"] + 2) * case["ny"] * case["aperture"]
        return dict(bytes=case["steps"] * k * (12 * 2 * 7 * 4 + 13 + 16) + n * 13 * 8,
                    flops=case["steps"] * k * (12 * 40 + (40 if case["solver"] == "newton" else 3) * 1000))
    es = STORED[case["precision"]]
    n, k = (case["nx"] + 2) * case["ny"] * case["nz"], _open(case)
    if kind in ("flow", "solve"):
        steps = case.get("steps", 5000)  # a solve from rest: 2,000 to 9,000 by the pack
        return dict(bytes=steps * k * 2 * 19 * es + 3 * n * max(4, es), flops=steps * k * 250)
    per = case["species"] * 2 * 7 * es + 3 * max(4, es) + 1
    fields = case["species"] + (2 if kind == "coupled" or case.get("law") == "dual" else 0)
    b, f = case["steps"] * k * per + fields * n * 8, case["steps"] * k * 40 * case["species"]
    if kind == "coupled":
        b, f = b + 0.7 * case["steps"] * k * 2 * 19 * es, f + 0.7 * case["steps"] * k * 250
    return dict(bytes=b, flops=f)


# ------------------------------------------------------------------ the same in plain torch, 64 bits
# Palabos' velocity order: rest, the negative half, its opposites.
C19 = [(0, 0, 0), (-1, 0, 0), (0, -1, 0), (0, 0, -1), (-1, -1, 0), (-1, 1, 0), (-1, 0, -1), (-1, 0, 1), (0, -1, -1),
       (0, -1, 1)]
C19 += [tuple(-v for v in c) for c in C19[1:]]
C7 = [(0, 0, 0), (-1, 0, 0), (0, -1, 0), (0, 0, -1), (1, 0, 0), (0, 1, 0), (0, 0, 1)]
W19 = [1 / 3] + [1 / 18 if sum(v * v for v in c) == 1 else 1 / 36 for c in C19[1:]]
W7 = [1 / 4] + [1 / 8] * 6


class _Lattice:
    """Streaming over the nodes `stored` of a box as one gather from (out of this step, out of the
    step before): from a stored neighbour its outgoing population; at the box's edge the node's own
    opposite one; from a wall the node's own opposite one of the step before (full-way bounce-back)."""

    def __init__(self, stored, C, dev):
        nx, ny, nz = stored.shape
        self.Q, self.C = len(C), C
        st = torch.from_numpy(np.ascontiguousarray(stored)).to(dev)
        self.node = torch.nonzero(st.reshape(-1)).reshape(-1)
        self.K = self.node.numel()
        idx = torch.full((nx * ny * nz,), -1, dtype=torch.long, device=dev)
        idx[self.node] = torch.arange(self.K, device=dev)
        self.idx = idx
        self.x, self.y, self.z = self.node // (ny * nz), self.node // nz % ny, self.node % nz
        self.shape = stored.shape
        self.opp = [C.index(tuple(-v for v in c)) for c in C]
        me = torch.arange(self.K, device=dev)
        self.src = torch.empty((self.Q, self.K), dtype=torch.long, device=dev)
        for i, c in enumerate(C):
            k, inside = self.neighbour(self.node, (-c[0], -c[1], -c[2]))
            s = torch.where(k >= 0, i * self.K + k, (self.Q + self.opp[i]) * self.K + me)
            self.src[i] = torch.where(inside, s, self.opp[i] * self.K + me)

    def neighbour(self, node, c):
        nx, ny, nz = self.shape
        x, y, z = node // (ny * nz) + c[0], node // nz % ny + c[1], node % nz + c[2]
        inside = (x >= 0) & (x < nx) & (y >= 0) & (y < ny) & (z >= 0) & (z < nz)
        n = torch.where(inside, (x * ny + y) * nz + z, torch.zeros_like(x))
        return torch.where(inside, self.idx[n], torch.full_like(n, -1)), inside

    def stream(self, buf):
        return buf.reshape(-1)[self.src]


class _Flow:
    def __init__(self, mats, taus, dev, bio_codes=(), perm_ratio=()):
        """One or several domains; several lie one after another along x with their own planes."""
        self.parts = []
        for mat, tau in zip(mats, taus):
            L = _Lattice(mat != WALL, C19, dev)
            code = torch.from_numpy(mat.reshape(-1).astype(np.int64)).to(dev)[L.node]
            om = torch.full((L.K,), 1.0 / tau, dtype=torch.float64, device=dev)
            for c, r in zip(bio_codes, perm_ratio):
                om[code == c] = 1.0 / (r * (tau - 0.5) + 0.5)
            self.parts.append((L, code != ROCK, om, mat.shape))
        self.dev = dev
        one = len(self.parts) == 1
        self.K = sum(L.K for L, *_ in self.parts)
        src, at = [], 0
        for L, *_ in self.parts:
            q = L.src // L.K
            src.append(q * self.K + at + (L.src - q * L.K))
            at += L.K
        self.src = src[0] if one else torch.cat(src, 1)
        self.bgk = torch.cat([p[1] for p in self.parts])
        self.omega = torch.cat([p[2] for p in self.parts])
        self.planes, at = [], 0
        rho = torch.empty(self.K, dtype=torch.float64, device=dev)
        rho_e = 1.0 - DELTA_P * 3.0
        for L, bgk, _, shape in self.parts:
            rho[at:at + L.K] = 1.0 - DELTA_P * 3.0 / (shape[0] - 1) * L.x.double()
            self.planes.append((at + torch.nonzero(bgk & (L.x == 0)).reshape(-1), -1, 0.0))
            self.planes.append((at + torch.nonzero(bgk & (L.x == shape[0] - 1)).reshape(-1), 1, rho_e - 1.0))
            at += L.K
        self.w = torch.tensor(W19, dtype=torch.float64, device=dev)
        self.c = torch.tensor(C19, dtype=torch.float64, device=dev)
        self.f = self.w[:, None] * (rho - 1.0)[None] * self.bgk.double()[None]
        self.buf = torch.zeros((2 * 19, self.K), dtype=torch.float64, device=dev)

    def _equilibrium(self, rb, j):
        cj = self.c @ j
        return self.w[:, None] * (rb + 3.0 * cj + 1.5 * (3.0 * cj * cj - (j * j).sum(0)))

    def _plane(self, g, o, rb):
        cx = self.c[:, 0]
        jx = o * (g[cx == 0].sum(0) + 2.0 * g[cx == o].sum(0) - rb)
        j = torch.zeros((3, g.shape[1]), dtype=torch.float64, device=self.dev)
        j[0] = jx
        return j

    def step(self, energy=False):
        g = self.f
        for at, o, rb in self.planes:
            gp = g[:, at]
            j = self._plane(gp, o, rb)
            feq = self._equilibrium(torch.full_like(j[0], rb), j)
            fac = (self.c[:, 0] == 0).double() + 2.0 * (self.c[:, 0] == o).double()
            fac[0] = 0.0  # the rest population carries no momentum
            neq = fac[:, None] * (gp - feq)
            pi = torch.einsum("ia,ib,ik->abk", self.c, self.c, neq)
            Q = self.c[:, :, None] * self.c[:, None, :] - torch.eye(3, dtype=torch.float64, device=self.dev) / 3.0
            g[:, at] = feq + 4.5 * self.w[:, None] * torch.einsum("iab,abk->ik", Q, pi)
        rb = g.sum(0)
        j = self.c.T @ g
        out = g + torch.where(self.bgk, self.omega, torch.zeros_like(self.omega)) * (self._equilibrium(rb, j) - g)
        e = 0.5 * ((j * j).sum(0) * self.bgk).sum() / self.bgk.sum() if energy else None
        self.buf[19:] = self.buf[:19]
        self.buf[:19] = out
        self.f = self.buf.reshape(-1)[self.src]
        return e

    def velocity(self):
        """[3][K]: j of the incoming populations; on the planes the imposed density's j_x; else 0."""
        j = (self.c.T @ self.f) * self.bgk
        for at, o, rb in self.planes:
            j[:, at] = self._plane(self.f[:, at], o, rb)
        return j

    def dense(self):
        """Per domain [3][N], as the library reads it out."""
        j, at, got = self.velocity(), 0, []
        for L, _, _, shape in self.parts:
            u = torch.zeros((3, int(np.prod(shape))), dtype=torch.float64, device=self.dev)
            u[:, L.node] = j[:, at:at + L.K]
            got.append(u)
            at += L.K
        return got


class _Transport:
    """One species on one domain: advection-diffusion BGK, x-faces, bounce-back walls."""

    def __init__(self, L, code, u, sp, bio_codes):
        self.L, self.sp = L, sp
        dev = code.device
        bio = torch.zeros_like(code, dtype=torch.bool)
        for c in bio_codes:
            bio |= code == c
        self.w = torch.full((L.K,), sp["omega_pore"], dtype=torch.float64, device=dev)
        self.w[bio] = sp["omega_biofilm"]
        self.u = u
        self.t = torch.tensor(W7, dtype=torch.float64, device=dev)
        self.c = torch.tensor(C7, dtype=torch.float64, device=dev)
        nx = L.shape[0]
        self.f = self.t[:, None] * torch.full((1, L.K), sp["c0"], dtype=torch.float64, device=dev)
        self.buf = torch.cat([self.f, self.f])
        self.faces = []
        for at_x, step, miss, kind, bc in ((0, 1, 4, sp["left_type"], sp["left_bc"]),
                                           (nx - 1, -1, 1, sp["right_type"], sp.get("right_bc", 0.0))):
            at = torch.nonzero(L.x == at_x).reshape(-1)
            inner, _ = L.neighbour(L.node[at], (step, 0, 0))
            value = torch.full((at.numel(),), bc if kind == clb.DIRICHLET else sp["c0"], dtype=torch.float64, device=dev)
            self.faces.append([at, inner, miss, kind, value])

    def refresh(self):
        for F in self.faces:
            if F[3] == clb.NEUMANN:
                F[4] = torch.where(F[1] >= 0, self.f[:, F[1].clamp(min=0)].sum(0), F[4])

    def density(self):
        """The incoming density of every node before a step, with the x-faces completed."""
        self.refresh()
        for at, _, miss, _, value in self.faces:
            g = self.f[:, at]
            g[miss] = 0.0
            g[miss] = value - g.sum(0)
            self.f[:, at] = g
        return self.f.sum(0)

    def collide(self, rho, dC):
        j = rho * self.u
        eq = self.t[:, None] * (rho + 4.0 * (self.c @ j))
        out = self.f + self.w * (eq - self.f)
        if dC is not None:
            out += self.t[:, None] * dC
        self.out = out

    def stream(self):
        self.buf[7:] = self.buf[:7]
        self.buf[:7] = self.out
        self.f = self.L.stream(self.buf)

    def dense(self):
        """Every voxel's density as the library reads it out: the faces' stored values, walls with
        what their open neighbours sent into them."""
        self.refresh()
        L = self.L
        n = int(np.prod(L.shape))
        d = torch.empty(n, dtype=torch.float64, device=self.f.device)
        d[L.node] = self.f.sum(0)
        for at, _, _, _, value in self.faces:
            d[L.node[at]] = value
        rest = torch.nonzero(L.idx < 0).reshape(-1)
        v = torch.full((rest.numel(),), self.sp["c0"] * W7[0], dtype=torch.float64, device=d.device)
        for i in range(1, 7):
            k, _ = L.neighbour(rest, tuple(-c for c in C7[i]))
            v += torch.where(k >= 0, self.buf[i, k.clamp(min=0)], torch.full_like(v, self.sp["c0"] * W7[i]))
        d[rest] = v
        return d


def _floor(c):
    return torch.where(c < 1e-12, torch.zeros_like(c), c)


def _clamped(d, c):
    d = torch.where(d.abs() > 1e-12, d, torch.zeros_like(d))
    d = torch.maximum(d, -c)
    return torch.where(d.abs() > 1e-12, d, torch.zeros_like(d))


def _kinetics(law, prm, rho, bio, react):
    """Increments of the species and the biomass advanced in place."""
    n = len(rho)
    if law == "none":
        return [None] * n
    C = [_floor(r) for r in rho]
    if law == "decay":
        R = [-prm[s] * C[s] for s in range(n)]
    elif law == "monod":
        R = [-prm[s] * C[s] / (prm[n + s] + C[s]) for s in range(n)]
    else:
        mu, ks, y, kd = prm
        R = [torch.zeros_like(C[0]) for _ in range(n)]
        for m in range(2):
            if 1 + m >= n:
                continue
            B = _floor(bio[m])
            growth = mu * C[0] / (ks + C[0]) * C[1 + m] / (ks + C[1 + m]) * B
            R[0] = R[0] - growth / y
            R[1 + m] = R[1 + m] - growth / y
            bio[m] += torch.where(react, _clamped(growth - kd * B, B), torch.zeros_like(B))
    return [torch.where(react, _clamped(R[s], C[s]), torch.zeros_like(C[s])) for s in range(n)]


def _speciate(S, logK, comp, c, tol=1e-10, most=200):
    """Newton-Raphson on log10 component concentrations with backtracking, every voxel at once."""
    T = (c.clamp(1e-30, 10.0) @ S).clamp(min=1e-30)
    x = torch.log10(c[:, comp].clamp(1e-30, 10.0))
    ln10 = math.log(10.0)
    nc = S.shape[1]
    SS = (S[:, :, None] * S[:, None, :]).reshape(S.shape[0], nc * nc)

    def residual(x, T):
        v = 10.0 ** (x @ S.T + logK).clamp(-300.0, 300.0)
        F = v @ S - T
        return v, F, F.norm(dim=1)

    act = torch.arange(x.shape[0], device=x.device)
    for _ in range(most):
        xa, Ta = x[act], T[act]
        v, F, fn = residual(xa, Ta)
        go = fn >= tol
        if not bool(go.any()):
            break
        act, xa, Ta, v, F, fn = act[go], xa[go], Ta[go], v[go], F[go], fn[go]
        J = ln10 * (v @ SS).reshape(-1, nc, nc)
        d, info = torch.linalg.solve_ex(J, -F)
        d = torch.where((info == 0)[:, None] & d.isfinite(), d, torch.zeros_like(d))
        big = d.abs().amax(1, keepdim=True)
        d = d * torch.where(big > 2.0, 2.0 / big, torch.ones_like(big))
        alpha = torch.ones_like(fn)
        for _ in range(40):
            xn = (xa + alpha[:, None] * d).clamp(-30.0, 1.0)
            bad = ~(residual(xn, Ta)[2] < fn * (1.0 - 1e-4 * alpha))
            if not bool(bad.any()):
                break
            alpha = torch.where(bad, alpha * 0.5, alpha)
        x[act] = (xa + alpha[:, None] * d).clamp(-30.0, 1.0)
    return (10.0 ** (x @ S.T + logK).clamp(-30.0, 1.0)).clamp(1e-30, 10.0)


def _exact_chemistry(case, seed, dev):
    x = _chemistry_inputs(case, seed)
    mat = x["mat"]
    F = _Flow([mat], [x["tau"]], dev)
    for _ in range(FLOW_BEFORE):
        F.step()
    code = torch.from_numpy(mat.reshape(-1).astype(np.int64)).to(dev)
    L = _Lattice(mat == PORE, C7, dev)
    u = F.dense()[0][:, L.node]
    ns = x["ns"]
    sp = [_Transport(L, code[L.node], u, s, ()) for s in x["species"][:ns]]
    mineral = torch.from_numpy(x["deposit"]).to(dev)
    react = (L.x > 0) & (L.x < mat.shape[0] - 1)
    S, logK = torch.from_numpy(x["S"]).to(dev), torch.from_numpy(x["logK"]).to(dev)
    k, ksp, nu = x["mineral"][0], x["mineral"][1], x["mineral"][3:]
    t = torch.tensor(W7, dtype=torch.float64, device=dev)[:, None]
    inner = torch.nonzero(react).reshape(-1)
    for _ in range(case["steps"]):
        rho = [s.density() for s in sp]
        la = sum(nu[i] * torch.log10(_floor(rho[i]).clamp(min=1e-30)) for i in range(ns) if nu[i])
        rm = k * (10.0 ** (la - ksp) - 1.0)
        for i, s in enumerate(sp):
            dC = torch.where(react, _clamped(-nu[i] * rm, _floor(rho[i])), torch.zeros_like(rm)) if nu[i] else None
            s.collide(rho[i], dC)
        m = mineral[L.node]
        mineral[L.node] = m + torch.where(react, _clamped(rm, _floor(m)), torch.zeros_like(rm))
        c = torch.stack([s.out[:, inner].sum(0) for s in sp], 1).clamp(min=1e-30)
        d = _speciate(S, logK, x["comp"], c) - c
        cap = (0.1 * c).clamp(min=1e-9)
        d = torch.maximum(torch.minimum(d, cap), -cap)
        d = torch.maximum(d, 1e-20 - c)
        d = torch.where(d.abs() > 1e-12, d, torch.zeros_like(d))
        for i, s in enumerate(sp):
            s.out[:, inner] += t * d[:, i]
            s.stream()
    return torch.stack([s.dense() for s in sp] + [mineral])


def _exact_ensemble(case, seed, dev):
    doms = _ensemble_inputs(case, seed)
    F = _Flow([x["mat"] for x in doms], [x["tau"] for x in doms], dev)
    for _ in range(20):
        F.step()
    us = F.dense()
    for _ in range(case["steps"]):
        F.step()
    out = []
    for x, u in zip(doms, us):
        out.append(_exact_species(x["mat"], u, x["species"], (), "monod", x["params"], None, case["steps"], dev)[0])
    return dict(u=torch.cat([u.reshape(-1) for u in F.dense()]), c=torch.cat(out, 1))


def _exact_species(mat, u, species, bio_codes, law, prm, biomass, steps, dev):
    code = torch.from_numpy(mat.reshape(-1).astype(np.int64)).to(dev)
    L = _Lattice((mat != WALL) & (mat != ROCK), C7, dev)
    sp = [_Transport(L, code[L.node], u[:, L.node], s, bio_codes) for s in species]
    react = (L.x > 0) & (L.x < mat.shape[0] - 1)
    bio = None if biomass is None else torch.from_numpy(biomass).to(dev)
    local = None if bio is None else [b[L.node] for b in bio]
    for _ in range(steps):
        rho = [s.density() for s in sp]
        dC = _kinetics(law, prm, rho, local, react)
        for s, r, d in zip(sp, rho, dC):
            s.collide(r, d)
            s.stream()
    if bio is not None:
        for m in range(bio.shape[0]):
            bio[m, L.node] = local[m]
    return torch.stack([s.dense() for s in sp]), bio


def exact(case, seed):
    kind, dev = case["kind"], _device()
    if kind == "coupled":
        return None  # the automaton's pushes choose neighbours by its own random numbers
    if kind == "chemistry":
        return _exact_chemistry(case, seed, dev)
    if kind == "ensemble":
        return _exact_ensemble(case, seed, dev)
    x = _inputs(case, seed)
    F = _Flow([x["mat"]], [case["tau"]], dev, x["bio_codes"], x["perm_ratio"])
    if kind == "solve":
        window = torch.zeros(500, dtype=torch.float64, device=dev)
        for k in range(20000):
            window[k % 500] = F.step(energy=True)
            if k >= 499 and float(window.std() / window.mean()) < case["eps"]:
                break
        return F.dense()[0].reshape(-1)
    for _ in range(case["steps"] if kind == "flow" else FLOW_BEFORE):
        F.step()
    u = F.dense()[0]
    if kind == "flow":
        return u.reshape(-1)
    del F
    c, bio = _exact_species(x["mat"], u, x["species"], x["bio_codes"], x["law"], x["params"], x["biomass"], case["steps"],
                            dev)
    return c if bio is None else torch.cat([c, bio])
