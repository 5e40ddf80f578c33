"""Performance cases: the calls a treatment-planning program makes on this engine, with their
inputs, their work and their results in 64 bits.

A case is a dict of plain values.  ``kind`` names the call:

  loss_grad   masked quadratic plan loss of one field with dL/dW and dL/dR (the inner step of a
              plan optimisation); ``graph``: replayed from a ``LossGradGraph`` as the
              optimisation loops do, else one eager ``DosePlan.loss_grad`` call
  dose        ``DosePlan.forward``: the dose of new weights on a resident plan
  dose_f64    ``DosePlan.forward_f64``: the float64 dose (commissioning, reference doses)
  dropin      ``torch_separable(problem)``: the one-call engine, problem arrays uploaded per call
  adjoint     ``DosePlan.adjoint``: dL/dW and dL/dR for a dL/dD of the caller's own objective
  robust      loss gradients of every (field, setup / range scenario) job of a robust plan
  tables      ``TableBuilder.build``: the depth tables and their range derivatives, rebuilt when
              range shifts move
  wed_dose    water-equivalent depths of a density map and the dose in that medium
  wed_grad    dL/dW and dL/dR of the dose in a medium
  gamma       gamma index of two doses with map, mask and statistics

Grids are voxels of 1-3 mm, lattices of 2.5-5 mm pitch, layers evenly spaced in range.
"""
from __future__ import annotations

import importlib
import math
import random

import numpy as np
import torch

pb = importlib.import_module("gpu-proton-dose-engine_b200")

FD_STEP = 0.005          # cm, step of the range-derivative tables
SIGMA_X0 = 0.30          # cm, beam width at the surface


# ------------------------------------------------------------------------------------ cases
def _field(kind, nx, ny, nz, vox, nsx, nsy, nl, pitch, r_min, r_max, **more):
    """Grid nx x ny x nz of ``vox`` cm, nsx x nsy spots of ``pitch`` cm, nl layers over r_min..r_max cm."""
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, vox=vox, nsx=nsx, nsy=nsy, nl=nl, pitch=pitch,
                r_min=r_min, r_max=r_max, **more)


def listed():
    return [
        # the smallest field (a unit test of a plan, one spot group of an adaptive loop): latency
        dict(_field("loss_grad", 32, 32, 64, 0.2, 11, 11, 8, 0.5, 4.0, 9.0, graph=False),
             name="small_loss_grad"),
        # the clinical field of plan optimisation, replayed as the optimiser's loop does
        dict(_field("loss_grad", 128, 128, 128, 0.2, 41, 41, 40, 0.25, 6.0, 16.0, graph=True),
             name="clinical_loss_grad"),
        # the dose of that field for new weights (dose display, line search)
        dict(_field("dose", 128, 128, 128, 0.2, 41, 41, 40, 0.25, 6.0, 16.0), name="clinical_dose"),
        # an objective of the caller's own: its dL/dD goes through the adjoint; uneven grid,
        # uneven lattice
        dict(_field("adjoint", 117, 93, 121, 0.2, 37, 29, 33, 0.3, 5.0, 17.0), name="uneven_adjoint"),
        # the 1 mm grid with the full lattice: the largest gradient of one field
        dict(_field("loss_grad", 200, 200, 256, 0.1, 61, 61, 60, 0.25, 4.0, 22.0, graph=False),
             name="large_loss_grad"),
        # robust optimisation: four uneven fields, nominal and shifted / scaled scenarios
        dict(kind="robust", nx=128, ny=128, nz=128, vox=0.2, pitch=0.25, r_min=5.0, r_max=17.0,
             fields=4, scenarios=5, name="robust_loss_grad"),
        # the drop-in call on a field wider than 64 spots (large target, fine pitch)
        dict(_field("dropin", 150, 142, 130, 0.2, 73, 69, 24, 0.25, 5.0, 18.0), name="wide_dropin"),
        # the float64 dose of a field
        dict(_field("dose_f64", 128, 128, 128, 0.2, 41, 41, 40, 0.25, 6.0, 16.0), name="dose_f64"),
        # depth tables of 40 layers with range derivatives (range-shift optimisation)
        dict(kind="tables", nz=128, vox=0.2, nl=40, r_min=6.0, r_max=16.0, name="tables"),
        # the clinical field in bone and lung slabs
        dict(_field("wed_dose", 128, 128, 128, 0.2, 41, 41, 40, 0.25, 6.0, 16.0), name="wed_dose"),
        dict(_field("wed_grad", 128, 128, 128, 0.2, 33, 33, 28, 0.25, 6.0, 16.0), name="wed_grad"),
        # plan check: 3 % / 3 mm on the clinical grid
        dict(kind="gamma", nx=128, ny=128, nz=128, vox=0.2, pct=3.0, dta_mm=3.0, dtype="float32",
             name="gamma"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["loss_grad", "loss_grad", "dose", "adjoint", "robust", "dropin", "dose_f64",
                       "tables", "wed_dose", "wed_grad", "gamma"])
    r_min = rng.uniform(3.0, 7.0)
    if kind == "tables":
        return dict(kind=kind, nz=_log_int(rng, 48, 256), vox=rng.choice([0.1, 0.15, 0.2]),
                    nl=_log_int(rng, 6, 60), r_min=r_min, r_max=r_min + rng.uniform(4.0, 15.0))
    if kind == "gamma":
        vox = rng.choice([0.1, 0.15, 0.2, 0.25])
        return dict(kind=kind, nx=rng.randint(48, 160), ny=rng.randint(48, 160),
                    nz=rng.randint(48, 160), vox=vox, pct=rng.choice([2.0, 3.0]),
                    dta_mm=rng.choice([2.0, 3.0]), dtype=rng.choice(["float32", "float64"]))
    if kind == "robust":
        return dict(kind=kind, nx=rng.randint(64, 128), ny=rng.randint(64, 128),
                    nz=rng.randint(64, 128), vox=rng.choice([0.2, 0.25]), pitch=0.25, r_min=r_min,
                    r_max=r_min + rng.uniform(4.0, 10.0), fields=rng.randint(1, 4),
                    scenarios=rng.randint(3, 6))
    big = kind in ("loss_grad", "dose", "dropin") and rng.random() < 0.4
    hi = 200 if big else 128
    nx, ny = _log_int(rng, 32, hi), _log_int(rng, 32, hi)
    nz = _log_int(rng, 48, 256 if big else 128)
    vox = rng.choice([0.1, 0.15, 0.2, 0.3])
    wide = kind == "dropin"
    nsx, nsy = (rng.randint(41, 81) if wide else _log_int(rng, 9, 61),
                rng.randint(17, 81) if wide else _log_int(rng, 9, 61))
    if rng.random() < 0.3 and not wide:          # the same grid and lattice along x and y
        ny, nsy = nx, nsx
    nl = _log_int(rng, 4, 32 if wide else 60)
    c = _field(kind, nx, ny, nz, vox, nsx, nsy, nl, rng.choice([0.25, 0.3, 0.5]), r_min,
               r_min + rng.uniform(3.0, 14.0))
    if kind == "loss_grad":
        c["graph"] = rng.random() < 0.5
    return c


# ------------------------------------------------------------------------------------ inputs
def _grid(c):
    return pb.model.DoseGrid(c["nx"], c["ny"], c["nz"], c["vox"], c["vox"], c["vox"],
                             -(c["nx"] - 1) * c["vox"] / 2.0, -(c["ny"] - 1) * c["vox"] / 2.0, 0.0)


def _weights_np(c, seed):
    """Spot weights: a spread-out Bragg peak (distal layers weighted most) with noise."""
    rng = np.random.default_rng(seed)
    sobp = 0.3 + 0.7 * np.arange(c["nl"]) / max(c["nl"] - 1, 1)
    w = sobp[:, None, None] * rng.uniform(0.6, 1.4, (c["nl"], c["nsy"], c["nsx"]))
    return w.astype(np.float32)


def _problem(c, w, tables=False):
    """PBProblem of a case.  Host tables are built only for the drop-in, which reads them."""
    grid = _grid(c)
    en = pb.model.clinical_layer_energies(c["nl"], c["r_min"], c["r_max"])
    lat = pb.model.SpotLattice(c["nsx"], c["nsy"], c["nl"], c["pitch"], c["pitch"], energies=en,
                               weights=w)
    idd = sig = np.zeros((c["nl"], c["nz"]))
    if tables:
        idd, sig = pb.physics.layer_luts(grid.z, en)
    return pb.model.PBProblem(grid, lat, idd, sig)


def _target(c):
    """Mask and prescription: a target box in the middle of the ranges, a shell around it."""
    mid = min(0.5 * (c["r_min"] + c["r_max"]), 0.6 * c["nz"] * c["vox"])
    g = dict(nx=c["nx"], ny=c["ny"], nz=c["nz"], dx=c["vox"], dy=c["vox"], dz=c["vox"],
             ox=-(c["nx"] - 1) * c["vox"] / 2.0, oy=-(c["ny"] - 1) * c["vox"] / 2.0, oz=0.0)
    half = min(3.0, 0.25 * c["vox"] * min(c["nx"], c["ny"]))
    eps = 1e-9
    ax = np.abs(g["ox"] + np.arange(c["nx"]) * c["vox"])[None, None, :]
    ay = np.abs(g["oy"] + np.arange(c["ny"]) * c["vox"])[None, :, None]
    az = np.abs(np.arange(c["nz"]) * c["vox"] - mid)[:, None, None]
    far = np.maximum(np.maximum(ax, ay), az)
    mask = np.where(far <= half + eps, 1.0, np.where(far <= half + 2.0 + eps, 0.2, 0.0))
    presc = np.where(far <= half + eps, 2.0, 0.0)
    return mask.astype(np.float32), presc.astype(np.float32)


def _grad_dose(c, seed, dev):
    """A dL/dD as a smooth objective gives it: signed, largest in and around the target."""
    gen = torch.Generator(device=dev).manual_seed(seed)
    mask, _ = _target(c)
    noise = torch.rand((c["nz"], c["ny"], c["nx"]), generator=gen, device=dev) - 0.4
    return noise * torch.as_tensor(mask, device=dev)


def _density(c, seed, dev):
    """Relative stopping power: water with noise, a bone slab, a lung half-slab behind it."""
    gen = torch.Generator(device=dev).manual_seed(seed + 77)
    rho = 1.0 + 0.04 * (torch.rand((c["nz"], c["ny"], c["nx"]), generator=gen, device=dev) - 0.5)
    z = (torch.arange(c["nz"], device=dev) * c["vox"]).view(-1, 1, 1)
    bone = (z >= 0.3 * c["r_min"]) & (z < 0.5 * c["r_min"])
    half = torch.arange(c["nx"], device=dev).view(1, 1, -1) < c["nx"] // 2
    lung = (z >= 0.6 * c["r_min"]) & (z < 0.9 * c["r_min"]) & half
    rho = torch.where(bone, rho * 1.6, rho)
    return torch.where(lung, rho * 0.25, rho).to(torch.float32).contiguous()


def _wed_plain(rho, vox):
    """Water-equivalent depth at the voxel centres, grid starting at depth 0 (float64)."""
    nz = rho.shape[0]
    z = torch.arange(nz, dtype=torch.float64, device=rho.device) * vox
    lo, mid, hi = ((z + s).clamp_min(0.0) for s in (-0.5 * vox, 0.0, 0.5 * vox))
    r = rho.to(torch.float64)
    full = r * (hi - lo).view(-1, 1, 1)
    return torch.cumsum(full, 0) - full + r * (mid - lo).view(-1, 1, 1)


ROBUST_LATTICES = ((21, 21, 16), (33, 33, 28), (41, 41, 40), (51, 41, 48))
# (dx, dy, dz, range scaling): setup shifts of 3 mm, range scaling of 3.5 %
SCENARIOS = ((0.0, 0.0, 0.0, 1.0), (0.3, 0.0, 0.0, 1.0), (0.0, -0.3, 0.0, 0.965),
             (0.0, 0.0, 0.3, 1.035), (-0.3, 0.3, -0.3, 1.035), (0.0, 0.3, 0.0, 1.0))


def _robust_fields(c):
    out = []
    for nsx, nsy, nl in ROBUST_LATTICES[:c["fields"]]:
        out.append(_field("dose", c["nx"], c["ny"], c["nz"], c["vox"], nsx, nsy, nl, c["pitch"],
                          c["r_min"], c["r_max"]))
    return out


def _gamma_doses(c, seed, dev):
    """Reference and evaluated dose: a spread-out field with noise; the second 1 mm off, 1 % higher."""
    gen = torch.Generator(device=dev).manual_seed(seed)
    x, y, z = (torch.arange(c[n], dtype=torch.float64, device=dev) * c["vox"] for n in ("nx", "ny", "nz"))
    lx, ly, lz = (c[n] * c["vox"] for n in ("nx", "ny", "nz"))

    def dose(shift):
        def edge(t, length):
            return 0.5 * (torch.erf((t - 0.25 * length) / 0.6) - torch.erf((t - 0.75 * length) / 0.6))
        depth = (0.6 + 0.4 * z / (0.7 * lz)) * 0.5 * (1.0 - torch.erf((z - 0.7 * lz) / 0.4))
        return 2.0 * depth.view(-1, 1, 1) * edge(y, ly).view(1, -1, 1) * edge(x - shift, lx).view(1, 1, -1)

    noise = torch.rand((c["nz"], c["ny"], c["nx"]), generator=gen, dtype=torch.float64, device=dev)
    dt = getattr(torch, c["dtype"])
    return (dose(0.0) * (1.0 + 0.01 * (noise - 0.5))).to(dt), (1.01 * dose(0.1)).to(dt)


def prepare(case, seed):
    c, dev = case, torch.device("cuda", torch.cuda.current_device())
    kind = c["kind"]
    s = {"case": c}
    if kind == "tables":
        en = pb.model.clinical_layer_energies(c["nl"], c["r_min"], c["r_max"])
        s["builder"] = pb.physics.TableBuilder(c["nz"], 0.0, c["vox"], en, fd_step=FD_STEP, device=dev)
        s["shift"] = torch.as_tensor(_shifts(c, seed), device=dev)
        return s
    if kind == "gamma":
        s["ref"], s["ev"] = _gamma_doses(c, seed, dev)
        spec = pb.gamma.gamma_spec((c["vox"],) * 3, c["pct"], c["dta_mm"])
        s["plan"] = pb.gamma.GammaPlan(s["ref"].shape, spec, device=dev)
        return s
    if kind == "robust":
        fields = _robust_fields(c)
        probs = [_problem(f, _weights_np(f, seed + k)) for k, f in enumerate(fields)]
        s["batch"] = pb.robust.ScenarioBatch(probs, [pb.robust.Scenario(*v) for v in SCENARIOS[:c["scenarios"]]],
                                             precision="fp16x3", device=dev, with_grad=True, fd_step=FD_STEP)
        s["mask"], s["presc"] = (torch.as_tensor(a, device=dev) for a in _target(c))
        return s
    w = _weights_np(c, seed)
    prob = _problem(c, w, tables=kind == "dropin")
    if kind == "dropin":
        s["problem"] = prob
        return s
    s["w"] = torch.as_tensor(w, device=dev)
    if kind in ("wed_dose", "wed_grad"):
        s["plan"] = pb.hetero.WedPlan(prob, device=dev)
        s["grid"] = prob.grid
        s["rho"] = _density(c, seed, dev)
        if kind == "wed_grad":
            s["wed"] = _wed_plain(s["rho"], c["vox"])
            s["g"] = _grad_dose(c, seed, dev)
        return s
    s["plan"] = pb.engines.DosePlan(prob, tables="device", fd_step=FD_STEP, device=dev)
    if kind == "loss_grad":
        s["mask"], s["presc"] = (torch.as_tensor(a, device=dev) for a in _target(c))
        if c["graph"]:
            s["graph"] = pb.engines.LossGradGraph(s["plan"], s["mask"], s["presc"])
            s["graph"].w.copy_(s["w"])
        else:
            s["out"] = s["plan"].alloc_outputs()
    elif kind == "adjoint":
        s["g"] = _grad_dose(c, seed, dev)
    elif kind == "dose":
        s["out"] = torch.empty((c["nz"], c["ny"], c["nx"]), dtype=torch.float32, device=dev)
    elif kind == "dose_f64":
        s["out"] = torch.empty((c["nz"], c["ny"], c["nx"]), dtype=torch.float64, device=dev)
    return s


def _shifts(c, seed):
    return np.random.default_rng(seed).uniform(-0.05, 0.05, c["nl"])


# ------------------------------------------------------------------------------------ one pass
RESULTS = ("dose", "grad_w", "grad_range", "loss")


def run(state):
    kind = state["case"]["kind"]
    if kind == "loss_grad":
        if state["case"]["graph"]:
            o = state["graph"].replay()
        else:
            o = state["plan"].loss_grad(state["mask"], state["presc"], w=state["w"], outputs=state["out"])
        return {k: o[k] for k in RESULTS}
    if kind == "dose":
        return state["plan"].forward(state["w"], out=state["out"])
    if kind == "dose_f64":
        return state["plan"].forward_f64(state["w"], out=state["out"])
    if kind == "dropin":
        return pb.engines.torch_separable(state["problem"])
    if kind == "adjoint":
        return state["plan"].adjoint(state["g"], state["w"])
    if kind == "robust":
        b = state["batch"]
        o = b.loss_grad_all(state["mask"], state["presc"])
        return {"dose": b.doses, "grad_w": b.field_grads, "loss": b.field_losses,
                "grad_range": [v["grad_range"] for v in o]}
    if kind == "tables":
        t = state["builder"].build(state["shift"])
        return {"idd": t.idd, "sigma": t.sigma, "didd_dr": t.didd_dr, "dsigma_dr": t.dsigma_dr}
    if kind == "wed_dose":
        wed = pb.hetero.wed_raytrace(state["rho"], state["grid"])
        return {"dose": state["plan"].forward(wed, state["w"]), "wed": wed}
    if kind == "wed_grad":
        return state["plan"].adjoint(state["g"], state["wed"], state["w"], with_range=True)
    if kind == "gamma":
        p = state["plan"]
        p.run(state["ref"], state["ev"])
        st = p.stats()
        return {"gamma": p.gamma, "mask": p.mask, "n_eval": st.n_eval, "n_pass": st.n_pass,
                "mean": st.gamma_mean, "p95": st.gamma_p95, "p99": st.gamma_p99, "max": st.gamma_max}
    raise ValueError(kind)


# ------------------------------------------------------------------------------------ work
def _pairs(c, scale=1.0, shift=0.0):
    """(layer, slice) pairs with depth dose: depths up to range + 8 sigma_R + 2 mm."""
    d = scale * (np.arange(c["nz"]) * c["vox"] - shift)
    n = 0
    for r in np.linspace(c["r_min"], c["r_max"], c["nl"]):
        zmax = r + 8.0 * 0.0135 * r + 0.2          # sigma_R is about 1.3 % of the range
        n += int(((d >= 0.0) & (d <= zmax)).sum())
    return n


def _fwd_flops(c, pairs):
    return 2.0 * pairs * c["nsy"] * c["nx"] * (c["nsx"] + c["ny"])


def _adj_flops(c, pairs):
    """dL/dW with the width derivative: [Gy | Gy']^T g, then its products with Gx and Gx'."""
    return 2.0 * pairs * c["nsy"] * c["nx"] * (2 * c["ny"] + 3 * c["nsx"])


def work(case):
    c, kind = case, case["kind"]
    if kind == "tables":
        lv, n_fine = 3 * c["nl"], 6000
        return {"bytes": 8.0 * (4 * c["nl"] * c["nz"] + 2 * c["nl"]),
                "flops": lv * (2 * 5.0 * 16384 * 14 + 60.0 * n_fine + 100.0 * 4000 + 20.0 * 6 * c["nz"])}
    nvox = float(c["nx"] * c["ny"] * c["nz"])
    if kind == "gamma":
        size = 4 if c["dtype"] == "float32" else 8
        return {"bytes": nvox * (2 * size + 9), "flops": nvox * 8.0}
    if kind == "robust":
        b = f = 0.0
        for fc in _robust_fields(c):
            for _, _, dz, sc in SCENARIOS[:c["scenarios"]]:
                p = _pairs(fc, sc, dz)
                f += _fwd_flops(fc, p) + _adj_flops(fc, p)
                b += 8.0 * 4 * fc["nl"] * fc["nz"] + 4.0 * fc["nl"] * fc["nsx"] * fc["nsy"] + 8.0 * nvox
            b += 4.0 * fc["nl"] * fc["nsx"] * fc["nsy"]
        return {"bytes": b + 8.0 * nvox, "flops": f}
    pairs = _pairs(c)
    wb = 4.0 * c["nl"] * c["nsx"] * c["nsy"]
    tb = 16.0 * c["nl"] * c["nz"]
    if kind == "loss_grad":
        return {"bytes": 2 * wb + 2 * tb + 16.0 * nvox, "flops": _fwd_flops(c, pairs) + _adj_flops(c, pairs)}
    if kind == "adjoint":
        return {"bytes": 2 * wb + 2 * tb + 4.0 * nvox, "flops": _adj_flops(c, pairs)}
    if kind == "dose_f64":
        return {"bytes": wb + tb + 8.0 * nvox, "flops": _fwd_flops(c, pairs)}
    if kind == "wed_dose":
        return {"bytes": wb + tb + 16.0 * nvox,
                "flops": _fwd_flops(c, pairs) + 8.0 * pairs * c["nx"] * c["ny"]}
    if kind == "wed_grad":
        return {"bytes": 2 * wb + 2 * tb + 12.0 * nvox,
                "flops": _adj_flops(c, pairs) + _fwd_flops(c, pairs) + 16.0 * pairs * c["nx"] * c["ny"]}
    return {"bytes": wb + tb + 4.0 * nvox, "flops": _fwd_flops(c, pairs)}      # dose, dropin


# ------------------------------------------------------------------------------------ 64 bits
MP, ME = 938.27208816, 0.51099895000
KZA = 0.307075 * (10.0 / 18.01528)


def _beta2(e):
    g = 1.0 + e / MP
    return g, np.clip(1.0 - 1.0 / g**2, 1e-14, 1.0)


def _stopping(e):
    """Bethe-Bloch stopping power of water, MeV / cm."""
    g, b2 = _beta2(e)
    t = 2.0 * ME * b2 * g**2
    arg = t * (t / (1.0 + 2.0 * g * ME / MP + (ME / MP) ** 2)) / 75.0e-6**2
    return KZA / b2 * (0.5 * np.log(np.clip(arg, 1.0 + 1e-12, None)) - b2)


_RANGE = []


def _range_table():
    if not _RANGE:
        e = np.unique(np.concatenate([np.linspace(0.5, 2.0, 800), np.linspace(2.0, 20.0, 900),
                                      np.linspace(20.0, 60.0, 900), np.linspace(60.0, 400.0, 1200)]))
        i = 1.0 / _stopping(e)
        _RANGE.extend([e, np.concatenate([[0.0], np.cumsum(0.5 * (i[1:] + i[:-1]) * np.diff(e))])])
    return _RANGE


def _energy(r):
    e, t = _range_table()
    return np.interp(np.clip(r, 0.0, t[-1]), t, e)


def _energies(c):
    return _energy(np.linspace(c["r_min"], c["r_max"], c["nl"]))


def _curve(e0):
    """(zmax, smoothed depth-dose curve on 6000 points of [0, zmax]) of one layer."""
    et, rt = _range_table()
    r0 = np.interp(e0, et, rt)
    e = np.linspace(0.5, e0, 4000)
    _, b2 = _beta2(e)
    f = KZA * ME / (np.clip(b2, 1e-12, None) * _stopping(e) ** 3)
    s = math.hypot(math.sqrt(np.trapezoid(f, e)), 1.77 * 0.0033 * r0)
    n, zmax = 6000, r0 + 8.0 * s + 0.2
    z = np.linspace(0.0, zmax, n)
    h = z[1] - z[0]
    edge = np.linspace(0.0, zmax, n + 1)
    ee = np.where(edge < r0, _energy(np.clip(r0 - edge, 0.0, None)), 0.0)
    binned = np.exp(-z / 150.0) * (ee[:-1] - ee[1:]) / h
    nfft = 16384
    ft = np.exp(-2.0 * (np.pi * np.fft.rfftfreq(nfft, d=h) * s) ** 2)
    return zmax, np.fft.irfft(np.fft.rfft(binned, nfft) * ft, nfft)[:n]


def _widths(z, e0, scale=1.0, anchored=False):
    """Lateral width at the depths ``z`` (water-equivalent); ``anchored``: scattering from depth 0."""
    d = z
    if anchored:
        pos = z[z > 0]
        d = np.concatenate([[0.0], pos]) if pos.size else np.array([0.0, 1e-6])
    span = d[-1] - d[0]
    nf = max((len(d) - 1) * 4 + 1, int(np.ceil(span / 0.02)) + 1, 2)
    zf = np.linspace(d[0], d[-1], nf)
    hf = np.gradient(zf)
    r0 = np.interp(e0, *_range_table())
    el = np.where(zf < r0, _energy(np.clip(r0 - zf, 0.0, None)), 0.0)
    g, b2 = _beta2(np.clip(el, 1e-3, None))
    bpc = np.clip(np.sqrt(b2) * np.sqrt(np.clip(g**2 - 1.0, 0.0, None)) * MP, 1e-9, None)
    th = np.where(zf < r0, (13.6 / bpc) ** 2 / 36.08 * 1.076, 0.0) * hf
    u = zf - zf[0]                      # sum over u' < u of (u - u')^2 T h, by running moments
    s0, s1, s2 = np.cumsum(th), np.cumsum(th * u), np.cumsum(th * u * u)
    b = np.interp(z, zf, np.clip(u * u * s0 - 2.0 * u * s1 + s2, 0.0, None))
    if anchored:
        b = np.where(z > 0, b, 0.0)
    return np.sqrt(np.clip(SIGMA_X0**2 + b / scale**2, 0.0, None))


def _tables(c, shift=None, scale=1.0, dz=0.0, anchored=False, derivative=True):
    """idd, sigma, didd_dr, dsigma_dr (L, nz) in float64."""
    z = scale * (np.arange(c["nz"]) * c["vox"] - dz)
    en, offs = _energies(c), (0.0, FD_STEP, -FD_STEP) if derivative else (0.0,)
    et, rt = _range_table()
    sh = np.zeros(c["nl"]) if shift is None else shift
    out = []
    for o in offs:
        tot = sh + o
        ev = np.where(tot == 0.0, en, _energy(np.interp(en, et, rt) + tot))
        idd = []
        for e in ev:
            zmax, f = _curve(e)
            idd.append(np.interp(z, np.linspace(0.0, zmax, len(f)), f, left=0.0, right=0.0))
        out.append((np.stack(idd), np.stack([_widths(z, e, scale, anchored) for e in ev])))
    if not derivative:
        return out[0]
    return (*out[0], (out[1][0] - out[2][0]) / (2 * FD_STEP), (out[1][1] - out[2][1]) / (2 * FD_STEP))


def _axes(c, dev, dx=0.0, dy=0.0):
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
    xv = (np.arange(c["nx"]) - (c["nx"] - 1) / 2.0) * c["vox"]
    yv = (np.arange(c["ny"]) - (c["ny"] - 1) / 2.0) * c["vox"]
    xs = dx + (np.arange(c["nsx"]) - (c["nsx"] - 1) / 2.0) * c["pitch"]
    ys = dy + (np.arange(c["nsy"]) - (c["nsy"] - 1) / 2.0) * c["pitch"]
    return (t(xv)[:, None] - t(xs)[None, :]) ** 2, (t(yv)[:, None] - t(ys)[None, :]) ** 2


def _gauss(d2, s):
    return torch.exp(-d2[None] / (2.0 * s[:, None, None] ** 2)) / (math.sqrt(2.0 * math.pi) * s[:, None, None])


def _lateral(gx, gy, w):
    return gy @ (w @ gx.transpose(1, 2))                     # (nz, ny, nx)


def _dose(c, w, idd, sig, dx=0.0, dy=0.0):
    dev = w.device
    dx2, dy2 = _axes(c, dev, dx, dy)
    d = torch.zeros((c["nz"], c["ny"], c["nx"]), dtype=torch.float64, device=dev)
    for l in range(c["nl"]):
        s = torch.as_tensor(sig[l], device=dev)
        d += torch.as_tensor(idd[l], device=dev)[:, None, None] * _lateral(_gauss(dx2, s), _gauss(dy2, s), w[l])
    return d


def _adjoint(c, w, g, idd, sig, didd, dsig, dx=0.0, dy=0.0, per_layer=None):
    """dL/dW and dL/dR; ``per_layer(l)``: maps that replace idd_l g and didd_l g (a medium)."""
    dev = w.device
    dx2, dy2 = _axes(c, dev, dx, dy)
    gw, gr = torch.zeros_like(w), torch.zeros(c["nl"], dtype=torch.float64, device=dev)
    for l in range(c["nl"]):
        s, ds = (torch.as_tensor(a[l], device=dev) for a in (sig, dsig))
        if per_layer is not None:
            m0, m1 = per_layer(l)
        else:
            m0, m1 = (g * torch.as_tensor(a[l], device=dev)[:, None, None] for a in (idd, didd))
        gx, gy = _gauss(dx2, s), _gauss(dy2, s)
        s3 = s[:, None, None]
        px, py = gx * (dx2[None] / s3**3 - 1.0 / s3), gy * (dy2[None] / s3**3 - 1.0 / s3)
        mx = m0 @ gx                                                     # (nz, ny, nsx)
        gw[l] = (gy.transpose(1, 2) @ mx).sum(0)
        per_z = ((gy @ w[l]) * (m0 @ px)).sum((1, 2)) + ((py @ w[l]) * mx).sum((1, 2))
        gr[l] = (per_z * ds).sum() + ((gy @ w[l]) * (m1 @ gx)).sum()
    return gw, gr


def _curve_at(e0, d, dev):
    """The layer's depth curve at the depths ``d`` (a tensor), linear between its points."""
    zmax, f = _curve(e0)
    f, n = torch.as_tensor(f, device=dev), len(f)
    h = zmax / (n - 1)
    k = (d / h).floor().clamp(0, n - 2).long()
    v = f[k] + (f[k + 1] - f[k]) / h * (d - k * h)
    return torch.where((d >= 0.0) & (d <= zmax), v, torch.zeros_like(v))


def _loss(d, mask, presc, dev):
    m, p = (torch.as_tensor(a, device=dev).to(torch.float64) for a in (mask, presc))
    r = d - p
    return (m * r * r).sum(), 2.0 * m * r


def _gamma(c, ref, ev):
    """Gamma index (global normalisation, 10 % threshold) by one shifted copy per search offset."""
    ref, ev = ref.to(torch.float64), ev.to(torch.float64)
    vox, dta = c["vox"], c["dta_mm"] / 10.0
    ref_max = ref.max()
    crit = c["pct"] / 100.0 * ref_max
    n = min(int(math.floor(dta / vox + 1e-9)), 6)
    padded = torch.nn.functional.pad(ev, (n,) * 6)
    g2 = torch.full_like(ref, math.inf)
    for a in range(-n, n + 1):
        for b in range(-n, n + 1):
            for k in range(-n, n + 1):
                dist = math.sqrt((a * vox) ** 2 + (b * vox) ** 2 + (k * vox) ** 2)
                if dist <= dta + 1e-12:
                    e = padded[n + a:n + a + c["nz"], n + b:n + b + c["ny"], n + k:n + k + c["nx"]]
                    g2 = torch.minimum(g2, (dist / dta) ** 2 + ((e - ref) / crit) ** 2)
    gamma, mask = g2.sqrt(), ref >= 0.1 * ref_max
    v = gamma[mask].sort().values

    def percentile(q):
        at = (v.numel() - 1) * q
        k = min(int(at), v.numel() - 2)
        return v[k] + (v[k + 1] - v[k]) * (at - k)

    return {"gamma": gamma, "mask": None, "n_eval": None, "n_pass": None, "mean": v.mean(),
            "p95": percentile(0.95), "p99": percentile(0.99), "max": v[-1]}


def exact(case, seed):
    c, kind = case, case["kind"]
    dev = torch.device("cuda", torch.cuda.current_device())
    if kind == "gamma":
        return _gamma(c, *_gamma_doses(c, seed, dev))
    if kind == "tables":
        return dict(zip(("idd", "sigma", "didd_dr", "dsigma_dr"), _tables(c, _shifts(c, seed))))
    if kind == "robust":
        mask, presc = _target(c)
        ds, gws, losses, grs = [], [], [], []
        for k, f in enumerate(_robust_fields(c)):
            w = torch.as_tensor(_weights_np(f, seed + k), device=dev).to(torch.float64)
            fg, fl = [], []
            for dx, dy, dz, sc in SCENARIOS[:c["scenarios"]]:
                t = _tables(f, None, sc, dz, True)
                d = _dose(f, w, t[0], t[1], dx, dy)
                loss, g = _loss(d, mask, presc, dev)
                gw, gr = _adjoint(f, w, g, *t, dx, dy)
                ds.append(d), fg.append(gw), fl.append(loss), grs.append(gr)
            gws.append(torch.stack(fg)), losses.append(torch.stack(fl))
        return {"dose": ds, "grad_w": gws, "loss": losses, "grad_range": grs}
    w = torch.as_tensor(_weights_np(c, seed), device=dev).to(torch.float64)
    if kind in ("dose", "dropin", "dose_f64"):
        return _dose(c, w, *_tables(c, derivative=False))
    t = _tables(c)
    if kind == "adjoint":
        return _adjoint(c, w, _grad_dose(c, seed, dev).to(torch.float64), *t)
    if kind == "loss_grad":
        d = _dose(c, w, t[0], t[1])
        loss, g = _loss(d, *_target(c), dev)
        gw, gr = _adjoint(c, w, g, *t)
        return {"dose": d, "grad_w": gw, "grad_range": gr, "loss": loss}
    wed = _wed_plain(_density(c, seed, dev), c["vox"])
    en = _energies(c)
    if kind == "wed_dose":
        dx2, dy2 = _axes(c, dev)
        d = torch.zeros(wed.shape, dtype=torch.float64, device=dev)
        for l in range(c["nl"]):
            s = torch.as_tensor(t[1][l], device=dev)
            d += _curve_at(en[l], wed, dev) * _lateral(_gauss(dx2, s), _gauss(dy2, s), w[l])
        return {"dose": d, "wed": wed}
    g = _grad_dose(c, seed, dev).to(torch.float64)
    rng = np.linspace(c["r_min"], c["r_max"], c["nl"])

    def maps(l):
        hi, lo = (_curve_at(float(_energy(rng[l] + o)), wed, dev) for o in (FD_STEP, -FD_STEP))
        return g * _curve_at(en[l], wed, dev), g * (hi - lo) / (2.0 * FD_STEP)

    return _adjoint(c, w, g, *t, per_layer=maps)
