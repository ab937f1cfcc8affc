"""Performance cases: the work a user of this framework has it do, through its
public entry points, and the same results in 64 bits by plain torch.

Systems are rigid-water boxes (optionally 2% Na+/Cl- ions) at 0.0334
molecules / A^3, jittered lattice sites and random orientations, atoms in
molecule order -- the recipe of ``protomoladdon_b200.water`` for any number of
molecules.

Kinds of case (``kind``):

* ``host``  -- ``SystemForce.evaluate`` on host arrays, as a ProtoMol integrator
  calls the force every step (forces and energies added to the caller's);
* ``step``  -- one device-resident leapfrog iteration with rigid waters and
  energies, from positions and velocities that the program has on the GPU;
* ``eval``  -- one device-resident evaluation (cutoff or real-space Ewald form;
  with or without energies, virials);
* ``batch`` -- many independent uneven boxes in one call;
* ``hvp``   -- the gradient and Hessian-vector products through torch.autograd
  (normal modes);
* ``fit``   -- one training step's gradients: energy and force matching loss,
  derivatives per charge and per Lennard-Jones type.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from protomoladdon_b200 import _lib, water
from protomoladdon_b200.autograd import NonbondedEnergy, lj_table
from protomoladdon_b200.batch import SystemBatch
from protomoladdon_b200.force import (EwaldRealB200SystemForce, NonbondedCutoffB200SystemForce,
                                      PeriodicTopology, ScalarStructure)

DEV = "cuda"
DENSITY = 0.0334         # molecules per cubic Angstrom
TIMEFACTOR = 0.02045482828087295  # one fs in ProtoMol's time unit
DT_FS = 1.0


def listed():
    return [
        # the plain FP64 method on the smallest box, called per step from the host
        dict(name="host_648_fp64", kind="host", waters=216, rc=8.0, precision="fp64"),
        # the host-integrated 41k-atom box: positions in, forces out every step
        dict(name="host_41k", kind="host", waters=13824, rc=10.0, precision="mixed"),
        # device-resident MD of a small box: launches and latency
        dict(name="step_648", kind="step", waters=216, rc=8.0, precision="mixed"),
        # device-resident MD of the 41k-atom box, energies every step
        dict(name="step_41k", kind="step", waters=13824, rc=10.0, precision="mixed"),
        # forces between energy outputs
        dict(name="forces_41k", kind="eval", waters=13824, rc=10.0, precision="mixed",
             form="cutoff", ions=False, energy=False, virial=False),
        # the plain FP64 evaluation of the same box
        dict(name="fp64_41k", kind="eval", waters=13824, rc=10.0, precision="fp64",
             form="cutoff", ions=False, energy=True, virial=False),
        # constant-pressure MD of an ordinary odd-sized box: atomic and
        # molecular virials
        dict(name="virials_15k", kind="eval", waters=5003, rc=9.0, precision="mixed",
             form="cutoff", ions=False, energy=True, virial=True),
        # the large ion box, both pair terms
        dict(name="ions_327k", kind="eval", waters=110592, rc=12.0, precision="mixed",
             form="cutoff", ions=True, energy=True, virial=False),
        dict(name="ewald_327k", kind="eval", waters=110592, rc=12.0, precision="mixed",
             form="ewald", ions=True, energy=True, virial=False),
        # 512 boxes of 300 to 6000 atoms
        dict(name="batch_512", kind="batch", boxes=512, rc=9.0, energy=True),
        # normal modes of the 41k-atom box
        dict(name="hvp_41k", kind="hvp", waters=13824, rc=10.0, precision="mixed", vectors=4),
        # parameter fitting on the 41k-atom box
        dict(name="fit_41k", kind="fit", waters=13824, rc=10.0, precision="mixed"),
    ]


def draw(rng):
    kind = rng.choice(["host", "step", "eval", "eval", "eval", "batch", "hvp", "fit"])
    if kind == "batch":
        return dict(kind=kind, boxes=int(round(math.exp(rng.uniform(math.log(16), math.log(512))))),
                    rc=round(rng.uniform(8.0, 9.0), 2), energy=rng.random() < 0.5)
    precision = rng.choice(["mixed", "mixed", "fp64"])
    most = 110592 if kind in ("step", "eval") and precision == "mixed" else 13824
    waters = int(round(math.exp(rng.uniform(math.log(216), math.log(most)))))
    half = 0.5 * (waters / DENSITY) ** (1.0 / 3.0)
    rc = round(rng.uniform(8.0, min(12.0 if precision == "mixed" else 10.0, half - 0.01)), 2)
    c = dict(kind=kind, waters=waters, rc=rc, precision=precision)
    if kind == "eval":
        c.update(form=rng.choice(["cutoff", "cutoff", "ewald"]), ions=rng.random() < 0.4,
                 energy=rng.random() < 0.6, virial=False)
        c["virial"] = c["energy"] and rng.random() < 0.4
    if kind == "hvp":
        c["vectors"] = rng.randint(1, 4)
    return c


# ---- systems ---------------------------------------------------------------

def _box(waters, seed, ions=False, edge=None):
    """One box of `waters` molecules (2% of them ions where asked), as arrays."""
    rng = np.random.Generator(np.random.PCG64(seed))
    edge = edge or (waters / DENSITY) ** (1.0 / 3.0)
    k = math.ceil(waters ** (1.0 / 3.0) - 1e-9)
    sites = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)
    if waters < k ** 3:
        sites = sites[rng.permutation(k ** 3)[:waters]]
    o = (sites + 0.5) * (edge / k) + rng.uniform(-0.1, 0.1, size=(waters, 3))
    quat = rng.standard_normal((waters, 4))
    w, x, y, z = (quat / np.linalg.norm(quat, axis=1, keepdims=True)).T
    # the H-H direction and the bisector, turned by the quaternion
    ex = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y + z * w), 2 * (x * z - y * w)], -1)
    ez = np.stack([2 * (x * z + y * w), 2 * (y * z - x * w), 1 - 2 * (x * x + y * y)], -1)
    half = 0.5 * water.THETA_HOH
    s, b = water.R_OH * math.sin(half), water.R_OH * math.cos(half)
    pos = np.stack([o, o + s * ex + b * ez, o - s * ex + b * ez], 1)
    typ = np.tile(np.array([water.T_O, water.T_H, water.T_H], dtype=np.int32), (waters, 1))
    q = np.tile(np.array([water.Q_O, water.Q_H, water.Q_H]), (waters, 1))
    mass = np.tile(np.array([water.MASS_O, water.MASS_H, water.MASS_H]), (waters, 1))
    keep = np.ones((waters, 3), dtype=bool)
    if ions:
        pairs = max(1, int(round(0.01 * waters)))
        pick = rng.permutation(waters)[:2 * pairs]
        keep[pick, 1:] = False
        for which, t, charge, m in ((pick[:pairs], water.T_NA, 1.0, water.MASS_NA),
                                    (pick[pairs:], water.T_CL, -1.0, water.MASS_CL)):
            typ[which, 0], q[which, 0], mass[which, 0] = t, charge, m
    first = np.cumsum(keep.sum(1)) - keep.sum(1)  # each molecule's first atom
    whole = first[keep.all(1)][:, None]
    excl = np.concatenate([np.stack([whole[:, 0] + a, whole[:, 0] + c,
                                     np.full(len(whole), 2)], -1)
                           for a, c in ((0, 1), (0, 2), (1, 2))])
    flat = keep.reshape(-1)
    mass = mass.reshape(-1)[flat]
    sig = np.array([water.SIG_O, 0.0] + ([water.SIG_NA, water.SIG_CL] if ions else []))
    eps = np.array([water.EPS_O, 0.0] + ([water.EPS_NA, water.EPS_CL] if ions else []))
    n = int(flat.sum())
    vel = rng.standard_normal((n, 3)) * np.sqrt(water.BOLTZMANN * 300.0 / mass)[:, None]
    return dict(pos=pos.reshape(-1, 3)[flat], vel=vel, type=typ.reshape(-1)[flat],
                qscaled=q.reshape(-1)[flat] * water.SQRT_COULOMB,
                mol=np.repeat(np.arange(waters, dtype=np.int32), 3)[flat], mass=mass,
                sigma=sig, epsilon=eps,
                lj=_mixed_table(torch.from_numpy(sig), torch.from_numpy(eps)).numpy(),
                excl=excl.astype(np.int32), box=np.full(3, edge), origin=np.full(3, 0.5 * edge),
                waters=(whole + np.arange(3)).astype(np.int32))


def _boxes(case, seed):
    """The uneven boxes of a batch: 300 to 6000 atoms, spread over the logarithm
    (the sizes are the case's, the molecules the seed's)."""
    rng = np.random.Generator(np.random.PCG64(case["boxes"]))
    out = []
    for b in range(case["boxes"]):
        w = max(1, int(round(math.exp(rng.uniform(math.log(300), math.log(6000))) / 3.0)))
        edge = max((w / DENSITY) ** (1.0 / 3.0), 2.0 * case["rc"])
        out.append(_box(w, seed * 7919 + b, edge=edge))
    return out


def _ewald(rc):
    """alpha and accuracy of the real-space Ewald term at this cutoff."""
    alpha = 3.6 / rc
    return alpha, math.exp(-(alpha * rc) ** 2)


def _force(case):
    rc = case["rc"]
    if case.get("form") == "ewald":
        return EwaldRealB200SystemForce(*_ewald(rc), precision=case["precision"])
    return NonbondedCutoffB200SystemForce(rc - 1.0, rc, rc, rc,
                                          precision=case.get("precision", "mixed"))


def _cuda(a):
    return torch.tensor(a, dtype=torch.float64, device=DEV)


def _flags(case):
    f = _lib.PMB200_ENERGY if case.get("energy") else 0
    if case.get("virial"):
        f |= _lib.PMB200_VIRIAL | _lib.PMB200_MOLVIRIAL
    return f


def _fit_inputs(sysd, case, seed):
    """Current parameters (5% off the true ones) and the targets."""
    rng = np.random.Generator(np.random.PCG64(seed + 1))

    def off(a):
        return _cuda(a * (1.0 + 0.05 * rng.standard_normal(a.shape)))
    frc, e = _plain(sysd, case["rc"], want=("forces", "energy"))
    return dict(q=off(sysd["qscaled"]), sigma=off(sysd["sigma"]), epsilon=off(sysd["epsilon"]),
                f0=frc, e0=e.sum())


# ---- what the program has before the call, and the call ------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        boxes = _boxes(case, seed)
        members = [(_force(case), PeriodicTopology.from_dict(b)) for b in boxes]
        pos = _cuda(np.concatenate([b["pos"] for b in boxes]))
        return dict(kind=kind, batch=SystemBatch(members), pos=pos, frc=torch.zeros_like(pos),
                    out=torch.zeros(len(boxes), 20, dtype=torch.float64, device=DEV),
                    flags=_flags(case), stream=torch.cuda.Stream())
    sysd = _box(case["waters"], seed, case.get("ions", False))
    topo = PeriodicTopology.from_dict(sysd)
    if kind == "hvp" or kind == "fit":
        rc = case["rc"]
        model = NonbondedEnergy(topo, rc - 1.0, rc, rc, rc, precision=case["precision"])
        model.force.number_of_blocks(topo)
        s = dict(kind=kind, model=model, pos=_cuda(sysd["pos"]).requires_grad_(kind == "hvp"))
        if kind == "hvp":
            s["q"], s["table"] = model.initial_params(DEV)
            rng = np.random.Generator(np.random.PCG64(seed + 1))
            v = rng.standard_normal((case["vectors"],) + sysd["pos"].shape)
            s["vectors"] = _cuda(v / np.linalg.norm(v, axis=(1, 2), keepdims=True))
        else:
            s.update(_fit_inputs(sysd, case, seed))
        return s
    force = _force(case)
    force.number_of_blocks(topo)
    if kind == "host":
        return dict(kind=kind, force=force, topo=topo, pos=sysd["pos"],
                    frc=np.zeros_like(sysd["pos"]), energies=ScalarStructure())
    s = dict(kind=kind, force=force, topo=topo, pos=_cuda(sysd["pos"]))
    s.update(frc=torch.zeros_like(s["pos"]),
             out=torch.zeros(20, dtype=torch.float64, device=DEV))
    if kind == "step":
        force.set_rigid_waters(topo, sysd["waters"], water.D_OH, water.D_HH)
        s.update(start=(s["pos"].clone(), _cuda(sysd["vel"]),
                        _plain(sysd, case["rc"], want=("forces",))[0]),
                 vel=torch.zeros_like(s["pos"]), stream=torch.cuda.Stream())
    else:
        s["flags"] = _flags(case)
    return s


def run(s):
    kind = s["kind"]
    if kind == "host":
        s["frc"].fill(0.0)
        s["energies"].clear()
        s["force"].evaluate(s["topo"], s["pos"], s["frc"], s["energies"])
        return s["frc"], s["energies"].table
    if kind == "step":
        st = s["stream"]
        st.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(st):
            for to, start in zip((s["pos"], s["vel"], s["frc"]), s["start"]):
                to.copy_(start)
            s["force"].step_device(s["topo"], s["pos"].data_ptr(), s["vel"].data_ptr(),
                                   s["frc"].data_ptr(), DT_FS, st.cuda_stream,
                                   s["out"].data_ptr(), _lib.PMB200_ENERGY)
        torch.cuda.current_stream().wait_stream(st)
        return s["pos"], s["vel"], s["frc"], s["out"]
    if kind == "eval":
        s["frc"].zero_()
        # torch's default stream is the legacy one: its explicit handle is 1
        s["force"].evaluate_device(s["topo"], s["pos"].data_ptr(), s["frc"].data_ptr(),
                                   s["out"].data_ptr(), s["flags"],
                                   torch.cuda.current_stream().cuda_stream or 1)
        return (s["frc"], s["out"]) if s["flags"] else s["frc"]
    if kind == "batch":
        st = s["stream"]
        st.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(st):
            s["frc"].zero_()
            s["batch"].eval_device(s["pos"].data_ptr(), s["frc"].data_ptr(), s["out"].data_ptr(),
                                   s["flags"], st.cuda_stream)
        torch.cuda.current_stream().wait_stream(st)
        return (s["frc"], s["out"]) if s["flags"] else s["frc"]
    if kind == "hvp":
        g = s["model"].gradient(s["pos"], s["q"], s["table"])
        return [g.detach()] + [torch.autograd.grad(g, s["pos"], grad_outputs=v,
                                                   retain_graph=True)[0] for v in s["vectors"]]
    q, sigma, epsilon = (s[k].detach().requires_grad_(True) for k in ("q", "sigma", "epsilon"))
    table = lj_table(sigma, epsilon)
    return _loss_and_gradients(s["model"].energy(s["pos"], q, table),
                               s["model"].forces(s["pos"], q, table), s["e0"], s["f0"],
                               (q, sigma, epsilon))


def _loss_and_gradients(e, f, e0, f0, params):
    """Energy and force matching; energies weigh in per squared force unit."""
    loss = (e - e0) ** 2 + ((f - f0) ** 2).sum()
    return [loss.detach()] + list(torch.autograd.grad(loss, params))


# ---- work ----------------------------------------------------------------------

def _pairs_of(atoms, edge, rc):
    return 0.5 * atoms * (atoms / edge ** 3) * 4.0 / 3.0 * math.pi * rc ** 3


def work(case):
    rc, kind = case["rc"], case["kind"]
    if kind == "batch":
        # atom counts spread over the logarithm: their mean, and the mean pairs
        atoms = case["boxes"] * (6000 - 300) / math.log(6000 / 300)
        pairs = 0.5 * atoms * 3.0 * DENSITY * 4.0 / 3.0 * math.pi * rc ** 3
    else:
        atoms = 3 * case["waters"]
        pairs = _pairs_of(atoms, (case["waters"] / DENSITY) ** (1.0 / 3.0), rc)
    # per unique pair: distance, LJ, Coulomb, switches, both forces
    flops, nbytes = 81.0, 24 + 8 + 4 + 4 + 24
    if kind == "step":
        nbytes += 4 * 24
    if kind == "hvp":
        flops += case["vectors"] * 120.0
        nbytes += case["vectors"] * 48
    if kind == "fit":
        flops += 81.0 + 60.0 + 150.0
        nbytes *= 3
    return {"bytes": float(nbytes * atoms), "flops": flops * pairs}


# ---- the same in 64 bits by plain torch -------------------------------------------

def _mixed_table(sigma, epsilon):
    """Lorentz-Berthelot table {A, B, A14, B14} per type pair."""
    s6 = (0.5 * (sigma[:, None] + sigma[None, :])) ** 6
    prod = epsilon[:, None] * epsilon[None, :]
    some = prod > 0
    e = torch.where(some, torch.sqrt(torch.where(some, prod, torch.ones_like(prod))), prod * 0.0)
    return torch.stack([4.0 * e * s6 * s6, 4.0 * e * s6] * 2, dim=-1)


def _near_pairs(pos, mol, edge, rc):
    """Chunks (i, j, d = x_j - x_i at the nearest image) of the unordered pairs
    of different molecules within rc; every pair of atoms is looked at."""
    n = pos.shape[0]
    x, y, z = (pos[:, a].contiguous() for a in range(3))
    i0 = 0
    while i0 < n:
        i1 = min(n, i0 + max(1, 60_000_000 // (n - i0)))
        d = []
        for a in (x, y, z):
            v = a[None, i0:] - a[i0:i1, None]
            d.append(v.sub_(torch.round(v / edge).mul_(edge)))
        near = (d[0] * d[0]).addcmul_(d[1], d[1]).addcmul_(d[2], d[2]) <= rc * rc
        near &= mol[None, i0:] != mol[i0:i1, None]
        near &= torch.arange(i0, n, device=pos.device)[None] > torch.arange(
            i0, i1, device=pos.device)[:, None]
        a, b = torch.nonzero(near, as_tuple=True)
        yield a + i0, b + i0, torch.stack([v[a, b] for v in d], -1)
        i0 = i1


def _lj_c2(r2, A, B, rc):
    """Lennard-Jones with the C2 switch from rc - 1: energy and force / r."""
    ron2, rc2 = (rc - 1.0) ** 2, rc * rc
    s6 = r2 ** -3
    e = (A * s6 - B) * s6
    f = (12.0 * A * s6 - 6.0 * B) * s6 / r2
    t3 = (rc2 - ron2) ** 3
    c2 = rc2 - r2
    c4 = c2 * (rc2 - 3.0 * ron2 + 2.0 * r2)
    on = r2 >= ron2
    sw = torch.where(on, c2 * c4 / t3, torch.ones_like(r2))
    dsw = torch.where(on, 4.0 / t3 * (c2 * c2 - c4), torch.zeros_like(r2))
    return e * sw, f * sw - e * dsw


def _coulomb_c1(r2, qq, rc):
    r = torch.sqrt(r2)
    return (qq * (1.0 / r - 1.5 / rc + 0.5 * r2 / rc ** 3), qq * (1.0 / (r2 * r) - 1.0 / rc ** 3))


def _ewald_real(r2, qq, rc):
    """The real-space Ewald term with erfc by Abramowitz & Stegun 7.1.26."""
    alpha = _ewald(rc)[0]
    r = torch.sqrt(r2)
    x = alpha * r
    t = 1.0 / (1.0 + 0.3275911 * x)
    g = torch.exp(-x * x)
    e = t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (
        -1.453152027 + t * 1.061405429)))) * g / r
    return qq * e, qq * (e + 2.0 * alpha / math.sqrt(math.pi) * g) / r2


def _plain(sysd, rc, form="cutoff", want=("forces", "energy"), pos=None):
    """Forces (n, 3) and the 20 results {Coulomb, LJ, virial, molecular virial}
    (the parts in `want`; the rest zero) of one box."""
    pos = _cuda(sysd["pos"]) if pos is None else pos
    n, edge = pos.shape[0], float(sysd["box"][0])
    mol = torch.tensor(sysd["mol"], device=DEV).long()
    typ = torch.tensor(sysd["type"], device=DEV).long()
    q, table = _cuda(sysd["qscaled"]), _cuda(sysd["lj"])
    frc = torch.zeros(n, 3, dtype=torch.float64, device=DEV)
    out = torch.zeros(20, dtype=torch.float64, device=DEV)
    com = None
    if "virial" in want:
        m = _cuda(sysd["mass"])[:, None]
        nm = int(mol.max()) + 1
        com = torch.zeros(nm, 3, dtype=torch.float64, device=DEV).index_add_(0, mol, pos * m)
        com /= torch.zeros(nm, 1, dtype=torch.float64, device=DEV).index_add_(0, mol, m)
    for i, j, d in _near_pairs(pos, mol, edge, rc):
        r2 = (d * d).sum(-1)
        qq = q[i] * q[j]
        if form == "ewald":
            e, f = _ewald_real(r2, qq, rc)
            el = torch.zeros_like(e)
        else:
            ab = table[typ[i], typ[j]]
            el, fl = _lj_c2(r2, ab[:, 0], ab[:, 1], rc)
            e, f = _coulomb_c1(r2, qq, rc)
            f = f + fl
        fv = f[:, None] * d
        frc.index_add_(0, j, fv)
        frc.index_add_(0, i, -fv)
        out[0] += e.sum()
        out[1] += el.sum()
        if "virial" in want:
            out[2:11] += (fv.T @ d).reshape(-1)
            c = com[mol[j]] - com[mol[i]]
            c = c - torch.round(c / edge) * edge
            u = torch.triu(fv.T @ c)
            out[11:20] += (u + torch.triu(u, 1).T).reshape(-1)
    if "energy" not in want:
        out.zero_()
    return frc, out


def _plain_energy(pos, q, table, sysd, rc):
    """The energy as a torch expression of positions, charges and LJ table."""
    edge = float(sysd["box"][0])
    mol = torch.tensor(sysd["mol"], device=DEV).long()
    typ = torch.tensor(sysd["type"], device=DEV).long()
    e = 0.0
    for i, j, _ in _near_pairs(pos.detach(), mol, edge, rc):
        d = pos[j] - pos[i]
        d = d - torch.round(d.detach() / edge) * edge
        r2 = (d * d).sum(-1)
        ab = table[typ[i], typ[j]]
        e = e + (_lj_c2(r2, ab[:, 0], ab[:, 1], rc)[0] +
                 _coulomb_c1(r2, q[i] * q[j], rc)[0]).sum()
    return e


def _shake(x0, x1, mass, waters):
    """x1 with the waters back on their bond lengths, corrections along the old
    bonds, iterated to convergence."""
    w = torch.tensor(waters, device=DEV).long()
    inv = 1.0 / mass
    lengths = ((0, 1, water.D_OH), (0, 2, water.D_OH), (1, 2, water.D_HH))
    old, new = x0[w], x1[w]
    im = inv[w][..., None]
    for _ in range(60):
        for a, b, length in lengths:
            r = new[:, b] - new[:, a]
            o = old[:, b] - old[:, a]
            g = ((r * r).sum(-1) - length ** 2) / (2.0 * (im[:, a, 0] + im[:, b, 0])
                                                   * (r * o).sum(-1))
            new[:, a] += im[:, a] * g[:, None] * o
            new[:, b] -= im[:, b] * g[:, None] * o
    x1 = x1.clone()
    x1[w] = new
    return x1


def exact(case, seed):
    kind = case["kind"]
    want = ("forces",) + (("energy",) if case.get("energy") else ()) + (
        ("virial",) if case.get("virial") else ())
    if kind == "batch":
        res = [_plain(b, case["rc"], want=want) for b in _boxes(case, seed)]
        frc = torch.cat([f for f, _ in res])
        return (frc, torch.stack([o for _, o in res])) if case["energy"] else frc
    sysd = _box(case["waters"], seed, case.get("ions", False))
    rc = case["rc"]
    if kind == "eval":
        frc, out = _plain(sysd, rc, case["form"], want)
        return (frc, out) if _flags(case) else frc
    if kind == "host":
        frc, out = _plain(sysd, rc)
        table = ScalarStructure().table
        table[:2] = out[:2].cpu().numpy()
        return frc.cpu().numpy(), table
    if kind == "step":
        h = DT_FS * TIMEFACTOR
        x0, mass = _cuda(sysd["pos"]), _cuda(sysd["mass"])
        v = _cuda(sysd["vel"]) + _plain(sysd, rc)[0] * h / mass[:, None]
        x1 = _shake(x0, x0 + v * h, mass, sysd["waters"])
        free = torch.ones(len(mass), dtype=torch.bool, device=DEV)
        free[torch.tensor(sysd["waters"], device=DEV).long().reshape(-1)] = False
        v = torch.where(free[:, None], v, (x1 - x0) / h)
        return (x1, v) + _plain(sysd, rc, pos=x1)
    pos = _cuda(sysd["pos"]).requires_grad_(True)
    if kind == "hvp":
        q, table = _cuda(sysd["qscaled"]), _cuda(sysd["lj"])
        (g,) = torch.autograd.grad(_plain_energy(pos, q, table, sysd, rc), pos, create_graph=True)
        rng = np.random.Generator(np.random.PCG64(seed + 1))
        v = rng.standard_normal((case["vectors"],) + sysd["pos"].shape)
        vectors = _cuda(v / np.linalg.norm(v, axis=(1, 2), keepdims=True))
        return [g.detach()] + [torch.autograd.grad(g, pos, grad_outputs=w, retain_graph=True)[0]
                               for w in vectors]
    p = _fit_inputs(sysd, case, seed)
    params = [p[k].detach().requires_grad_(True) for k in ("q", "sigma", "epsilon")]
    e = _plain_energy(pos, params[0], _mixed_table(*params[1:]), sysd, rc)
    (g,) = torch.autograd.grad(e, pos, create_graph=True)
    return _loss_and_gradients(e, -g, p["e0"], p["f0"], params)
