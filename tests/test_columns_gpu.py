"""The column kernels (the evaluation path of orthogonal periodic boxes) at the
shapes where their layout has edges: clusters of 8 atoms and blocks of 32 staged
ones that do not fill, boxes of exactly two cutoffs, columns that are their own
opposite, columns whose atoms overflow their bucket, the sort's shared memory or both,
clusters taller than the cutoff, exclusion lists longer than a warp, a buffer that
is nearly full at the end -- against the FP64 oracle.

Tolerances: forces 1e-5 RMS relative (the mixed kernels' bound; FP32 pair
arithmetic leaves about 1e-6); energies 1e-6 of the pair magnitudes, about
100 kcal/mol per atom; the pair set is the oracle's up to one pair in 1e6 at the
cutoff.  FP64 kernel: forces 1e-12 RMS relative, energies 1e-11 of the pair
magnitudes (only the order of the sums differs from the oracle's).
Hessian-vector products: 1e-6 of |Hv| against central differences of the oracle's
forces, h = 1e-4 (the h^2/6 term is below 1e-7 for r^-13 at 2.4 A; the directions
move no pair across the cutoff, where the C1 force's slope jumps).
Batches: the mixed bounds."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as O
from protomoladdon_b200 import _lib, water
from protomoladdon_b200.autograd import NonbondedEnergy
from protomoladdon_b200.batch import SystemBatch
from protomoladdon_b200.force import (EwaldRealB200SystemForce, NonbondedCutoffB200PairForce,
                                      NonbondedCutoffB200SystemForce, PeriodicTopology,
                                      ScalarStructure)

pytestmark = pytest.mark.gpu


def _waters(n, edges, region=None, seed=3, rc=8.0):
    """n waters in a box of the given edges, on a jittered lattice filling
    `region` (the whole box by default) at most as densely as water."""
    edges = np.asarray(edges, dtype=np.float64)
    region = edges if region is None else np.asarray(region, dtype=np.float64)
    k = np.maximum(1, np.floor(region / (np.prod(region) / n) ** (1 / 3.0)).astype(int))
    while np.prod(k) < n:
        k[np.argmax(region / k)] += 1
    rng = np.random.default_rng(seed)
    sites = np.stack(np.meshgrid(*[np.arange(q) for q in k], indexing="ij"), -1).reshape(-1, 3)
    sites = sites[np.sort(rng.permutation(len(sites))[:n])]
    s = water.water_box(2, rc=rc, ron=rc - 1.0, seed=seed, nmol=1, box=20.0)
    o, h = s["pos"][0], s["pos"][1:3] - s["pos"][0]
    first = (sites + 0.5) * (region / k) + rng.uniform(-0.1, 0.1, (n, 3)) + 0.5 * (edges - region)
    turn = np.linalg.qr(rng.standard_normal((n, 3, 3)))[0]
    pos = np.concatenate([first[:, None], first[:, None] + np.einsum("nij,hj->nhi", turn, h)], 1)
    s.update(pos=pos.reshape(-1, 3), type=np.tile(s["type"], n), qscaled=np.tile(s["qscaled"], n),
             mass=np.tile(s["mass"], n), mol=np.repeat(np.arange(n, dtype=np.int32), 3),
             excl=(np.tile(s["excl"], (n, 1)) +
                   np.repeat(3 * np.arange(n), 3)[:, None] * np.array([1, 1, 0])).astype(np.int32),
             box=edges, origin=0.5 * edges, n=3 * n)
    return s


def _merged(s, size, modified):
    """`size` neighbouring waters as one molecule, all its pairs excluded or (one
    in three between different waters, where asked) modified."""
    n = s["n"]
    s["mol"] = (np.arange(n) // (3 * size)).astype(np.int32)
    a, b = np.triu_indices(3 * size, 1)
    kind = np.where(modified & (a // 3 != b // 3) & ((a + b) % 3 == 0), 1, 2)
    base = np.arange(0, n, 3 * size)
    e = np.stack([(base[:, None] + a).ravel(), (base[:, None] + b).ravel(),
                  np.tile(kind, len(base))], -1)
    s["excl"] = e[(e[:, 0] < n) & (e[:, 1] < n)].astype(np.int32)
    s["lj"] = s["lj"] * np.array([1.0, 1.0, 0.5, 0.5])
    s["coulomb_scaling"] = 0.8
    return s


def _unwrapped(s):
    rng = np.random.default_rng(5)
    s["pos"] = s["pos"] + np.repeat(rng.integers(-2, 3, (s["n"] // 3, 3)), 3, 0) * s["box"]
    return s


def _ball(n, light):
    """n single atoms on a jittered 1.9 A lattice inside one column, each within
    the cutoff of all others of the lowest cluster; `light` of them without a
    Lennard-Jones term.  The lowest cluster stages 7 + n - 8 atoms, at most 96 of
    them before its last round: the buffer is fuller than a last flush may find it."""
    s = _waters(1, (16.5, 16.5, 100.0))
    rng = np.random.default_rng(n + light)
    sites = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3)
    sites = sites[np.sort(rng.permutation(125)[:n])]
    typ = np.zeros(n, dtype=np.int32)
    typ[rng.permutation(n)[:light]] = 1
    a, b = 4.0 * 0.2 * 1.7 ** 12, 4.0 * 0.2 * 1.7 ** 6
    s.update(pos=0.4 + 1.9 * sites + rng.uniform(-0.05, 0.05, (n, 3)), type=typ,
             qscaled=water.SQRT_COULOMB * rng.uniform(-0.5, 0.5, n), mass=np.full(n, 16.0),
             mol=np.arange(n, dtype=np.int32), excl=np.zeros((0, 3), dtype=np.int32), n=n)
    s["lj"] = np.zeros((2, 2, 4))
    s["lj"][0, 0] = a, b, a, b
    return s


CASES = {
    "one_water": lambda: _waters(1, (16.0, 16.0, 16.0)),
    "three_waters": lambda: _waters(3, (17.0, 19.0, 16.5)),
    "two_cutoffs": lambda: _waters(136, (16.0, 16.0, 16.0)),
    "odd_edges_unwrapped": lambda: _unwrapped(_waters(509, (16.1, 22.3, 45.0))),
    "dilute_tall_clusters": lambda: _waters(61, (27.0, 33.0, 46.0), rc=12.0),
    "one_full_column": lambda: _waters(331, (60.0, 60.0, 100.0), (9.0, 9.0, 99.0)),
    "long_columns": lambda: _waters(10007, (16.5, 16.5, 1110.0)),
    "long_exclusion_lists": lambda: _merged(_waters(400, (20.0, 25.0, 24.0)), 4, False),
    "modified_pairs": lambda: _merged(_waters(399, (20.0, 25.0, 24.0)), 3, True),
    "flat": lambda: _waters(700, (60.0, 21.0, 16.0)),
    "tall_block_in_vacuum": lambda: _waters(727, (150.0, 140.0, 400.0), (11.0, 11.0, 180.0)),
    "thread_in_vacuum": lambda: _waters(1540, (52.5, 52.5, 1250.0), (6.2, 6.2, 1197.0), rc=11.0),
    "many_columns": lambda: _waters(4500, (1000.0, 1000.0, 16.5), (300.0, 300.0, 16.5)),
    "short_cutoff": lambda: _waters(400, (40.0, 23.0, 40.0), (22.0, 23.0, 24.0), rc=3.0),
    "full_last_flush_104_37": lambda: _ball(104, 37),
    "full_last_flush_99_5": lambda: _ball(99, 5),
    "full_last_flush_104_95": lambda: _ball(104, 95),
}


@pytest.mark.parametrize("name", CASES)
def test_against_oracle(name):
    s = CASES[name]()
    n = s["n"]
    topo = PeriodicTopology.from_dict(s)
    f = NonbondedCutoffB200SystemForce(s["ron"], s["rc_lj"], s["rc_coul"], s["rc_alg"])
    F = np.zeros_like(s["pos"])
    E = ScalarStructure(virial=True, molecular_virial=True)
    f.evaluate(topo, s["pos"], F, E)
    pairs = f.last_pair_count()
    F2, E2 = np.zeros_like(F), ScalarStructure()
    f.evaluate(topo, s["pos"], F2, E2)  # the instance without virial, the counts cleared
    f.close()
    fo, eo, vo, mo = O.restate_eval(s, s["pos"], virial_mode=2)
    assert np.array_equal(F, F2)
    scale = max(np.sqrt((fo ** 2).sum()), 1e-30)
    assert np.sqrt(((F - fo) ** 2).sum()) <= 1e-5 * scale
    for e in (E, E2):
        assert abs(e[0] - eo[0]) <= 1e-4 * n and abs(e[1] - eo[1]) <= 1e-4 * n
    po = O.restate_count_pairs(s, s["pos"])
    assert abs(pairs - po) <= 1 + 1e-6 * po
    for got, want in ((E.virial_matrix(), vo), (E.molvirial_matrix(), mo)):
        want = np.asarray(want).reshape(3, 3)
        assert np.abs(got - want).max() <= 1e-5 * max(np.abs(want).max(), 1.0)


@pytest.mark.parametrize("name", CASES)
def test_fp64_against_oracle(name):
    s = CASES[name]()
    n = s["n"]
    f = NonbondedCutoffB200SystemForce(s["ron"], s["rc_lj"], s["rc_coul"], s["rc_alg"],
                                       precision="fp64")
    F, E = np.zeros_like(s["pos"]), ScalarStructure()
    f.evaluate(PeriodicTopology.from_dict(s), s["pos"], F, E)
    pairs = f.last_pair_count()
    f.close()
    fo, eo, _, _ = O.restate_eval(s, s["pos"], virial_mode=0)
    scale = max(np.sqrt((fo ** 2).sum()), 1e-30)
    assert np.sqrt(((F - fo) ** 2).sum()) <= 1e-12 * scale
    assert abs(E[0] - eo[0]) <= 1e-9 * n and abs(E[1] - eo[1]) <= 1e-9 * n
    assert pairs == O.restate_count_pairs(s, s["pos"])


@pytest.mark.parametrize("precision,length,tol", [
    ("mixed", 1279.0, 2e-6), ("mixed", 1281.0, 2e-6), ("mixed", 19200.0, 2e-6),
    ("fp64", 1281.0, 1e-12), ("fp64", 32760.0, 1e-12), ("fp64", 32800.0, 1e-12),
    ("fp64", 6e5, 1e-12)])
def test_long_boxes(precision, length, tol):
    """The column kernels hold a coordinate to 2^-32 of its edge (at 19,200 A three
    times the FP32 force error of about 1e-6): mixed evaluations of longer boxes, and
    FP64 ones from 4,096 cutoffs on, run on the cell kernels, with the same errors as
    short ones."""
    s = _waters(400, (20.0, 20.0, length), (20.0, 20.0, 30.0), rc=8.0)
    s["pos"] = s["pos"] + np.array([0.0, 0.0, 0.37 * length])
    f = NonbondedCutoffB200SystemForce(s["ron"], s["rc_lj"], s["rc_coul"], s["rc_alg"],
                                       precision=precision)
    F, E = np.zeros_like(s["pos"]), ScalarStructure()
    f.evaluate(PeriodicTopology.from_dict(s), s["pos"], F, E)
    pairs = f.last_pair_count()
    f.close()
    fo, eo, _, _ = O.restate_eval(s, s["pos"], virial_mode=0)
    assert np.sqrt(((F - fo) ** 2).sum()) <= tol * np.sqrt((fo ** 2).sum())
    assert max(abs(E[0] - eo[0]), abs(E[1] - eo[1])) <= tol * 100.0 * s["n"]
    assert abs(pairs - O.restate_count_pairs(s, s["pos"])) <= (precision == "mixed")


HVP_CASES = ["full_last_flush_104_37", "full_last_flush_104_95", "three_waters", "two_cutoffs", "odd_edges_unwrapped", "one_full_column",
             "long_exclusion_lists", "modified_pairs"]
H = 1e-4


def _direction(s):
    v = np.random.default_rng(12).standard_normal(s["pos"].shape)
    return v / np.linalg.norm(v)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", HVP_CASES)
def test_hvp_against_differences(name, precision):
    s = CASES[name]()
    m = NonbondedEnergy.from_system(s, precision=precision)
    q, t = m.initial_params()
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda", requires_grad=True)
    v = _direction(s)
    (g,) = torch.autograd.grad(m.energy(pos, q, t), pos, create_graph=True)
    (hv,) = torch.autograd.grad(g, pos, grad_outputs=torch.tensor(v, device="cuda"))
    m.close()
    fp, fm = (O.restate_eval(s, s["pos"] + d * v, virial_mode=0)[0] for d in (H, -H))
    ref = -(fp - fm) / (2 * H)
    assert np.linalg.norm(hv.cpu().numpy() - ref) <= 1e-6 * np.linalg.norm(ref)


def test_batch_against_oracle():
    boxes = [make() for make in CASES.values()]
    want = [O.restate_eval(s, s["pos"], virial_mode=0)[:2] for s in boxes]
    b = SystemBatch([(NonbondedCutoffB200SystemForce(s["ron"], s["rc_lj"], s["rc_coul"],
                                                     s["rc_alg"]),
                      PeriodicTopology.from_dict(s)) for s in boxes])
    pos = torch.tensor(np.concatenate([s["pos"] for s in boxes]), device="cuda")
    out = torch.zeros((len(boxes), 20), dtype=torch.float64, device="cuda")
    for parts in (1, 2, 8):
        b.set_schedule(parts=parts, order=1)
        frc = torch.zeros_like(pos)
        b.eval_device(pos.data_ptr(), frc.data_ptr(), out.data_ptr(), _lib.PMB200_ENERGY, None)
        b.sync()
        F, at = frc.cpu().numpy(), 0
        for k, (s, (fo, eo)) in enumerate(zip(boxes, want)):
            got = F[at:at + s["n"]]
            at += s["n"]
            assert np.sqrt(((got - fo) ** 2).sum()) <= 1e-5 * max(np.sqrt((fo ** 2).sum()), 1e-30)
            assert np.abs(out[k, :2].cpu().numpy() - eo[:2]).max() <= 1e-4 * s["n"]
    b.close()


FORM_CASES = ["one_water", "two_cutoffs", "odd_edges_unwrapped", "dilute_tall_clusters",
              "long_exclusion_lists", "modified_pairs", "tall_block_in_vacuum"]


def _form(form, s, precision):
    """A force of the form, and the oracle's forces, energies, virials and pairs."""
    rc = s["rc_coul"]
    if form in ("poly5", "exact"):
        alpha, acc = 3.0 / rc, float(np.exp(-9.0))
        fo, eo, vo, mo = O.restate_ewald_real(s, s["pos"], alpha, acc, form == "exact", 2)
        return (EwaldRealB200SystemForce(alpha, acc, precision=precision, erfc=form), fo,
                np.array([eo, 0.0]), vo, mo)
    fo, eo, vo, mo = O.restate_eval(s, s["pos"], virial_mode=2)
    if form == "switches":  # the same potential through the general switches
        f = NonbondedCutoffB200PairForce(("C2", s["ron"], rc), ("C1", 0.0, rc), rc,
                                         precision=precision)
    else:
        f = NonbondedCutoffB200SystemForce(s["ron"], rc, rc, rc, precision=precision)
    return f, fo, np.asarray(eo), vo, mo


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("form", ["poly5", "exact", "switches", "many_types"])
@pytest.mark.parametrize("name", FORM_CASES)
def test_forms_against_oracle(name, form, precision):
    """The other forms and tables beyond shared memory at the same edges; with the
    general switches energies to 1e-6 of the unswitched pair magnitudes, about
    1,000 kcal/mol per atom."""
    s = CASES[name]()
    if form == "many_types":
        s = water.many_types(s)
    f, fo, eo, vo, mo = _form(form, s, precision)
    topo = PeriodicTopology.from_dict(s)
    F, E = np.zeros_like(s["pos"]), ScalarStructure()
    f.evaluate(topo, s["pos"], F, E)
    Fv, Ev = np.zeros_like(F), ScalarStructure(virial=True, molecular_virial=True)
    f.evaluate(topo, s["pos"], Fv, Ev)
    f.close()
    tol, etol = (1e-5, 1e-3 if form == "switches" else 1e-4) if precision == "mixed" else (1e-12,
                                                                                         1e-9)
    for got, e in ((F, E), (Fv, Ev)):
        assert np.sqrt(((got - fo) ** 2).sum()) <= tol * max(np.sqrt((fo ** 2).sum()), 1e-30)
        assert max(abs(e[0] - eo[0]), abs(e[1] - eo[1])) <= etol * s["n"]
    for got, want in ((Ev.virial_matrix(), vo), (Ev.molvirial_matrix(), mo)):
        want = np.asarray(want).reshape(3, 3)
        assert np.abs(got - want).max() <= 1e-5 * max(np.abs(want).max(), 1.0)


@pytest.mark.parametrize("name", ["tall_block_in_vacuum", "thread_in_vacuum", "two_cutoffs"])
def test_shares_sum_to_one_evaluation(name):
    """Shards (bit for bit) and cell ranges (host sums) on overfull layouts."""
    s = CASES[name]()
    topo = PeriodicTopology.from_dict(s)
    f = NonbondedCutoffB200SystemForce(s["ron"], s["rc_lj"], s["rc_coul"], s["rc_alg"])
    pos = torch.tensor(s["pos"], device="cuda")
    frc = torch.zeros_like(pos)
    out = torch.zeros(20, dtype=torch.float64, device="cuda")
    f.evaluate_device(topo, pos.data_ptr(), frc.data_ptr(), out.data_ptr(), _lib.PMB200_ENERGY, 1)
    total = torch.zeros(3 * s["n"], dtype=torch.int64, device="cuda")
    for k in range(3):
        facc = torch.full_like(total, 12345)  # (overwritten)
        f.shard_eval_device(topo, pos.data_ptr(), k, 3, facc.data_ptr(), None, 0, 1)
        total += facc
    sharded = torch.zeros_like(pos)
    f.shard_finalize(total.data_ptr(), sharded.data_ptr(), 1)
    torch.cuda.synchronize()
    want = frc.cpu().numpy()
    scale = np.abs(want).max()
    # (a launch without energies takes the same pairs in the same groups)
    assert np.abs(sharded.cpu().numpy() - want).max() <= 1e-6 * scale
    blocks = f.number_of_blocks(topo)
    F, E = np.zeros_like(want), ScalarStructure()
    for lo, hi in ((0, blocks // 3), (blocks // 3, blocks // 2), (blocks // 2, blocks)):
        f.evaluate_cells(topo, s["pos"], F, E, lo, hi)
    f.close()
    assert np.abs(F - want).max() <= 1e-12 * scale
    e = out.cpu().numpy()
    assert max(abs(E[0] - e[0]), abs(E[1] - e[1])) <= 1e-12 * max(abs(e[0]), abs(e[1]), 1.0)


def _derivatives(s, v, padded):
    """H v and the parameter derivatives of E and of v . G; padded: five types in the
    table, which the general derivative kernel serves."""
    s = dict(s)
    nt = len(s["lj"])
    if padded:
        lj = np.zeros((5, 5, 4))
        lj[:nt, :nt] = s["lj"]
        s["lj"] = lj
    m = NonbondedEnergy.from_system(s, precision="fp64")
    q, t = (x.requires_grad_(True) for x in m.initial_params())
    pos = torch.tensor(s["pos"], device="cuda", requires_grad=True)
    first = torch.autograd.grad(m.energy(pos, q, t), (q, t))
    g = m.gradient(pos, q, t)
    second = torch.autograd.grad(g, (pos, q, t), grad_outputs=torch.tensor(v, device="cuda"))
    m.force.sync()
    m.close()
    cut = lambda x: x[:nt, :nt] if x.dim() == 3 else x  # noqa: E731
    return [cut(x.detach()).cpu().numpy() for x in first + second]


@pytest.mark.parametrize("name", HVP_CASES)
def test_derivatives_against_the_general_kernel(name):
    """Products and parameter derivatives on the column walk, modified pairs among
    them, against the cell walk that serves larger tables: the same FP64 terms in
    another order."""
    s = CASES[name]()
    v = _direction(s)
    for a, b in zip(_derivatives(s, v, False), _derivatives(s, v, True)):
        assert np.linalg.norm(a - b) <= 1e-12 * max(np.linalg.norm(b), 1e-30)


def test_a_direction_that_is_not_finite_stays_local():
    """A NaN in the direction reaches the products of the atoms within the cutoff of
    its atom, and no others."""
    s = CASES["odd_edges_unwrapped"]()
    m = NonbondedEnergy.from_system(s, precision="fp64")
    q, t = m.initial_params()
    pos = torch.tensor(s["pos"], device="cuda", requires_grad=True)
    g = m.gradient(pos, q, t)
    v = torch.tensor(_direction(s), device="cuda")
    (want,) = torch.autograd.grad(g, pos, grad_outputs=v, retain_graph=True)
    m.force.sync()
    bad = v.clone()
    bad[7, 1] = float("nan")
    (got,) = torch.autograd.grad(g, pos, grad_outputs=bad)
    with pytest.raises(_lib.PmbError):
        m.force.sync()
    m.close()
    d = s["pos"] - s["pos"][7]
    d -= s["box"] * np.rint(d / s["box"])
    far = torch.tensor(np.sqrt((d ** 2).sum(1)) > s["rc_coul"] + 1e-6, device="cuda")
    assert torch.equal(got[far], want[far]) and far.sum() > s["n"] // 4
