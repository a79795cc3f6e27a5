"""The work that users of this package have it do, as cases that can be timed.

A case is a dict of plain values.  ``prepare`` makes what a program holds before
the call (seeded inputs and handles), ``run`` is one pass through the package's
public entry points and returns what that pass computes, ``work`` counts the
bytes and operations a pass cannot do without, and ``exact`` gives a pass's
results in 64 bits from plain numpy and torch.

The systems are glycine in SPC/E water at 1 g/cm^3 (``system.make_system``), cut-off
10 A, skin 2 A, DSF alpha 0.2/A.  One system per composition is generated
(clash-free lattice, random orientations); a seed gives other inputs of that
composition: the axes permuted and mirrored, every atom translated, every
molecule displaced a little, velocities drawn for 300 K.
"""
from __future__ import annotations

import functools
import dataclasses
import math
import random

import numpy as np
import torch

from molecular_simulation_code_b200 import batch, mixed, nonbond, system

ALPHA, CUT, SKIN = 0.2, 10.0, 2.0
CLUSTER = dict(mrcut=9.0, denscut=6.0, densmin=11)  # the reference input's criterion
TERMS = {"mixed": mixed.MIXED, "fp64": mixed.FP64}


def listed():
    return [
        # Device-resident Langevin segments, read back at their end.  9,000 atoms is the
        # single small replica (launches and latency), in both precisions; 275,000 atoms
        # is the throughput workload.
        dict(name="md_9k_fp64", kind="md", n_gly=150, n_wat=2500, precision="fp64", steps=40,
             rattle=False),
        dict(name="md_9k_mixed", kind="md", n_gly=150, n_wat=2500, precision="mixed", steps=40,
             rattle=False),
        dict(name="md_275k_mixed", kind="md", n_gly=3500, n_wat=80000, precision="mixed", steps=20,
             rattle=False),
        # A batch of independent replicas of 3,000 to 30,000 atoms advanced together, as a
        # server does between membership changes.
        dict(name="batch_16_mixed", kind="batch", replicas=16, mix=1, precision="mixed", steps=25),
        # The drop-in force call of a host code: positions from host memory, forces and
        # energies back.  One call on a small system, and a short trajectory (list kept,
        # pruned again as atoms move) on a large one.
        dict(name="forces_9k_host", kind="forces", n_gly=150, n_wat=2500, precision="mixed",
             frames=1, virial=False, memory="host"),
        dict(name="forces_275k_host", kind="forces", n_gly=3500, n_wat=80000, precision="mixed",
             frames=4, virial=False, memory="host"),
        # Single-point evaluation of a trial configuration in FP64: new state in, list build,
        # energies, virial and forces out.
        dict(name="point_90k_fp64", kind="point", n_gly=1500, n_wat=25000, precision="fp64"),
        # The reference's own data structures: full Verlet list and FP64 LJ + DSF forces on
        # device arrays (45,255 atoms: the composition of the reference's input file).
        dict(name="verlet_45k_device", kind="verlet", n_gly=1500, n_wat=10085, term="dsf"),
        # The PME path's real-space term over the same list, at an odd size.
        dict(name="verlet_21k_long", kind="verlet", n_gly=401, n_wat=5731, term="long"),
        # A host code's whole list step on host arrays: wrap, cell sort, permute the per-atom
        # arrays, full list and forces back to the host.
        dict(name="host_step_9k", kind="host_step", n_gly=150, n_wat=2500),
        # Torsions with 1-4 pairs, impropers and the excluded-pair corrections on host arrays.
        dict(name="bonded_1500", kind="bonded", n_gly=1500, n_wat=3000),
        # Largest-cluster analysis of 3,500 glycines with a crystalline nucleus.
        dict(name="cluster_3500", kind="cluster", n_gly=3500, n_wat=10000, nucleus=200),
    ]


def _composition(rng: random.Random, n_min: int, n_max: int) -> dict:
    """Atoms spread over the logarithm of [n_min, n_max], 5-20 % of the molecules glycine."""
    n = math.exp(rng.uniform(math.log(n_min), math.log(n_max)))
    f = rng.uniform(0.05, 0.20)
    g = max(1, round(f * n / (10 * f + 3 * (1 - f))))
    return dict(n_gly=g, n_wat=max(1, round((n - 10 * g) / 3)))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["md", "md", "batch", "forces", "forces", "point", "verlet", "verlet",
                       "host_step", "bonded", "cluster"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "md":
        c = _composition(rng, 3000, 250000)
        n = 10 * c["n_gly"] + 3 * c["n_wat"]
        most = min(40, int((1.0 if precision == "mixed" else 0.4) * 5.5e6 / n))
        return dict(kind=kind, **c, precision=precision, steps=rng.randint(5, max(5, most)),
                    rattle=rng.random() < 0.25)
    if kind == "batch":
        return dict(kind=kind, replicas=rng.randint(2, 16), mix=rng.randint(2, 10 ** 6),
                    precision=precision, steps=rng.randint(5, 25 if precision == "mixed" else 10))
    if kind == "forces":
        return dict(kind=kind, **_composition(rng, 3000, 250000), precision=precision,
                    frames=rng.randint(1, 4), virial=rng.random() < 0.3,
                    memory=rng.choice(["host", "device"]))
    if kind == "point":
        return dict(kind=kind, **_composition(rng, 3000, 100000), precision="fp64")
    if kind == "verlet":
        return dict(kind=kind, **_composition(rng, 3000, 60000), term=rng.choice(["dsf", "long"]))
    if kind == "host_step":
        return dict(kind=kind, **_composition(rng, 3000, 20000))
    if kind == "bonded":
        return dict(kind=kind, n_gly=rng.randint(50, 2000), n_wat=rng.randint(1000, 5000))
    g = rng.randint(200, 3500)
    return dict(kind=kind, n_gly=g, n_wat=rng.randint(2 * g, 3 * g),
                nucleus=rng.choice([0, rng.randint(30, 200)]))


# ---------------------------------------------------------------------------
# inputs

@functools.lru_cache(maxsize=24)
def _base(n_gly: int, n_wat: int, nucleus: int = 0):
    return system.make_system(n_gly, n_wat, 17, nucleus=nucleus)


def _seeded(n_gly: int, n_wat: int, seed: int, nucleus: int = 0):
    """The composition's system with the seed's coordinates and velocities."""
    s = _base(n_gly, n_wat, nucleus)
    rng = np.random.default_rng([seed, n_gly, n_wat])
    box = float(s.box)
    x = s.xyz.astype(np.float64)[:, rng.permutation(3)] * rng.choice([-1.0, 1.0], 3)
    x = x + rng.uniform(0.0, box, 3) + rng.uniform(-0.04, 0.04, (s.n_mol, 3))[s.mol_id()]
    xyz = system.wrap_positions(np.mod(x, box).astype(np.float32), s.box)
    sigma = np.sqrt(0.001987204181 * 300.0 * 0.0004184 / s.mass_type[s.types - 1])
    v = (rng.normal(size=(s.np_atoms, 3)) * sigma[:, None]).astype(np.float32)
    return dataclasses.replace(s, xyz=xyz, velocity=v, seed=seed)


def _dsf(s):
    return nonbond.DsfParams(ALPHA, s.box, CUT, CUT, SKIN)


def _md_system(ctx, s, precision, seed, rattle=False):
    m = mixed.System(ctx, s, alpha=ALPHA, cut=CUT, skin=SKIN, precision=TERMS[precision])
    m.set_state(s.xyz.astype(np.float64), s.velocity.astype(np.float64))
    # strong coupling, as segments that bring a start to 300 K use it
    m.md_setup(s, dt=2.0, temperature=300.0, gamma=0.02, seed=seed + 1, rattle=rattle)
    return m


def _replicas(case):
    rng = random.Random(case["mix"])
    return [_composition(rng, 3000, 30000) for _ in range(case["replicas"])]


def _frames(case, s):
    """Positions along a straight flight of 2 fs steps, as 16-byte reference records."""
    out = []
    for k in range(case["frames"]):
        x = s.xyz.astype(np.float64) + 2.0 * k * s.velocity.astype(np.float64)
        f = dataclasses.replace(s, xyz=system.wrap_positions(x.astype(np.float32), s.box))
        out.append(f.position_aos())
    return out


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=True)
    t.copy_(torch.from_numpy(a))
    return t.numpy()


def _torsion_coeff(s, seed):
    return np.random.default_rng(seed + 5).uniform(-1.0, 1.0, (s.dihed_coeff.shape[0], 4))


def _gewald():
    return nonbond.calculate_gewald(CUT)


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, ctx=nonbond.Context(0))
    if kind == "batch":
        st["systems"] = [_md_system(st["ctx"], _seeded(c["n_gly"], c["n_wat"], seed + 97 * k),
                                    case["precision"], seed + k)
                         for k, c in enumerate(_replicas(case))]
        st["batch"] = batch.Batch(st["ctx"], st["systems"])
        st["batch"].set_segment(min(25, case["steps"]))
        return st
    s = st["s"] = _seeded(case["n_gly"], case["n_wat"], seed, case.get("nucleus", 0))
    if kind == "md":
        st["system"] = _md_system(st["ctx"], s, case["precision"], seed, case["rattle"])
    elif kind == "forces":
        st["system"] = mixed.System(st["ctx"], s, alpha=ALPHA, cut=CUT, skin=SKIN,
                                    precision=TERMS[case["precision"]])
        frames = _frames(case, s)
        if case["memory"] == "device":
            st["frames"] = [torch.from_numpy(f).cuda() for f in frames]
            st["ff"] = [torch.zeros((s.np_atoms, 3), device="cuda") for f in frames]
        else:
            st["frames"] = [_pinned(f) for f in frames]
            st["ff"] = [_pinned(np.zeros((s.np_atoms, 3), np.float32)) for f in frames]
    elif kind == "point":
        st["system"] = mixed.System(st["ctx"], s, alpha=ALPHA, cut=CUT, skin=SKIN,
                                    precision=TERMS[case["precision"]])
        st["x"] = s.xyz.astype(np.float64)
    else:
        st["p"] = _dsf(s)
        st["pos"] = s.position_aos()
        st["lj"] = (s.lj1, s.lj2, s.lj3, s.lj4)
        if kind == "verlet":
            dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
            st["pos"], st["q"] = dev(st["pos"]), dev(s.q)
            st["lj"] = tuple(dev(a) for a in st["lj"])
            st["specbond"], st["num3bond"] = dev(s.specbond), dev(s.num3bond)
            st["ff"] = torch.zeros((s.np_atoms, 3), device="cuda")
            st["gewald"] = _gewald()
        elif kind == "bonded":
            st["dihed_coeff"], st["gewald"] = _torsion_coeff(s, seed), _gewald()
        elif kind == "cluster":
            st["pos"] = torch.from_numpy(st["pos"]).cuda()
            st["ids"] = torch.arange(1, s.np_atoms + 1, dtype=torch.int32, device="cuda")
            st["ptta0"] = torch.from_numpy(s.xyz[:10 * s.n_gly].astype(np.float64)).cuda()
            st["ptta"] = torch.empty_like(st["ptta0"])
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# passes

def _state(m):
    """A trajectory frame: coordinates and velocities as the writers store them (real*4)."""
    x, v, _ = m.get_state()
    return x.astype(np.float32), v.astype(np.float32)


def _run_md(st):
    e = st["system"].md_run(st["case"]["steps"], energy_every=st["case"]["steps"])
    x, v = _state(st["system"])
    return dict(energies=e, x=x, v=v)


def _run_batch(st):
    e = st["batch"].run(st["case"]["steps"], energy_every=1)
    frames = [_state(m) for m in st["systems"]]
    names = list(e[0])
    return dict(energies=np.array([[row[k] for k in names] for row in e], np.float32),
                x=np.concatenate([f[0] for f in frames]), v=np.concatenate([f[1] for f in frames]))


def _run_forces(st):
    out = []
    for pos, ff in zip(st["frames"], st["ff"]):
        f, pot, ec, vir = st["system"].forces_dropin(pos, ff, virial=st["case"]["virial"])
        out.append(dict(ff=f, pot=pot, ecoul=ec,
                        virial=None if vir is None else [float(a) for a in vir]))
    return out


def _run_point(st):
    m = st["system"]
    m.set_state(st["x"])
    e = m.compute(virial=True)
    return dict(e=e, f=m.get_state()[2])


def _run_verlet(st):
    c, n = st["ctx"], st["s"].ntypes
    _, _, alloc = nonbond.neighbor_wrapper(c, st["pos"], st["specbond"], st["num3bond"], st["p"],
                                           neigh_alloc=1024, want_host=False)
    if st["case"]["term"] == "dsf":
        r = nonbond.lj_cut_coul_dsf_nonewton(c, st["pos"], st["q"], st["lj"], n, None, None, alloc,
                                             st["p"], ff=st["ff"])
    else:
        r = nonbond.lj_cut_coul_long_nonewton(c, st["pos"], st["q"], st["lj"], n, None, None,
                                              alloc, st["p"], st["gewald"], ff=st["ff"])
    return dict(ff=r[0], pot=r[1], ecoul=r[2], virial=r[3])


def _run_host_step(st):
    c, s, p = st["ctx"], st["s"], st["p"]
    pos = nonbond.pbc(c, st["pos"], s.box)
    tt, ttb, start, end, atombin, pos = nonbond.cell_sort(c, pos, p)
    q = nonbond.sort_posit(c, ttb, s.q)
    v = nonbond.sort_posit(c, ttb, s.velocity)
    spec, n1, n2, n3 = nonbond.sort_specbond_numbond(c, tt, s.specbond, s.num1bond, s.num2bond,
                                                     s.num3bond)
    bonds = nonbond.sort_list(c, tt, s.bonds, 2)
    moved = nonbond.check_neighbor(c, *(np.ascontiguousarray(2.0 * v[:, d]) for d in range(3)),
                                   p.rvrc2)
    nlist, numneigh, alloc = nonbond.neighbor_wrapper(c, pos, spec, n3, p, neigh_alloc=1024)
    ff, pot, ec, vir = nonbond.lj_cut_coul_dsf_nonewton(c, pos, q, st["lj"], s.ntypes, nlist,
                                                        numneigh, alloc, p)
    return dict(order=[tt, ttb, start, end, atombin], pos=pos, q=q, v=v, spec=[spec, n1, n2, n3],
                bonds=bonds, moved=moved, nlist=nlist, numneigh=numneigh, ff=ff, pot=pot, ecoul=ec,
                virial=vir)


def _run_bonded(st):
    c, s, p, pos, g = st["ctx"], st["s"], st["p"], st["pos"], st["gewald"]
    tor = nonbond.dihedral_opls_dsf(c, pos, s.q, s.ntypes, s.lj14, s.dihedrals, st["dihed_coeff"],
                                    p)
    imp = nonbond.improper_harmonic(c, pos, s.impropers, s.impro_coeff, p)
    c12 = nonbond.correct_12_bonds(c, pos, s.q, s.bonds, g, 0.0, p)
    c13 = nonbond.correct_13_bonds(c, pos, s.q, s.angles, g, 0.0, p)
    c14 = nonbond.correct_14_bonds(c, pos, s.q, s.dihedrals, g, 0.5, p)
    return dict(torsion=tor, improper=imp, c12=c12, c13=c13, c14=c14)


def _run_cluster(st):
    s = st["s"]
    st["ptta"].copy_(st["ptta0"])
    torch.cuda.current_stream().synchronize()  # the analysis runs on the context's stream
    size, greatest, dens, belongs = nonbond.get_greatest_cluster(
        st["ctx"], st["pos"], st["ids"], s.n_gly, 10, s.box, ptta_full=st["ptta"], **CLUSTER)
    return dict(size=size, greatest=greatest, dens=dens, belongs=belongs, ptta=st["ptta"])


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


# ---------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    if case["kind"] == "batch":
        n = sum(10 * c["n_gly"] + 3 * c["n_wat"] for c in _replicas(case))
    else:
        n = 10 * case["n_gly"] + 3 * case["n_wat"]
    density = 0.1  # atoms per A^3 at 1 g/cm^3
    pairs = 0.5 * n * density * 4.0 / 3.0 * math.pi * CUT ** 3
    near = pairs * ((CUT + SKIN) / CUT) ** 3
    flop = 60.0  # per pair inside the cut-off: displacement, LJ, DSF Coulomb, accumulation
    kind = case["kind"]
    if kind in ("md", "batch"):
        k = case["steps"]
        return dict(bytes=n * (96.0 * k + 48.0), flops=k * (flop * pairs + 200.0 * n))
    if kind == "forces":
        return dict(bytes=28.0 * n * case["frames"], flops=case["frames"] * flop * pairs)
    if kind == "point":
        return dict(bytes=48.0 * n, flops=flop * pairs + 10.0 * near)
    if kind == "verlet":
        return dict(bytes=n * 90.0 + 8.0 * near, flops=2 * flop * pairs + 20.0 * near)
    if kind == "host_step":
        return dict(bytes=n * 200.0 + 8.0 * near, flops=2 * flop * pairs + 20.0 * near)
    if kind == "bonded":
        terms = 15 * case["n_gly"], 9 * case["n_gly"] + 2 * case["n_wat"]
        return dict(bytes=5 * 40.0 * n + 20.0 * sum(terms), flops=300.0 * terms[0] + 80.0 * terms[1])
    g = case["n_gly"]
    return dict(bytes=20.0 * n + 480.0 * g, flops=g * (100.0 + 27 * 8 * 12.0))


# ---------------------------------------------------------------------------
# the same results in 64 bits

F32 = lambda v: float(np.float32(v))  # noqa: E731
P_ERFC = F32(0.3275911)
A_ERFC = [F32(a) for a in (0.254829592, -0.284496736, 1.421413741, -1.453152027, 1.061405429)]
ROOT_PI = F32(1.77245385090551602729)
COULPRE = F32(332.06371)


def _erfc(z, e):
    """Abramowitz and Stegun 7.1.26 with e = exp(-z^2), the reference's erfc."""
    t = 1.0 / (1.0 + P_ERFC * z)
    return t * (A_ERFC[0] + t * (A_ERFC[1] + t * (A_ERFC[2] + t * (A_ERFC[3] + t * A_ERFC[4])))) * e


def _shifts():
    e = math.exp(-(ALPHA * CUT) ** 2)
    c = math.erfc(ALPHA * CUT)
    f = -(c / CUT ** 2 + 2.0 / ROOT_PI * ALPHA * e / CUT)
    return c / CUT - f * CUT, f


def _pair_terms(r2, qq, lj, term):
    """F/r, LJ energy and Coulomb energy of pairs at squared distance r2."""
    r = torch.sqrt(r2)
    i6 = 1.0 / r2 ** 3
    flj, elj = i6 * (lj[0] * i6 - lj[1]), i6 * (lj[2] * i6 - lj[3])
    pref = COULPRE * qq / r
    if term == "long":
        g = _gewald() * r
        e = torch.exp(-g * g)
        c = _erfc(g, e)
        return (pref * (c + F32(1.12837917) * g * e) + flj) / r2, elj, pref * c
    e_shift, f_shift = _shifts()
    e = torch.exp(-ALPHA * ALPHA * r2)
    c = _erfc(ALPHA * r, e)
    fc = pref * (c / r + 2.0 * ALPHA / ROOT_PI * e + r * f_shift) * r
    return (fc + flj) / r2, elj, pref * (c - r * e_shift - r2 * f_shift)


def _nonbonded(s, xyz, term="dsf"):
    """Forces (n,3), LJ and Coulomb energies and diagonal virial over all pairs inside the
    cut-off that are not excluded."""
    n, box = s.np_atoms, float(s.box)
    x = torch.from_numpy(np.asarray(xyz, np.float64)).cuda()
    q = torch.from_numpy(s.q).cuda().double()
    ty = torch.from_numpy(s.types.astype(np.int64) - 1).cuda()
    tab = [torch.from_numpy(t).cuda().double() for t in (s.lj1, s.lj2, s.lj3, s.lj4)]
    spec = torch.from_numpy(np.where(np.arange(12)[None] < s.num3bond[:, None],
                                     s.specbond.astype(np.int64) - 1, -1)).cuda()
    order = torch.argsort(x[:, 2])  # rows of one slab look at a z window of atoms only
    z = x[order, 2].contiguous()
    zz = torch.cat([z - box, z, z + box])
    f = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    sums = torch.zeros(5, dtype=torch.float64, device="cuda")
    rows = max(64, int(3e7 * box / (n * (2 * CUT + 2.0))))
    for a in range(0, n, rows):
        i = order[a:a + rows]
        lo = int(torch.searchsorted(zz, z[a] - CUT - 1e-3))
        hi = int(torch.searchsorted(zz, z[min(a + rows, n) - 1] + CUT + 1e-3))
        j = order[(torch.arange(lo, min(hi, lo + n), device="cuda")) % n]
        r2 = torch.zeros((len(i), len(j)), dtype=torch.float64, device="cuda")
        for d in range(3):
            t = x[i, d][:, None] - x[j, d][None, :]
            t -= box * torch.round(t / box)
            r2 += t * t
        k, m = torch.nonzero((r2 <= CUT * CUT) & (i[:, None] != j[None, :]), as_tuple=True)
        del r2
        k, m = i[k], j[m]
        keep = ~(spec[k] == m[:, None]).any(1)
        k, m = k[keep], m[keep]
        dx = x[k] - x[m]
        dx -= box * torch.round(dx / box)
        o = ty[k] * s.ntypes + ty[m]
        fr, elj, ec = _pair_terms((dx * dx).sum(1), q[k] * q[m], [t[o] for t in tab], term)
        f.index_add_(0, k, dx * fr[:, None])
        sums += 0.5 * torch.stack([elj.sum(), ec.sum(), *(dx * dx * fr[:, None]).sum(0)])
    e = [float(v) for v in sums]
    return f.cpu().numpy(), e[0], e[1], np.array(e[2:])


def _minimum(d, box):
    return d - box * torch.round(d / box)


def _scattered(n, ids, parts):
    f = torch.zeros((n, 3), dtype=torch.float64)
    for k, p in zip(ids, parts):
        f.index_add_(0, k, p)
    return f.numpy()


def _exact_bonded(s, coeff):
    x = torch.from_numpy(s.xyz.astype(np.float64))
    q, ty = torch.from_numpy(s.q).double(), torch.from_numpy(s.types.astype(np.int64) - 1)
    box, n, g = float(s.box), s.np_atoms, _gewald()
    ids = lambda lst, cols: [torch.from_numpy(lst[:, c].astype(np.int64) - 1) for c in cols]  # noqa: E731

    def angle(y, quad):
        a, b, c, d = (y[k] for k in quad)
        v1, v2, v3 = _minimum(a - b, box), _minimum(c - b, box), _minimum(d - c, box)
        u, w = torch.cross(v1, v2, dim=1), torch.cross(v2, v3, dim=1)
        return -(u * w).sum(1) / (u.norm(dim=1) * w.norm(dim=1))

    def minus_gradient(energy):
        y = x.clone().requires_grad_(True)
        e = energy(y)
        e.backward()
        return -y.grad, float(e.detach())

    quad = ids(s.dihedrals, range(4))
    k = torch.from_numpy(coeff)[torch.from_numpy(s.dihedrals[:, 4].astype(np.int64) - 1)]

    def torsion(y):
        c = angle(y, quad)
        c2, c3, c4 = 2 * c * c - 1, 4 * c ** 3 - 3 * c, 8 * c ** 4 - 8 * c * c + 1
        return (k[:, 0] * (1 + c) + k[:, 1] * (1 - c2) + k[:, 2] * (1 + c3)
                + k[:, 3] * (1 - c4)).sum()

    ft, et = minus_gradient(torsion)
    i, j = quad[0], quad[3]
    d = _minimum(x[i] - x[j], box)
    lj14 = torch.from_numpy(np.asarray(s.lj14, np.float64))
    half = [t[ty[i], ty[j]] for t in lj14]
    fr, elj, ec = _pair_terms((d * d).sum(1), 0.5 * q[i] * q[j], half, "dsf")
    f14 = _scattered(n, [i, j], [d * fr[:, None], -d * fr[:, None]])
    out = dict(torsion=[ft.numpy() + f14, et, float(ec.sum()), float(elj.sum())], improper=None)
    for name, lst, cols, fudge in (("c12", s.bonds, (0, 1), 0.0), ("c13", s.angles, (0, 2), 0.0),
                                   ("c14", s.dihedrals, (0, 3), 0.5)):
        i, j = ids(lst, cols)
        d = _minimum(x[i] - x[j], box)
        r2 = (d * d).sum(1)
        r = torch.sqrt(r2)
        pref, e = COULPRE * q[i] * q[j] / r, torch.exp(-(g * r) ** 2)
        c = _erfc(g * r, e)
        fr = pref * (c + F32(1.12837917) * g * r * e - (1.0 - fudge)) / r2
        out[name] = [_scattered(n, [i, j], [d * fr[:, None], -d * fr[:, None]]),
                     float((pref * (c - (1.0 - fudge))).sum()),
                     (d * d * fr[:, None]).sum(0).numpy()]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("md", "batch"):
        return None  # trajectories
    s = _seeded(case["n_gly"], case["n_wat"], seed, case.get("nucleus", 0))
    if kind == "forces":
        out = []
        for pos in _frames(case, s):
            f, pot, ec, vir = _nonbonded(s, pos[:, :3])
            out.append(dict(ff=f, pot=pot, ecoul=ec,
                            virial=[float(a) for a in vir] if case["virial"] else None))
        return out
    if kind == "point":
        f, pot, ec, vir = _nonbonded(s, s.xyz)
        return dict(e=np.array([pot, ec, *vir]), f=f)
    if kind == "verlet":
        f, pot, ec, vir = _nonbonded(s, s.xyz, case["term"])
        return dict(ff=f, pot=pot, ecoul=ec, virial=vir)
    if kind == "host_step":
        f, pot, ec, vir = _nonbonded(s, s.xyz)
        width = float(np.float32(s.box) / np.float32(int(np.float32(s.box) / np.float32(CUT))))
        side = int(float(s.box) / CUT)
        c = np.minimum((s.xyz.astype(np.float64) * (1.0 / width)).astype(np.int64), side - 1)
        cell = c[:, 0] + side * (c[:, 1] + side * c[:, 2])
        order = np.lexsort((-np.arange(s.np_atoms), cell))  # descending index inside a cell
        return dict(ff=f[order], pot=pot, ecoul=ec, virial=vir)
    if kind == "bonded":
        return _exact_bonded(s, _torsion_coeff(s, seed))
    x = s.xyz[:10 * s.n_gly].astype(np.float64).reshape(-1, 10, 3)
    d = x - x[:, :1]
    return dict(ptta=(x - float(s.box) * np.round(d / float(s.box))).reshape(-1, 3))
