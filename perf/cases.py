"""Timed cases: the work a program built on this framework has it do.

Every case is one rebuild period of a simulation (20 timesteps, the first of
them with the scheduled rebuild) through the public classes System,
ClusterSystem and Ensemble, ending with the atoms' state in the caller's
buffers, or one single-point evaluation of a configuration. Sizes are fcc cells
per side (4 atoms each); states are perturbed fcc lattices with Maxwell
velocities: disordered neighbour lists and forces, no overlapping atoms.

exact() integrates the same inputs in FP64 with plain torch operations.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "md-bench_b200"))
import mdb  # noqa: E402
import workloads  # noqa: E402

RHO, TEMP, SKIN, DT = 0.8442, 1.44, 0.3, 0.005   # the reference's LJ defaults
EAM_FILE = os.path.join("md-bench_b200", "data", "Cu_u3.eam")
EAM_A, EAM_T, EAM_DT, EAM_SKIN = 3.615, 1600.0, 0.001, 1.0
EV, BOLTZ = 1.036427e-4, 8.617343e-5             # amu (A/ps)^2 in eV; eV/K
PERIOD, REBUILD_STEP = 20, 19                    # a run of PERIOD steps opens with the rebuild
CHECK = 0.15                                     # displacement limit: half the skin


def _case(name, kind, nx, ny, nz, precision, half, **more):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=precision, half=half)
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the benchmark's system: LJ liquid, 1,048,576 atoms, cluster pairs
        _case("cp44_half_1m", "cp", 64, 64, 64, "mixed", 1, n=4),
        # the smallest boxes the cutoff allows: launches and latency
        _case("cp44_half_840", "cp", 6, 5, 7, "mixed", 1, n=4),
        # an ordinary liquid in an odd box, rebuilt when an atom moved too far
        _case("cp44_half_checked", "cp", 23, 17, 29, "mixed", 1, n=4, check=CHECK),
        # the wider cluster shape with full lists
        _case("cp48_full", "cp", 40, 40, 40, "mixed", 0, n=8),
        # the reference's precision: bit-identical double-precision runs
        _case("cp44_full_fp64", "cp", 31, 27, 22, "fp64", 0, n=4),
        # the multi-type liquid (four species), two million atoms
        _case("cp44_types_2m", "cp", 80, 80, 80, "mixed", 1, n=4, types=4),
        # the Verlet-list scheme on the benchmark's system, state on the GPU
        _case("vl_full_1m", "vl", 64, 64, 64, "mixed", 0),
        # Verlet lists in double precision, half lists, an odd box
        _case("vl_half_fp64", "vl", 20, 26, 23, "fp64", 1),
        # the benchmark's copper crystal at 1600 K (embedded atom)
        _case("eam_mixed_131k", "eam", 32, 32, 32, "mixed", 0),
        # a small copper crystal in double precision
        _case("eam_fp64_4k", "eam", 9, 10, 11, "fp64", 0),
        # many independent liquids of 500 to 32,000 atoms advanced together
        _case("ensemble_32", "ens", 0, 0, 0, "mixed", 1, n=4, replicas=32),
        # energies and forces of one given configuration (no timesteps)
        _case("vl_point", "point", 48, 40, 52, "mixed", 0),
    ]


def draw(rng):
    def box(lo, hi):
        n = round(math.exp(rng.uniform(math.log(lo), math.log(hi))))
        f = [rng.uniform(0.85, 1.18) for _ in range(3)]
        return [max(lo, min(hi, round(n * k))) for k in f]

    kind = rng.choice(["cp", "cp", "cp", "vl", "vl", "eam", "ens", "point"])
    if kind == "cp":
        prec = rng.choice(["mixed", "mixed", "mixed", "fp64"])
        types = rng.choice([1, 1, 4])
        nx, ny, nz = box(6 if types == 1 else 7, 64 if prec == "mixed" else 40)
        more = dict(n=rng.choice([4, 4, 8]))
        if types > 1:
            more["types"] = types
        elif rng.random() < 0.25:
            more["check"] = CHECK
        return _case("", kind, nx, ny, nz, prec, rng.choice([0, 1]), **more)
    if kind == "vl":
        return _case("", kind, *box(7, 60), rng.choice(["mixed", "fp64"]), rng.choice([0, 1]))
    if kind == "eam":
        return _case("", kind, *box(6, 36), rng.choice(["mixed", "mixed", "fp64"]), 0)
    if kind == "ens":
        return _case("", kind, 0, 0, 0, "mixed", rng.choice([0, 1, 1]), n=4,
                     replicas=rng.randint(6, 40))
    return _case("", kind, *box(7, 60), rng.choice(["mixed", "fp64"]), rng.choice([0, 1]))


# ---- the physical system of a case --------------------------------------------------
class _Sys:
    """Box, parameters and initial state (device tensors) of one system."""

    def __init__(self, cells, seed, types=1, eam=False, rho=RHO, temp=TEMP):
        self.eam = eam
        self.a = EAM_A if eam else (4.0 / rho) ** (1.0 / 3.0)
        self.box = [n * self.a for n in cells]
        self.n = 4 * cells[0] * cells[1] * cells[2]
        self.eps, self.sig = [1.0], [1.0]
        if types > 1:
            self.eps, self.sig = workloads.c5_types(ntypes=types)
        if eam:
            self.mass, self.cut, self.dt, self.skin = 63.55, _eam_header()[4], EAM_DT, EAM_SKIN
            self.dtf = 0.5 * self.dt / self.mass / EV
            sv = math.sqrt(BOLTZ * EAM_T / (self.mass * EV))
        else:
            self.mass, self.cut, self.dt, self.skin = 1.0, 2.5 * max(self.sig), DT, SKIN
            self.dtf = 0.5 * self.dt
            sv = math.sqrt(temp)
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = _fcc(cells).double() * (0.5 * self.a)
        # displacements of a few percent of the nearest-neighbour distance
        amp = (0.02 if types > 1 else 0.06) * self.a
        x += amp * (2.0 * torch.rand(x.shape, generator=g, device="cuda",
                                     dtype=torch.float64) - 1.0)
        L = torch.tensor(self.box, device="cuda", dtype=torch.float64)
        self.x = x - L * torch.floor(x / L)
        v = sv * torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64)
        self.v = v - v.mean(0)
        self.t = torch.randint(0, types, (self.n,), generator=g, device="cuda",
                               dtype=torch.int32)

    def params(self):
        return dict(xprd=self.box[0], yprd=self.box[1], zprd=self.box[2], cutforce=self.cut,
                    cutneigh=self.cut + self.skin, dt=self.dt, dtforce=self.dtf,
                    natoms=self.n, mass=self.mass, ntypes=len(self.eps),
                    epsilon_per_type=self.eps, sigma_per_type=self.sig)

    def host(self):
        return self.x.cpu().numpy(), self.v.cpu().numpy(), self.t.cpu().numpy()


def _fcc(cells):
    """fcc sites in units of half the lattice constant, in createAtom's order
    (blocks of 8^3 half-cells, x fastest)."""
    r = [torch.arange(2 * n, device="cuda") for n in cells]
    z, y, x = torch.meshgrid(r[2], r[1], r[0], indexing="ij")
    p = torch.stack([x, y, z], -1).reshape(-1, 3)
    p = p[p.sum(1) % 2 == 0]
    b, nb = p // 8, [(2 * n + 7) // 8 for n in cells]
    key = ((b[:, 2] * nb[1] + b[:, 1]) * nb[0] + b[:, 0]) * 512
    w = p % 8
    return p[torch.argsort(key + (w[:, 2] * 8 + w[:, 1]) * 8 + w[:, 0])]


def _systems(case, seed):
    """The case's systems: one, or the ensemble's replicas."""
    if case["kind"] == "ens":
        return [_Sys((n, n, n), seed * 1000 + k, rho=rho, temp=temp)
                for k, (n, rho, temp) in enumerate(workloads.c4_replicas(case["replicas"]))]
    return [_Sys((case["nx"], case["ny"], case["nz"]), seed, types=case.get("types", 1),
                 eam=case["kind"] == "eam")]


# ---- the framework's side -------------------------------------------------------------
def prepare(case, seed):
    kind, prec, half = case["kind"], case["precision"], case["half"]
    ps = _systems(case, seed)
    if kind in ("cp", "ens"):
        total = sum(p.n for p in ps)
        out = [torch.empty((total, 3), dtype=torch.float64).pin_memory().numpy(),
               torch.empty((total, 3), dtype=torch.float64).pin_memory().numpy(),
               torch.empty(total, dtype=torch.int32).pin_memory().numpy()]
        members, views, at = [], [], 0
        for p in ps:
            s = mdb.ClusterSystem(cluster_n=case["n"], half_neigh=half, precision=prec,
                                  **p.params())
            if case.get("check"):
                s.set_rebuild_check(case["check"])
            s.set_atoms(*p.host())
            s.setup()
            members.append(s)
            views.append(tuple(o[at:at + p.n] for o in out))
            at += p.n
        ens = mdb.Ensemble(members) if kind == "ens" else None
        return dict(kind=kind, members=members, views=views, out=out, ens=ens)
    p = ps[0]
    tables = mdb.read_funcfl(EAM_FILE) if kind == "eam" else None
    # a generated crystal's bins; a single point comes as a configuration file does
    s = mdb.System(force_field=mdb.FF_EAM if kind == "eam" else mdb.FF_LJ, half_neigh=half,
                   precision=prec, nx=case["nx"], ny=case["ny"], nz=case["nz"],
                   bin_rule=mdb.BINS_FILE if kind == "point" else mdb.BINS_LATTICE,
                   eam=tables, **p.params())
    st = dict(kind=kind, s=s, n=p.n, x=p.x, v=p.v, t=p.t)
    st["out"] = [torch.empty_like(p.x) for _ in range(3)]
    torch.cuda.synchronize()
    s.set_atoms_ptr(p.n, p.x.data_ptr(), p.v.data_ptr(), p.t.data_ptr())
    if kind != "point":
        s.setup()
    return st


def run(state):
    kind = state["kind"]
    if kind in ("cp", "ens"):
        if kind == "ens":
            state["ens"].run(2 * PERIOD, first_step=REBUILD_STEP)
        else:
            state["members"][0].run(PERIOD, first_step=REBUILD_STEP)
        for s, view in zip(state["members"], state["views"]):
            s.update_single_atoms()
            s.atoms(out=view)
        x, v, t = state["out"]
        return {"x": x, "v": v, "t": t}
    s, (x, v, f) = state["s"], state["out"]
    if kind == "point":
        s.set_atoms_ptr(state["n"], state["x"].data_ptr(), state["v"].data_ptr(),
                        state["t"].data_ptr())
        s.setup()
        th = s.thermo()
        s.atoms_ptr(f=f.data_ptr())
        return {"f": f, "pe": th["PE"], "ke": th["KE"]}
    s.run(PERIOD, first_step=REBUILD_STEP)
    s.atoms_ptr(x=x.data_ptr(), v=v.data_ptr(), f=f.data_ptr())
    return {"x": x, "v": v, "f": f}


def work(case):
    """State in and out once; each pair inside the cutoff once per evaluation."""
    if case["kind"] == "ens":
        atoms = [(4 * n ** 3, rho) for n, rho, _ in workloads.c4_replicas(case["replicas"])]
    else:
        atoms = [(4 * case["nx"] * case["ny"] * case["nz"], RHO)]
    evals = {"ens": 2 * PERIOD, "point": 1}.get(case["kind"], PERIOD)
    by = fl = 0.0
    for n, rho in atoms:
        cut = 2.5
        if case["kind"] == "eam":
            rho, cut = 4.0 / EAM_A ** 3, _eam_header()[4]
        elif case.get("types", 1) > 1:
            cut = 2.5 * max(workloads.c5_types(ntypes=case["types"])[1])
        pairs = 0.5 * n * rho * 4.0 / 3.0 * math.pi * cut ** 3
        fl += evals * (pairs * (70.0 if case["kind"] == "eam" else 27.0) + 18.0 * n)
        by += n * (52.0 + (24.0 if case["kind"] == "point" else 48.0))
    return {"bytes": by, "flops": fl}


def tolerance(case):
    # measured against exact(): FP64 forces 3e-14 after a period; FP32 pair
    # forces 1e-6 to 4e-6, single atoms up to the force's jump at the cutoff
    # (3e-3 of the mean force) where an FP32 distance falls on its other side
    if case["precision"] == "fp64":
        return {"rel": 2e-13, "max": 1e-10}
    return {"rel": 1.5e-5, "max": 1e-2}


# ---- the same in FP64 with plain torch ----------------------------------------------------
def _eam_lines():
    with open(EAM_FILE) as f:
        return f.read().split("\n")


def _eam_header():
    h = _eam_lines()[2].split()
    return int(h[0]), float(h[1]), int(h[2]), float(h[3]), float(h[4])


def _pairs(x, box, cut):
    """(i, j, s): pairs within cut of each other, each once; x[i] - x[j] - s L is
    the difference to the nearest periodic image."""
    n = x.shape[0]
    L = torch.tensor(box, device="cuda", dtype=torch.float64)

    def near(i, j):
        d = x[i] - x[j]
        s = torch.round(d / L)
        k = ((d - s * L) ** 2).sum(-1) < cut * cut
        return i[k].int(), j[k].int(), s[k].to(torch.int8)

    nc = [int(b / cut) for b in box]
    if min(nc) < 3:
        i, j = torch.triu_indices(n, n, 1, device="cuda")
        return near(i, j)
    m = torch.tensor(nc, device="cuda")
    c = torch.minimum((x / L * m).long().clamp_(min=0), m - 1)
    cell = (c[:, 2] * nc[1] + c[:, 1]) * nc[0] + c[:, 0]
    order = torch.argsort(cell, stable=True)
    count = torch.bincount(cell, minlength=nc[0] * nc[1] * nc[2])
    start = torch.cumsum(count, 0) - count
    cap = int(count.max())
    tab = torch.full((count.numel(), cap), -1, device="cuda", dtype=torch.long)
    tab[cell[order], torch.arange(n, device="cuda") - start[cell[order]]] = order
    tab = tab.reshape(nc[2], nc[1], nc[0], cap)
    found = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if (dz, dy, dx) < (0, 0, 0):
                    continue
                other = torch.roll(tab, (-dz, -dy, -dx), (0, 1, 2))
                for z in range(nc[2]):  # one plane of cells at a time bounds the memory
                    a, b = tab[z].reshape(-1, cap, 1), other[z].reshape(-1, 1, cap)
                    a, b = torch.broadcast_tensors(a, b)
                    ok = (a >= 0) & (b >= 0)
                    if (dz, dy, dx) == (0, 0, 0):
                        ok &= a < b
                    found.append(near(a[ok], b[ok]))
    return tuple(torch.cat(c) for c in zip(*found))


def _cluster_pairs(x, box, cut, col, edge2, N, half):
    """(i, j, s, mutual): every atom pair of the listed cluster pairs (4 x N
    atoms), for atoms sorted by column col and height: those with an atom pair
    within cut, and those whose bounding boxes are closer than cut less half a
    column's diagonal (edge2 = its square). Full lists: the pair acts on i. Half
    lists: on both atoms (mutual), once, except across the periodic boundary,
    where both atoms list it."""
    i, j, s = _pairs(x, box, cut + 0.7)  # the boxes' pairs hold one this close
    L = torch.tensor(box, device="cuda", dtype=torch.float64)
    n = len(col)
    _, col, count = torch.unique_consecutive(col, return_inverse=True, return_counts=True)
    r = torch.arange(n, device="cuda") - (torch.cumsum(count, 0) - count)[col]
    nj = (count + N - 1) // N
    J = (torch.cumsum(nj, 0) - nj)[col] + r // N
    ic = J * (N // 4) + (r % N) // 4
    tab = torch.full(((int(nj.sum())) * N,), -1, device="cuda", dtype=torch.long)
    tab[J * N + r % N] = torch.arange(n, device="cuda")
    nJ = int(nj.sum())

    def key(i, j, s):
        s = s.long() + 1
        return ((ic[i] * nJ + J[j]) * 3 + s[:, 0]) * 9 + s[:, 1] * 3 + s[:, 2]

    def extent(c, clusters):
        e = x.new_full((2, clusters, 3), math.inf)
        for k, sign in enumerate((1.0, -1.0)):
            e[k].scatter_reduce_(0, c[:, None].expand(-1, 3), sign * x, "amin")
        return e[0], -e[1]

    def parts(k):
        c = k % 27
        return k // 27 // nJ, k // 27 % nJ, torch.stack([c // 9, c // 3 % 3, c % 3], 1) - 1

    a = torch.arange(n, device="cuda")
    keys = torch.unique(torch.cat([key(i, j, s), key(j, i, -s),
                                   key(a, a, s.new_zeros(n, 3))]))
    hit = torch.zeros(len(keys), device="cuda", dtype=torch.bool)
    for c in zip(*(torch.split(q, 1 << 25) for q in (i, j, s))):
        k = ((x[c[0]] - x[c[1]] - c[2] * L) ** 2).sum(-1) <= cut * cut
        for u, v, w in ((c[0][k], c[1][k], c[2][k]), (c[1][k], c[0][k], -c[2][k])):
            hit[torch.searchsorted(keys, key(u, v, w))] = True
    del i, j, s
    imin, imax = extent(ic, nJ * (N // 4))
    jmin, jmax = extent(J, nJ)
    rbb = max(0.0, cut - 0.5 * math.sqrt(edge2))
    out = []
    for k, h in zip(torch.split(keys, 1 << 20), torch.split(hit, 1 << 20)):
        I, jc, sh = parts(k)
        gap = torch.maximum(imin[I] - jmax[jc] - sh * L, jmin[jc] + sh * L - imax[I])
        k = k[h | ((gap.clamp_(min=0.0) ** 2).sum(1) < rbb * rbb)]
        I, jc, sh = parts(k)
        local = (sh == 0).all(1)
        if half:
            keep = ~local | (I // (N // 4) <= jc)
            sh, I, jc, local = sh[keep], I[keep], jc[keep], local[keep]
        sa = (I[:, None] * 4 + torch.arange(4, device="cuda"))[:, :, None]
        sb = (jc[:, None] * N + torch.arange(N, device="cuda"))[:, None, :]
        diag = (local & (I // (N // 4) == jc))[:, None, None]
        ok = (tab[sa] >= 0) & (tab[sb] >= 0) & ~(diag & ((sa >= sb) if half else (sa == sb)))
        w = ok.nonzero()
        out.append((tab[sa[w[:, 0], w[:, 1], 0]].int(), tab[sb[w[:, 0], 0, w[:, 2]]].int(),
                    sh[w[:, 0]].to(torch.int8), local[w[:, 0]] & bool(half)))
    return tuple(torch.cat(c) for c in zip(*out))


def _spline(f, delta):
    """Cubic through tabulated values: rows (c0, c1, c2, c3) of c0 p^3 + ...,
    p in [0, 1) from the row's point (five-point slopes inside)."""
    n = len(f)
    s = np.zeros(n)
    s[2:n - 2] = ((f[:n - 4] - f[4:]) + 8.0 * (f[3:n - 1] - f[1:n - 3])) / 12.0
    s[0], s[1] = f[1] - f[0], 0.5 * (f[2] - f[0])
    s[n - 2], s[n - 1] = 0.5 * (f[n - 1] - f[n - 3]), f[n - 1] - f[n - 2]
    c = np.zeros((n, 4))
    d = f[1:] - f[:-1]
    c[:-1, 0] = s[:-1] + s[1:] - 2.0 * d
    c[:-1, 1] = 3.0 * d - 2.0 * s[:-1] - s[1:]
    c[:, 2], c[:, 3] = s, f
    return torch.tensor(c, device="cuda")


class _Eam:
    """Tables of the funcfl file, resampled as the potential defines them: all
    but the last point of each table, the charge function squared."""

    def __init__(self):
        nrho, self.drho, nr, self.dr, self.cut = _eam_header()
        v = np.array(" ".join(_eam_lines()[3:]).split(), dtype=float)
        frho, zr, rhor = v[:nrho], v[nrho:nrho + nr], v[nrho + nr:nrho + 2 * nr]
        self.f = _spline(frho[:-1], self.drho)
        self.r = _spline(rhor[:-1], self.dr)
        self.z = _spline(27.2 * 0.529 * zr[:-1] ** 2, self.dr)

    def at(self, c, u, lo):
        m = u.long().clamp_(lo, c.shape[0] - 2)
        p = (u - m).clamp_(max=1.0)
        k = c[m]
        return (((k[:, 0] * p + k[:, 1]) * p + k[:, 2]) * p + k[:, 3],
                (3.0 * k[:, 0] * p + 2.0 * k[:, 1]) * p + k[:, 2])


class _Exact:
    """Velocity Verlet in FP64 over the pairs that the last rebuild listed."""

    def __init__(self, p, case):
        self.p, self.x, self.v, self.t = p, p.x.clone(), p.v.clone(), p.t.clone()
        self.cluster, self.half, self.check = case.get("n", 0), case["half"], case.get("check")
        self.L = torch.tensor(p.box, device="cuda", dtype=torch.float64)
        self.eps = torch.tensor(p.eps, device="cuda", dtype=torch.float64)
        self.sig = torch.tensor(p.sig, device="cuda", dtype=torch.float64)
        self.tab = _Eam() if p.eam else None
        self.rebuild()

    def rebuild(self):
        """Wrap into the box; cluster pairs: atoms by column, then z; the list."""
        p, L = self.p, self.L
        self.x = torch.where(self.x < 0, self.x + L, torch.where(self.x >= L, self.x - L, self.x))
        if self.cluster:
            # a lattice constant may divide the box: the column count hangs on the rounding
            edge = math.cbrt(self.cluster / (p.n / (p.box[0] * p.box[1] * p.box[2])))
            nb = [max(1, math.ceil(b / edge)) for b in p.box]
            ix = (self.x[:, 0] * (nb[0] / p.box[0])).long()
            iy = (self.x[:, 1] * (nb[1] / p.box[1])).long()
            col = iy * (nb[0] + 1) + ix
            o = torch.argsort(self.x[:, 2])
            o = o[torch.argsort(col[o], stable=True)]
            self.x, self.v, self.t = self.x[o], self.v[o], self.t[o]
        if self.cluster:
            edge2 = sum((b / k) ** 2 for b, k in zip(p.box[:2], nb))
            self.pairs = _cluster_pairs(self.x, p.box, p.cut + p.skin, col[o], edge2,
                                        self.cluster, self.half)
        else:
            self.pairs = _pairs(self.x, p.box, p.cut + p.skin)
        self.xb = self.x

    def chunks(self):
        """(i, j, difference, rsq, mutual) of the listed pairs inside the cutoff."""
        for c in zip(*(torch.split(q, 1 << 25) for q in self.pairs)):
            i, j = c[0].long(), c[1].long()
            d = self.x[i] - self.x[j] - c[2] * self.L
            rsq = (d * d).sum(-1)
            k = rsq < self.p.cut ** 2
            yield i[k], j[k], d[k], rsq[k], c[3][k] if self.cluster else None

    def force(self):
        f = torch.zeros_like(self.x)
        pe = 0.0
        if self.tab:
            rho = torch.zeros_like(self.x[:, 0])
            for i, j, _, rsq, _ in self.chunks():
                w, _ = self.tab.at(self.tab.r, rsq.sqrt() / self.tab.dr, 0)
                rho.index_add_(0, i, w)
                rho.index_add_(0, j, w)
            e, fp = self.tab.at(self.tab.f, rho / self.tab.drho, 0)
            fp /= self.tab.drho
            pe += float(e.sum())
        for i, j, d, rsq, mutual in self.chunks():
            if self.tab:
                r = rsq.sqrt()
                _, dr = self.tab.at(self.tab.r, r / self.tab.dr, 0)
                z, dz = self.tab.at(self.tab.z, r / self.tab.dr, 0)
                e = z / r
                fr = -((fp[i] + fp[j]) * dr / self.tab.dr + (dz / self.tab.dr - e) / r) / r
            else:
                ti, tj = self.t[i].long(), self.t[j].long()
                ep = torch.sqrt(self.eps[ti] * self.eps[tj])
                sr6 = (self.sig[ti] * self.sig[tj]) ** 3 / rsq ** 3
                e = 4.0 * ep * sr6 * (sr6 - 1.0)
                fr = 48.0 * ep * sr6 * (sr6 - 0.5) / rsq
            pe += float(e.sum())
            f.index_add_(0, i, d * fr[:, None])
            if mutual is not None:
                j, d, fr = j[mutual], d[mutual], fr[mutual]
            f.index_add_(0, j, d * fr[:, None], alpha=-1.0)
        self.pe = pe
        return f

    def steps(self, count):
        p, f = self.p, self.force()
        for n in range(REBUILD_STEP, REBUILD_STEP + count):
            self.v = self.v + p.dtf * f
            self.x = self.x + p.dt * self.v
            moved = self.check and ((self.x - self.xb) ** 2).sum(1).max() > self.check ** 2
            if (n + 1) % PERIOD == 0 or moved:
                self.rebuild()
            f = self.force()
            self.v = self.v + p.dtf * f
        return f


def exact(case, seed):
    kind = case["kind"]
    out = []
    for p in _systems(case, seed):
        e = _Exact(p, case)
        if kind == "point":
            f = e.force()
            return {"f": f, "pe": e.pe, "ke": 0.5 * p.mass * float((p.v ** 2).sum())}
        f = e.steps(2 * PERIOD if kind == "ens" else PERIOD)
        out.append((e.x, e.v, e.t, f))
    x, v, t, f = (torch.cat(c) for c in zip(*out))
    return {"x": x, "v": v, "t": t} if kind in ("cp", "ens") else {"x": x, "v": v, "f": f}
