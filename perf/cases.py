"""Timed workloads of the mechanics path, through its public entry points.

Every case is one kind of call on a synthetic actin network of n_fil filaments
of n_cyl cylinders (the generator and the composition of the benchmark
workloads: linkers, motors, branch points, excluded volume and a cubic
boundary from the device neighbor list):

  evaluate   energy, per-force-field energies and forces at host coordinates
             (ForceFieldManager.evaluate, one call per step of a host program)
  resident   the same at coordinates that live on the device
             (medyan_mech_enqueue_evaluate and the handle's device buffers)
  minimize   conjugate-gradient minimization from host coordinates, to the
             reference's tolerances or to a limit on the energy calls
  batch      an ensemble of independent networks minimized together
  step       neighbor-list rebuild, then energy and forces with the new lists
  hvp        Hessian-vector product (the backward pass of an implicit adjoint)

A network's topology depends on the case alone and is kept per process; the
bead coordinates (thermal displacements around the generator's positions) are
drawn from the seed. An ensemble's displacements are fixed and the seed moves
each replica as a whole: in some displaced ensembles a coplanar pair's force
leaves the fixed-point range of the deterministic sums, which ends the batch.
"""
from __future__ import annotations

import ctypes as C
from functools import lru_cache

import numpy as np
import torch

from medyan_b200._abi import FF_COUNT, SystemView
from medyan_b200.forcefield import BatchMinimizer, ForceFieldManager, conjugate_gradient_params
from medyan_b200.network import CYL_LEN, CylindersView, NetworkSpec, batch_specs, make_network

JITTER = 0.5        # nm, standard deviation of a coordinate's displacement
TILE_LIMIT = 3000   # networks with more filaments are 2 x 2 x 2 blocks of an eighth each


def listed() -> list[dict]:
    return [
        # the smallest networks of the test suite: one call per step, latency counts
        dict(name="evaluate_50x10_fp64", kind="evaluate", n_fil=50, n_cyl=10, prec="fp64"),
        # a mid-size network (the differentiation workload's size) in the mixed mode
        dict(name="evaluate_500x20_mixed", kind="evaluate", n_fil=500, n_cyl=20, prec="mixed"),
        # an odd size: no filament or record count is a multiple of a block
        dict(name="resident_1237x17_fp64", kind="resident", n_fil=1237, n_cyl=17, prec="fp64"),
        # the benchmark's 400k-cylinder network in both precisions
        dict(name="resident_20000x20_mixed", kind="resident", n_fil=20000, n_cyl=20, prec="mixed"),
        dict(name="resident_20000x20_fp64", kind="resident", n_fil=20000, n_cyl=20, prec="fp64"),
        # whole minimizations to the reference's tolerances
        dict(name="minimize_50x10_fp64", kind="minimize", n_fil=50, n_cyl=10, prec="fp64", limit=0),
        dict(name="minimize_500x20_mixed", kind="minimize", n_fil=500, n_cyl=20, prec="mixed", limit=0),
        # the first iterations of larger ones (a call limit is what a user sets
        # to bound the time of a mechanics step)
        dict(name="minimize_2000x20_fp64", kind="minimize", n_fil=2000, n_cyl=20, prec="fp64", limit=400),
        dict(name="minimize_20000x20_mixed", kind="minimize", n_fil=20000, n_cyl=20, prec="mixed", limit=100),
        # an ensemble of replicas, sizes log-uniform over a factor of 20
        dict(name="batch_128_fp64", kind="batch", replicas=128, lo=200, hi=4000, prec="fp64", limit=100),
        # once per mechanics step: the lists follow the moved beads
        dict(name="step_2000x20_fp64", kind="step", n_fil=2000, n_cyl=20, prec="fp64"),
        # the backward direction
        dict(name="hvp_500x20_fp64", kind="hvp", n_fil=500, n_cyl=20, prec="fp64"),
    ]


def draw(rng) -> dict:
    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["evaluate", "resident", "resident", "minimize", "minimize", "batch", "step", "hvp"])
    prec = rng.choice(["fp64", "mixed"])
    n_cyl = rng.randint(6, 20)
    if kind == "batch":
        return dict(kind=kind, replicas=log_int(8, 96), lo=200, hi=rng.randint(800, 4000), prec=prec,
                    limit=rng.randint(40, 100))
    if kind == "minimize":
        n_fil = log_int(40, 2500)
        return dict(kind=kind, n_fil=n_fil, n_cyl=n_cyl, prec=prec, limit=0 if n_fil < 300 else rng.randint(60, 300))
    top = {"evaluate": 2500, "resident": 20000, "step": 2500, "hvp": 1000}[kind]
    return dict(kind=kind, n_fil=log_int(50, top), n_cyl=n_cyl, prec="fp64" if kind == "hvp" else prec)


# ------------------------------------------------------------------ networks
def spec_of(n_fil: int, n_cyl: int) -> NetworkSpec:
    """The medium workload's composition at its cylinder density (40,000 in a
    5 um cube), in a box that holds the filaments."""
    n = n_fil * n_cyl
    box = max(5000.0 * (n / 40000.0) ** (1.0 / 3.0), 1.39 * n_cyl * CYL_LEN, 1500.0)
    return NetworkSpec(f"net_{n_fil}x{n_cyl}", n_fil, n_cyl, box, n_linker=n // 10, n_motor=n // 100,
                       n_branch=n // 100, seed=n_fil + 7 * n_cyl)


class Net:
    """Arrays of one network: coordinates, topology, records."""

    def __init__(self, net, tiles: int = 1):
        s = net.spec
        nb, nc, nf = net.n_beads, net.n_cyl, s.n_fil
        m = tiles ** 3
        shift = np.array([(i, j, k) for i in range(tiles) for j in range(tiles) for k in range(tiles)], float) * s.box
        self.box, self.spec, self.n_beads, self.n_cyl = s.box * tiles, s, m * nb, m * nc
        self.coords = (net.coords[None] + shift[:, None, :]).reshape(-1, 3)

        def rep(a, step):  # one copy per tile, indices shifted
            a = np.asarray(a)
            return np.concatenate([np.where(a >= 0, a + t * step, a) for t in range(m)]).astype(np.int32)

        self.bead1, self.bead2 = rep(net.cyl_bead1, nb), rep(net.cyl_bead2, nb)
        self.fil, self.pos = rep(net.cyl_fil, nf), np.tile(net.cyl_pos, m)
        self.branching, self.minus = rep(net.cyl_branching, nc), np.tile(net.cyl_minus_end, m)
        self.eqlen, self.exclk = np.tile(net.cyl_eqlen, m), np.tile(net.cyl_exclk, m)
        self.ff = {k: v if np.ndim(v) == 0 else rep(v, 3 * nb) if k.endswith("_beads") else np.tile(v, m)
                   for k, v in net.ff.items()}
        for k in [k for k in self.ff if k.endswith("_beads")]:
            self.ff[k] = self.ff[k].reshape(-1, net.ff[k].shape[1])
        self.net = net

    def cylinders(self):
        n = self.n_cyl
        return CylindersView(self.bead1, self.bead2, np.arange(n, dtype=np.int32), self.fil, self.pos,
                             np.zeros(n, np.int32), self.branching, self.minus, self.eqlen, self.exclk)

    def planes(self):
        lo, hi, rows = 25.0, self.box - 25.0, []
        for axis in range(3):
            for point, sign in ((lo, 1.0), (hi, -1.0)):
                n = [0.0, 0.0, 0.0]
                n[axis] = sign
                rows.append(n + [-sign * point])
        return np.asarray(rows)

    def lists(self):
        """(cylinders, neighbor-list parameters, boundary parameters, keep-alive)."""
        nl = self.net.nl_params()
        for k in range(3):
            nl.grid_size[k] = self.box
        b, _ = self.net.boundary_params()
        planes = np.ascontiguousarray(self.planes())
        b.plane_eq = planes.ctypes.data_as(C.POINTER(C.c_double))
        return self.cylinders(), nl, b, planes


@lru_cache(maxsize=16)
def network(n_fil: int, n_cyl: int) -> Net:
    if n_fil <= TILE_LIMIT:
        return Net(make_network(spec_of(n_fil, n_cyl)))
    return Net(make_network(spec_of(max(n_fil // 8, 1), n_cyl)), tiles=2)


@lru_cache(maxsize=8)
def ensemble(replicas: int, lo: int, hi: int) -> list:
    """An ensemble's replicas: up to 32 networks, each the start of several replicas."""
    nets = [Net(make_network(s)) for s in batch_specs(min(replicas, 32), cyl_range=(lo, hi))]
    return [nets[r % len(nets)] for r in range(replicas)]


def positions(net: Net, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    return np.ascontiguousarray((net.coords + rng.normal(0.0, JITTER, net.coords.shape)).reshape(-1))


def replica_positions(nets: list, seed: int) -> list:
    shifts = np.random.default_rng(seed).uniform(-5.0, 5.0, (len(nets), 3))
    return [(positions(n, r).reshape(-1, 3) + shifts[r]).reshape(-1) for r, n in enumerate(nets)]


class _Device:
    """A device array of the library as torch sees it; a tensor made from it
    keeps the handle that owns the memory."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 2}


def params_of(case: dict):
    return conjugate_gradient_params(energy_call_limit=case["limit"] if "limit" in case else 0)


# ------------------------------------------------------------- state and run
def prepare(case: dict, seed: int) -> dict:
    if case["kind"] == "batch":
        nets = ensemble(case["replicas"], case["lo"], case["hi"])
        b = BatchMinimizer([SystemView(n.n_beads, **n.ff) for n in nets], case["prec"])
        b.set_deterministic(True)
        xs = replica_positions(nets, seed)
        for r, n in enumerate(nets):
            b.rebuild_neighbor_lists(r, xs[r], *n.lists()[:3])
        return dict(case=case, batch=b, x=xs, params=params_of(case))
    net = network(case["n_fil"], case["n_cyl"])
    ffm = ForceFieldManager(case["prec"])
    ffm.vectorize_all_force_fields(SystemView(net.n_beads, **net.ff))
    x = positions(net, seed)
    ffm.set_coords(x)
    keep = net.lists()
    ffm.set_cylinders(*keep[:3])
    ffm.rebuild_neighbor_lists()
    state = dict(case=case, ffm=ffm, x=x, keep=keep, params=params_of(case))
    if case["kind"] == "minimize":
        ffm.set_deterministic(True)  # a long path is only repeatable with order-independent sums
    if case["kind"] == "hvp":
        state["v"] = np.random.default_rng(seed + 1).normal(size=x.size)
    if case["kind"] in ("resident", "step"):
        p = [C.c_void_p() for _ in range(3)]
        ffm.lib.medyan_mech_device_buffers(ffm.handle, *(C.byref(q) for q in p))
        state["forces"] = torch.as_tensor(_Device(ffm, p[1].value, x.size), device="cuda")
        state["energies"] = torch.as_tensor(_Device(ffm, p[2].value, FF_COUNT + 1), device="cuda")
    return state


def run(s: dict):
    kind = s["case"]["kind"]
    if kind == "evaluate":
        total, per, f = s["ffm"].evaluate(s["x"])
        return dict(total=total, energies=per, forces=f)
    if kind == "resident":
        s["ffm"].lib.medyan_mech_enqueue_evaluate(s["ffm"].handle)
        return dict(energies=s["energies"], forces=s["forces"])
    if kind == "step":
        n_excl, n_boundary = s["ffm"].rebuild_neighbor_lists()
        s["ffm"].lib.medyan_mech_enqueue_evaluate(s["ffm"].handle)
        return dict(n_excl=n_excl, n_boundary=n_boundary, energies=s["energies"], forces=s["forces"])
    if kind == "hvp":
        return dict(hv=s["ffm"].hvp(s["v"]))
    if kind == "minimize":
        status, x, f, r = s["ffm"].minimize(s["x"], s["params"])
        return dict(status=status, coords=x, forces=f, before=np.array(r.energy_before),
                    after=np.array(r.energy_after), calls=np.array([r.num_iter, r.num_energy_call, r.num_force_call]))
    status, xs, fs, rs = s["batch"].minimize(s["x"], s["params"])
    return dict(status=np.array(status), coords=np.concatenate(xs), forces=np.concatenate(fs),
                before=np.array([list(r.energy_before) for r in rs]),
                after=np.array([list(r.energy_after) for r in rs]),
                calls=np.array([[r.num_iter, r.num_energy_call, r.num_force_call] for r in rs]))


# ---------------------------------------------------------------------- work
def work(case: dict) -> dict:
    """Bytes: coordinates in, forces out, every record read once per
    evaluation; a minimization also reads and writes its search direction and
    both force vectors per iteration. Flops: the potentials' FP64 operations."""
    if case["kind"] == "batch":
        n = case["replicas"] * (case["hi"] - case["lo"]) / np.log(case["hi"] / case["lo"])  # mean of a log-uniform size
        n_fil = n / 10
    else:
        n, n_fil = case["n_fil"] * case["n_cyl"], case["n_fil"]
    beads = n + n_fil
    pairs = 0.12 * n  # excluded-volume pairs at this density
    ev = 48 * beads + 33 * beads + 48 * 0.11 * n + 80 * 0.01 * n + 24 * pairs
    fl = 150 * n + 150 * 0.11 * n + 600 * 0.01 * n + 2500 * pairs
    times = 1
    if case["kind"] in ("minimize", "batch"):
        times = case["limit"] // 2 if case.get("limit") else 400
        ev += 7 * 24 * beads
    return {"bytes": float(ev * times), "flops": float(fl * times)}


# --------------------------------------------------- 64-bit reference values
def _dot(a, b):
    return (a * b).sum(-1)


def _close_pairs(net: Net, x: torch.Tensor) -> torch.Tensor:
    """Excluded-volume pairs (key, neighbor): key id > neighbor id, midpoints
    within the cutoff, not within two positions on one filament, and not a
    branch's first cylinder with the parent it branches off."""
    dev = x.device
    b1, b2, fil, pos, br = (torch.as_tensor(a, device=dev, dtype=torch.long)
                            for a in (net.bead1, net.bead2, net.fil, net.pos, net.branching))
    mid = 0.5 * (x[b1] + x[b2])
    cut = float(net.spec.volume_cutoff)
    g = int(net.box // cut) + 2
    cell = (mid / cut).floor().long() + 1
    key = (cell[:, 0] * (g + 2) + cell[:, 1]) * (g + 2) + cell[:, 2]
    order = torch.argsort(key)
    skey = key[order]
    found = []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                k = key + (dx * (g + 2) + dy) * (g + 2) + dz
                lo, hi = torch.searchsorted(skey, k), torch.searchsorted(skey, k, right=True)
                n = hi - lo
                i = torch.repeat_interleave(torch.arange(key.numel(), device=dev), n)
                j = order[torch.arange(i.numel(), device=dev) - torch.repeat_interleave(n.cumsum(0) - n, n)
                          + torch.repeat_interleave(lo, n)]
                keep = (i > j) & ~((fil[i] == fil[j]) & ((pos[i] - pos[j]).abs() <= 2)) & (br[j] != i)
                i, j = i[keep], j[keep]
                d = mid[j] - mid[i]
                near = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]) <= cut * cut
                found.append(torch.stack([i[near], j[near]], 1))
    return torch.cat(found)


def _excl_energy(c, krs):
    """Repulsion of two segments c[:, 0:2], c[:, 2:4]: the analytic integral of 1/r^4."""
    c1, c2, c3, c4 = c.unbind(1)
    r12, r34, r31, r14, r32 = c2 - c1, c4 - c3, c1 - c3, c4 - c1, c2 - c3
    a, b, cc, d, e, F = _dot(r12, r12), _dot(r34, r34), _dot(r31, r31), _dot(r12, r34), _dot(r12, r31), _dot(r34, r31)
    g, h, i = _dot(r12, r14), _dot(r34, r32), _dot(r34, r14)
    root = lambda p, q, s: torch.sqrt((torch.sqrt(p * q) + s) * (torch.sqrt(p * q) - s))  # noqa: E731
    AA, BB, EE, FF = root(a, cc, e), root(b, cc, F), root(a, _dot(r14, r14), g), root(b, _dot(r32, r32), h)
    CC, DD, GG = d * e - a * F, b * e - d * F, d * g - a * i
    HH = CC + GG - DD
    jj = _dot(torch.linalg.cross(r12, r34), r31)
    at = torch.atan
    return 0.5 * krs / (-jj * jj) * (CC / AA * (at((a + e) / AA) - at(e / AA))
                                     + GG / EE * (at((a + e - d) / EE) - at((e - d) / EE))
                                     + DD / BB * (at(F / BB) - at((F - b) / BB))
                                     + HH / FF * (at((d + F) / FF) - at((d + F - b) / FF)))


def _out_of_plane(c):
    """The force path moves bead 2 of a nearly coplanar pair 0.01 nm along the plane's normal."""
    v1, v2, v3 = c[:, 1] - c[:, 0], c[:, 2] - c[:, 0], c[:, 3] - c[:, 0]
    n = torch.linalg.cross(v1, v2)
    n = n / torch.sqrt(_dot(n, n))[:, None]
    flat = (_dot(v3, n) / torch.sqrt(_dot(v3, v3))).abs() < 0.1
    return torch.stack([c[:, 0], c[:, 1] + 0.01 * n * flat[:, None], c[:, 2], c[:, 3]], 1)


def _terms(net: Net, x: torch.Tensor):
    """(slot, bead indices [n, k], energy of beads [n, k, 3], bead shift or None) of every force field."""
    dev = x.device
    t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
    idx = lambda a: torch.as_tensor(np.asarray(a) // 3, device=dev, dtype=torch.long)  # noqa: E731
    ff, out = net.ff, []
    length = lambda r: torch.sqrt(_dot(r, r))  # noqa: E731

    def bend(r1, r2, k, th):
        cos = _dot(r1, r2) / (length(r1) * length(r2))
        if not bool((th != 0).any()):
            return k * (1 - cos)
        return k * (1 - (cos * torch.cos(th) + torch.sqrt(1 - cos * cos) * torch.sin(th)))

    def at(c, i, j, p):
        return c[:, i] * (1 - p)[:, None] + c[:, j] * p[:, None]

    k, l0 = t(ff["stretch_k"]), t(ff["stretch_l0"])
    out.append((0, idx(ff["stretch_beads"]), lambda c, k=k, l0=l0: 0.5 * k * (length(c[:, 1] - c[:, 0]) - l0) ** 2, None))
    bk, th = t(ff["bend_k"]), t(ff["bend_theta0"])
    out.append((1, idx(ff["bend_beads"]), lambda c: bend(c[:, 1] - c[:, 0], c[:, 2] - c[:, 1], bk, th), None))
    for slot, name in ((2, "linker"), (3, "motor")):
        if name + "_beads" in ff:
            k, l0, p, q = (t(ff[name + s]) for s in ("_k", "_l0", "_pos1", "_pos2"))
            out.append((slot, idx(ff[name + "_beads"]), lambda c, k=k, l0=l0, p=p, q=q:
                        0.5 * k * (length(at(c, 2, 3, q) - at(c, 0, 1, p)) - l0) ** 2, None))
    if "branch_beads" in ff:
        b, p = idx(ff["branch_beads"]), t(ff["branch_pos"])
        sk, sl, ck, ct, dk = (t(ff["branch_" + s]) for s in
                              ("stretch_k", "stretch_l0", "bend_k", "bend_theta0", "dihedral_k"))

        def dihedral(c):
            m = at(c, 0, 1, p)
            n1 = torch.linalg.cross(c[:, 1] - m, c[:, 2] - m)
            n2 = torch.linalg.cross(c[:, 3] - c[:, 2], c[:, 2] - m)
            return dk * (1 - _dot(n1, n2) / (length(n1) * length(n2)))

        out.append((4, b, lambda c: 0.5 * sk * (length(c[:, 2] - at(c, 0, 1, p)) - sl) ** 2, None))
        out.append((5, b, lambda c: bend(c[:, 1] - c[:, 0], c[:, 3] - c[:, 2], ck, ct), None))
        out.append((6, b, dihedral, None))
    pr = _close_pairs(net, x)
    b1, b2 = (torch.as_tensor(a, device=dev, dtype=torch.long) for a in (net.bead1, net.bead2))
    krs = t(net.exclk)[pr[:, 0]] * t(net.eqlen)[pr[:, 0]] * t(net.eqlen)[pr[:, 1]]
    beads = torch.stack([b1[pr[:, 0]], b2[pr[:, 0]], b1[pr[:, 1]], b2[pr[:, 1]]], 1)
    out.append((8, beads, lambda c: _excl_energy(c, krs), _out_of_plane))
    mid, minus = 0.5 * (x[b1] + x[b2]), torch.as_tensor(net.minus, device=dev) != 0
    for pl in t(net.planes()):
        near = mid @ pl[:3] + pl[3] < net.spec.boundary_cutoff
        on = torch.cat([b2[near], b1[near & minus]])[:, None]
        s = net.spec
        out.append((9, on, lambda c, pl=pl: s.boundary_k * torch.exp(-(c[:, 0] @ pl[:3] + pl[3]) / s.boundary_slen), None))
    return out


def _energies(terms, x) -> torch.Tensor:
    e = torch.zeros(FF_COUNT, dtype=torch.float64, device=x.device)
    for slot, beads, energy, _ in terms:
        e[slot] += energy(x[beads]).sum()
    return e


def _forces(terms, x) -> torch.Tensor:
    f = torch.zeros_like(x)
    for _, beads, energy, shift in terms:
        if beads.numel():
            c = x[beads] if shift is None else shift(x[beads])
            g = torch.func.grad(lambda q: energy(q).sum())(c)
            f = f.index_add(0, beads.reshape(-1), -g.reshape(-1, 3))
    return f


def exact(case: dict, seed: int):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "batch":  # only the start's energies are no outcome of a chaotic path
        before = []
        nets = ensemble(case["replicas"], case["lo"], case["hi"])
        for net, at in zip(nets, replica_positions(nets, seed)):
            x = torch.as_tensor(at, device=dev).view(-1, 3)
            before.append(_energies(_terms(net, x), x).cpu().numpy())
        return dict(status=None, coords=None, forces=None, before=np.stack(before), after=None, calls=None)
    net = network(case["n_fil"], case["n_cyl"])
    x = torch.as_tensor(positions(net, seed), device=dev).view(-1, 3)
    terms = _terms(net, x)
    if case["kind"] == "hvp":
        v = torch.as_tensor(np.random.default_rng(seed + 1).normal(size=x.numel()), device=dev).view(-1, 3)
        return dict(hv=-torch.func.jvp(lambda q: _forces(terms, q), (x,), (v,))[1].reshape(-1).cpu().numpy())
    e = _energies(terms, x)
    if case["kind"] == "minimize":
        return dict(status=None, coords=None, forces=None, before=e.cpu().numpy(), after=None, calls=None)
    f = _forces(terms, x).reshape(-1)
    if case["kind"] == "evaluate":
        return dict(total=float(e.sum()), energies=e.cpu().numpy(), forces=f.cpu().numpy())
    got = dict(energies=torch.cat([e, e.sum()[None]]), forces=f)
    return got if case["kind"] == "resident" else dict(n_excl=None, n_boundary=None, **got)
