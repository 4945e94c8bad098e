"""The pieces of a neighbor-list step that depend on sizes: bins that hold from
none to hundreds of cylinders (a lane walks a bin), key counts around a warp's
block, and the first pass of a vectorization (sent as launches) against the
later ones (a captured graph)."""
import ctypes as C

import numpy as np
import pytest

from medyan_b200._abi import BoundaryParams, CylindersView, NLParams, SystemView
from medyan_b200.forcefield import ForceFieldManager, neighbor_pairs
from medyan_b200.lib import MedyanError
from medyan_b200.network import make_workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,box", [(1, 60.0), (7, 60.0), (8, 60.0), (9, 100.0), (33, 150.0), (700, 120.0), (700, 600.0)])
def test_bins_of_every_fill_match_oracle(gpu_lib, oracle, n, box):
    rng = np.random.default_rng(n)
    mid = 300.0 + rng.uniform(0.0, box, (n, 3))
    off = rng.normal(size=(n, 3)) * 5.0
    x = np.stack([mid - off, mid + off], 1).reshape(-1)
    cv = CylindersView(2 * np.arange(n), 2 * np.arange(n) + 1, np.arange(n), np.arange(n) // 5, np.arange(n) % 5,
                       np.zeros(n), np.full(n, -1), np.ones(n), np.full(n, 10.0), np.full(n, 1e5))
    p = NLParams()
    p.rmax, p.rmin = 54.0, 0.0
    for d in range(3):
        p.grid_size[d] = 1000.0
    st, want = oracle.neighbor_pairs(cv, x, 2 * n, p)
    assert st == 0
    assert np.array_equal(neighbor_pairs(cv, x, 2 * n, p), want)


@pytest.mark.parametrize("cfg", [0, 1])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_first_pass_is_the_later_passes(gpu_lib, oracle, cfg, precision):
    net = make_workload(cfg)
    x = net.flat_coords()
    with ForceFieldManager(precision) as ff:
        ff.vectorize_all_force_fields(net.system_view())
        ff.set_deterministic(True)  # whole-number sums: equal results are equal bits
        ff.set_coords(x)
        ff.set_cylinders(net.cylinders_view(), net.nl_params(), net.boundary_params()[0])
        for _ in range(2):  # the second rebuild starts over with launches
            ff.rebuild_neighbor_lists()
            passes = [ff.evaluate(x) for _ in range(3)]
            alone = [(ff.compute_energy(), ff.compute_forces()) for _ in range(3)]
            for e, _, f in passes[1:]:
                assert e == passes[0][0] and np.array_equal(f, passes[0][2])
            for e, f in alone[1:]:
                assert e == alone[0][0] and np.array_equal(f, alone[0][1])


@pytest.mark.parametrize("n", [31, 683, 2049])  # cylinders: below a warp, around a scan tile of 2,048 counts
@pytest.mark.parametrize("planes", [0, 2, 3])
def test_records_follow_the_lists(gpu_lib, oracle, n, planes):
    """Rebuilds whose lists grow (from none, past what counting keeps of a key),
    shrink, and fail (a midpoint outside the grid): the records are the
    oracle's pairs and the planes' terms, and a failed rebuild changes neither."""
    rng = np.random.default_rng(n + planes)
    unit, off = rng.uniform(0.0, 1.0, (n, 3)), rng.normal(size=(n, 3)) * 2.0
    minus = (np.arange(n) % 3 == 0).astype(np.int32)
    cv = CylindersView(2 * np.arange(n), 2 * np.arange(n) + 1, np.arange(n), np.arange(n) // 5, np.arange(n) % 5,
                       np.zeros(n), np.full(n, -1), minus, np.full(n, 10.0), np.full(n, 1e5))
    p = NLParams()
    p.rmax, p.rmin = 54.0, 0.0
    for d in range(3):
        p.grid_size[d] = 1000.0
    eq = np.array([[1.0, 0.0, 0.0, 0.0], [0.0, -1.0, 0.0, 1000.0], [0.0, 0.0, 1.0, -200.0]])[:planes]
    bp = BoundaryParams()
    bp.n_planes, bp.cutoff, bp.k, bp.screen_length = planes, 250.0, 40.0, 2.7
    bp.plane_eq = eq.ctypes.data_as(C.POINTER(C.c_double)) if planes else None

    def coords(box):
        mid = 300.0 + unit * box
        return np.stack([mid - off, mid + off], 1).reshape(-1)

    def in_order(pairs):
        q = np.asarray(pairs, np.int64).reshape(-1, 2)
        return q[np.lexsort((q[:, 1], q[:, 0]))]

    def records(ff):
        beads, krs, _ = ff.excluded_volume_interactions()
        assert np.all(krs == 1e5 * 10.0 * 10.0)
        return in_order(beads[:, ::2] // 6)  # a cylinder is two beads, three offsets each

    with ForceFieldManager("fp64") as ff:
        ff.vectorize_all_force_fields(SystemView(2 * n))
        ff.set_cylinders(cv, p, bp if planes else None)
        want = []
        for box in (650.0, 200.0, 120.0, 400.0, 2000.0, 300.0):
            x = coords(box)
            ff.set_coords(x)
            if box > 1000.0:
                with pytest.raises(MedyanError):
                    ff.rebuild_neighbor_lists()
                assert np.array_equal(records(ff), want)
                continue
            st, pairs = oracle.neighbor_pairs(cv, x, 2 * n, p)
            assert st == 0
            want = in_order(pairs)
            b = x.reshape(-1, 2, 3)
            near = (0.5 * b[:, 0] + 0.5 * b[:, 1]) @ eq[:, :3].T + eq[:, 3] < 250.0
            terms = int((near * (1 + minus)[:, None]).sum())
            assert ff.rebuild_neighbor_lists() == (len(want), terms)
            assert np.array_equal(records(ff), want)
            if box < 650.0:
                continue  # crowded cylinders overlap: thousands of quadratures
            d = b @ eq[:, :3].T + eq[:, 3]  # distances of both beads; a minus end adds its first
            u = 40.0 * np.exp(-d / 2.7)
            exact = float((near * (u[:, 1] + minus[:, None] * u[:, 0])).sum())
            got = ff.compute_individual_energies(x).as_array()[9]
            # positive terms, each an exp of an argument below 100 that is a few ulp off
            assert abs(got - exact) <= 1e-12 * exact
