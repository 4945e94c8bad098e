"""The pieces of a neighbor-list step that depend on sizes: bins that hold from
none to hundreds of cylinders (a lane walks a bin), key counts around a warp's
block, and the first pass of a vectorization (sent as launches) against the
later ones (a captured graph)."""
import numpy as np
import pytest

from medyan_b200._abi import CylindersView, NLParams
from medyan_b200.forcefield import ForceFieldManager, neighbor_pairs
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
