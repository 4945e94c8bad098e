"""Neighbor lists of bundles, where a few bins hold all cylinders: every lane of
a key's warp takes its share of them, whatever the bins."""
import time

import numpy as np
import pytest

from medyan_b200._abi import SystemView
from medyan_b200.forcefield import ForceFieldManager, neighbor_pairs
from medyan_b200.network import CylindersView, make_workload

pytestmark = pytest.mark.gpu

N_FIL, N_CYL = 100, 20


def cylinders(x):
    fil, pos = np.repeat(np.arange(N_FIL), N_CYL), np.tile(np.arange(N_CYL), N_FIL)
    b1, n = fil * (N_CYL + 1) + pos, N_FIL * N_CYL
    return CylindersView(b1, b1 + 1, np.arange(n), fil, pos, np.zeros(n), np.full(n, -1), pos == 0,
                         np.full(n, 108.0), np.full(n, 1e5)), np.ascontiguousarray(x.reshape(-1))


def bundle(side):
    """Filaments along z through a square of this side, ends within a cylinder's length."""
    rng = np.random.default_rng(0)
    x = np.empty((N_FIL, N_CYL + 1, 3))
    x[:, :, :2] = rng.uniform(200.0, 200.0 + side, (N_FIL, 1, 2))
    x[:, :, 2] = 200.0 + 107.9 * np.arange(N_CYL + 1) + rng.uniform(0.0, 100.0, (N_FIL, 1))
    return cylinders(x)


@pytest.mark.parametrize("side", [100.0, 300.0])
def test_bundle_pairs_match_oracle(gpu_lib, oracle, side):
    cv, x = bundle(side)
    net = make_workload(0, n_fil=1, cyl_per_fil=1, box=3000.0, n_linker=0, n_motor=0, n_branch=0)
    st, want = oracle.neighbor_pairs(cv, x, x.size // 3, net.nl_params())
    assert st == 0
    assert np.array_equal(neighbor_pairs(cv, x, x.size // 3, net.nl_params()), want)


def test_bundle_takes_little_longer(gpu_lib):
    """A rebuild of the bundle's 35,000 pairs against one of as many cylinders
    spread over the box: 9 times as long with a lane per bin, under 3 now."""
    net = make_workload(0, n_fil=N_FIL, cyl_per_fil=N_CYL, box=3000.0, n_linker=0, n_motor=0, n_branch=0)
    spread = (net.cylinders_view(), net.flat_coords())
    t = []
    for cv, x in (spread, bundle(100.0)):
        with ForceFieldManager("fp64") as ff:
            ff.vectorize_all_force_fields(SystemView(x.size // 3))
            ff.set_coords(x)
            ff.set_cylinders(cv, net.nl_params(), None)
            for _ in range(3):
                ff.rebuild_neighbor_lists()
            best = np.inf
            for _ in range(30):
                a = time.perf_counter()
                ff.rebuild_neighbor_lists()
                best = min(best, time.perf_counter() - a)
            t.append(best)
    assert t[1] <= 4.0 * t[0], t
