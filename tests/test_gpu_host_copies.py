"""What host coordinates and results cost: the bead order does not change the
time of a call, and a call that only brings coordinates takes what the copy
takes. Bounds stand between what is measured and what the slower forms took."""
import time

import numpy as np
import pytest

from medyan_b200._abi import SystemView
from medyan_b200.forcefield import ForceFieldManager

pytestmark = pytest.mark.gpu


def chain(n, shuffled):
    rng = np.random.default_rng(n)
    x = np.cumsum(rng.normal([27.0, 0.0, 0.0], 2.0, (n, 3)), 0)
    at = rng.permutation(n) if shuffled else np.arange(n)
    ext = np.empty_like(x)
    ext[at] = x
    return SystemView(n, stretch_beads=3 * np.stack([at[:-1], at[1:]], 1), stretch_k=np.full(n - 1, 100.0),
                      stretch_l0=np.full(n - 1, 27.0)), ext.reshape(-1)


def best(f, reps=60):
    for _ in range(5):
        f()
    t = []
    for _ in range(reps):
        a = time.perf_counter()
        f()
        t.append(time.perf_counter() - a)
    return min(t)


def test_bead_order_costs_little(gpu_lib):
    """Gathered bead by bead on the host, 21,000 beads in random order took 1.25
    times as long; the device's gather takes 1.03."""
    t = []
    for shuffled in (False, True):
        sv, x = chain(21000, shuffled)
        with ForceFieldManager("fp64") as ff:
            ff.vectorize_all_force_fields(sv)
            t.append(best(lambda: ff.evaluate(x)))
    assert t[1] <= 1.15 * t[0], t


def test_large_arrays_take_the_copies_time(gpu_lib):
    """126,000 beads: coordinates alone took 1.7 times the plain copy through the
    staging, an evaluation 1.6 times the two copies and the pass; 1.05 and 1.1
    without it."""
    import torch

    n = 126000
    sv, x = chain(n, False)
    host, dev, back = torch.from_numpy(x), torch.empty(3 * n, dtype=torch.float64, device="cuda"), torch.empty(3 * n, dtype=torch.float64)

    def copy_in():
        dev.copy_(host)
        torch.cuda.synchronize()

    def copy_out():
        back.copy_(dev)
        torch.cuda.synchronize()

    with ForceFieldManager("fp64") as ff:
        ff.vectorize_all_force_fields(sv)
        t_in, t_out = best(copy_in), best(copy_out)
        t_set, t_eval = best(lambda: ff.set_coords(x)), best(lambda: ff.evaluate(x))
    assert t_set <= 1.35 * t_in, (t_set, t_in)
    assert t_eval <= 1.35 * (t_in + t_out), (t_eval, t_in, t_out)


def test_coordinates_alone_cost_no_launch(gpu_lib):
    """Through the staging, 504 beads took 1.25 times as long as 312, which took
    the plain copy; 1.03 when both do."""
    t = []
    for n in (312, 504):
        sv, x = chain(n, False)
        with ForceFieldManager("fp64") as ff:
            ff.vectorize_all_force_fields(sv)
            t.append(best(lambda: ff.set_coords(x), reps=1000))
    assert t[1] <= 1.13 * t[0], t
