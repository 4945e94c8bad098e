"""Host coordinates and results through the handle's pinned staging: bead counts
around one piece, around the four pieces that are in flight together, and far
more; the caller's bead order permuted; memory that is copied plainly (pinned).
Everything is one copy of the same numbers, so all ways agree bit for bit with
whole-number force sums."""
import ctypes as C

import numpy as np
import pytest

from medyan_b200._abi import FF_COUNT, SystemView
from medyan_b200.forcefield import ForceFieldManager

pytestmark = pytest.mark.gpu

PIECE = 5460


def chain(n, shuffled):
    """One filament of n beads (one bead: no interaction), its beads numbered
    along it or at random."""
    rng = np.random.default_rng(n)
    x = np.cumsum(rng.normal([27.0, 0.0, 0.0], 2.0, (n, 3)), 0)
    at = rng.permutation(n) if shuffled else np.arange(n)
    ext = np.empty_like(x)
    ext[at] = x
    sv = SystemView(n, stretch_beads=3 * np.stack([at[:-1], at[1:]], 1), stretch_k=np.full(n - 1, 100.0),
                    stretch_l0=np.full(n - 1, 27.0))
    return sv, ext.reshape(-1)


@pytest.mark.parametrize("n", [1, 2, 85, PIECE - 1, PIECE, PIECE + 1, 4 * PIECE, 4 * PIECE + 1, 5 * PIECE, 60001])
@pytest.mark.parametrize("shuffled", [False, True])
def test_staged_calls_match_plain_copies(gpu_lib, oracle, n, shuffled):
    import torch

    sv, x = chain(n, shuffled)
    fo = oracle.forces(sv, x)
    eo, _ = oracle.energy(sv, x)
    with ForceFieldManager("fp64") as ff:
        ff.vectorize_all_force_fields(sv)
        ff.set_deterministic(True)
        e, per, f = ff.evaluate(x)
        e2, per2, f2 = ff.evaluate(x[::-1].copy())
        ff.set_coords(x)
        assert np.array_equal(ff.get_coords(), x)
        f3 = ff.compute_forces()
        xp, fp = torch.from_numpy(x).pin_memory(), torch.empty(3 * n, dtype=torch.float64).pin_memory()
        tot, pp = C.c_double(), (C.c_double * FF_COUNT)()
        ptr = lambda t: C.cast(t.data_ptr(), C.POINTER(C.c_double))
        assert ff.lib.medyan_mech_evaluate(ff.handle, ptr(xp), C.byref(tot), pp, ptr(fp)) == 0
    assert np.array_equal(f3, f) and np.array_equal(fp.numpy(), f) and tot.value == e
    assert abs(e - eo) <= 1e-12 * abs(eo)
    assert np.abs(f - fo).max() <= 1e-9 * max(np.abs(fo).max(), 1.0)  # whole-number force sums
    assert n == 1 or not np.array_equal(f2, f)
