"""Cylinder pairs on four lanes each and on one thread each: the pair counts
where a warp, a block or the choice between the two forms is partly filled,
against the oracle. The pairs are skew cylinders at 30-90 degrees, where the
formula is well conditioned, so the tolerance is the golden networks' 1e-12
(1e-6 for the mixed mode's forces, its stated bound)."""
import numpy as np
import pytest

from medyan_b200._abi import SystemView
from medyan_b200.forcefield import ForceFieldManager

pytestmark = pytest.mark.gpu


def pairs(n, seed=0):
    rng = np.random.default_rng(seed)
    at = 500.0 * np.stack([np.arange(n) % 20, np.arange(n) // 20 % 20, np.arange(n) // 400], 1)
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    w = np.cross(u, rng.normal(size=(n, 3)))
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    ang = rng.uniform(np.pi / 6, np.pi / 2, (n, 1))
    v = np.cos(ang) * u + np.sin(ang) * w
    off = rng.uniform(10.0, 50.0, (n, 1)) * np.cross(u, w) + rng.uniform(-30.0, 30.0, (n, 1)) * u
    x = np.stack([at - 54 * u, at + 54 * u, at + off - 54 * v, at + off + 54 * v], 1)
    beads = 12 * np.arange(n)[:, None] + 3 * np.arange(4)[None]
    return SystemView(4 * n, excl_beads=beads, excl_k=np.full(n, 1e5), excl_eqlen=np.full(2 * n, 108.0)), x.reshape(-1)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 15, 16, 17, 65, 8000, 8001])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_pair_counts_match_oracle(gpu_lib, oracle, n, precision):
    sv, x = pairs(n)
    eo, per = oracle.energy(sv, x)
    fo = oracle.forces(sv, x)
    with ForceFieldManager(precision) as ff:
        ff.vectorize_all_force_fields(sv)
        e, p, f = ff.evaluate(x)
        e1, f1 = ff.compute_energy(), ff.compute_forces()
    assert abs(e - eo) <= 1e-12 * abs(eo) and e1 == e
    tol = 1e-12 if precision == "fp64" else 1e-6
    assert np.abs(f - fo).max() <= tol * np.abs(fo).max()
    assert np.abs(f1 - f).max() <= 1e-12 * np.abs(fo).max()
