"""Floating-point force sums in the resident loop: a small network's minimization
does not depend on the order in which its blocks add."""
import numpy as np
import pytest

from medyan_b200.forcefield import BatchMinimizer, ForceFieldManager, conjugate_gradient_params as cgp
from medyan_b200.network import make_workload

pytestmark = pytest.mark.gpu


def network(oracle, **kw):
    net = make_workload(0, **{**dict(n_fil=12, cyl_per_fil=6, box=700.0, n_linker=16, seed=3), **kw})
    st, extra = oracle.complete(net)
    assert st == 0
    return net.system_view(**extra), net.flat_coords()


def test_runs_end_alike(gpu_lib, oracle):
    """To the tolerances, 100 times: 8 to 10 of them ended at other energies, by 5
    to 35 %, when other last bits of the forces led them another way."""
    sv, x = network(oracle)
    so, xo, fo, ro = oracle.minimize(sv, x, cgp())
    with ForceFieldManager("fp64") as ff:
        ff.vectorize_all_force_fields(sv)
        runs = [ff.minimize(x, cgp()) for _ in range(100)]
    for s, xg, f, r in runs:
        assert s == so == 0 and r.num_iter == ro.num_iter
        assert abs(r.energy_after_total - ro.energy_after_total) <= 1e-2 * ro.energy_after_total
    assert len({r.energy_after_total for _, _, _, r in runs}) <= 2


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_runs_end_alike(gpu_lib, oracle, precision):
    reps = [network(oracle, n_fil=12 + 3 * k, seed=3 + k, box=800.0) for k in range(6)]
    with BatchMinimizer([sv for sv, _ in reps], precision) as b:
        runs = [b.minimize([x for _, x in reps], cgp(energy_call_limit=400)) for _ in range(8)]
    for s, xs, _, rs in runs[1:]:
        assert s == runs[0][0] == [0] * len(reps)
        for r, r0 in zip(rs, runs[0][3]):
            assert (r.num_iter, r.num_energy_call) == (r0.num_iter, r0.num_energy_call)


@pytest.mark.parametrize("size", [1e9, 1e-9])
def test_large_and_small_forces(gpu_lib, size):
    """Springs whose forces lie beyond the exact sums' range (2^25 pN) and below their
    last place (2^-26): the forces of a fresh evaluation, to rounding."""
    from medyan_b200._abi import SystemView
    n = 40
    rng = np.random.default_rng(1)
    x = rng.uniform(0.0, 100.0, (n, 3)).reshape(-1)
    pairs = np.array([(a, b) for a in range(n) for b in range(a + 1, n)])
    sv = SystemView(n, stretch_beads=3 * pairs, stretch_k=np.full(len(pairs), size), stretch_l0=np.full(len(pairs), 30.0))
    with ForceFieldManager("fp64") as ff:
        ff.vectorize_all_force_fields(sv)
        s, xg, f, r = ff.minimize(x, cgp(energy_call_limit=3, grad_tol=0.0, energy_rel_tol=0.0, max_dist=1e-3))
        want = ff.compute_forces(xg)
    # a bead's force is a sum of 39 contributions of up to 75 size, each rounded once or twice
    assert s == 0 and np.abs(f - want).max() <= 2 * 39 * 39 * 75.0 * size * 2.0 ** -53
