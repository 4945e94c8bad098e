"""The resident minimizer loop (one kernel per minimization) against the
oracle's CGMethod, at the sizes where its team of blocks changes: one block, a
cluster, the largest cluster, a cooperative grid, and partial warps and tiles
at each. Tolerances are those of the short runs in test_gpu_cg.py."""
import numpy as np
import pytest

from medyan_b200._abi import SystemView
from medyan_b200.forcefield import ForceFieldManager, conjugate_gradient_params as cgp
from medyan_b200.network import make_workload

pytestmark = pytest.mark.gpu

# filaments, cylinders per filament, box (nm)
SIZES = [(1, 1, 500.0), (2, 3, 700.0), (7, 6, 800.0), (31, 9, 1500.0), (83, 10, 1600.0), (160, 13, 2200.0)]


def network(oracle, n_fil, n_cyl, box):
    net = make_workload(0, n_fil=n_fil, cyl_per_fil=n_cyl, box=box, n_linker=n_fil if n_fil > 20 else 0,
                        n_branch=n_fil // 10, n_motor=0, seed=11)
    net.coords += np.random.default_rng(4).normal(0.0, 0.5, net.coords.shape)
    st, extra = oracle.complete(net)
    assert st == 0
    return net.system_view(**extra), net.flat_coords()


def counts(r):
    return r.num_energy_call, r.num_force_call, r.num_iter


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("line_search", ["BACKTRACKING", "QUADRATIC"])
def test_short_run_matches_oracle(gpu_lib, oracle, size, line_search):
    sv, x = network(oracle, *size)
    p = cgp(grad_tol=1e-4, energy_rel_tol=1e-14, energy_call_limit=40, line_search=line_search)
    so, xo, fo, ro = oracle.minimize(sv, x, p)
    tol = 1e-7 if line_search == "BACKTRACKING" else 1e-6
    for deterministic in (False, True):
        with ForceFieldManager("fp64") as ff:
            ff.vectorize_all_force_fields(sv)
            ff.set_deterministic(deterministic)
            sg, xg, fg, rg = ff.minimize(x, p)
            again = ff.minimize(x, p)
        assert sg == so and counts(rg) == counts(ro)
        assert np.abs(xg - xo).max() <= tol
        assert np.abs(fg - fo).max() <= tol * max(np.abs(fo).max(), 1.0)
        if deterministic:  # the same bits on every run
            assert np.array_equal(again[1], xg) and np.array_equal(again[2], fg) and counts(again[3]) == counts(rg)


def test_mixed_forces_reproduce(gpu_lib, oracle):
    """Mixed precision with fixed-point sums: a second run gives the same bits,
    and forces equal a fresh evaluation at the returned coordinates."""
    sv, x = network(oracle, 83, 10, 1600.0)
    with ForceFieldManager("mixed") as ff:
        ff.vectorize_all_force_fields(sv)
        ff.set_deterministic(True)
        s, xg, fg, r = ff.minimize(x, cgp(energy_call_limit=60))
        s2, x2, f2, r2 = ff.minimize(x, cgp(energy_call_limit=60))
        f = ff.compute_forces(xg)
    assert s == s2 == 0 and np.array_equal(xg, x2) and np.array_equal(fg, f2)
    assert np.array_equal(fg, f)


@pytest.mark.parametrize("tilt", [0.0, 1e-3])
def test_rejected_pair_is_finished_by_the_graph_loop(gpu_lib, oracle, tilt):
    """A collinear cylinder pair needs the reference's quadrature: the loop
    hands over, in its setup when the pair starts collinear (tilt 0), in front
    of the pass that meets it when springs pull it collinear. The stretched
    springs' energy must fall and every call be counted as the oracle does."""
    x = np.array([0, 0, 0, 10, 0, 0, 20, 0, 0, 30, tilt, 0, 30, -tilt, 0], float)
    sv = SystemView(5, excl_beads=[0, 3, 6, 9], excl_k=[1e-4], excl_eqlen=[10.0, 10.0],
                    stretch_beads=[9, 12], stretch_k=[50.0], stretch_l0=[0.0])
    p = cgp(grad_tol=1e-12, energy_rel_tol=0.0, energy_call_limit=4)
    so, xo, fo, ro = oracle.minimize(sv, x, p)
    with ForceFieldManager("fp64") as ff:
        ff.vectorize_all_force_fields(sv)
        sg, xg, fg, rg = ff.minimize(x, p)
    assert sg == so and counts(rg) == counts(ro)
    assert np.isfinite(xg).all() and np.abs(xg - xo).max() <= 1e-7
    assert abs(rg.energy_after_total - ro.energy_after_total) <= 1e-9 * max(abs(ro.energy_after_total), 1.0)


def test_forces_after_failed_line_searches(gpu_lib):
    """Springs minimized past what rounding allows: line searches fail, safe
    mode and recovery steps follow. Wherever a call limit ends the run, the
    returned forces are a fresh evaluation's, bit for bit (fixed-point sums)."""
    rng = np.random.default_rng(0)
    n = 5
    x = (np.array([[0, 0, 0], [10, 0, 0], [5, 8, 0]], float)[None] + rng.normal(0, 1.0, (n, 3, 3)) +
         np.arange(n)[:, None, None] * np.array([50.0, 0, 0])).reshape(-1)
    b = 9 * np.arange(n)[:, None]
    beads = np.stack([b + [0, 3], b + [3, 6], b + [6, 0]], 1).reshape(-1, 2)
    sv = SystemView(3 * n, stretch_beads=beads, stretch_k=np.tile([100.0, 50.0, 20.0], n),
                    stretch_l0=np.tile([10.0, 10.0, 25.0], n))
    with ForceFieldManager("fp64") as ff:
        ff.vectorize_all_force_fields(sv)
        ff.set_deterministic(True)
        failed = 0
        for limit in range(300, 1500, 37):
            s, xg, fg, r = ff.minimize(x, cgp(grad_tol=1e-14, energy_rel_tol=0.0, energy_call_limit=limit,
                                              force_call_limit=10 ** 6))
            assert s == 0 and np.array_equal(fg, ff.compute_forces(xg)), (limit, counts(r))
            failed += r.num_force_call < r.num_iter
        assert failed > 0  # some runs ended after a failed line search


@pytest.mark.parametrize("size", [(7, 6, 800.0), (83, 10, 1600.0), (500, 20, 3200.0), (2400, 20, 5500.0)])
def test_energies_are_the_energy_kernels(gpu_lib, size):
    """The loop's energies are the per-potential kernels' bit for bit, from a few
    energy rows to shares of more than 32 rows (the largest size), and on teams
    where the rounds have blocks of their own and where they do not."""
    n_fil, n_cyl, box = size
    net = make_workload(0, n_fil=n_fil, cyl_per_fil=n_cyl, box=box, n_linker=n_fil, n_branch=n_fil // 4,
                        n_motor=n_fil // 8, seed=11)
    with ForceFieldManager("fp64") as ff:
        ff.vectorize_all_force_fields(net.system_view())
        ff.set_coords(net.flat_coords())
        ff.set_cylinders(net.cylinders_view(), net.nl_params(), net.boundary_params()[0])
        ff.rebuild_neighbor_lists()
        s, x, f, r = ff.minimize(net.flat_coords(), cgp(energy_call_limit=30))
        ff.set_shapes(pass_layout=1)
        before = ff.compute_individual_energies(net.flat_coords()).as_array()
        after = ff.compute_individual_energies(x).as_array()
    assert s == 0
    assert np.array_equal(before, np.array(r.energy_before)) and np.array_equal(after, np.array(r.energy_after))
