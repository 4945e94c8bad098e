"""Where a minimization runs: in the resident loop, or, where the device does not
hold its blocks at once, in the graph loop (a batch: packed). Both are the same
minimization: with fixed-point force sums the same bits."""
import ctypes as C

import numpy as np
import pytest

from medyan_b200.forcefield import BatchMinimizer, ForceFieldManager, conjugate_gradient_params as cgp
from medyan_b200.network import make_batch, make_workload

pytestmark = pytest.mark.gpu


def set_room(lib, handle, cluster, grid):
    f = lib.medyan_internal_loop_room
    f.argtypes, f.restype = [C.c_void_p, C.c_int32, C.c_int32], C.c_int32
    assert f(handle, cluster, grid) == 0


def counts(r):
    return r.num_energy_call, r.num_force_call, r.num_iter


def network(ff, n_fil, n_cyl, box):
    net = make_workload(0, n_fil=n_fil, cyl_per_fil=n_cyl, box=box, n_linker=n_fil if n_fil > 20 else 0,
                        n_branch=n_fil // 10, n_motor=0, seed=11)
    x = (net.coords + np.random.default_rng(4).normal(0.0, 0.5, net.coords.shape)).reshape(-1)
    ff.vectorize_all_force_fields(net.system_view())
    ff.set_coords(x)
    ff.set_cylinders(net.cylinders_view(), net.nl_params(), net.boundary_params()[0])
    ff.rebuild_neighbor_lists()
    return x


# one block, a cluster, a grid; below and above the size of the 512-thread blocks, and
# above the size where a vector pass has more components than threads
SIZES = [(2, 3, 700.0), (31, 9, 1500.0), (160, 13, 2200.0), (3500, 20, 6100.0), (3700, 20, 6200.0), (5000, 20, 6900.0)]


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("line_search", ["BACKTRACKING", "QUADRATIC"])
def test_graph_loop_is_the_resident_loop(gpu_lib, size, precision, line_search):
    p = cgp(grad_tol=1e-4, energy_rel_tol=1e-14, energy_call_limit=40, line_search=line_search)
    with ForceFieldManager(precision) as ff:
        x = network(ff, *size)
        ff.set_deterministic(True)
        s1, x1, f1, r1 = ff.minimize(x, p)
        set_room(ff.lib, ff.handle, 0, 0)
        s2, x2, f2, r2 = ff.minimize(x, p)
    assert s1 == s2 == 0 and counts(r1) == counts(r2)
    assert np.array_equal(x1, x2) and np.array_equal(f1, f2)
    assert np.array_equal(np.array(r1.energy_before), np.array(r2.energy_before))
    assert np.array_equal(np.array(r1.energy_after), np.array(r2.energy_after))


@pytest.mark.parametrize("size,room", [((31, 9, 1500.0), (0, 148)), ((160, 13, 2200.0), (16, 20)), ((160, 13, 2200.0), (0, 0))])
def test_too_little_room(gpu_lib, oracle, size, room):
    """Fewer SMs than the team needs: the launch would be refused, the
    minimization runs all the same, as on the whole device."""
    p = cgp(energy_call_limit=20)
    with ForceFieldManager("fp64") as ff:
        x = network(ff, *size)
        ff.set_deterministic(True)
        want = ff.minimize(x, p)
        set_room(ff.lib, ff.handle, *room)
        got = ff.minimize(x, p)
    assert got[0] == want[0] == 0 and np.array_equal(got[1], want[1]) and counts(got[3]) == counts(want[3])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("line_search", ["BACKTRACKING", "QUADRATIC"])
def test_packed_batch_is_the_resident_batch(gpu_lib, precision, line_search):
    """The packed conjugate-gradient loop against the resident one, in the default
    and in other packed shapes (records padded to other blocks), fixed-point sums."""
    nets = make_batch(6, 5, (200, 800))
    xs = [net.flat_coords() for net in nets]
    p = cgp(grad_tol=1e-4, energy_rel_tol=1e-14, energy_call_limit=40, line_search=line_search)
    tol = 1e-7 if line_search == "BACKTRACKING" else 1e-6
    runs = []
    with BatchMinimizer([net.system_view() for net in nets], precision) as b:
        b.set_deterministic(True)
        for r, net in enumerate(nets):
            b.rebuild_neighbor_lists(r, xs[r], net.cylinders_view(), net.nl_params(), net.boundary_params()[0])
        runs.append(b.minimize(xs, p))
        set_room(b.lib, b.replica(3), 0, 0)
        runs.append(b.minimize(xs, p))
        b.set_shapes(bonded_threads=128, excl_threads=32, chain_threads=512, chain_chunk=1024)
        runs.append(b.minimize(xs, p))
        runs.append(b.minimize(xs, p))
    (s0, x0, f0, r0), packed = runs[0], runs[1:]
    for s, x, f, r in packed:
        for i in range(len(nets)):
            assert s[i] == s0[i] == 0 and counts(r[i]) == counts(r0[i])
            assert np.abs(x[i] - x0[i]).max() <= tol and np.abs(f[i] - f0[i]).max() <= tol * np.abs(f0[i]).max()
    for i in range(len(nets)):
        assert np.array_equal(packed[1][1][i], packed[2][1][i])
        if line_search == "BACKTRACKING":  # default shapes: the resident batch's order of sums
            assert np.array_equal(packed[0][1][i], x0[i])
