"""What a minimization leaves in the handle: its device buffers hold the final
coordinates, the forces there and the energies there, whatever ended the run."""
import ctypes as C

import numpy as np
import pytest

from medyan_b200._abi import FF_COUNT, SystemView
from medyan_b200.forcefield import ForceFieldManager, conjugate_gradient_params as cgp
from medyan_b200.network import make_workload

pytestmark = pytest.mark.gpu


def device_energies(ff):
    import torch
    p = [C.c_void_p() for _ in range(3)]
    ff.lib.medyan_mech_device_buffers(ff.handle, *(C.byref(q) for q in p))

    class Array:
        __cuda_array_interface__ = {"shape": (FF_COUNT + 1,), "typestr": "<f8", "data": (p[2].value, False), "version": 2}
    return torch.as_tensor(Array(), device="cuda").cpu().numpy().copy()


def degenerate():
    """A bend whose first two beads coincide (NaN energy) and a stretched spring."""
    x = np.array([0, 0, 0, 0, 0, 0, 10, 0, 0, 30, 5, 0, 60, 5, 0], float)
    return SystemView(5, bend_beads=[0, 3, 6], bend_k=[10.0], bend_theta0=[0.0], stretch_beads=[9, 12],
                      stretch_k=[5.0], stretch_l0=[20.0]), x


@pytest.mark.parametrize("end", ["limit", "converged", "failed"])
def test_energy_buffer_holds_the_final_energies(gpu_lib, end):
    if end == "failed":
        sv, x = degenerate()
        p = cgp(grad_tol=1e-3, try_to_recover=False)
    else:
        net = make_workload(0)
        sv, x = net.system_view(), net.flat_coords()
        p = cgp(energy_call_limit=30) if end == "limit" else cgp(grad_tol=1e30)
    with ForceFieldManager("fp64") as ff:
        ff.vectorize_all_force_fields(sv)
        ff.evaluate(x + np.random.default_rng(0).normal(0.0, 0.5, x.shape))  # other energies in the buffer
        st, xg, fg, r = ff.minimize(x, p)
        got = device_energies(ff)
        assert st == (7 if end == "failed" else 0)
        # the minimizer's energies are those of the per-potential kernels, bit for bit
        ff.set_shapes(pass_layout=1)
        ff.set_coords(xg)
        total, per = ff._energy()
    assert np.array_equal(got, np.append(per, total), equal_nan=True), (got, per, total)
