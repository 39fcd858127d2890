"""What one half step leaves and reads between its kernels, on the GPU."""
import ctypes

import numpy as np
import pytest

from parity_util import inputs


class _DevArray:
    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (int(ptr), False), "version": 3,
                                         "strides": None}


def _device(r, shape_states=None, typestr="<c16"):
    """the context's states (if a shape is given) and densities as torch views"""
    import torch
    st, de, po = ctypes.c_void_p(), ctypes.POINTER(ctypes.c_double)(), ctypes.POINTER(ctypes.c_double)()
    r._check(r.lib.wtd_device_pointers(r.h, ctypes.byref(st), ctypes.byref(de), ctypes.byref(po)))
    dens = torch.as_tensor(_DevArray(ctypes.addressof(de.contents), (12 * r.N,), "<f8"), device="cuda")
    states = torch.as_tensor(_DevArray(st.value, shape_states, typestr), device="cuda") if shape_states else None
    return states, dens


@pytest.mark.gpu
@pytest.mark.parametrize("name,nwf", [("t1d_sldae_a1", 40), ("t3d_sldae_a1_sym", 24), ("t2d_slda", 24)])
def test_half_step_without_gradients_clears_tau_before_the_functional(has_gpu, name, nwf):
    """a half step without gradients sets tau and j to zero before the functional reads them: what an
    earlier call left there (here NaN) reaches neither the potentials nor the states"""
    import torch
    from wslda_b200 import TDRun

    def run(poison):
        proj, d = inputs(name, nwf)
        r = TDRun(name, nwf)
        r.setup(d["states"], d["pots"], d["occ"], d["params"], d["extra"])
        r.initial_measurement()
        r.sync()
        if poison:
            _, dens = _device(r)
            N = r.N
            dens[3 * N:7 * N] = float("nan")      # tau_a, j_a
            dens[8 * N:] = float("nan")           # tau_b, j_b
            torch.cuda.synchronize()
        r.steps(3)
        out = r.potentials(), r.states(), r.densities()
        r.close()
        return out
    for a, b in zip(run(False), run(True)):
        assert np.array_equal(a, b)
