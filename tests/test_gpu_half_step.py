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


@pytest.mark.gpu
def test_stream_path_takes_more_than_65535_states(has_gpu):
    """the state count is no grid extent limited to 65,535: 20 x 18 x 22 with 65,540 complex64 states
    (50 GB), normalised from arbitrary norms, measured and stepped"""
    import torch
    from wslda_b200 import MIXED_H32, TDRun
    from wslda_b200.projects import Project, make_potentials
    proj, S = Project("t3d_ragged"), 65540
    if torch.cuda.mem_get_info()[0] < 70e9:
        pytest.skip("needs 70 GB of free device memory")
    r = TDRun(proj, S, precision=MIXED_H32)
    states, dens = _device(r, (2, S, r.N), "<c8")
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    parts = [(a, min(a + 4096, S)) for a in range(0, S, 4096)]

    def norms():
        return torch.cat([(states[:, a:b].abs() ** 2).sum(dim=(0, 2), dtype=torch.float64) for a, b in parts]) * proj.dv
    for a, b in parts:
        states[:, a:b] = torch.randn((2, b - a, r.N), dtype=torch.complex64, device="cuda", generator=g)
    # the component that a state adds to the densities is its small one, so that 65,540 states on
    # 7,920 points stay dilute (0.04 per point and spin)
    occ = (np.arange(S) % 2 == 0).astype(float)
    states[0, 0::2] *= 0.1
    states[1, 1::2] *= 0.1
    r.setup_fields(make_potentials(proj), occ, proj.params)
    torch.cuda.synchronize()
    for call in (r.initial_measurement, lambda: r.steps(1)):
        call()
        r.sync()
        n = norms()
        assert float((n - 1.0).abs().max()) < 1e-6
        # rho_a = sum f |u|^2, rho_b = sum (1 - f) |v|^2, over all the states
        f = torch.tensor(occ, device="cuda")
        want = torch.zeros(2, r.N, dtype=torch.float64, device="cuda")
        for a, b in parts:
            want[0] += ((states[0, a:b].abs() ** 2).double() * f[a:b, None]).sum(0)
            want[1] += ((states[1, a:b].abs() ** 2).double() * (1.0 - f[a:b, None])).sum(0)
        for k, off in ((0, 2), (1, 7)):
            got = dens[off * r.N:(off + 1) * r.N]
            assert float(torch.linalg.vector_norm(got - want[k]) / torch.linalg.vector_norm(want[k])) < 1e-6
    r.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name,nwf,prec", [("t3d_ragged", 9, 2), ("c3_aslda3d", 8, 1), ("c3_aslda3d", 8, 2), ("c5_slda3d", 4, 2)])
def test_densities_are_those_of_the_returned_states(has_gpu, name, nwf, prec):
    """the complex64 forms sum the densities of the states that the call leaves, not of states rounded
    once more afterwards: rho and nu formed from the returned states agree to FP64 rounding of sums of
    nwf terms.  And the returned states are normalised: rounding the 4 N reals of a state once each
    (2^-25 rms / sqrt 3 relative and independent) leaves its norm off by 2^-24 / sqrt(4 N) or less,
    2e-9 is five times that at the smallest N; a state scaled after it was rounded keeps up to 3e-8"""
    from wslda_b200 import TDRun
    proj, d = inputs(name, nwf)
    N = proj.numel
    r = TDRun(name, nwf, precision=prec)
    r.setup(d["states"], d["pots"], d["occ"], d["params"], d["extra"])
    for call in (r.initial_measurement, lambda: r.steps(2), lambda: r.steps(1)):
        call()
        y, dens = r.states().reshape(2, nwf, N), r.densities()
        f = np.asarray(d["occ"])[:, None]
        u, v = y[0], y[1]
        assert np.abs((np.abs(y) ** 2).sum(axis=(0, 2)) * proj.dv - 1.0).max() < 2e-9
        nu = ((u * v.conj()) * (1.0 - 2.0 * f) * 0.5).sum(0)
        got = dens[:2 * N].view(np.complex128)
        # relative to sum |u v|, which the signed sum nu cancels from
        scale = np.sqrt(((np.abs(u) * np.abs(v) * 0.5).sum(0) ** 2).sum())
        assert np.linalg.norm(got - nu) < 1e-14 * scale
        for want, off in (((np.abs(u) ** 2 * f).sum(0), 2), ((np.abs(v) ** 2 * (1.0 - f)).sum(0), 7)):
            assert np.linalg.norm(dens[off * N:(off + 1) * N] - want) < 1e-14 * np.linalg.norm(want)
    r.close()


def _h_psi_ragged(proj, psi, pots, params):
    """H psi of t3d_ragged (3D ASLDA, variable mass, Delta_ext) in numpy: psi [2, S, N], FP64"""
    n = (proj.nx, proj.ny, proj.nz)
    N, S = proj.numel, psi.shape[1]
    c = proj.constants()
    k, kd = [], []
    for m, d in zip(n, (proj.dx, proj.dy, proj.dz)):
        q = np.where(np.arange(m) < m // 2, np.arange(m), np.arange(m) - m) * (2.0 * np.pi / (m * d))
        k.append(q)
        kd.append(np.where(np.arange(m) == m // 2, 0.0, q))
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    kd = [kd[0][:, None, None], kd[1][None, :, None], kd[2][None, None, :]]

    def spectral(f, mul):
        g = np.fft.fftn(f.reshape(-1, *n), axes=(1, 2, 3)) * mul
        return np.fft.ifftn(g, axes=(1, 2, 3)).reshape(f.shape)
    x = [(np.arange(m) - m // 2) * d for m, d in zip(n, (proj.dx, proj.dy, proj.dz))]
    L = [m * d for m, d in zip(n, (proj.dx, proj.dy, proj.dz))]
    dext = params[3] * (1.0 + 0.5j * np.sin(2 * np.pi * x[0] / L[0]))[:, None, None] * np.cos(2 * np.pi * x[1] / L[1])[None, :, None]
    D = pots[2 * N:4 * N].view(np.complex128) + np.broadcast_to(dext, n).reshape(N)
    H = np.empty_like(psi)
    for s in range(2):
        V, al, A = pots[s * N:(s + 1) * N] - (c["mu_a"], c["mu_b"])[s], pots[(4 + s) * N:(5 + s) * N], pots[(6 + 3 * s) * N:(9 + 3 * s) * N].reshape(3, N)
        sgn, y, o = (1.0, -1.0)[s], psi[s], psi[1 - s]
        lap_al = spectral(al[None].astype(complex), -k2)[0].real
        div = sum(spectral(A[a][None].astype(complex), 1j * kd[a])[0].real for a in range(3))
        H[s] = sgn * (-0.25 * (al * spectral(y, -k2) + spectral(al * y, -k2)) + (V + 0.25 * lap_al) * y) + (D, D.conj())[s] * o
        H[s] += -1j * sum(A[a] * spectral(y, 1j * kd[a]) for a in range(3)) - 0.5j * div * y
    return H


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1])
def test_mixed_h64_forms_h_in_fp64_where_the_line_path_does_not_fit(has_gpu, prec):
    """f = (H - <H>) psi of the stored states, formed on demand and kept in FP64: on 20 x 18 x 22, which
    the line path does not take, WTD_MIXED_H64 computes it from the complex64 states in FP64.  Two
    FP64 evaluations of sums of at most 3 x 22 products per point differ by less than 1e-13 of f;
    FP32 arithmetic would differ by 1e-7."""
    from wslda_b200 import TDRun
    nwf = 7
    proj, d = inputs("t3d_ragged", nwf)
    r = TDRun("t3d_ragged", nwf, precision=prec)
    r.setup(d["states"], d["pots"], d["occ"], d["params"], d["extra"])
    r.initial_measurement()
    r.steps(2)
    f, psi, E = r.history(0).reshape(2, nwf, -1), r.states().reshape(2, nwf, -1), r.qpe()
    h = _h_psi_ragged(proj, psi, r.potentials(), d["params"])
    r.close()
    e = (psi.conj() * h).real.sum(axis=(0, 2)) * proj.dv
    assert np.abs(E - e).max() < 1e-12 * np.abs(e).max()
    want = h - e[None, :, None] * psi
    assert np.linalg.norm(f - want) < 1e-13 * np.linalg.norm(want)


@pytest.mark.gpu
@pytest.mark.parametrize("name,nwf,fail_at", [("t3d_ragged", 9, 1), ("t3d_ragged", 9, 2), ("t2d_slda", 24, 1)])
def test_failed_density_exchange_leaves_normalised_states(has_gpu, name, nwf, fail_at):
    """a density exchange that fails inside a block ends the call with an error; the states are left
    normalised, and the context then runs new states as a fresh one does"""
    from wslda_b200 import TDRun, WtdError
    proj, d = inputs(name, nwf)
    calls = [0]

    def hook(ptr, count, stream):
        calls[0] += 1
        if calls[0] > fail_at:
            raise RuntimeError("exchange refused by the test")

    def fresh(r):
        r.setup(d["states"], d["pots"], d["occ"], d["params"], d["extra"])
        r.initial_measurement()
        r.steps(2)
        return r.states(), r.densities(), r.potentials()
    r = TDRun(name, nwf)
    r.setup(d["states"], d["pots"], d["occ"], d["params"], d["extra"])
    r.set_density_exchange(hook)
    r.initial_measurement()
    with pytest.raises(WtdError):
        r.steps(3)
    y = r.states().reshape(2, nwf, -1)
    norms = (np.abs(y) ** 2).sum(axis=(0, 2)) * proj.dv
    assert np.abs(norms - 1.0).max() < 1e-12
    r.set_density_exchange(None)
    got = fresh(r)
    r.close()
    other = TDRun(name, nwf)
    want = fresh(other)
    other.close()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("name,nwf,prec,path", [("c3_aslda3d", 400, 0, None), ("c3_aslda3d", 400, 1, None), ("c3_aslda3d", 400, 2, None),
                                                ("c3_aslda3d", 400, 0, "staged"), ("c3_aslda3d", 400, 2, "line"),
                                                ("t3d_ragged", 1500, 1, None), ("t2d_big", 600, 0, None), ("t2d_big", 600, 1, None),
                                                ("c2_slda2d", 3000, 0, None)])
def test_device_bytes_are_those_of_the_path(has_gpu, monkeypatch, name, nwf, prec, path):
    """wtd_device_bytes against the device memory that a context takes, on every path.  It leaves out
    nothing that grows with the states, so the two differ by the rounding of two dozen allocations
    (2 MiB each) and by the estimate of the density slots (300 CTAs; the paths take between 148 and
    600 of 12 to 16 words a point): 600 x 16 x N doubles."""
    import torch
    from wslda_b200 import TDRun
    if path:
        monkeypatch.setenv("WTD_3D_PATH", path)
    TDRun(name, 1, precision=prec).close()          # modules loaded, context created
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    r = TDRun(name, nwf, precision=prec)
    used = free - torch.cuda.mem_get_info()[0]
    N = r.N
    want = r.lib.wtd_device_bytes(nwf, prec)
    r.close()
    assert abs(used - want) < 24 * 2 ** 21 + 300 * 16 * N * 8, (used, want)
    assert abs(used - want) < 0.1 * used, (used, want)


@pytest.mark.gpu
@pytest.mark.parametrize("name,nwf", [("t3d_ragged", 9), ("t2d_slda", 24)])
def test_subset_densities_report_a_failed_wait(has_gpu, name, nwf):
    """the error of the call's last wait is returned and not dropped.  The wait is made to fail on the
    host, without a fault: a stream in capture refuses to be waited for, and nothing of what was
    queued runs; the context is used on afterwards"""
    from wslda_b200 import TDRun, WtdError
    import torch  # noqa: F401  (its CUDA runtime is the one loaded here)
    rt = ctypes.CDLL("libcudart.so.12")
    proj, d = inputs(name, nwf)
    r = TDRun(name, nwf)
    r.setup(d["states"], d["pots"], d["occ"], d["params"], d["extra"])
    r.initial_measurement()
    w = np.ones(nwf)
    want = r.subset_densities(w)
    st, graph = ctypes.c_void_p(r.stream()), ctypes.c_void_p()
    assert rt.cudaStreamBeginCapture(st, 2) == 0          # relaxed: allocations stay allowed
    try:
        with pytest.raises(WtdError):
            r.subset_densities(w)
    finally:
        rt.cudaStreamEndCapture(st, ctypes.byref(graph))   # the refused wait has ended the capture
        rt.cudaGetLastError()
    assert np.array_equal(r.subset_densities(w), want)
    r.close()
