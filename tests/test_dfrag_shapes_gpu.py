"""The FP64 fragment kernel on every form it takes (3 to 12 orbitals, boxes 1 to 7 cells high, one to three
field axes, both solvers, ragged columns, slabs, chunk tails, long pulses through the allocation-free entry
point), against the CPU oracle and the element-group kernel.

Tolerances: 1e-10 relative L2 per current axis against the oracle (the parity bar), and 1e-11 against the
element-group kernel, both FP64: 130 steps of four stages with sums of at most 12 x 12 x 8 terms round by
about sqrt(5e5) x 1.1e-16 = 8e-14."""
import ctypes as ct
import os

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _param(path, n1, n2, steps, pol, lam=3000.0):
    dt = 0.02197
    return {"path_tb": path, "nr1": n1, "nr2": n2, "nr3": 1, "tmax": (steps + 0.5) * dt, "dt": dt, "intensity": 2e12,
            "lambda": lam, "tmax_field": (steps + 0.5) * dt, "pol_vec": np.array(pol), "phi_vec": np.array([0.1, 0.4, 0.0])}


def _run(param, solver="rspace", group=False, k_rows=None):
    from pySWE import pyswe

    if group:
        os.environ["HHG_DFRAG"] = "0"
    try:
        s = pyswe.SWE(pyswe.Settings(dict(param)), solver=solver, k_rows=k_rows)
    finally:
        os.environ.pop("HHG_DFRAG", None)
    s.run_simulation()
    J, rho, name = np.stack(s.get_current()[1:]), s.get_rho_k(), s.launch_shape()["kernel_name"]
    s.delete()
    return J, rho, name


CASES = [  # orbitals, box, rows, columns, steps, polarisation, solver
    (3, 7, 18, 8, 66, [0.0, 1.0, 0.0], "rspace"), (4, 3, 10, 12, 65, [0.6, 0.8, 0.0], "rspace"),
    (5, 5, 46, 6, 20, [0.6, 0.8, 0.0], "rspace"), (6, 7, 16, 16, 130, [0.0, 1.0, 0.0], "kspace"),
    (7, 5, 14, 14, 64, [0.8, 0.6, 0.0], "kspace"), (8, 7, 34, 8, 63, [1.0, 0.0, 0.0], "rspace"),
    (8, 5, 8, 8, 17, [0.5, 0.5, 0.7], "rspace"), (9, 7, 10, 14, 66, [0.0, 1.0, 0.0], "rspace"),
    (9, 1, 8, 6, 16, [0.6, 0.8, 0.0], "rspace"), (10, 5, 12, 12, 65, [0.6, 0.8, 0.0], "kspace"),
    (11, 3, 18, 4, 33, [0.5, 0.5, 0.7], "rspace"), (12, 5, 10, 10, 129, [0.6, 0.8, 0.0], "kspace"),
    (12, 7, 20, 10, 30, [0.6, 0.8, 0.0], "rspace"),
]


@pytest.mark.parametrize("nw,window,n1,n2,steps,pol,solver", CASES)
def test_shapes_against_oracle_and_element_groups(nw, window, n1, n2, steps, pol, solver, tmp_path, oracle_mod):
    import tbgen

    path = str(tmp_path / "m_tb.dat")
    tbgen.random_tmd(path, nw=nw, seed=20 + nw, window=window)
    param = _param(path, n1, n2, steps, pol)
    J, rho, name = _run(param, solver)
    assert name == "propagate_dfrag_kernel"
    Jg, rho_g, name_g = _run(param, solver, group=True)
    assert name_g == "propagate_group_kernel<double>"
    Jo = (oracle_mod.run_kspace if solver == "kspace" else oracle_mod.run)(path, param)[1]
    for a in range(3):
        if np.abs(Jo[a]).max() == 0:
            assert np.abs(J[a]).max() == 0
        else:
            assert rel_l2(J[a], Jo[a]) < 1e-10, (a, rel_l2(J[a], Jo[a]))
            assert rel_l2(J[a], Jg[a]) < 1e-11, (a, rel_l2(J[a], Jg[a]))
    assert rel_l2(rho, rho_g) < 1e-11
    m = rho.reshape(-1, nw, nw)
    assert np.abs(m - m.conj().transpose(0, 2, 1)).max() < 1e-13


def test_slabs_and_chunks(tmp_path):
    """Row slabs add up to the full current; a pulse served in chunks that start inside a flush ring gives
    the same bits."""
    import tbgen
    from pySWE import pyswe

    for nw, solver in ((5, "rspace"), (10, "rspace"), (10, "kspace")):
        path = str(tmp_path / f"m{nw}_tb.dat")
        tbgen.random_tmd(path, nw=nw, seed=3, window=5)
        param = _param(path, 22, 22, 70, [0.6, 0.8, 0.0])
        J, _, _ = _run(param, solver)
        parts = [_run(param, solver, k_rows=r)[0] for r in ((0, 3), (3, 20), (20, 22))]
        assert rel_l2(sum(parts), J) < 1e-12
        srv = pyswe.SWEServer(device=0, chunk_steps=19)
        r = pyswe.SWE(pyswe.Settings(dict(param)), solver=solver, defer_init=True)
        tk = srv.submit(r)
        assert srv.wait(tk, timeout=120.0)
        assert np.array_equal(np.stack(r.get_current()[1:]), J)
        srv.close()


def test_allocation_free_entry_splits_over_fewer_ctas(tmp_path):
    """More virtual CTAs than the fixed scratch has rows for: the solve runs on fewer of them."""
    import tbgen
    import torch
    from pySWE import pyswe

    path = str(tmp_path / "m_tb.dat")
    tbgen.random_tmd(path, nw=9, seed=5, window=3)
    param = _param(path, 60, 60, 4600, [0.0, 1.0, 0.0])
    swe = pyswe.SWE(pyswe.Settings(dict(param)), device=0)
    shape = swe.launch_shape()
    assert shape["kernel_name"] == "propagate_dfrag_kernel" and shape["ctas"] * swe.settings.nt * 48 > 32 << 20
    rho0 = swe.get_rho_k()
    swe.run_simulation()
    J = swe.get_current()[1:]
    L = ct.CDLL(pyswe.default_library())
    L.SWESim_run_simulation_noalloc.argtypes = [ct.c_void_p] * 4
    L.SWESim_last_error.argtypes, L.SWESim_last_error.restype = [ct.c_void_p], ct.c_char_p
    rho = torch.from_numpy(rho0.copy()).cuda()
    cur = torch.zeros((3, swe.settings.nt), dtype=torch.complex128, device="cuda")
    rc = L.SWESim_run_simulation_noalloc(swe.ptr, rho.data_ptr(), cur.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0, L.SWESim_last_error(swe.ptr)
    torch.cuda.synchronize()
    assert rel_l2(cur.cpu().numpy()[:2], J[:2]) < 1e-12
    swe.delete()
