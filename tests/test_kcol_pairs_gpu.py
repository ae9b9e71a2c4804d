"""The pair form of the column-tile kernel (two orbitals) over the forms it takes: boxes of 1, 3, 5 and 7 cells, one
to three field axes, both solvers, tiles of 1 to 32 pairs with one and two warps, slabs whose rows have a partner,
none or some, and chunk tails, against the CPU oracle and the thread-per-k-point kernel.

Tolerances: 1e-10 relative L2 per current axis against the oracle (the parity bar), 1e-11 against the other FP64
kernel: 600 steps round by about sqrt(600 x 200) x 1.1e-16 = 4e-14."""
import os

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _param(path, n1, n2, steps, pol):
    dt = 0.02197
    return {"path_tb": path, "nr1": n1, "nr2": n2, "nr3": 1, "tmax": (steps + 0.5) * dt, "dt": dt, "intensity": 2e12,
            "lambda": 3000.0, "tmax_field": (steps + 0.5) * dt, "pol_vec": np.array(pol), "phi_vec": np.array([0.1, 0.4, 0.0])}


def _run(param, solver="rspace", kernel=None, k_rows=None):
    from pySWE import pyswe

    if kernel:
        os.environ["HHG_KERNEL"] = kernel
    try:
        s = pyswe.SWE(pyswe.Settings(dict(param)), solver=solver, k_rows=k_rows)
    finally:
        os.environ.pop("HHG_KERNEL", None)
    s.run_simulation()
    out = np.stack(s.get_current()[1:]), s.get_rho_k(), s.launch_shape()
    s.delete()
    return out


@pytest.mark.parametrize("window,n1,n2,steps,pol,solver", [
    (5, 16, 10, 257, [0.0, 1.0, 0.0], "rspace"), (7, 22, 8, 66, [0.6, 0.8, 0.0], "rspace"),
    (3, 14, 14, 5, [0.6, 0.8, 0.0], "kspace"), (1, 18, 10, 9, [0.0, 1.0, 0.0], "rspace"),
    (5, 16, 16, 258, [0.5, 0.5, 0.7], "kspace"), (7, 14, 14, 31, [1.0, 0.0, 0.0], "kspace"),
    (5, 66, 4, 20, [0.5, 0.5, 0.7], "rspace"), (5, 66, 6, 20, [0.5, 0.5, 0.7], "rspace"), (5, 8, 240, 18, [0.6, 0.8, 0.0], "rspace")])
def test_pair_form_against_oracle_and_thread_per_kpt(window, n1, n2, steps, pol, solver, tmp_path, oracle_mod):
    import tbgen

    path = str(tmp_path / "m_tb.dat")
    tbgen.random_tmd(path, nw=2, seed=40 + window, window=window)
    param = _param(path, n1, n2, steps, pol)
    J, rho, shape = _run(param, solver, "kcol")
    Jo = (oracle_mod.run_kspace if solver == "kspace" else oracle_mod.run)(path, param)[1]
    if n2 < window:  # the box folds onto the grid: the placement is not Hermitian, and no two-orbital kernel takes it
        assert shape["kernel_name"] == "propagate_group_kernel<double>"
        assert max(rel_l2(J[a], Jo[a]) for a in range(2)) < 1e-10
        return
    assert shape["kernel_name"] == "propagate_kcol_kernel"
    # one warp a tile from 1.5 tiles an SM on (240 columns on 148 SMs), else two
    assert shape["threads"] == (32 if n2 >= 240 else 64)
    Jk, rho_k, shape_k = _run(param, solver, "kpt")
    assert shape_k["kernel_name"] == "propagate_kpt_kernel"
    for a in range(3):
        if np.abs(Jo[a]).max() == 0:
            assert np.abs(J[a]).max() == 0
        else:
            assert rel_l2(J[a], Jo[a]) < 1e-10, (a, rel_l2(J[a], Jo[a]))
            assert rel_l2(J[a], Jk[a]) < 1e-11, (a, rel_l2(J[a], Jk[a]))
    assert rel_l2(rho, rho_k) < 1e-11


def test_slabs_tiles_and_chunks():
    """Slabs with rows of both halves of the grid, of one, and of a row without its partner add up; split tiles and
    chunks that start inside a staged interval: rounding of the k-sum's order, and the same bits."""
    import tbgen
    from pySWE import pyswe

    param = _param(tbgen.model_path("haldane"), 20, 18, 600, [0.6, 0.8, 0.0])
    J, _, _ = _run(param, kernel="kcol")
    parts = [_run(param, kernel="kcol", k_rows=r)[0] for r in ((0, 3), (3, 17), (17, 18), (18, 20))]
    assert rel_l2(sum(parts), J) < 1e-12
    os.environ["HHG_KCOL_PARTS"] = "3"
    try:
        assert rel_l2(_run(param, kernel="kcol")[0], J) < 1e-12
    finally:
        del os.environ["HHG_KCOL_PARTS"]
    for solver in ("rspace", "kspace"):
        p = dict(param, nr2=20)
        J, _, _ = _run(p, solver)
        srv = pyswe.SWEServer(device=0, chunk_steps=13)
        r = pyswe.SWE(pyswe.Settings(dict(p)), solver=solver, defer_init=True)
        tk = srv.submit(r)
        assert srv.wait(tk, timeout=120.0)
        assert np.array_equal(np.stack(r.get_current()[1:]), J)
        srv.close()
