"""The mixed form's tile kernel on the forms of its outer sums: elements shared by the lanes of two k-points
(k-space solver, 11 and 12 orbitals), each lane its own tile (real-space solver; 6 orbitals), on columns whose last
tile holds an odd or a small number of k-points, against the FP64 form.

Tolerance: the state after at most 70 steps of dt |H| < 1 rounds by at most 70 x 2 sqrt(12) x 6e-8 = 3e-5 in FP32
products; 1e-5 relative L2 is a third of that, a misplaced element is above 1e-3.  Slabs propagate the same k-points
to the same bits and differ by the order of FP64 sums only: 1e-12."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _run(path, n1, n2, steps, pol, solver, precision, k_rows=None):
    from pySWE import pyswe

    dt = 0.02197
    param = {"path_tb": path, "nr1": n1, "nr2": n2, "nr3": 1, "tmax": (steps + 0.5) * dt, "dt": dt, "intensity": 2e12,
             "lambda": 3000.0, "tmax_field": (steps + 0.5) * dt, "pol_vec": np.array(pol), "phi_vec": np.array([0.1, 0.4, 0.0])}
    s = pyswe.SWE(pyswe.Settings(param), solver=solver, precision=precision, k_rows=k_rows)
    s.run_simulation()
    J, rho, name = np.stack(s.get_current()[1:]), s.get_rho_k(), s.launch_shape()["kernel_name"]
    s.delete()
    return J, rho, name


@pytest.mark.parametrize("nw,n1,n2,steps,pol,solver", [
    (11, 10, 10, 70, [0.0, 1.0, 0.0], "kspace"), (11, 14, 14, 65, [0.6, 0.8, 0.0], "kspace"),
    (12, 18, 18, 66, [0.0, 1.0, 0.0], "kspace"), (12, 6, 6, 17, [0.6, 0.8, 0.0], "kspace"),
    (6, 34, 34, 65, [0.6, 0.8, 0.0], "kspace"), (11, 18, 6, 66, [0.0, 1.0, 0.0], "rspace"),
    (11, 12, 10, 65, [0.6, 0.8, 0.0], "rspace"), (12, 10, 4, 33, [0.6, 0.8, 0.0], "rspace"),
    (6, 38, 4, 65, [0.0, 1.0, 0.0], "rspace"), (12, 10, 10, 17, [0.6, 0.8, 0.0], "kspace"),
    (11, 18, 8, 66, [0.0, 1.0, 0.0], "rspace"), (12, 10, 8, 33, [0.6, 0.8, 0.0], "rspace"),
    (6, 38, 8, 65, [0.0, 1.0, 0.0], "rspace")])
def test_forms_of_the_outer_sums(nw, n1, n2, steps, pol, solver, tmp_path):
    import tbgen

    path = str(tmp_path / "m_tb.dat")
    tbgen.random_tmd(path, nw=nw, seed=40 + nw, window=7)
    J, rho, name = _run(path, n1, n2, steps, pol, solver, "mixed")
    # (a grid narrower than the cell box folds it, and the element-group kernel takes the solve)
    assert name == ("propagate_mtile_kernel" if min(n1, n2) > 7 else "propagate_group_kernel<float>")
    _, rho64, _ = _run(path, n1, n2, steps, pol, solver, "fp64")
    assert rel_l2(rho, rho64) < 1e-5
    parts = [_run(path, n1, n2, steps, pol, solver, "mixed", k_rows=r)[0] for r in ((0, 1), (1, 4), (4, n1))]
    assert rel_l2(sum(parts), J) < 1e-12
