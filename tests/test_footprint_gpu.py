"""The server's admission estimate bounds the device memory of a solve from above for every kernel's split of the
current partials: a solve beside an equal one is admitted only if both fit the budget."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _settings(pyswe, path, n1, n2, steps, pol):
    dt = 0.02197
    return pyswe.Settings({"path_tb": path, "nr1": n1, "nr2": n2, "nr3": 1, "tmax": (steps + 0.5) * dt, "dt": dt,
                           "intensity": 1e12, "lambda": 3000.0, "tmax_field": (steps + 0.5) * dt,
                           "pol_vec": np.array(pol), "phi_vec": np.zeros(3)})


# Column tiles of one warp (8 CTAs per SM), both solvers; tiles of one warp of the general form (one orbital); two-warp
# tiles; the fragment, tile and element-group kernels.
@pytest.mark.parametrize("nw,window,n1,n2,steps,pol,solver,precision", [
    (2, 5, 300, 300, 8192, [0.0, 1.0, 0.0], "rspace", "fp64"), (2, 7, 300, 300, 8192, [0.6, 0.8, 0.0], "kspace", "fp64"),
    (2, 5, 300, 300, 8192, [0.0, 1.0, 0.0], "rspace", "mixed"), (1, 5, 32, 1200, 4096, [0.6, 0.8, 0.0], "rspace", "fp64"),
    (2, 5, 40, 150, 2048, [0.6, 0.8, 0.0], "rspace", "fp64"), (2, 5, 12, 12, 4096, [0.0, 1.0, 0.0], "rspace", "fp64"),
    (3, 5, 60, 60, 1024, [0.6, 0.8, 0.0], "kspace", "fp64"), (12, 7, 40, 40, 256, [0.6, 0.8, 0.0], "rspace", "fp64"),
    (6, 7, 60, 60, 1024, [0.6, 0.8, 0.0], "rspace", "mixed"), (13, 3, 16, 16, 256, [0.6, 0.8, 0.0], "rspace", "fp64")])
def test_the_estimate_is_an_upper_bound(nw, window, n1, n2, steps, pol, solver, precision, tmp_path):
    import tbgen
    from pySWE import pyswe

    path = str(tmp_path / "m_tb.dat")
    tbgen.random_tmd(path, nw=nw, seed=nw, window=window)

    def serve(budget, count):
        srv = pyswe.SWEServer(device=0, hbm_budget=budget, max_active=4)
        reqs = [pyswe.SWE(_settings(pyswe, path, n1, n2, steps, pol), precision=precision, solver=solver, defer_init=True)
                for _ in range(count)]
        for t in [srv.submit(r) for r in reqs]:
            assert srv.wait(t, timeout=120.0)
        st = srv.stats()
        srv.close()
        for r in reqs:
            r.delete()
        return st

    actual = serve(0, 1)["peak_bytes"]  # the exact figure after setup
    st = serve(2 * actual - 1, 2)
    assert st["completed"] == 2 and st["peak_running"] == 1 and st["peak_bytes"] == actual
