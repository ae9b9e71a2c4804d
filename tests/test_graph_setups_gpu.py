"""Runs of one object across setups: a setup's first run launches directly, the second captures a CUDA graph, later ones
replay it; a new setup captures again.  Each gives the bits and the launch count of direct launches (HHG_GRAPH=0)."""
import os

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


def _runs(param, precision, solver, graph):
    from pySWE import pyswe

    os.environ["HHG_GRAPH"] = "1" if graph else "0"
    try:
        s = pyswe.SWE(pyswe.Settings(dict(param)), precision=precision, solver=solver)
        out = []
        for nt_factor in (1.0, 0.5, 1.0):  # a new setup with fewer steps, and the first one's again
            if out:
                s.settings = pyswe.Settings(dict(param, tmax=param["tmax"] * nt_factor))
                s.set_settings(s.settings.ptr)
                s.restart()
            for _ in range(3):
                s.reset()
                s.run_simulation()
                out.append((np.stack(s.get_current()[1:]), np.array(s.get_rho_k()), s.last_launches()))
        s.delete()
    finally:
        os.environ.pop("HHG_GRAPH", None)
    return out


@pytest.mark.parametrize("name,precision", [("haldane_12_pol", "fp64"), ("c1", "fp64"), ("tmd11_10", "mixed"),
                                            ("tmd11_10", "fp64"), ("ks_tmd11_10", "mixed")])
def test_captured_and_replayed_runs_of_every_setup(name, precision):
    _, param, _, _ = load_golden(name)
    param = dict(param, tmax=min(param["tmax"], 4.4))
    solver = param.get("solver", "rspace")
    g, d = (_runs(param, precision, solver, graph) for graph in (True, False))
    for (J, rho, n), (Jd, rho_d, nd) in zip(g, d):
        assert np.array_equal(J, Jd) and np.array_equal(rho, rho_d)
        assert n == nd
