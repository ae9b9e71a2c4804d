"""Host threads that set up and run solves of different sizes at once: a kernel's dynamic shared-memory limit is one
value per function and device, so a thread with a small solve must not lower it under another's launches.  Each solve
gives, bit for bit, what it gives alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _param(path, n, steps):
    dt = 0.02197
    return {"path_tb": path, "nr1": n, "nr2": n, "nr3": 1, "tmax": (steps + 0.5) * dt, "dt": dt, "intensity": 2e12,
            "lambda": 3000.0, "tmax_field": (steps + 0.5) * dt, "pol_vec": np.array([0.6, 0.8, 0.0]), "phi_vec": np.zeros(3)}


# (orbitals of the solves with the larger and the smaller shared memory, precision, the kernel both run)
@pytest.mark.parametrize("large,small,precision,kernel", [
    (8, 3, "fp64", "propagate_dfrag_kernel"), (12, 9, "fp64", "propagate_dfrag_kernel"),
    (13, 16, "fp64", "propagate_group_kernel<double>"), (10, 7, "mixed", "propagate_group_kernel<float>")])
def test_setups_and_runs_of_two_sizes_side_by_side(large, small, precision, kernel, tmp_path):
    import tbgen
    from pySWE import pyswe

    solves, alone = [], []
    for nw, steps in ((large, 2048), (small, 64)):
        path = str(tmp_path / f"m{nw}_tb.dat")
        tbgen.random_tmd(path, nw=nw, seed=nw, window=5)
        s = pyswe.SWE(pyswe.Settings(_param(path, 12, steps)), precision=precision)
        assert s.launch_shape()["kernel_name"] == kernel
        s.run_simulation()
        solves.append(s)
        alone.append(np.stack(s.get_current()[1:]))
    assert solves[0].launch_shape()["smem_bytes"] > solves[1].launch_shape()["smem_bytes"]
    errors, done = [], threading.Event()

    def work(i, again):
        try:
            while again():
                solves[i].restart()
                solves[i].run_simulation()
                assert np.array_equal(np.stack(solves[i].get_current()[1:]), alone[i])
        except Exception as e:  # noqa: BLE001
            errors.append(e)
        finally:
            done.set()

    rounds = iter(range(30))
    threads = [threading.Thread(target=work, args=(0, lambda: next(rounds, None) is not None and not errors)),
               threading.Thread(target=work, args=(1, lambda: not done.is_set()))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for s in solves:
        s.delete()
