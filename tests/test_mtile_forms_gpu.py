"""The tile kernel's two forms of the commutator product (packed pairs; scalar operations where one field axis leaves a
CTA alone on its SM) give the same bits: a slab of a solve, small enough for the scalar form, against the whole solve in
the packed one."""
import numpy as np
import pytest

from test_mtile_shapes_gpu import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw,n1,n2,cut,solver", [
    (6, 38, 80, 32, "rspace"), (6, 100, 100, 32, "kspace"), (11, 42, 40, 23, "rspace"), (11, 40, 40, 24, "kspace"),
    (12, 42, 40, 17, "rspace"), (12, 40, 40, 24, "kspace")])
def test_packed_and_scalar_products_give_the_same_bits(nw, n1, n2, cut, solver, tmp_path):
    import tbgen

    path = str(tmp_path / "m_tb.dat")
    tbgen.random_tmd(path, nw=nw, seed=60 + nw, window=7)
    kpc = 32 if nw == 6 else 8
    assert n2 * -(-n1 // kpc) > 148 >= n2 * -(-cut // kpc)  # tiles of the solve and of the slab, SMs
    args = (path, n1, n2, 66, [0.0, 1.0, 0.0], solver, "mixed")
    _, rho, name = _run(*args)
    assert name == "propagate_mtile_kernel"
    _, part, _ = _run(*args, k_rows=(0, cut))
    assert np.array_equal(part[:cut * n2], rho[:cut * n2])
