"""Spectra at the limits of their launches: calls of different lengths from several threads, many signals of a few
samples, and more harmonic values than a 32-bit thread index counts."""
import threading
import time

import numpy as np
import pytest

from conftest import rel_l2
from test_spectrum_gpu import numpy_harmonics, numpy_spectrum

pytestmark = pytest.mark.gpu


def test_transforms_of_several_lengths_side_by_side():
    """The block transform's shared memory grows with the length; a call must not lower the limit another launches
    with.  Every call gives the bits of the first one; that one within 1e-13 relative L2 of numpy (rounding of a
    length-7000 transform: below 1e-14)."""
    from pySWE import pyswe

    rng = np.random.default_rng(11)
    signals = [rng.standard_normal((3, n)) + 1j * rng.standard_normal((3, n)) for n in (7000, 512, 64)]
    first = [pyswe.spectrum(J, 0.02) for J in signals]
    for J, S in zip(signals, first):
        assert rel_l2(S, numpy_spectrum(J, 0.02)) < 1e-13
    errors, stop = [], time.monotonic() + 4.0
    lib, _ = pyswe._load(pyswe.default_library())

    def work(i):
        J, out = signals[i].reshape(-1), np.zeros(signals[i].size, dtype=np.complex128)
        while time.monotonic() < stop and not errors:
            rc = lib.HHG_spectrum(J, signals[i].shape[1], 3, 0.02, out)
            if rc != 0 or not np.array_equal(out, first[i].reshape(-1)):
                errors.append((i, rc, lib.HHG_last_error()))

    threads = [threading.Thread(target=work, args=(i,)) for i in (0, 1, 2, 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_more_harmonic_values_than_2_to_the_27():
    """A warp per value: 2^27 of them are 2^32 threads.  Eleven samples whose orders reach the last harmonic; the
    expected sums take each sample's order (exact to 1e-7) to its window, and hold one sample each."""
    from pySWE import pyswe

    nh, n, tmax = (1 << 27) + 1000, 11, 1.0
    top = 2 * nh - 1
    lam = 600.0 * tmax * top / n  # the last sample has the last harmonic's order
    rng = np.random.default_rng(5)
    S = rng.standard_normal((1, n)) + 1j * rng.standard_normal((1, n))
    order = np.linspace(-top, top, n)
    near = np.rint(order).astype(np.int64)
    held = [(int(near[i] // 2), abs(S[0, i]) ** 2) for i in range(n)
            if near[i] > 0 and near[i] % 2 == 1 and abs(order[i] - near[i]) < 0.49]
    assert np.all(np.abs(np.abs(order - near) - 0.5) > 1e-3) and len(held) >= 2 and held[-1][0] == nh - 1
    I = pyswe.harmonic_intensities(S, tmax, lam, nh)[0]
    where = np.flatnonzero(I)
    assert where.tolist() == [k for k, _ in held]
    for k, v in held:
        assert abs(I[k] - v) <= 1e-14 * v


@pytest.mark.parametrize("n,count,tmax,nh", [(2, 4001, 0.04, 25), (3, 1000, 0.06, 7), (8, 2000, 0.16, 25), (16, 500, 0.32, 25),
                                             (31, 300, 2.0, 3), (33, 300, 40.0, 2), (130, 99, 9.0, 40)])
def test_many_short_signals(n, count, tmax, nh):
    """Blocks of a warp up to 16 of them, windows of none to some samples, uploaded whole or in part.  Transforms
    1e-13 relative L2 (below 1e-15 x log2 n of rounding), sums of non-negative terms 1e-12."""
    from pySWE import pyswe

    rng = np.random.default_rng(n)
    J = rng.standard_normal((count, n)) + 1j * rng.standard_normal((count, n))
    S, ref = pyswe.spectrum(J, tmax / n), numpy_spectrum(J, tmax / n)
    assert max(rel_l2(S[a], ref[a]) for a in range(count)) < 1e-13
    I, I_ref = pyswe.harmonic_intensities(S, tmax, 3000.0, nh), numpy_harmonics(S, tmax, 3000.0, nh)
    assert np.array_equal(I == 0, I_ref == 0)
    assert np.all(np.abs(I - I_ref) <= 1e-12 * I_ref)
