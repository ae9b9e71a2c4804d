"""Spectra at the limits of their launches: calls of different lengths from several threads."""
import threading
import time

import numpy as np
import pytest

from conftest import rel_l2
from test_spectrum_gpu import numpy_spectrum

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
