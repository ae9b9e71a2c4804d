"""Forms of the device spectrum that the block transform and the pass-by-pass one split: lengths on both sides of the
shared-memory limit, a large prime radix first, in the middle and last, and harmonic windows that begin before the
axis, end after it or hold no sample.

Tolerances: a transform of length n with radix sums of at most R terms rounds by about (log2 n + sqrt(R)) x 1.1e-16,
below 2e-14 for R = 7043, so 1e-13 relative L2 as for the other lengths; harmonic sums of non-negative terms 1e-12."""
import numpy as np
import pytest

from conftest import rel_l2
from test_spectrum_gpu import numpy_harmonics, numpy_spectrum

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count", [(7040, 2), (7041, 2), (7043, 1), (7042, 3), (2 * 1009, 2), (11 * 640, 1), (8192, 5),
                                     (9, 300), (3, 1), (7 * 11 * 13, 4)])
def test_lengths_around_the_block_limit(n, count):
    from pySWE import pyswe

    rng = np.random.default_rng(n)
    J = rng.standard_normal((count, n)) + 1j * rng.standard_normal((count, n))
    S, ref = pyswe.spectrum(J, 0.02197), numpy_spectrum(J, 0.02197)
    assert max(rel_l2(S[a], ref[a]) for a in range(count)) < 1e-13


@pytest.mark.parametrize("n,tmax,lam,nh", [(512, 11.0, 3000.0, 25), (64, 0.5, 800.0, 200), (2, 1.0, 2000.0, 3),
                                           (4095, 90.0, 2000.0, 40), (100, 0.01, 3000.0, 5), (1000, 4000.0, 3000.0, 7)])
def test_harmonic_windows(n, tmax, lam, nh):
    from pySWE import pyswe

    rng = np.random.default_rng(nh)
    S = rng.standard_normal((5, n)) + 1j * rng.standard_normal((5, n))
    I, ref = pyswe.harmonic_intensities(S, tmax, lam, nh), numpy_harmonics(S, tmax, lam, nh)
    assert np.array_equal(I == 0, ref == 0)
    assert np.all(np.abs(I - ref) <= 1e-12 * ref)
