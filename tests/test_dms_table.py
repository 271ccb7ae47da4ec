"""The distance pair scores that the score kernel's length arithmetic counts
on: scaled by 2^-7, the scores and the means of two are multiples of 2^-48, so
the bits of a positive running sum, as an integer, exceed the longest segment
(99 elements and 6 past the end of a list) in units of 2^22; and sums stay
below 1."""
import numpy as np


def test_pair_scores(oracle_lib):
    d = [*range(21), 255]
    T = np.array([[oracle_lib.lib().orc_dms_pair_score(a, b) for b in d] for a in d], np.float32).ravel()
    v = T.astype(np.float64) * 2.0**40
    assert np.array_equal(v, np.rint(v))
    means = np.float32(0.5) * (T[:, None] * np.float32(2.0**-7) + T[None] * np.float32(2.0**-7))
    m = means.astype(np.float64) * 2.0**48
    assert np.array_equal(m, np.rint(m))
    assert int(np.float32(2.0**-48).view(np.int32)) >= 105 * 2**22
    assert T.max() * 105 < 2.0**7
