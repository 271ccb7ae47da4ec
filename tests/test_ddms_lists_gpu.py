"""The distance term at every list length: lists of 0..99 distances on both
sides (values at and past the saturation point, runs without data, long runs
of similar values), DSTSEGM in each of the kernel's compile-time cases and at
its ends, a database whose last block of columns is partial. Scores and
modular scores equal the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _set_lists(ps, rng, first):
    n = ps.npositions
    cnt = (first + np.arange(n)) % 100
    v = rng.integers(3, 26, size=(99, n))
    for c in range(n):
        kind = c % 4
        if kind == 1:                      # long similar stretches: segments that span many steps
            v[:, c] = 8 + rng.integers(0, 2, 99)
        elif kind == 2:                    # a chain's walk
            v[:, c] = np.clip(8 + np.cumsum(rng.integers(-2, 3, 99)), 0, 30)
        elif kind == 3:                    # stretches without data
            v[rng.random(99) < 0.3, c] = 255
    ps.dd[0] = cnt
    ps.dd[1:] = np.where(np.arange(99)[:, None] < cnt[None], v, 255)


@pytest.mark.parametrize("dstsegm", [1, 2, 4, 5, 6, 7, 13, 20])
def test_all_list_lengths(ss_table, oracle_lib, dstsegm):
    import cother_b200 as cb
    from cother_b200 import synth
    rng = np.random.default_rng(100 + dstsegm)
    q = synth.make_profiles([101], 61, True)
    db = synth.make_profiles([1, 2, 31, 64, 107, 3, 119], 62, False)
    _set_lists(q, rng, 99)
    _set_lists(db, rng, 37)
    o = cb.Options.defaults()
    o.dstsegm = dstsegm
    o.autotune = 0
    with cb.BatchProcessing(ss_table, o) as bp:
        bp.transfer_cpm_data(db)
        bp.process_score_matrix(q)
        sc, ms, _ = bp.read_score_matrix(q.npositions, db.npositions)
    want = oracle_lib.score_matrix(q, db, ss_table, dstsegm=dstsegm, nthreads=4)
    assert np.array_equal(ms, want[1])
    assert np.array_equal(sc, want[0])
