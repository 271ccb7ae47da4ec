"""What the kernel tuner times and how it chooses: no launch for a choice that
the search does not depend on, the phase-1 DP's warps per block only where a
warp sweeps a profile of its own, in that form; and the unshared DP kernels,
which take more than 9,472 profiles, with 1 and 2 warps a block."""
import numpy as np
import pytest

from test_dp1_gpu import _compare

pytestmark = pytest.mark.gpu

MARGIN = 0.015      # a candidate must be this much faster to replace the preferred one


def _context(ss, **opt):
    import cother_b200 as cb
    o = cb.Options.defaults()
    for k, v in opt.items():
        setattr(o, k, v)
    return cb.BatchProcessing(ss, o)


def _launches(bp, q):
    """Kernel launches of a first search beyond those of the next."""
    n = []
    for _ in range(2):
        bp.process_score_matrix(q)
        n.append(bp.launch_count())
    return n[0] - n[1]


# ten score launches with their column orders (twenty), and of the DP two
# repetitions of its two launches, for one launch form or two
@pytest.mark.parametrize("ddmswgt,Lq,want", [(0.2, 100, 20 + 4), (0.0, 100, 4), (0.2, 60, 20 + 8), (0.0, 60, 8)])
def test_timed_launches(ss_table, ddmswgt, Lq, want):
    from cother_b200 import synth
    q = synth.make_profiles([Lq], 2000 + Lq, True)
    db = synth.make_profiles([30, 77, 120, 45], 2001, False)
    with _context(ss_table, ddmswgt=ddmswgt) as bp:
        bp.transfer_cpm_data(db)
        assert _launches(bp, q) == want
        t = bp.tuning(Lq)
        assert all((x > 0) == (ddmswgt > 0) for x in t["score_candidates_ms"])
        two, one = t["dp_candidates_ms"]
        assert two > 0 and one > 0
        if Lq > 64:
            assert two == one          # one launch, timed once
        # one warp a block unless two are clearly faster; untouched where warps share a profile
        assert t["dp_warps"] == (2 if Lq > 64 or two <= (1.0 - MARGIN) * one else 1)


def test_large_chunk_after_a_small_one(ss_table):
    """The DP's choice waits for a chunk that depends on it."""
    from cother_b200 import synth
    rng = np.random.default_rng(2010)
    q = synth.make_profiles([70], 2011, True)
    small = synth.make_profiles([30, 77], 2012, False)
    large = synth.make_profiles(rng.integers(1, 24, size=9500).astype(np.int32), 2013, False)
    with _context(ss_table, ddmswgt=0.0) as bp:
        bp.transfer_cpm_data(small)
        assert _launches(bp, q) == 4
        assert bp.tuning(70)["dp_warps"] == 2
        bp.transfer_cpm_data(large)
        assert _launches(bp, q) == 8
        t = bp.tuning(70)
        two, one = t["dp_candidates_ms"]
        assert t["dp_warps"] == (2 if two <= (1.0 - MARGIN) * one else 1)


def test_unshared_dp_kernels(oracle_lib, ss_table):
    """More than 9,472 profiles with codes for all of them, some of several
    64-column rings: scores, codes, records and pass list equal the oracle's
    with 1 and with 2 warps a block."""
    from cother_b200 import synth
    rng = np.random.default_rng(2020)
    lens = rng.integers(1, 6, size=9500).astype(np.int32)
    lens[::190] = rng.integers(64, 330, size=50)
    q = synth.make_profiles([200], 2021, True)
    db = synth.make_profiles(lens, 2022, False)
    synth.plant_homologs(q, db, 0.01, seed=2023)
    for warps in (1, 2):
        with _context(ss_table, ddmswgt=0.0, all_codes=1) as bp:
            bp.set_kernels(200, 16, 1024, warps)
            bp.set_score_threshold(3.0)
            bp.transfer_cpm_data(db)
            bp.process_score_matrix(q)
            assert bp.tuning(200)["dp_warps"] == warps
            _compare(bp, oracle_lib, q, db, 3.0)
