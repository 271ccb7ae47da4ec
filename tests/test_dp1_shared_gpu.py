"""Phase-1 DP with several warps to a profile (few profiles) and one warp each
(many): query lengths at the ends of 64-row bands and of the rules that choose
the number of warps, profile lengths around the 16-column pieces, every first
column mod 4. Scores, backtrack codes, records and the pass list equal the
oracle's bit for bit, with codes for all profiles and for the candidates
only."""
import numpy as np
import pytest

from test_dp1_gpu import _compare, _search

pytestmark = pytest.mark.gpu

# profile lengths: single columns, piece ends, wavefront (32) ends, long ones
LENS = [1, 15, 16, 17, 2, 31, 32, 33, 64, 47, 300, 3, 129, 5, 77, 451]


@pytest.mark.parametrize("Lq", [64, 65, 128, 129, 256, 257, 320, 513, 577, 1030])
def test_warps_share_a_profile(oracle_lib, ss_table, Lq):
    from cother_b200 import synth
    q = synth.make_profiles([Lq], 800 + Lq, True)
    db = synth.make_profiles(LENS, 900 + Lq, False)
    synth.plant_homologs(q, db, 0.4, seed=Lq)
    for thld, all_codes in ((-1.0, 1), (3.0, 0)):
        bp = _search(q, db, ss_table, thld, all_codes=all_codes)
        _compare(bp, oracle_lib, q, db, thld, all_codes=bool(all_codes), mixed=False)
        bp.close()


@pytest.mark.parametrize("nprof,Lq", [(450, 330), (2400, 140), (9500, 70)])
def test_many_profiles(oracle_lib, ss_table, nprof, Lq):
    """Past each rule's line: fewer warps a profile, the longest first, in one
    slab and (as they come) in several."""
    from cother_b200 import synth
    rng = np.random.default_rng(nprof)
    q = synth.make_profiles([Lq], 820 + Lq, True)
    db = synth.make_profiles(rng.integers(1, 24, size=nprof).astype(np.int32), 920 + Lq, False)
    bp = _search(q, db, ss_table, 1.5, all_codes=0)
    _compare(bp, oracle_lib, q, db, 1.5, all_codes=False, mixed=False)
    whole = bp.hit_records()
    bp.close()
    bp = _search(q, db, ss_table, 1.5, max_slab=20000, all_codes=0)
    assert np.array_equal(bp.hit_records(), whole)
    bp.close()
