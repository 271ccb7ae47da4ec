"""MAP realignment of more than four pairs an SM (592), which takes every step
with its column checks: profile lengths around 32-column chunks, one band,
more bands than warps. Every realigned pair's rows, counts and coordinates
equal the oracle's."""
import pytest

from test_map_gpu import _check_map, _search

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lq", [31, 97, 290])
def test_more_than_four_pairs_an_sm(oracle_lib, ss_table, Lq):
    from cother_b200 import synth
    q = synth.make_profiles([Lq], 1700 + Lq, True)
    db = synth.make_profiles([1, 2, *range(26, 38), *range(58, 70), 93, 96, 97, 100] * 22, 1800 + Lq, False)
    synth.plant_homologs(q, db, 1.0, seed=Lq)
    bp = _search(q, db, ss_table, thld=-1.0, logethld=1e9, minpp=0.05, all_codes=1)
    try:
        assert len(bp.hit_records()) >= 592
        assert _check_map(bp, oracle_lib, q, db, minpp=0.05, logethld=1e9) >= 100
    finally:
        bp.close()
