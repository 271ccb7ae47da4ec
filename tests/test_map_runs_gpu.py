"""MAP realignment at the ends of its chunks: profile lengths around 32-column
chunks and their runs (the cell-score kernel splits a band's chunks into 16
runs), and query lengths around 32-row bands. Every realigned pair's rows,
counts and coordinates equal the oracle's."""
import numpy as np
import pytest

from test_map_gpu import _check_map, _search

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lq", [31, 32, 33, 64, 97, 290])
def test_profile_lengths_around_chunks(oracle_lib, ss_table, Lq):
    from cother_b200 import synth
    q = synth.make_profiles([Lq], 1100 + Lq, True)
    db = synth.make_profiles([33, 1, 32, 31, 64, 65, 95, 481, 482, 511, 513, 545, 30, 2], 1200 + Lq, False)
    synth.plant_homologs(q, db, 0.6, seed=Lq)
    bp = _search(q, db, ss_table, thld=-1.0, logethld=1e9, minpp=0.05, all_codes=1)
    try:
        assert _check_map(bp, oracle_lib, q, db, minpp=0.05, logethld=1e9) >= 4
    finally:
        bp.close()


@pytest.mark.parametrize("Lq", [33, 97, 290])
def test_many_pairs(oracle_lib, ss_table, Lq):
    """More pairs than one and a half an SM take the steps in groups of four:
    chunks that end inside and between groups, and more bands than warps."""
    from cother_b200 import synth
    q = synth.make_profiles([Lq], 1300 + Lq, True)
    db = synth.make_profiles([*range(26, 38), *range(58, 70), 93, 96, 97, 100] * 12, 1400 + Lq, False)
    synth.plant_homologs(q, db, 1.0, seed=Lq)
    bp = _search(q, db, ss_table, thld=-1.0, logethld=1e9, minpp=0.05, all_codes=1)
    try:
        assert _check_map(bp, oracle_lib, q, db, minpp=0.05, logethld=1e9) > 222
    finally:
        bp.close()
