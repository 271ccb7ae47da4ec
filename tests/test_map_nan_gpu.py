"""MAP realignment with transitions that are not numbers: the log-sum of two
terms keeps a NaN of its first term and leaves out one of its second, as the
oracle's (and the reference's a < b ? b : a) does. Forward-backward values
equal the oracle's bit for bit, alignments and counts too."""
import numpy as np
import pytest

from test_map_gpu import _check_map, _search

pytestmark = pytest.mark.gpu

LENS = [33, 1, 64, 200, 97, 150, 31, 80]


# transitions MM, MI, MD, IM, II, DM, DD: II and DD are second terms, the
# others enter first terms too
@pytest.mark.parametrize("kinds", [(4,), (6,), (4, 6), (1, 2), (0, 3, 5)])
@pytest.mark.parametrize("copies", [1, 32])       # a pair for every SM and fewer; more
def test_nan_transitions(oracle_lib, ss_table, kinds, copies):
    import cother_b200 as cb
    from cother_b200 import synth
    lens = LENS * copies
    q = synth.make_profiles([97], 1500, True)
    db = synth.make_profiles(lens, 1501, False)
    synth.plant_homologs(q, db, 0.6, seed=1502)
    rng = np.random.default_rng(1503)
    for k in kinds:
        q.trn[k, rng.random(q.trn.shape[1]) < 0.03] = np.nan
        db.trn[k, rng.random(db.trn.shape[1]) < 0.03] = np.nan
    bp = _search(q, db, ss_table, thld=-1.0, logethld=1e9, minpp=0.05, all_codes=1)
    try:
        assert _check_map(bp, oracle_lib, q, db, minpp=0.05, logethld=1e9) >= 3 * copies
        st = cb.records_table(bp.read_statistics())
        sc, ms, _ = bp.read_score_matrix(q.npositions, db.npositions)
        for i in range(0, len(st["score"]), 7):
            p = int(st["org_pro_no"][i])
            s0, Ld = int(db.starts[p]), int(db.lens[p])
            want = oracle_lib.map_pair(q, db, p, sc[:, s0:s0 + Ld], ms[:, s0:s0 + Ld],
                                       float(st["log_evalue_pair"][i]), minpp=0.05)["fb"]
            fb = bp.map_fb(i, q.npositions)
            assert np.array_equal(np.isnan(fb), np.isnan(want))
            assert np.array_equal(fb[~np.isnan(fb)].view(np.uint32), want[~np.isnan(want)].view(np.uint32))
    finally:
        bp.close()
