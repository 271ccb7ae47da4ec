"""Contexts of one device searching at the same time from several threads,
with realignments of different sizes (the MAP kernel's shared memory depends
on the query length and on the number of pairs): every search succeeds and
gives the records and alignments it gives alone."""
import threading

import numpy as np
import pytest

from test_map_gpu import _search

pytestmark = pytest.mark.gpu


def test_realignments_of_different_sizes(ss_table):
    from cother_b200 import synth
    opt = dict(thld=-1.0, logethld=1e9, minpp=0.05, ddmswgt=0.0)
    work = []
    # query length, profiles, searches: 16 warps a pair, then two, one, and
    # with more than 148 pairs eight
    for k, (Lq, nprof, n) in enumerate([(530, 10, 400), (60, 4, 0), (30, 4, 0), (290, 150, 0)]):
        q = synth.make_profiles([Lq], 1600 + k, True)
        db = synth.make_profiles([40 + 7 * (i % 9) for i in range(nprof)], 1610 + k, False)
        synth.plant_homologs(q, db, 0.6, seed=1620 + k)
        bp = _search(q, db, ss_table, **opt)
        work.append((bp, q, n, bp.hit_records(), bp.alignment_rows()))
    failed = []
    done = threading.Event()

    def searches(bp, q, n, recs, rows):
        try:
            i = 0
            while (i < n) if n else not done.is_set():
                bp.process_score_matrix(q)
                assert np.array_equal(bp.hit_records().view(np.uint32), recs.view(np.uint32))
                assert np.array_equal(bp.alignment_rows(), rows)
                i += 1
        except Exception as e:
            failed.append(e)
        if n or failed:
            done.set()

    threads = [threading.Thread(target=searches, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for w in work:
        w[0].close()
    assert not failed, failed[0]
