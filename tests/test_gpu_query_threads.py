"""One-launch queries of several handles and a batch in flight at the same time, from threads of their own: each
takes the whole GPU for a cooperative launch or a cluster of it, and gives what it gives alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _records(V, n, seed):
    from graphzeppelin_b200 import streams as S
    rng = np.random.default_rng(seed)
    return S.make_records(rng.integers(0, V, n).astype(np.uint32), rng.integers(0, V, n).astype(np.uint32))


def test_queries_of_many_threads(gz):
    sizes = [900, 5000, 60000, 60000, 300000]
    parts = [[_records(V, V // 2, 10 * i + k) for k in range(6)] for i, V in enumerate(sizes)]
    want = []
    for V, p in zip(sizes, parts):
        with gz.CCSketchAlg(V, 5) as a:
            w = []
            for rec in p:
                a.ingest_records(rec)
                cc = a.connected_components()
                w.append((cc.parent_arr.tobytes(), cc.size(), a.last_query_rounds))
            want.append(w)
    Vs = [500] * 60
    batch = [[_records(500, 300, 1000 * k + g) for g in range(60)] for k in range(6)]
    with gz.CCSketchBatch(Vs, list(range(60))) as b:
        bwant = []
        for recs in batch:
            b.ingest(recs)
            r = b.connected_components()
            bwant.append((r.num_cc.tobytes(), r.rounds.tobytes(), b"".join(x.tobytes() for x in r.labels)))
    errors = []

    def single(i):
        try:
            for _ in range(3):
                with gz.CCSketchAlg(sizes[i], 5) as a:
                    for k, rec in enumerate(parts[i]):
                        a.ingest_records(rec)
                        if k % 2:
                            cc, rounds = a.query_wait(a.query_submit())
                        else:
                            cc = a.connected_components()
                            rounds = a.last_query_rounds
                        assert (cc.parent_arr.tobytes(), cc.size(), rounds) == want[i][k]
        except BaseException as e:  # noqa: BLE001
            errors.append((i, e))

    def many():
        try:
            for _ in range(3):
                with gz.CCSketchBatch(Vs, list(range(60))) as b:
                    for k, recs in enumerate(batch):
                        b.ingest(recs)
                        r = b.connected_components()
                        assert (r.num_cc.tobytes(), r.rounds.tobytes(),
                                b"".join(x.tobytes() for x in r.labels)) == bwant[k]
        except BaseException as e:  # noqa: BLE001
            errors.append(("batch", e))

    threads = [threading.Thread(target=single, args=(i,)) for i in range(len(sizes))] + [threading.Thread(target=many)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(300)
    assert not errors, errors
    assert not any(t.is_alive() for t in threads)
