"""Queries that follow one another on one handle: the one-launch query keeps its accumulators between
queries and leaves each clear for the next, also after a query that ran out of samples. Answers equal
those of a fresh handle's per-phase kernels (whole numbers: no tolerance). Sizes: one cluster, the
first cooperative launch, warps that keep their vertices' roots in registers, and more vertices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _records(V, n, seed):
    from graphzeppelin_b200 import streams as S
    rng = np.random.default_rng(seed)
    u = np.minimum((V * rng.random(n) ** 2).astype(np.int64), V - 1)
    return S.make_records(u.astype(np.uint32), rng.integers(0, V, n).astype(np.uint32))


def _fresh(gz, V, seed, parts):
    with gz.CCSketchAlg(V, seed) as a:
        a.set_query_graph(0)
        for p in parts:
            a.ingest_records(p)
        cc = a.connected_components()
        return cc.parent_arr.tobytes(), cc.size(), a.last_query_rounds


def _ticket(a):
    cc, rounds = a.query_wait(a.query_submit())
    return cc.parent_arr.tobytes(), cc.size(), rounds


@pytest.mark.parametrize("V", [700, 2049, 5000, 120000])
def test_queries_follow_one_another(gz, V):
    parts = [_records(V, V // 2, 1), _records(V, V // 3, 2), _records(V, 2 * V, 3)]
    rng = np.random.default_rng(V)
    with gz.CCSketchAlg(V, 19) as a:
        a.set_query_graph(2)
        for k in range(len(parts)):
            a.ingest_records(parts[k])
            want = _fresh(gz, V, 19, parts[:k + 1])
            assert _ticket(a) == want
            assert _ticket(a) == want  # again, on the same sketches
            # two sketches of noise: they FAIL in every round, with whatever merged into them
            noise = {v: rng.integers(0, 256, a.params.sketch_bytes, dtype=np.uint8) for v in (1, V // 2)}
            for v, x in noise.items():
                a.apply_raw_buckets_update(v, x)
            with pytest.raises(gz.OutOfSamplesException):
                a.query_wait(a.query_submit())
            for v, x in noise.items():
                a.apply_raw_buckets_update(v, x)
            assert _ticket(a) == want
            cc = a.connected_components()  # the blocking query's own buffers
            assert (cc.parent_arr.tobytes(), cc.size(), a.last_query_rounds) == want
