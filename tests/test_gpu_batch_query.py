"""The batched query's two forms (one launch up to 2^23 vertices, grouping rounds beyond) and batches
whose graphs take different sketch-update forms give what each graph gives alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_grouping_rounds_equal_one_launch(gz):
    from graphzeppelin_b200 import streams as S
    V, n = 1024, 8200  # 8.4e6 vertices together; halves below 2^23
    kinds = [S.planted_partition_stream(V, k, 7 + k, mean_degree=6, min_size=5)[0].records for k in (1, 9, 60)]
    kinds.append(np.zeros(0, dtype=S.RECORD_DTYPE))
    sts = [kinds[i % 4] for i in range(n)]
    seeds = [31 + i for i in range(n)]
    with gz.CCSketchBatch([V] * n, seeds) as b:
        b.ingest(sts)
        whole = [b.connected_components() for _ in range(2)]  # launched, then as a captured round
    for lo, hi in ((0, n // 2), (n // 2, n)):
        with gz.CCSketchBatch([V] * (hi - lo), seeds[lo:hi]) as b:
            b.ingest(sts[lo:hi])
            part = b.connected_components()
        for w in whole:
            assert (w.num_cc[lo:hi] == part.num_cc).all() and (w.rounds[lo:hi] == part.rounds).all()
            assert (w.status[lo:hi] == part.status).all()
            assert all((w.labels[lo + i] == part.labels[i]).all() for i in range(hi - lo))


# factor 2: 28 columns at 1000 vertices (bucket planes), 44 at 70000 (staged tiles)
@pytest.mark.parametrize("Vs,factor", [([2, 70000, 31, 33, 9001], 1.0), ([1000, 70000, 40, 5003], 2.0)])
def test_mixed_graphs_match_single_handles(gz, Vs, factor):
    from graphzeppelin_b200 import streams as S
    sts = [S.erdos_renyi_stream(V, min(0.9, 3.0 / V), seed=3 + V, churn_fraction=0.2).records for V in Vs]
    seeds = [77 + V for V in Vs]
    with gz.CCSketchBatch(Vs, seeds, sketches_factor=factor) as b:
        b.set_route(0.0)  # every record through the gutter
        b.ingest(sts)
        res = [b.connected_components() for _ in range(2)][1]
        for g, V in enumerate(Vs):
            with gz.CCSketchAlg(V, seeds[g], gz.CCAlgConfiguration().sketches_factor(factor)) as alg:
                alg.ingest_records(sts[g])
                cc = alg.connected_components()
                assert b.dump_sketches(g).tobytes() == alg.dump_sketches().tobytes()
                assert int(res.num_cc[g]) == cc.size() and (res.labels[g] == cc.parent_arr).all()
                assert int(res.rounds[g]) == alg.last_query_rounds
