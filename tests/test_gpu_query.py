"""The one-launch query (mode 2) against the per-phase kernels with the round loop on the host
(mode 0): labels, component count, rounds, sample traces, spanning forest and out-of-samples
outcome are equal bit for bit (whole numbers: no tolerance). Sizes sit at the edges of its launch
shapes: a batch of 4 or 8 members and its remainder, the largest single cluster and one vertex
more, the last size whose warps keep their vertices' roots in registers and one batch more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 31, 33, 2048, 2049, 8191, 113664, 113673]


def _edges(kind, V, rng):
    if kind == "path":  # every round halves the components at best
        p = rng.permutation(V)
        return p[:-1], p[1:]
    if kind == "islands":  # many finished components early, some still growing
        k = max(1, V // 40)
        c = rng.integers(0, k, V)
        order = np.argsort(c, kind="stable")
        same = c[order][:-1] == c[order][1:]
        keep = same & (rng.random(V - 1) < 0.9)
        return order[:-1][keep], order[1:][keep]
    n = 8 * V  # giant: a power-law graph, one component over half the vertices, isolated vertices
    a = np.minimum((V * 0.9 * rng.random(n) ** 3).astype(np.int64), V - 1)
    b = rng.integers(0, max(1, int(V * 0.9)), n)
    keep = a != b
    return a[keep], b[keep]


def _answers(gz, alg, mode, trace):
    alg.set_query_graph(mode)
    alg.set_trace(trace)
    try:
        cc = alg.connected_components()
    except gz.OutOfSamplesException:
        return "out of samples", alg.last_query_rounds
    forest = {(min(e), max(e)) for e in alg.calc_spanning_forest().get_edges()}
    assert len(forest) == alg.get_num_vertices() - cc.size()
    return (cc.parent_arr.tobytes(), cc.size(), alg.last_query_rounds,
            alg.get_trace().tobytes() if trace else b"")


@pytest.mark.parametrize("kind", ["path", "islands", "giant"])
@pytest.mark.parametrize("V", SIZES)
def test_one_launch_equals_host_loop(V, kind):
    import graphzeppelin_b200 as gz
    from graphzeppelin_b200 import streams as S
    rng = np.random.default_rng(V)
    u, v = _edges(kind, V, rng)
    rec = S.make_records(u.astype(np.uint32), v.astype(np.uint32))
    algs = [gz.CCSketchAlg(V, 77) for _ in range(3)]
    for a in algs:
        a.ingest_records(rec)
    want = _answers(gz, algs[0], 0, True)
    got = _answers(gz, algs[1], 2, True)
    assert got == want
    assert _answers(gz, algs[2], 2, False)[:3] == want[:3]
    for a in algs:
        a.close()


@pytest.mark.parametrize("factor", [1.0, 2.5])
@pytest.mark.parametrize("V", [60, 3000])
def test_one_endpoint_updates(V, factor):
    """Updates that reach one endpoint only (apply_update_batch): no complement merge, vertices whose
    empty sketch samples ZERO are linked by others later, and sampling may run out."""
    import graphzeppelin_b200 as gz
    rng = np.random.default_rng(V + int(factor))
    u, v = _edges("giant", V, rng)
    order = np.argsort(u, kind="stable")
    u, v = u[order], v[order]
    cuts = np.flatnonzero(np.diff(u)) + 1
    got = []
    for mode in (0, 2):
        a = gz.CCSketchAlg(V, 5, gz.CCAlgConfiguration().sketches_factor(factor))
        for src, dst in zip(u[np.r_[0, cuts]], np.split(v, cuts)):
            a.apply_update_batch(0, int(src), dst)
        got.append(_answers(gz, a, mode, True))
        a.close()
    assert got[0] == got[1]


def test_query_after_a_failed_one():
    """An out-of-samples query and an aborted one leave the accumulators clean for the next."""
    import graphzeppelin_b200 as gz
    from graphzeppelin_b200 import streams as S
    rng = np.random.default_rng(3)
    V = 5000
    u, v = _edges("islands", V, rng)
    rec = S.make_records(u.astype(np.uint32), v.astype(np.uint32))
    a = gz.CCSketchAlg(V, 9)
    a.ingest_records(rec)
    first = a.connected_components().parent_arr.copy()
    bad = S.make_records(np.array([V + 5], np.uint32), np.array([1], np.uint32))
    a.ingest_records(bad)  # reported by the query, which is not run
    with pytest.raises(gz.BadVertexError):
        a.connected_components()
    assert (a.connected_components().parent_arr == first).all()
    a.close()
