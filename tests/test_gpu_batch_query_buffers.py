"""Where the batched query keeps its accumulators -- the gutter's entry buffer where that is large enough, a
block of its own otherwise -- changes no answer, over ingests and queries in any order, and a batch whose
entry buffer holds them takes next to no memory for its first query."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _records(V, n, seed):
    from graphzeppelin_b200 import streams as S
    rng = np.random.default_rng(seed)
    u = np.minimum((V * rng.random(n) ** 2).astype(np.int64), V - 1)
    return S.make_records(u.astype(np.uint32), rng.integers(0, V, n).astype(np.uint32))


def _equal(x, y):
    assert (x.num_cc == y.num_cc).all() and (x.rounds == y.rounds).all() and (x.status == y.status).all()
    assert all((a == b).all() for a, b in zip(x.labels, y.labels))


@pytest.mark.parametrize("Vs", [[2, 33, 1024, 1024, 300], [40, 20000, 1031]])
def test_shared_and_own_block_agree(gz, Vs):
    seeds = [9 + i for i in range(len(Vs))]
    none = np.zeros(0, np.uint8)
    with gz.CCSketchBatch(Vs, seeds) as a, gz.CCSketchBatch(Vs, seeds) as b:
        b.set_route(1e9)  # records straight to the sketches: no entry buffer
        # dense (the entries outgrow the accumulators), one graph alone, sparse, nothing, dense again
        steps = [lambda V, i, k: _records(V, 40 * V, k), lambda V, i, k: _records(V, 30 * V, k) if i == 1 else none,
                 lambda V, i, k: _records(V, max(1, V // 8), k), lambda V, i, k: none,
                 lambda V, i, k: _records(V, 90 * V, k)]
        for k, make in enumerate(steps):
            recs = [make(V, i, 100 * k + i) for i, V in enumerate(Vs)]
            a.ingest(recs)
            b.ingest(recs)
            want = b.connected_components()
            _equal(a.connected_components(), want)
            _equal(a.connected_components(), want)
        for g in range(len(Vs)):
            with gz.CCSketchAlg(Vs[g], seeds[g]) as s:
                for k, make in enumerate(steps):
                    r = make(Vs[g], g, 100 * k + g)
                    if r.size:
                        s.ingest_records(r)
                cc = s.connected_components()
                assert cc.size() == int(want.num_cc[g]) and (cc.parent_arr == want.labels[g]).all()


def test_own_block_of_changing_sizes(gz):
    """A server's queries take one block with many small graphs, few large ones and both in turn: the
    accumulators of one query lie where the states of another did."""
    from graphzeppelin_b200.serve import SketchServer
    sizes = [512] * 40 + [20000, 9000]
    recs = [_records(V, 3 * V, 50 + i) for i, V in enumerate(sizes)]
    want = []
    for i, V in enumerate(sizes):
        with gz.CCSketchAlg(V, 70 + i) as s:
            s.ingest_records(recs[i])
            cc = s.connected_components()
            want.append((cc.parent_arr.copy(), cc.size(), s.last_query_rounds))
    with SketchServer(1 << 30, 1 << 20) as srv:
        srv.set_query_snapshot(False)
        ids = [srv.admit(V, 70 + i) for i, V in enumerate(sizes)]
        srv.ingest(ids, recs)
        everyone, small = list(range(42)), list(range(40))
        for ask in (small, [40], [41, 0], small, everyone, [40, 41], small[:3], everyone, [40], small):
            out = srv.query_wait(srv.query_submit([ids[k] for k in ask]), [ids[k] for k in ask])
            for k, (lab, ncc, rounds, status) in zip(ask, out):
                assert status == 0 and ncc == want[k][1] and rounds == want[k][2] and (lab == want[k][0]).all()


def test_first_query_memory(gz):
    torch = pytest.importorskip("torch")
    V, G, n = 1024, 600, 16384
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    u = torch.randint(0, V, (n * G,), generator=gen, device="cuda", dtype=torch.int32)
    v = torch.randint(0, V, (n * G,), generator=gen, device="cuda", dtype=torch.int32)
    rec = torch.zeros((n * G, 9), dtype=torch.uint8, device="cuda")
    rec[:, 1:5] = u.view(torch.uint8).view(-1, 4)
    rec[:, 5:9] = v.view(torch.uint8).view(-1, 4)
    torch.cuda.synchronize()
    with gz.CCSketchBatch([V] * G, list(range(G))) as b:
        b.ingest_device(rec.data_ptr(), [n * i for i in range(G + 1)])
        before = torch.cuda.mem_get_info()[0]
        res = b.connected_components()
        taken = before - torch.cuda.mem_get_info()[0]
        # labels, parents and what the pool takes at a time; the accumulators alone are 157 MB
        assert taken < 80 << 20
        assert (res.num_cc >= 1).all()
