"""Small graphs are tiled for whole staged sketches in calls that bring them few entries a vertex, and for
bucket planes otherwise: the tiling a call leaves behind says which, and calls in any order -- in place,
staged, planes, small and large graphs together -- give the sketches and answers of single handles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _records(V, n, seed):
    from graphzeppelin_b200 import streams as S
    rng = np.random.default_rng(seed)
    u = np.minimum((V * rng.random(n) ** 2).astype(np.int64), V - 1)
    return S.make_records(u.astype(np.uint32), rng.integers(0, V, n).astype(np.uint32))


def _tiles(b):
    b._refresh_params()
    return [p.vertices_per_tile for p in b.params]


@pytest.mark.parametrize("V,entries,staged", [(256, 8, True), (33, 47, True), (256, 47, True), (256, 49, False),
                                              (512, 8, False), (512, 39, True), (512, 41, False), (1024, 39, False)])
def test_form_of_small_graphs(gz, V, entries, staged):
    G = (160 << 20) // (V * 2172) + 1  # more than L2 holds, so that nothing goes in place
    n = V * entries // 2
    rec = _records(V, n, V)
    with gz.CCSketchBatch([V] * G, [7] * G) as b:
        assert set(_tiles(b)) == {8}
        b.ingest([rec] * G)
        t = _tiles(b)[0]
        assert (t > 8) == staged
        with gz.CCSketchAlg(V, 7) as a:
            a.ingest_records(rec)
            want = a.dump_sketches().tobytes()
        for g in (0, G // 2, G - 1):
            assert b.dump_sketches(g).tobytes() == want


def test_forms_follow_the_calls(gz):
    Vs = [2, 3, 31, 64, 200, 256, 300, 512] * 40 + [9001, 20000]
    seeds = [11 + i for i in range(len(Vs))]
    small = range(len(Vs) - 2)
    # entries a vertex of the small and the large graphs: too few for the graphs of 300 and 512, too many, a large
    # graph among them, staged, a large one again, one graph alone, too few
    plan = [(12, 0), (60, 10), (1, 1), (30, 0), (12, 300), (0, 0), (20, 0)]
    fed = [[] for _ in Vs]
    forms = []
    with gz.CCSketchBatch(Vs, seeds) as b:
        b.set_route(0.0)  # every record through the gutter
        for k, (few, many) in enumerate(plan):
            recs = [_records(V, V * (few if g in small else many) // 2, 1000 * k + g) for g, V in enumerate(Vs)]
            if k == 5:
                recs[40] = _records(Vs[40], 5, 3)
            b.ingest(recs)
            forms.append(_tiles(b)[4] > 8)
            for g, r in enumerate(recs):
                fed[g].append(r)
            res = b.connected_components()
        assert forms == [False, False, False, True, False, True, False]
        for g in list(range(8)) + [40, len(Vs) - 2, len(Vs) - 1]:
            with gz.CCSketchAlg(Vs[g], seeds[g]) as a:
                for r in fed[g]:
                    if len(r):
                        a.ingest_records(r)
                assert b.dump_sketches(g).tobytes() == a.dump_sketches().tobytes()
                cc = a.connected_components()
                assert int(res.num_cc[g]) == cc.size() and (res.labels[g] == cc.parent_arr).all()


def test_asked_tiles_stay(gz):
    Vs = [200] * 700
    rec = _records(200, 800, 5)
    with gz.CCSketchBatch(Vs, [7] * 700, vertices_per_tile=[16] * 700) as b:
        b.ingest([rec] * 700)
        assert set(_tiles(b)) == {16}
        b.set_tuning(512, 2)
        before = _tiles(b)
        b.ingest([rec] * 700)
        assert _tiles(b) == before


@pytest.mark.parametrize("V,entries,direct", [(16, 16, True), (16, 24, False), (32, 9, True), (32, 11, False),
                                              (64, 4, True), (64, 6, False), (100, 3, True), (100, 5, False)])
def test_records_of_tiny_graphs_go_in_place(gz, V, entries, direct):
    """One kernel for records in place, several for the gutter and its tiles."""
    G = (300 << 20) // (V * 2604)  # more than L2 holds, less than 1 GB
    rec = _records(V, V * entries // 2, V)
    with gz.CCSketchBatch([V] * G, [7] * G) as b:
        b.ingest([rec] * G)
        at = b.get_profile()["kernel_launches"]
        b.ingest([rec] * G)
        assert (b.get_profile()["kernel_launches"] - at == 1) == direct
        b.ingest([rec] * G)
        with gz.CCSketchAlg(V, 7) as a:
            a.ingest_records(rec)
            assert b.dump_sketches(G - 1).tobytes() == a.dump_sketches().tobytes()


def test_params_while_another_thread_ingests(gz):
    """The tiling is read whole while calls of other densities change it."""
    import threading
    V, G = 256, 300
    few, many = _records(V, 8 * V // 2, 1), _records(V, 60 * V // 2, 2)
    with gz.CCSketchBatch([V] * G, [7] * G) as b:
        b.set_route(0.0)
        done = threading.Event()
        seen, errors = set(), []

        def read():
            try:
                while not done.is_set():
                    b._refresh_params()
                    p = b.params[G // 2]
                    seen.add((p.vertices_per_tile, p.num_tiles, p.vertices_per_bin, p.num_bins))
            except BaseException as e:  # noqa: BLE001
                errors.append(e)

        t = threading.Thread(target=read)
        t.start()
        for _ in range(20):
            b.ingest([few] * G)
            b.ingest([many] * G)
        done.set()
        t.join(60)
        assert not errors and not t.is_alive()
        assert seen <= {(8, 32, 8, 32), (32, 8, 32, 8)}
