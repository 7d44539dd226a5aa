"""Records of small graphs that go straight to the sketches are spread over the GPU as those of large ones are:
the same number of records takes about as long in thousands of small graphs as in a few large ones. And the
split changes nothing: sketch bytes equal single handles', at the edges of warps, record tiles and parts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _records(V, n, seed):
    from graphzeppelin_b200 import streams as S
    rng = np.random.default_rng(seed)
    return S.make_records(rng.integers(0, V, n).astype(np.uint32), rng.integers(0, V, n).astype(np.uint32))


@pytest.mark.parametrize("counts", [[0, 1, 31, 32, 33], [255, 256, 257, 4095], [4096, 4097, 8193, 0, 5],
                                    [1] * 700 + [4096, 300], [20000, 3]])
def test_direct_bytes(gz, counts):
    Vs = [[2, 64, 300, 1031][i % 4] for i in range(len(counts))]
    recs = [_records(V, n, 5 + i) for i, (V, n) in enumerate(zip(Vs, counts))]
    with gz.CCSketchBatch(Vs, [3 + i for i in range(len(Vs))]) as b:
        b.set_route(1e9)
        b.ingest(recs)
        for g in list(range(min(8, len(Vs)))) + [len(Vs) - 2, len(Vs) - 1]:
            with gz.CCSketchAlg(Vs[g], 3 + g) as a:
                a.ingest_records(recs[g])
                assert b.dump_sketches(g).tobytes() == a.dump_sketches().tobytes()


def test_small_graphs_take_no_longer(gz):
    torch = pytest.importorskip("torch")
    total, best = 1 << 19, {}
    for V in (64, 4096):
        G = total // V
        n = V // 2  # one entry a vertex: the direct route
        rec = torch.zeros((n * G, 9), dtype=torch.uint8, device="cuda")
        gen = torch.Generator(device="cuda")
        gen.manual_seed(V)
        for at in (1, 5):
            ids = torch.randint(0, V, (n * G,), generator=gen, device="cuda", dtype=torch.int32)
            rec[:, at:at + 4] = ids.view(torch.uint8).view(-1, 4)
        torch.cuda.synchronize()
        with gz.CCSketchBatch([V] * G, list(range(G))) as b:
            b.set_profiling(True)
            times = []
            for _ in range(6):
                b.set_profiling(True)
                b.ingest_device(rec.data_ptr(), np.arange(G + 1, dtype=np.uint64) * n)
                times.append(b.get_profile()["sketch_update_ms"])
            best[V] = min(times[1:])
    # a warp per record tile, which a small graph's records do not fill: 5 to 10 times as long
    assert best[64] < 2.5 * best[4096]
