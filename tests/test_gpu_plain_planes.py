"""Bucket planes fed with plain entries (CubeSketch, sketches of more than 31 columns, large graphs,
the no-allocation ingest), the coded path's small tiles, and calls that go straight to the sketches,
against the oracle: sketch bytes equal (no tolerance). Sizes sit at the edges of tiles, of groups of
32 slots and of the planes' depth (11 rows)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _records(V, n, seed):
    from graphzeppelin_b200 import streams as S
    rng = np.random.default_rng(seed)
    u = np.minimum((V * rng.random(n) ** 2).astype(np.int64), V - 1)  # some tiles heavy, some light
    v = rng.integers(0, V, n)
    return S.make_records(u.astype(np.uint32), v.astype(np.uint32))  # self-loops among them


def _raw(rec):
    return np.ascontiguousarray(rec).view(np.uint8).reshape(-1)


# 31, 32 and 33 columns: one group with the deterministic slot, one full group and the slot alone, two
@pytest.mark.parametrize("V,factor,cube", [
    (2, 1.0, True), (9, 1.0, True), (40, 1.0, True), (64, 1.0, True), (300, 1.0, True), (1031, 1.0, True),
    (40, 4.5, False), (1024, 2.25, False), (1024, 2.3, False), (1024, 2.4, False), (777, 5.0, False),
    (2, 1.0, False), (9, 1.0, False), (33, 1.0, False), (4735, 1.0, False), (4737, 1.0, False),
    (9471, 1.0, False), (9473, 1.0, False)])
def test_sketch_bytes(V, factor, cube, oracle_mod):
    import graphzeppelin_b200 as gz
    alg = gz.CCSketchAlg(V, 31, gz.CCAlgConfiguration().sketches_factor(factor),
                         sketch_algorithm="cube" if cube else "cameo")
    alg.set_direct_factor(0)  # everything through the planes
    rec = _records(V, 40000 if V < 2000 else 150000, V)  # depths past the planes' rows occur
    cut = rec.size // 3
    osk = oracle_mod.OracleSketches(V, 31, factor, cube=cube)
    for part in (rec[:cut], rec[cut:cut + 1], rec[cut + 1:]):
        alg.ingest_records(part)
    osk.apply_records(_raw(rec))
    assert alg.dump_sketches().tobytes() == osk.data.tobytes()
    alg.close()


@pytest.mark.parametrize("V", [2, 31, 1024, 20000])
def test_direct_calls(V, oracle_mod):
    """Calls too small for the gutter: one record, a few, up to the threshold and past it; records
    naming a vertex >= V are dropped and reported."""
    import graphzeppelin_b200 as gz
    from graphzeppelin_b200 import streams as S
    alg = gz.CCSketchAlg(V, 8)
    alg.set_direct_factor(1e6)  # straight to the sketches at any density
    rec = _records(V, 5000, V + 1)
    for a, b in ((0, 1), (1, 2), (2, 33), (33, 1000), (1000, 5000)):
        alg.ingest_records(rec[a:b])
    osk = oracle_mod.OracleSketches(V, 8)
    osk.apply_records(_raw(rec))
    assert alg.dump_sketches().tobytes() == osk.data.tobytes()
    alg.ingest_records(S.make_records(np.array([V, 0], np.uint32), np.array([0, V + 7], np.uint32)))
    with pytest.raises(gz.BadVertexError):
        alg.flush()
    assert alg.dump_sketches().tobytes() == osk.data.tobytes()
    alg.close()


def test_direct_threshold_routes_agree():
    import graphzeppelin_b200 as gz
    V = 3000
    rec = _records(V, 20000, 4)
    got = []
    for factor in (0.0, 1.0, 1e6):
        alg = gz.CCSketchAlg(V, 3)
        alg.set_direct_factor(factor)
        at = 0
        for n in (1, 5, 100, 2000, 5000, 12894):
            alg.ingest_records(rec[at:at + n])
            at += n
        got.append(alg.dump_sketches().tobytes())
        alg.close()
    assert got[0] == got[1] == got[2]


@pytest.mark.parametrize("V,n", [(9, 3000), (1000, 50001), (65535, 200000), (65544, 200000)])
def test_noalloc_tiles(V, n):
    """65,536 vertices are the most with a bin per 8 vertices; the caller's buffer ends at the last
    sketch."""
    torch = pytest.importorskip("torch")
    import graphzeppelin_b200 as gz
    from graphzeppelin_b200 import _lib
    lib = _lib.load()
    rec = _records(V, n, n)
    alg = gz.CCSketchAlg(V, 12)
    alg.ingest_records(rec)
    want = torch.from_numpy(alg.dump_sketches()).cuda()
    got = torch.zeros_like(want)
    dev = torch.from_numpy(_raw(rec).copy()).cuda()
    torch.cuda.synchronize()
    assert lib.gz_ingest_records_noalloc(ctypes.c_void_p(got.data_ptr()), V, 12, 1.0,
                                         ctypes.c_void_p(dev.data_ptr()), n, None) == 0
    assert torch.equal(got, want)
    alg.close()
