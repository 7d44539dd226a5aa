"""Graphs past 2^18 vertices at default settings, against the oracle byte for byte: plain entries through bucket
planes (bins beyond the shared-memory sort: global scatter; between 2^16 and 2^18 with more than 31 columns:
tiles of 16), sparse tiles in place, calls that go straight to the sketches, several gutter chunks to a wave;
the no-allocation ingest where its bins hold several tiles; the default query form on both sides of 2^21."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _among(ids, n, seed):
    """n records among the given vertex ids, repeats and self-loops among them."""
    from graphzeppelin_b200 import streams as S
    rng = np.random.default_rng(seed)
    k = np.minimum((ids.size * rng.random(n) ** 2).astype(np.int64), ids.size - 1)
    return S.make_records(ids[k].astype(np.uint32), ids[rng.integers(0, ids.size, n)].astype(np.uint32))


def _raw(rec):
    return np.ascontiguousarray(rec).view(np.uint8).reshape(-1)


def _ids(V, n):
    """n vertices: the first and last, runs across tile and bin edges, and others spread."""
    rng = np.random.default_rng(V)
    edge = [v for b in (8, 16, 32, 64, 4096, V // 2 // 64 * 64) for v in range(b - 2, b + 3)]
    ids = np.unique(np.concatenate([np.arange(4), np.arange(V - 9, V), edge, rng.integers(0, V, n)]))
    return rng.permutation(ids)


# 26 columns: one group of slots and the in-place route of sparse tiles; 36 (factor 1.6): two groups
@pytest.mark.parametrize("V,factor", [((1 << 18) + 1, 1.0), (70001, 1.6)])
@pytest.mark.parametrize("direct", [0.0, 1.0])
def test_plain_planes_bytes(gz, oracle_mod, V, factor, direct):
    osk = oracle_mod.OracleSketches(V, 23, factor)
    with gz.CCSketchAlg(V, 23, gz.CCAlgConfiguration().sketches_factor(factor)) as a:
        a.set_direct_factor(direct)
        everyone = np.random.default_rng(1).permutation(V)
        waves = [[_among(everyone, 300000, 1), _among(everyone, 40000, 2), _among(everyone, 7, 3)],  # three chunks
                 [_among(_ids(V, 300), 20000, 4)],  # few tiles, many entries in each
                 [_among(_ids(V, 3000), 900, 5)],   # few entries to a tile
                 [_among(everyone, 1, 6), _among(everyone, 33, 7)]]
        for wave in waves:
            for rec in wave:
                a.ingest_records(rec)
                osk.apply_records(_raw(rec))
            a.flush()
        a.apply_update_batch(0, V - 1, np.arange(500, dtype=np.uint32))
        osk.apply_batch(V - 1, np.arange(500, dtype=np.uint32))
        got = a.dump_sketches()
        assert np.array_equal(got, osk.data)


def test_noalloc_several_tiles_a_bin(gz, oracle_mod):
    torch = pytest.importorskip("torch")
    from graphzeppelin_b200 import _lib
    V = (1 << 21) + 5  # 65,537 tiles of 32 in bins of two
    try:
        osk = oracle_mod.OracleSketches(V, 4)  # pages that no record touches stay unmapped
    except MemoryError:
        pytest.skip("no address space for the oracle's sketches")
    ids = _ids(V, 2500)
    rec = _among(ids, 60000, 8)
    osk.apply_records(_raw(rec))
    sk = torch.zeros(V * osk.sketch_bytes, dtype=torch.uint8, device="cuda")
    dev = torch.from_numpy(_raw(rec).copy()).cuda()
    torch.cuda.synchronize()
    lib = _lib.load()
    half = rec.size // 2
    for at, n in ((0, half), (half, rec.size - half)):
        assert lib.gz_ingest_records_noalloc(ctypes.c_void_p(sk.data_ptr()), V, 4, 1.0,
                                             ctypes.c_void_p(dev.data_ptr() + 9 * at), n, None) == 0
    rows = sk.view(V, osk.sketch_bytes)
    at = np.sort(ids)
    got = rows[torch.from_numpy(at).cuda()].cpu().numpy()
    want = np.stack([osk.sketch(int(v)) for v in at])
    assert np.array_equal(got, want)
    rows[torch.from_numpy(at).cuda()] = 0
    words = sk.view(torch.int32) if sk.numel() % 4 == 0 else sk
    step = 1 << 30
    assert not any(bool(words[i:i + step].any()) for i in range(0, words.numel(), step))
    del rows, words, sk
    torch.cuda.empty_cache()


@pytest.mark.parametrize("V,one_launch", [(1 << 21, True), ((1 << 21) + 3, False)])
def test_default_query_form_past_its_switch(gz, V, one_launch):
    rec = _among(_ids(V, 200000), 300000, V)
    got = []
    with gz.CCSketchAlg(V, 2) as a:
        a.ingest_records(rec)
        a.flush()
        for mode in (-1, 2, 1):
            a.set_query_graph(mode)
            a.ingest_records(rec[:1])  # the same update twice: the answer is asked for anew
            a.ingest_records(rec[:1])
            a.flush()
            before = a.get_profile()["kernel_launches"]
            cc = a.connected_components()
            launches = a.get_profile()["kernel_launches"] - before
            if mode == -1:
                assert (launches <= 2) == one_launch
            got.append((cc.parent_arr.tobytes(), cc.size(), a.last_query_rounds))
    assert got[0] == got[1] == got[2]
