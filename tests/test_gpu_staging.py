"""apply_update_batch stages a whole call at once: calls that end at, cross or fill the staging buffer
(2^20 entries) give the sketches of the same updates in small calls, and a refused call adds nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CAP = 1 << 20


@pytest.mark.parametrize("sizes", [[0, 1, 3], [CAP], [CAP - 1, 1, 1], [5, CAP], [7, 2 * CAP + 3, 2]])
def test_staged_calls_equal_small_calls(gz, sizes):
    V = 3000
    rng = np.random.default_rng(len(sizes) + sum(sizes))
    calls = [(int(rng.integers(V)), rng.integers(0, V, n).astype(np.uint32)) for n in sizes]
    calls = [(s, d[d != s]) for s, d in calls]
    with gz.CCSketchAlg(V, 11) as a, gz.CCSketchAlg(V, 11) as b:
        for s, d in calls:
            a.apply_update_batch(0, s, d)
            with pytest.raises(gz.BadVertexError):
                a.apply_update_batch(0, s, np.append(d[:100], np.uint32(V)))
            # an update that occurs an even number of times cancels: small calls of the odd ones
            ids, cnt = np.unique(d, return_counts=True)
            for part in np.array_split(ids[cnt % 2 == 1], 3):
                b.apply_update_batch(0, s, part)
        a.flush()
        b.flush()
        assert a.dump_sketches().tobytes() == b.dump_sketches().tobytes()
