"""The autotuner compares the whole device time of an ingest call -- gutter and sketch update, since each form
hashes in a different one of them -- over a scratch batch with as many sketches as the real one has (up to 1 GB):
what it picks is no slower than the default."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_autotune_picks_no_slower_form(gz):
    torch = pytest.importorskip("torch")
    V, G, n = 1024, 400, 2048  # 1.7 GB of sketches, 4 entries a vertex
    rec = torch.zeros((n * G, 9), dtype=torch.uint8, device="cuda")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    for at in (1, 5):
        rec[:, at:at + 4] = torch.randint(0, V, (n * G,), generator=gen, device="cuda",
                                          dtype=torch.int32).view(torch.uint8).view(-1, 4)
    torch.cuda.synchronize()
    off = np.arange(G + 1, dtype=np.uint64) * n
    with gz.CCSketchBatch([V] * G, list(range(G))) as b:
        def call():
            times = []
            for _ in range(6):
                b.set_profiling(True)
                b.ingest_device(rec.data_ptr(), off)
                p = b.get_profile()
                times.append(p["gutter_ms"] + p["sketch_update_ms"])
            return min(times[1:])

        default = call()
        b.autotune(4)
        assert call() < 1.25 * default  # staged tiles: 1.5 to 1.7 times as long
