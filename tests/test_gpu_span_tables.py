"""The spans as an engine reports them (Engine.spans): which batches run as spans
and at what size, and the bands that the device cut, which have to obey what
test_span_layout.py asks of its restatement of the cuts."""
import numpy as np
import pytest

from test_span_layout import BATCHES, check, setup

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _engine(shapes, slots, **kw):
    from jellyfih_b200 import Engine, InstanceSpec
    return Engine([InstanceSpec(slots, nx, ny, ny / nx) for nx, ny in shapes], **kw)


# the engine refuses a batch whose cluster layout does not fit, and runs one of several n_grid as clusters
REFUSED = [[(1000, 40)], [(256, 256)] * 40]


@pytest.mark.parametrize("shapes", [b for b in BATCHES if b not in REFUSED and len({nx for nx, _ in b}) == 1],
                         ids=lambda s: f"{len(s)}x{s[0][0]}x{s[0][1]}")
def test_the_bands_on_the_device_cover_the_rows_and_fit(shapes):
    n_sm = torch.cuda.get_device_properties(0).multi_processor_count
    groups, cap, rowoff, _ = setup(shapes, n_sm)
    slots = 400
    e = _engine(shapes, slots)
    s = e.spans()
    assert len(s["bands"]) == 0  # nothing sorted yet
    assert (s["launches"], s["ctas"], s["block_threads"], s["window_nodes"]) == (
        len(groups), max(g[4] for g in groups), 512, cap)
    rng = np.random.default_rng(len(shapes))
    for kind in range(3):
        for m, (nx, ny) in enumerate(shapes):
            lo, hi = np.array([1.0, 1.0]) / nx, np.array([nx - 2.0, ny - 2.0]) / nx
            if kind == 1:  # all of a few tanks' particles in a few rows
                hi[1] = lo[1] + 4.0 / nx if m % 3 else hi[1]
            n = slots if kind < 2 else (0 if m % 2 else slots)
            e.load(m, rng.uniform(lo, hi, (n, 2)).astype(np.float32), rng.choice([0, 1], n).astype(np.int32))
        e.step(1)
        bands = e.spans()["bands"]
        assert e.sync()
        for k, g in enumerate(groups):
            b = bands[bands[:, 0] == k]
            per_cta = [b[b[:, 1] == c] for c in range(g[4])]
            assert sum(len(p) for p in per_cta) == len(b)
            cuts = [0]
            for p in per_cta:
                at = cuts[-1]
                for _, _, m, first, end in p:  # one after the other from where the CTA before ended
                    assert rowoff[m] - g[2] + first == at
                    at = rowoff[m] - g[2] + end
                cuts.append(at)
            check(shapes, g, rowoff, cap, cuts)
    e.close()


@pytest.mark.parametrize("threads,runs", [(0, 512), (256, 256), (768, 768)])
def test_which_layout_a_batch_runs_as(threads, runs):
    e = _engine([(128, 128)] * 32, 1000, block_threads=threads)
    assert e.spans()["block_threads"] == runs
    e.close()
    for shapes, kw in (([(64, 64), (128, 128)], {}), ([(8, 8)] * 2000, {}), ([(128, 128)] * 2, {"cluster_size": 4}),
                       ([(128, 128)], {"path": "plain"})):
        e = _engine(shapes, 100, block_threads=threads, **kw)
        assert e.spans() is None
        e.close()
