"""The batched path's spans (jellyfih_b200/csrc/jf_span.cu) against one cluster
per instance, over the batches whose layouts differ most: bands of four rows,
several instances in one CTA, cuts inside instances, partial 32-cell segments,
several groups.  One substep from the same moving state: both layouts sum the
same contributions in different orders, so every field agrees within the 1e-5
of its max-norm that one substep's summation orders are held to against the
oracle, and positions within 4 ulp; a chunk across re-sorts keeps the payload's
centre within 1e-6 (the order spread of 48 substeps is about 1e-9 of it)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BATCHES = {  # (instances, slots, n_grid, n_grid_y)
    "one tank": [(1, 80000, 128, 128)],
    "eight rows": [(3, 200, 16, 8)],
    "several in a CTA": [(300, 300, 16, 12)],
    "partial segments": [(5, 9000, 40, 52)],
    "uneven": [(3, 30000, 64, 64), (2, 40000, 64, 128), (1, 0, 64, 64)],
    "groups": [(52, 1500, 128, 128)],
}


def _inputs(shapes, seed):
    from jellyfih_b200 import InstanceSpec
    rng = np.random.default_rng(seed)
    specs, states = [], []
    for count, n, nx, ny in shapes:
        h = ny / nx
        for _ in range(count):
            specs.append(InstanceSpec(n, nx, ny, h))
            lo = 2.0 / nx
            x = rng.uniform([lo, lo], [1 - lo, h - lo], (n, 2)).astype(np.float32)
            mat = rng.choice([0, 0, 0, 0, 1, 2, 3, -1], n).astype(np.int32)
            fib = rng.normal(size=(n, 2)).astype(np.float32)
            fib /= np.maximum(np.linalg.norm(fib, axis=1, keepdims=True), 1e-6)
            states.append((x, mat, fib, rng.normal(0, 0.3, (n, 2)).astype(np.float32),
                           rng.normal(0, 2.0, (n, 2, 2)).astype(np.float32),
                           (np.eye(2) + rng.normal(0, 2e-3, (n, 2, 2))).astype(np.float32)))
    return specs, states


def _engine(specs, states, **kw):
    from jellyfih_b200 import Engine
    e = Engine(specs, **kw)
    for m, (x, mat, fib, v, C, F) in enumerate(states):
        e.load(m, x, mat, fib)
        e.write(m, v=v, C=C, F=F)
    e.time = 0.02
    return e


@pytest.mark.parametrize("threads", [0, 256, 768])
@pytest.mark.parametrize("batch", BATCHES)
def test_spans_match_clusters(batch, threads):
    specs, states = _inputs(BATCHES[batch], 7)
    a = _engine(specs, states, block_threads=threads, resort_interval=16)
    b = _engine(specs, states, cluster_size=4, resort_interval=16)
    a.step(1)
    b.step(1)
    for m in range(len(specs)):
        live = states[m][1] >= 0
        p, q = a.read(m), b.read(m)
        assert np.abs(p["x"] - q["x"]).max(initial=0.0) <= 4 * np.spacing(np.float32(specs[m].domain_height))
        for k in ("v", "C", "F", "Jp"):
            scale = np.abs(q[k][live]).max(initial=1e-30)
            assert np.abs(p[k][live].astype(np.float64) - q[k][live]).max(initial=0.0) <= 1e-5 * scale, (m, k)
        (gv, gm), (hv, hm) = a.read_grid(m), b.read_grid(m)
        assert np.array_equal(gm > 0, hm > 0)
        assert np.abs(gm - hm).max() <= 1e-5 * max(np.abs(hm).max(), 1e-30)
    assert not a.error_flags().any()
    a.close()
    b.close()


def test_spans_carry_a_chunk_as_clusters_do():
    from jellyfih_b200 import Engine, InstanceSpec, tank
    tanks = [tank.fill_tank(g, 80000) for g in tank.gaussian_genomes(9, 3)]
    rows = []
    for cs in (0, 8):
        e = Engine([InstanceSpec(80000)] * 9, cluster_size=cs, resort_interval=16)
        for m, t in enumerate(tanks):
            e.load(m, *t[:3])
        rows.append(e.run_headless(48))
        e.close()
    assert np.abs(rows[0] - rows[1]).max() <= 1e-6


@pytest.mark.parametrize("cluster_size", [0, 4])
def test_a_smaller_engine_leaves_the_larger_one_its_shared_memory(cluster_size):
    from jellyfih_b200 import Engine, InstanceSpec
    big = Engine([InstanceSpec(2000, 128, 256, 2.0)] * 32, cluster_size=cluster_size)
    small = Engine([InstanceSpec(500, 32, 32, 1.0)], cluster_size=cluster_size)
    big.step(3)
    small.step(3)
    big.step(3)
    assert big.sync() and small.sync()
    big.close()
    small.close()
