"""Slot-order reads and writes on the device (slots_out_kernel, slots_in_kernel,
the position adjoint and the packed frame), after re-sorts have permuted the
engine's order: what is written comes back bit for bit, fields that are not
given stay, and every size about the kernels' blocks."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "C", "F", "Jp", "glow")


@pytest.mark.parametrize("path", ["batched", "plain"])
@pytest.mark.parametrize("n", [1, 3, 255, 256, 257, 5001])
def test_written_fields_come_back(n, path):
    from jellyfih_b200 import Engine, InstanceSpec
    rng = np.random.default_rng(n)
    e = Engine([InstanceSpec(64, 32, 32), InstanceSpec(n, 32, 32)], path=path, resort_interval=2)
    x = rng.uniform(0.1, 0.9, (n, 2)).astype(np.float32)
    mat = rng.choice([0, 1, 2, 3, -1], n).astype(np.int32)
    fib = rng.normal(size=(n, 2)).astype(np.float32)
    e.load(1, x, mat, fib)
    e.step(5)  # the order is no longer the slots'
    shapes = {"x": (n, 2), "v": (n, 2), "C": (n, 2, 2), "F": (n, 2, 2), "Jp": (n,), "glow": (n,)}
    want = {k: rng.uniform(0.2, 0.8, shapes[k]).astype(np.float32) for k in FIELDS}
    e.write(1, **want)
    got = e.read(1)
    for k in FIELDS:
        assert np.array_equal(got[k], want[k]), k
    assert np.array_equal(got["material"], mat) and np.array_equal(got["fiber"], fib)
    new = rng.uniform(0.2, 0.8, (n, 2)).astype(np.float32)
    for k in ("v", "x"):  # one half of a packed pair at a time
        want[k] = new
        e.write(1, **{k: new})
        got = e.read(1)
        for q in FIELDS:
            assert np.array_equal(got[q], want[q]), (k, q)
    e.close()


@pytest.mark.parametrize("res", [1, 17, 256])
def test_frame_comes_back_whole(res):
    from jellyfih_b200 import Engine, InstanceSpec
    e = Engine([InstanceSpec(1)])
    e.load(0, np.full((1, 2), 0.5, np.float32), np.array([2], np.int32))
    e.frame_create(res)
    e.frame_clear(0.25)
    e.render_flat(res, 1, 2.0, 2, 0.1, 0.2, 0.3)
    f = e.read_frame()
    hit = (f != 0.25).any(-1)
    assert hit.any() and np.array_equal(f[hit], np.broadcast_to(np.float32([0.1, 0.2, 0.3]), f[hit].shape))
    e.close()
