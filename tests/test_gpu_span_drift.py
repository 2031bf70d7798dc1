"""Particles that leave their CTA's window within a chunk of the batched path's
spans (jellyfih_b200/csrc/jf_span.cu): they scatter into the spill grid and
gather the rows that the other CTAs publish."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_a_slow_pass_gathers_what_the_substep_before_published():
    """A CTA whose pass takes far longer than its neighbours' (60,000 overflow
    particles on four rows) and whose fast particles come last in it: the rows
    they gather are still those of the substep before when the chunk's last
    grid is published.  The fast ones fly alone, so that they keep their velocity
    (64 substeps of about 10 ulp of weights, and stresses of rounding, are 1e-4 of
    it); a gather from the next grid, which does not hold them yet, gives 0."""
    from jellyfih_b200 import Engine, InstanceSpec
    n, fast, v0 = 60000, 6, 60.0
    rng = np.random.default_rng(1)
    x = np.empty((n + fast, 2), np.float32)
    x[:n, 0] = rng.uniform(8 / 128, 80 / 128, n)
    x[:n, 1] = rng.uniform(60.3 / 128, 64.2 / 128, n)
    x[n:, 0] = (np.linspace(96, 121, fast) + 0.4) / 128
    x[n:, 1] = 62.4 / 128
    v = np.zeros((n + fast, 2), np.float32)
    v[n:, 1] = v0
    e = Engine([InstanceSpec(n + fast)], cell_cap=1, resort_interval=64)
    e.load(0, x, np.r_[np.zeros(n, np.int32), np.ones(fast, np.int32)])
    e.write(0, v=v)
    e.step(64)
    got, counts = e.read(0), e.path_counts()
    assert not e.error_flags().any() and counts["remote_gathers"] > 0
    e.close()
    assert np.abs(got["v"][n:] - v[n:]).max() <= 1e-3 * v0
    assert np.abs(got["x"][n:, 1] - (x[n:, 1] + 64 * 2e-5 * v0)).max() <= 1e-3 * (64 * 2e-5 * v0)
