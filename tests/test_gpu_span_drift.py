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


@pytest.mark.parametrize("axisym", [False, True])
@pytest.mark.parametrize("threads", [0, 768])
@pytest.mark.parametrize("batch,cluster", [("one tank", 0), ("several in a CTA", 0), ("groups", 0), ("mixed n_grid", 0),
                                           ("one tank", 4), ("one tank", 16), ("several in a CTA", 2)])
def test_tanks_that_drift_beside_tanks_that_do_not(batch, cluster, threads, axisym):
    """One tank of three moves up three rows in a chunk of eight substeps, all its
    particles at one velocity; a contribution that is lost costs them most of it.
    Clusters have the same far rows and are held to the same.  Against the FP32
    oracle: the 1e-5 of the max-norm that one substep's summation orders are held
    to, for eight substeps, and ten times what the oracle's two precisions differ
    by, which is what these tanks make of a rounding."""
    from jellyfih_b200 import Engine, InstanceSpec
    from oracle import oracle as O
    shapes = {"one tank": [(128, 128)], "several in a CTA": [(16, 12)] * 300, "groups": [(128, 128)] * 52,
              "mixed n_grid": [(64, 64), (128, 128), (32, 48)]}[batch]
    n, steps, dt = 60, 8, 2e-5
    rng = np.random.default_rng(4)
    states = []
    for m, (nx, ny) in enumerate(shapes):
        lo, hi = np.array([0.3, 0.3 * ny / nx]), np.array([0.7, 0.5 * ny / nx])
        x = rng.uniform(lo, hi, (n, 2)).astype(np.float32)
        v = np.tile(np.float32([0.0, 3.0 / nx / (steps * dt)]), (n, 1)) if m % 3 == 0 else \
            rng.normal(0, 0.01, (n, 2)).astype(np.float32)
        states.append((x, rng.choice([0, 1, 2, 3], n).astype(np.int32), v))
    e = Engine([InstanceSpec(n, nx, ny, ny / nx) for nx, ny in shapes], axisym=axisym, cluster_size=cluster,
               block_threads=threads)
    for m, (x, mat, v) in enumerate(states):
        e.load(m, x, mat)
        e.write(m, v=v)
    prm = e.get_params()
    e.step(steps)
    got = [e.read(m) for m in range(len(shapes))]
    assert not e.error_flags().any()
    assert (e.spans() is None) == (cluster > 0 or batch == "mixed n_grid")
    assert e.path_counts()["remote_gathers"] > 0
    assert batch != "groups" or e.spans()["launches"] > 1
    e.close()
    for m, (nx, ny) in enumerate(shapes):
        want = []
        for prec, t0 in (("f32", np.float32(0)), ("f64", 0.0)):
            s = O.new_state(states[m][0], states[m][1], np.tile(np.float32([0, 1]), (n, 1)), prec, nx, ny)
            s["v"][:] = states[m][2]
            O.run(O.Instance(nx=nx, ny=ny, domain_h=ny / nx, axisym=axisym, contraction=float(prm["contraction"][m]),
                             freq=float(prm["freq"][m])), s, t0, steps)
            want.append(s)
        tol = 10 * np.abs(want[0]["v"] - want[1]["v"]).max() + steps * 1e-5 * np.abs(want[0]["v"]).max()
        assert np.abs(got[m]["v"] - want[0]["v"]).max() <= tol, m
        assert np.abs(got[m]["x"] - want[0]["x"]).max() <= steps * dt * tol + 4 * np.spacing(np.float32(2.0)), m
