"""The differentiable forward's block sums (jf_grad.cu: Tile) at the ends of what
they hold: particles outside the lower walls, whose weights exceed 1, with
momenta about 1, and positions that are not finite."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("speed", [20.0, 120.0, 240.0, 900.0])
def test_block_sums_match_the_oracle_outside_the_lower_walls(speed):
    """Bit for bit the oracle's fixed-point sums: a particle of the 8x8 grid weighs
    1/256, so that these speeds give contributions of 0.1 to 8."""
    from jellyfih_b200 import Engine, InstanceSpec
    from oracle import oracle as O
    rng = np.random.default_rng(int(speed))
    n, dx = 300, 1.0 / 8
    x = rng.uniform(-0.45 * dx, 1.4 * dx, (n, 2)).astype(np.float32)
    x[100:] = rng.uniform(2 * dx, 6 * dx, (n - 100, 2)).astype(np.float32)
    mat = rng.choice([0, 1, 3], n).astype(np.int32)
    fib = np.tile(np.float32([0.6, 0.8]), (n, 1))
    v = rng.uniform(-speed, speed, (n, 2)).astype(np.float32)
    e = Engine([InstanceSpec(n, 8, 8)], path="plain")
    e.load(0, x, mat, fib)
    e.write(0, v=v)
    e.time = 0.0
    e.grad_forward(1, 1)
    got = e.read(0)
    assert not e.error_flags().any()
    c, f = float(e.get_params()["contraction"][0]), float(e.get_params()["freq"][0])
    e.close()
    s = O.new_state(x, mat, fib, "f32", 8, 8)
    s["v"][:] = v
    O.run(O.Instance(nx=8, ny=8, contraction=c, freq=f, fixed_p2g=True), s, np.float32(0), 1)
    for k in ("x", "v", "C", "F"):
        assert np.array_equal(got[k], s[k]), k


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_position_that_is_not_finite_is_flagged_and_moves_nothing_else(bad, fp64):
    """The other particles end where they do with the particle left out.  A NaN
    has the stencil of node 0 in FP32, and is flagged; in FP64, as an infinity in
    both, it has none."""
    from jellyfih_b200 import Engine, InstanceSpec
    rng = np.random.default_rng(3)
    n = 200
    x = rng.uniform(0.02, 0.3, (n, 2)).astype(np.float32)
    states = []
    for left_out in (False, True):
        p, mat = x.copy(), np.zeros(n, np.int32)
        if left_out:
            mat[7] = -1
        else:
            p[7] = bad
        e = Engine([InstanceSpec(n, 16, 16)], path="plain", grad_fp64=fp64)
        e.load(0, p, mat)
        e.grad_forward(1, 1)
        states.append((e.read(0), int(e.error_flags()[0])))
        e.close()
    (got, flags), (want, none) = states
    assert none == 0 and (flags != 0) == (np.isnan(bad) and not fp64)
    rest = np.arange(n) != 7
    tol = 1e-12 if fp64 else 0.0  # FP64 sums depend on their order
    for k in ("x", "v", "C", "F"):
        assert np.abs(got[k][rest].astype(np.float64) - want[k][rest]).max() <= tol * max(1.0, np.abs(want[k]).max()), k
