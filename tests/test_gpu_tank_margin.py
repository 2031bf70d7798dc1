"""The water exclusion's boxes (robot_margin_kernel): margins below and far above
the lattice spacing, lattices of other spacings, and robot particles at the
walls and outside the lattice, against tank.fill_tank bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("margin", [0.0011, 0.005, 0.08])
@pytest.mark.parametrize("div", [1.3, 2.0, 3.7])
def test_margins_and_spacings_match_the_host_fill(margin, div, monkeypatch):
    from jellyfih_b200 import Engine, InstanceSpec, tank
    rng = np.random.default_rng(int(margin * 1e4) + int(10 * div))
    robot = np.concatenate([rng.uniform(0.3, 0.7, (150, 2)), rng.uniform(-0.1, 1.1, (60, 2)),
                            [[0.0, 0.5], [1.0, 0.5], [0.5, 0.0], [1.0, 1.0]]])
    mat = np.ones(len(robot), np.int32)
    fib = np.tile(np.float32([0.0, 1.0]), (len(robot), 1))
    monkeypatch.setattr(tank, "generate_phenotype", lambda *a, **k: (robot, mat, fib, False))
    slots = 20000
    pos, m, f, st = tank.fill_tank(np.zeros(11), slots, grid_res=32, water_margin=margin, spacing_div=div)
    e = Engine([InstanceSpec(slots, 32, 32)])
    counts = e.load_robot(0, robot, mat, fib, water_margin=margin, spacing_div=div)
    got = e.read(0)
    e.close()
    assert counts == (st["n_robot"], st["n_water"])
    assert np.array_equal(got["x"], pos) and np.array_equal(got["material"], m) and np.array_equal(got["fiber"], f)
