"""Bounded waits of the batched path's spans (jellyfih_b200/csrc/jf_span.cu) that
run out: with a limit of a few polls the ordinary waits for a neighbour's rows
give up.  The run returns, says so, stays refused until the flags are cleared,
and steps as ever after a clear and a reload."""
import time

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _drifting_tank(seed=31):
    from jellyfih_b200 import tank
    pos, mat, fib, _ = tank.fill_tank(tank.uniform_genomes(1, seed)[0], 80000, jitter=0.25, seed=seed)
    v = np.zeros_like(pos)
    live = mat >= 0
    v[live] = np.random.default_rng(0).normal(0, 10.0, (int(live.sum()), 2)).astype(np.float32)
    return pos, mat, fib, v


def _load(e, tank):
    e.load(0, *tank[:3])
    e.write(0, v=tank[3])
    e.time = 0.0


@pytest.mark.parametrize("threads", [0, 768])
def test_a_wait_that_runs_out_ends_the_run_until_the_flags_are_cleared(threads):
    """The reference after the reload is the plain path, at the bounds that the
    drift test of the golden suite has for the same tank and substeps."""
    from jellyfih_b200 import Engine, InstanceSpec, JfError
    from jellyfih_b200 import _lib as L
    tank = _drifting_tank()
    p = Engine([InstanceSpec(80000)], path="plain")
    _load(p, tank)
    p.step(64)
    want = p.read(0)
    p.close()
    e = Engine([InstanceSpec(80000)], block_threads=threads, resort_interval=16)
    for limit in (1, 3, 10, 40):  # give up at different places of a substep
        _load(e, tank)
        e.set_wait_limit(limit)
        t = time.perf_counter()
        e.step(2000)  # 125 chunks, most of them replayed from a graph
        try:
            e.sync()
        except JfError as err:
            assert err.code == L.JF_ERR_CUDA and "instance 0" in str(err) and "clear" in str(err)
        else:
            assert limit > 1, "no wait of one poll ran out"
            continue
        assert time.perf_counter() - t < 2.0
        assert e.error_flags()[0] & L.JF_ERRFLAG_ABANDONED
        e.set_wait_limit(0)
        x = e.read(0)["x"]
        e.step(64)  # refused: nothing moves
        with pytest.raises(JfError):
            e.sync()
        assert np.array_equal(e.read(0)["x"], x)
        e.clear_error_flags()
        _load(e, tank)
        e.step(64)
        assert e.sync() and not e.error_flags().any()
        got, live = e.read(0), tank[1] >= 0
        assert np.abs(got["x"][live] - want["x"][live]).max() < 1e-4
        assert np.abs(got["v"][live] - want["v"][live]).max() < 1e-2 * np.abs(want["v"][live]).max()
    e.close()


@pytest.mark.parametrize("count,n,nx,ny", [(300, 300, 16, 12), (52, 1500, 128, 128)], ids=["several in a CTA", "groups"])
def test_every_instance_is_finished_or_flagged(count, n, nx, ny):
    """One substep: an instance without the flag has the state of an undisturbed
    run (4 ulp, the bound of one substep elsewhere); one left in the middle, or
    behind the give-up in a later launch, carries the flag.  Four rows of the
    first instance hold 20,000 particles that are scattered one by one, so that
    the neighbouring band waits for them."""
    from jellyfih_b200 import Engine, InstanceSpec, JfError
    from jellyfih_b200 import _lib as L
    h, rng = ny / nx, np.random.default_rng(5)
    xs = [rng.uniform([2 / nx, (ny // 2 - 1.7) / nx], [1 - 2 / nx, (ny // 2 + 2.2) / nx], (20000, 2))]
    xs += [rng.uniform([2 / nx, 2 / nx], [1 - 2 / nx, h - 2 / nx], (n, 2))] * (count - 1)
    states = []
    for limit in (0, 1):
        e = Engine([InstanceSpec(len(x), nx, ny, h) for x in xs], cell_cap=1)
        for m, x in enumerate(xs):
            e.load(m, x, np.zeros(len(x), np.int32))
            e.write(m, v=np.random.default_rng(m).normal(0, 0.3, (len(x), 2)).astype(np.float32))
        e.set_wait_limit(limit)
        e.step(1)
        if limit:
            with pytest.raises(JfError):
                e.sync()
        else:
            assert e.sync()
        states.append(([e.read(m)["x"] for m in range(count)], e.error_flags()))
        e.close()
    (want, none), (got, flags) = states
    assert not none.any() and set(flags) <= {0, L.JF_ERRFLAG_ABANDONED}
    assert flags[0] and (flags[-1] or nx < 128)  # the last group runs behind the give-up
    for m in range(count):
        if not flags[m]:
            assert np.abs(got[m] - want[m]).max() <= 4 * np.spacing(np.float32(h)), m
