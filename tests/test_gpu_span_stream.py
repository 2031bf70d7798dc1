"""A stream that may use only some of the SMs (of a green context): the batched
path's spans, which need an SM for each CTA, are laid out for those."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
driver = pytest.importorskip("cuda.bindings.driver")
pytestmark = pytest.mark.gpu


def _ok(result):
    err, *rest = result
    if err != driver.CUresult.CUDA_SUCCESS:
        pytest.skip(f"no green context here: {err}")
    return rest[0] if len(rest) == 1 else rest


@pytest.mark.parametrize("count,sms", [(1, 16), (3, 16), (3, 64)])
def test_spans_follow_a_stream_with_fewer_sms(count, sms):
    from jellyfih_b200 import Engine, InstanceSpec, tank
    tanks = [tank.fill_tank(g, 80000)[:3] for g in tank.gaussian_genomes(count, 3)]
    e = Engine([InstanceSpec(80000)] * count)
    full = e.spans()["ctas"]

    def rows(steps=130):  # graph replays among them
        for m, t in enumerate(tanks):
            e.load(m, *t)
        return e.run_headless(steps)
    want = rows()
    res = _ok(driver.cuDeviceGetDevResource(0, driver.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    parts, _, _ = _ok(driver.cuDevSmResourceSplitByCount(1, res, 0, sms))
    desc = _ok(driver.cuDevResourceGenerateDesc(parts, 1))
    green = _ok(driver.cuGreenCtxCreate(desc, 0, driver.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = _ok(driver.cuGreenCtxStreamCreate(green, driver.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    e.set_wait_limit(1000000)  # a second or so
    e.set_stream(int(stream))
    has = parts[0].sm.smCount
    ctas = e.spans()["ctas"] if e.spans() else 0
    assert ctas <= has and (ctas > 0 or has < full)
    few = rows()
    e.set_stream(0)
    assert e.spans()["ctas"] == full
    again = rows()
    assert not e.error_flags().any()
    e.close()
    driver.cuStreamDestroy(stream)
    driver.cuGreenCtxDestroy(green)
    # the bound that a chunk has against the clusters in test_gpu_span.py
    assert np.abs(few - want).max() <= 1e-6 and np.abs(again - want).max() <= 1e-6


def test_engines_side_by_side_on_threads_and_streams():
    """Three engines, whose launches each take every SM, from three threads at
    once: a cooperative launch is placed whole, so that no wait runs out, and the
    rows are those of a run alone (the bound of a chunk, as above)."""
    import threading

    from jellyfih_b200 import Engine, InstanceSpec, tank
    tanks = [tank.fill_tank(g, 80000)[:3] for g in tank.gaussian_genomes(8, 5)]
    engines = [Engine([InstanceSpec(80000)] * 8) for _ in range(3)]
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1, 0)]
    got = [[] for _ in engines]

    def run(k, times):
        for _ in range(times):
            for m, t in enumerate(tanks):
                engines[k].load(m, *t)
            got[k].append(engines[k].run_headless(192))
    for e, s in zip(engines, streams):
        e.set_stream(s)
        e.set_wait_limit(3000000)  # some two seconds
    run(0, 1)
    want = got[0].pop()
    threads = [threading.Thread(target=run, args=(k, 6)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for e, rows in zip(engines, got):
        assert len(rows) == 6 and not e.error_flags().any()
        assert max(np.abs(r - want).max() for r in rows) <= 1e-6
        e.close()
