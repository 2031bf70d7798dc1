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
