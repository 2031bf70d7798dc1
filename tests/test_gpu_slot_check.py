"""A slot permutation that is broken is refused by the reads and writes that go
by it, and nothing outside the instance's arrays is touched.  (The kernels check
the slot before they use it, so that the broken one is never an address.)"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def poke(tmp_path_factory):
    from jellyfih_b200 import build
    lib = str(tmp_path_factory.mktemp("poke") / "engine_poke.so")
    subprocess.run([build.nvcc_path(), *build.ARCH, "-std=c++17", "--shared", "-Xcompiler", "-fPIC", "-I", build.CSRC,
                    "-I", os.path.join(build.REPO, "include"), "-o", lib, os.path.join(HERE, "engine_poke.cu")],
                   check=True, timeout=300)
    fn = ctypes.CDLL(lib).poke_slot
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int32, ctypes.c_void_p]

    def set_slot(e, m, k, slot):
        old = ctypes.c_int32()
        assert fn(e._h, m, k, slot, ctypes.byref(old)) == 0
        return old.value
    return set_slot


@pytest.mark.parametrize("path", ["batched", "plain"])
@pytest.mark.parametrize("slot", [-1, 300, 2 ** 31 - 1])
def test_a_broken_permutation_is_refused(path, slot, poke):
    from jellyfih_b200 import Engine, InstanceSpec, JfError
    rng = np.random.default_rng(2)
    n = 300
    e = Engine([InstanceSpec(n, 32, 32), InstanceSpec(n, 32, 32)], path=path)
    x = rng.uniform(0.2, 0.8, (n, 2)).astype(np.float32)
    for m in range(2):
        e.load(m, x, rng.choice([0, 2], n).astype(np.int32))
    e.grad_forward(1, 1)
    e.grad_backward()
    want, gx = [e.read(m) for m in range(2)], e.grad_positions(0)
    old = poke(e, 0, 257, slot)
    for call in (lambda: e.read(0), lambda: e.write(0, v=x), lambda: e.grad_positions(0)):
        with pytest.raises(JfError, match="slot permutation"):
            call()
    got = e.read(1)
    assert all(np.array_equal(got[k], want[1][k]) for k in want[1])
    poke(e, 0, 257, old)
    e.write(0, v=want[0]["v"])
    got = e.read(0)
    assert all(np.array_equal(got[k], want[0][k]) for k in want[0])
    assert np.array_equal(e.grad_positions(0), gx)
    e.close()
