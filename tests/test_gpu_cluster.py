"""The cluster layout of the batched path (jf_batched.cu: chunk_kernel), asked for
with a cluster size: the reference-recorded substeps with every cell cap, at the
bounds of test_gpu_parity.py.  (test_gpu_span_drift.py has its far rows.)"""
import pytest

import golden_io as G

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["batched_regs", "batched_tmem"])
@pytest.mark.parametrize("cluster", [4, 8])
@pytest.mark.parametrize("cap", [0, 1, 2, 16])
@pytest.mark.parametrize("case", G.STEP_CASES)
def test_clusters_match_reference_goldens(case, cap, cluster, layout):
    from test_gpu_parity import _check_goldens
    _check_goldens(case, layout, cell_cap=cap, cluster_size=cluster)
