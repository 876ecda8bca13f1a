import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "glu-hcu_b200"))
sys.path.insert(0, ROOT)
GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")
    config.addinivalue_line("markers", "ref: needs the reference built into oracle/_ref")


def _has_gpu():
    try:
        import torch

        return torch.cuda.is_available()
    except Exception:
        return False


HAS_GPU = _has_gpu()


# What needs third-party code that is built only where its sources are: the
# preprocessing library behind pyglu's analysis, the command line tool linked to it.
def _without_preprocessing():
    from pyglu import _capi

    if os.path.exists(_capi.NICSLU_PATH):
        return

    def load_preprocess():
        pytest.skip(f"{os.path.basename(_capi.NICSLU_PATH)} not built (its sources are not here)")

    _capi.load_preprocess = load_preprocess


_without_preprocessing()
LU_CMD = os.path.join(ROOT, "glu-hcu_b200", "bin", "lu_cmd")
NEEDS_FILE = {
    "test_cli.py::test_usage_and_bad_arguments": LU_CMD,
    "test_cli.py::test_lu_cmd_solves_and_writes_x": LU_CMD,
    "test_zz_no_alloc.py::test_noalloc_rejects_dense_tail_beyond_its_array": os.path.join(
        ROOT, "glu-hcu_b200", "lib", "libglu_nicslu.so"),
    "test_cpu_dist.py::test_reference_arm_runs_on_rank_zero_only": os.path.join(ROOT, "oracle", "_ref", "libglu_ref.so"),
}


def pytest_collection_modifyitems(config, items):
    import oracle

    skip_gpu = pytest.mark.skip(reason="no CUDA device")
    skip_ref = pytest.mark.skip(reason="reference not built into oracle/_ref")
    for it in items:
        if "gpu" in it.keywords and not HAS_GPU:
            it.add_marker(skip_gpu)
        if "ref" in it.keywords and not oracle.ref_available():
            it.add_marker(skip_ref)
        path = NEEDS_FILE.get(f"{it.path.name}::{it.name}")
        if path and not os.path.exists(path):
            it.add_marker(pytest.mark.skip(reason=f"{os.path.basename(path)} not built"))
