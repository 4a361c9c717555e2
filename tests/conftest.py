import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")
    config.addinivalue_line("markers", "slow: takes more than a few seconds")


def _has_gpu() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


def pytest_collection_modifyitems(config, items):
    if _has_gpu():
        return
    skip = pytest.mark.skip(reason="no CUDA device visible")
    for it in items:
        if "gpu" in it.keywords:
            it.add_marker(skip)


@pytest.fixture(autouse=True)
def _skip_at_a_missing_reference_build(monkeypatch):
    """A test that comes to need the reference's own build (oracle/_ref, made
    from its sources) where there is none is skipped there, not failed."""
    po = sys.modules.get("oracle.pyoracle")
    if po is None:
        return
    ref_lib = po.ref_lib

    def lib(simple=False):
        if not po.ref_available(simple):
            pytest.skip("oracle/_ref not built (needs the reference's sources)")
        return ref_lib(simple)

    monkeypatch.setattr(po, "ref_lib", lib)
