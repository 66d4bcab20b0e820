import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
for p in (str(ROOT), str(ROOT / "tests")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on a B200)")


def pytest_collection_modifyitems(config, items):
    import torch
    if torch.cuda.is_available():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


@pytest.fixture
def plain_kernels(monkeypatch):
    """The engine's kernels replaced by their plain PyTorch statements (CPU)."""
    import plain_ops
    plain_ops.install(monkeypatch)
    return plain_ops


@pytest.fixture(params=["tcgen05", "mma.sync"])
def prefill_form(request):
    """Steps that either of two prefill kernels can serve all go to the one or the other: both are compared at every size."""
    from llm_b200.ops import tactics
    names = {"tcgen05": ("attention_prefill_window_mma", "diff_attention_mma", "sigmoid_attention_mma"),
             "mma.sync": ("attention_prefill_window_tc", "diff_attention_tc", "sigmoid_attention_tc")}[request.param]
    for name in names:
        tactics.disable(name)
    yield request.param
    for name in names:
        tactics.enable(name)
