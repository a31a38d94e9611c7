"""Shared fixtures. GPU tests carry @pytest.mark.gpu; everything else runs on CPU."""
from __future__ import annotations

import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))

GOLDEN = Path(__file__).resolve().parent / "golden"


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")


def pytest_collection_modifyitems(items):
    """The drop-in program is built against Remora's headers. Where they are missing its test fails; it
    comes last then, so that a run that stops at the first failure has done all the others."""
    if not (ROOT / "tests" / "cpp" / "_build" / "dropin_test").exists():
        items.sort(key=lambda item: item.name == "test_dropin_program")


@pytest.fixture(scope="session")
def orc():
    import oracle
    return oracle.Oracle()


@pytest.fixture(scope="session")
def golden():
    def load(name: str):
        return np.load(GOLDEN / f"{name}.npz")
    return load


@pytest.fixture(scope="session")
def cuda():
    """The CUDA device and the loaded product library (fails loudly if either is missing)."""
    import torch
    if not torch.cuda.is_available():
        pytest.fail("GPU test run without a CUDA device")
    import remora_b200
    remora_b200.lib()
    return torch.device("cuda:0")
