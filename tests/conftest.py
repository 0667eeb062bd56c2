"""Shared pytest configuration.

Tests marked ``gpu`` call the CUDA library through its C ABI and need a B200;
everything else runs on the CPU (oracle pins, host logic, ABI exports).
"""

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
    config.addinivalue_line("markers", "gpu: needs a CUDA device (sm_100a)")
    config.addinivalue_line("markers", "slow: long-running")


# Holds an FP64 oracle to 1e-9 of the effective degrees of freedom. The device's B_n are
# float32 as the reference's: at the stamps that the reference selects that moves them
# by less, at the fixed ones used without it by 1.6e-8 (49.801186822 in FP64 rows,
# 49.801187657 in float32 rows, 49.801187648 on the device).
NEEDS_REFERENCE_STAMPS = "test_stamp_gcv_matches_fp64_oracle_and_central_differences"


def pytest_collection_modifyitems(items):
    """Without the oracle built from the reference that test misses its bound: it runs
    last, so that a run that stops at the first failure has run all the others."""
    from oracle import refbuild

    if not refbuild.available():
        items.sort(key=lambda item: item.name == NEEDS_REFERENCE_STAMPS)


@pytest.fixture
def rng():
    return np.random.default_rng(12345)


def load_golden(name: str) -> dict:
    with np.load(GOLDEN / f"{name}.npz", allow_pickle=False) as z:
        return {k: z[k] for k in z.files}
