"""The work counts of the tensor-core sweeps as they run (CPU): products of more than 32 modes in modular arithmetic at every
setting, leaves and the products among them in digits."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


@pytest.mark.parametrize("levels, M, fp64, fp16", [
    ("0", 256, 4 * 256 ** 3, 48 * 256 ** 3),
    ("1", 256, 2 * 4 * 128 ** 3, 48 * 256 ** 3 + 4 * 48 * 128 ** 3),
    ("2", 512, 4 * 4 * 128 ** 3, 48 * 512 ** 3 + 4 * 48 * 256 ** 3 + 8 * 48 * 128 ** 3),
])
def test_fewer_levels_run_modular_products(monkeypatch, levels, M, fp64, fp16):
    monkeypatch.setenv("RG_SPLIT_INVERSE", levels)
    monkeypatch.delenv("RG_TENSOR_R", raising=False)
    assert bench.executed_flops(M, 2, "blocked_symmetric", bench.MODULAR_PRODUCT) == (2.0 * fp64, 2.0 * fp16)


@pytest.mark.parametrize("M, fp16", [
    # 65 -> two blocks of 32.5 -> four of 16.25: the products of a half of 32.5 are modular, those of 16.25 in digits
    (65, 48 * 65 ** 3 + 4 * 48 * 32.5 ** 3 + 8 * 208 * 16.25 ** 3 + 4 * 296 * 16.25 ** 3),
    (100, 48 * 100 ** 3 + 4 * 48 * 50 ** 3 + 8 * 208 * 25 ** 3 + 4 * 296 * 25 ** 3),
    (256, 48 * 256 ** 3 + 4 * 48 * 128 ** 3 + 8 * 48 * 64 ** 3 + 16 * 208 * 32 ** 3 + 8 * 296 * 32 ** 3),
    (512, 48 * 512 ** 3 + 4 * 48 * 256 ** 3 + 8 * 48 * 128 ** 3 + 16 * 48 * 64 ** 3 + 32 * 208 * 32 ** 3 + 16 * 296 * 32 ** 3),
])
def test_default_levels(monkeypatch, M, fp16):
    monkeypatch.delenv("RG_SPLIT_INVERSE", raising=False)
    monkeypatch.delenv("RG_TENSOR_R", raising=False)
    assert bench.executed_flops(M, 1, "blocked_symmetric", bench.MODULAR_PRODUCT) == (0.0, pytest.approx(fp16, rel=1e-12))


def test_shared_memory_sweep_and_eigenvalues():
    assert bench.executed_flops(64, 5, "symmetric") == (0.0, 5 * (26 + 37) * 8.0 * 64 ** 3)
    assert bench.flops_eigenvalues(30) == pytest.approx(16 * sum(2.0 * k ** 2 for k in range(1, 31)), rel=0.06)
