"""The roofline block of the benchmark names what bounds the kernels that ran."""
import pytest

import bench


@pytest.fixture
def rates(monkeypatch):
    monkeypatch.setattr(bench, "measure_fp64_rates", lambda d: {"dfma_tflops": 1.25, "dmma_tflops": 1.2})
    monkeypatch.setattr(bench, "measure_imad_rate", lambda d: 9.0)


def test_fixed_point_kernels(rates):
    N, nnz = 36_000_000, 2_800_000_000
    r = bench.sigma_roofline({"beta_shape": "slab"}, 3.6, N, nnz, 24 * N + 8 * nnz, 6682.5, "measured", None, 0)
    assert r["bound"] == "integer multiply-adds" and abs(r["achieved"] - 3 * nnz / 3.6e-3 / 1e12) < 1e-9
    assert r["frac"] == r["achieved"] / 9.0 and r["hbm"]["bytes"] == 24 * N
    assert "frac" not in r["read_per_nonzero"]


def test_fp64_kernels(rates):
    N, nnz = 144_000_000, 72_000_000
    r = bench.sigma_roofline({"beta_shape": "stream"}, 1.2, N, nnz, 24 * N + 8 * nnz, 6682.5, "measured", 1.0, 0)
    assert r["bound"] == "hbm" and r["algorithmic_bytes"] == 24 * N + 8 * nnz and r["traffic"] == 1.0


@pytest.mark.gpu
def test_measured_integer_rate():
    """Between a half and one and a quarter of 32 a clock and SM (152 SMs at 2.07 GHz)."""
    assert 5.0 < bench.measure_imad_rate(0) < 12.6
