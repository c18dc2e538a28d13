"""The small symmetric eigenproblem of the Rayleigh-Ritz steps (rr_dev.cuh), in the
blocks of both solvers: every size around those of its padding, its FP32 sweeps and
its thread counts, and spectra that are clustered, spread over many orders of
magnitude, degenerate, or far from 1.

Tolerance: the rotations end at off-diagonal elements of 1e-15 of the norm, and each
of some ten sweeps of n rotations an index rounds every column a few times: 16 n
2^-53 of the norm for the residual, 16 n 2^-53 for the orthonormality.
"""
import os
import subprocess

import numpy as np
import pytest

from sbd_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rr") / "rr_jacobi")
    subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, os.path.join(ROOT, "tests", "cpp", "rr_jacobi.cu"),
                    "-o", out, "-lcudart"], check=True)
    return out


def _matrices(n, rng):
    q = np.linalg.qr(rng.normal(size=(n, n)))[0]

    def of(w):
        a = (q * np.asarray(w)) @ q.T
        return 0.5 * (a + a.T)

    a = rng.normal(size=(n, n))
    tall = -45.0 + 1e-3 * (a + a.T)  # a subspace's: one shift, small differences
    yield a + a.T
    yield of(np.where(np.arange(n) % 3 == 0, 1.0, 1.0 + 1e-10 * np.arange(n)))  # clustered
    yield of(10.0 ** -np.linspace(0, 14, n))
    yield of(np.where(np.arange(n) < n // 2, 1.0, -1.0))  # two degenerate levels
    yield np.where(np.eye(n) > 0, np.diag(np.linspace(-3, 9, n)), 1e-9 * tall)
    yield tall
    yield np.diag(rng.normal(size=n))
    yield np.zeros((n, n))
    yield 1e200 * (a + a.T)
    yield 1e-200 * (a + a.T)


@pytest.mark.parametrize("nmax,sizes", [(32, (1, 2, 5, 6, 7, 16, 23, 24, 31, 32)),
                                        (64, (1, 2, 3, 6, 31, 32, 33, 45, 48, 49, 63, 64))])
def test_eigenpairs(exe, tmp_path, nmax, sizes):
    rng = np.random.default_rng(nmax)
    mats = [a for n in sizes for a in _matrices(n, rng)]
    with open(tmp_path / "in", "wb") as f:
        np.array([float(len(mats))]).tofile(f)
        for a in mats:
            np.array([float(len(a))]).tofile(f)
            np.ascontiguousarray(a.T).tofile(f)
    subprocess.run([exe, str(tmp_path / "in"), str(tmp_path / "out"), str(nmax)], check=True)
    out, at = np.fromfile(tmp_path / "out"), 0
    for a in mats:
        n = len(a)
        w, v = out[at:at + n], out[at + n:at + n + n * n].reshape(n, n).T
        at += n + n * n
        scale = np.abs(a).max() or 1.0  # (1e200: its squares overflow)
        b, u = a / scale, w / scale
        bound = 16 * n * 2.0 ** -53
        assert np.abs(v.T @ v - np.eye(n)).max() <= bound
        assert np.linalg.norm(b @ v - v * u) <= bound * max(np.linalg.norm(b), 1e-300)
        assert np.abs(np.sort(u) - np.linalg.eigvalsh(b)).max() <= bound * max(np.linalg.norm(b), 1e-300)
    assert at == out.size
