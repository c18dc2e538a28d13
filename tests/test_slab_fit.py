"""Which forms' kernels of sigma_slab.cu a problem's sizes leave room for: the FP32
ones take at least 16 bytes of shared memory a row of a sweep and always keep the
alpha x beta sums, the 8-byte ones can do with 8 and without."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIMIT = 232448 - 1024  # opt-in shared memory of a CTA less the kernels' static part


@pytest.fixture(scope="module")
def fits(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fit") / "slab_fit")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "sbd_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "slab_fit.cpp"), "-o", exe], check=True)

    def ask(norb, na, nb, sa, sb):
        """(8-byte forms, FP32) for sa and sb singles a string."""
        r = subprocess.run([exe] + [str(x) for x in (norb, na, nb, int(sa * na), int(sb * nb), LIMIT)],
                           capture_output=True, text=True, check=True)
        return tuple(int(x) for x in r.stdout.split())

    return ask


def test_sizes(fits):
    assert fits(36, 6000, 6000, 4, 4) == (1, 1)
    assert fits(40, 12000, 12000, 2, 2) == (1, 0)  # FP32 alpha x beta: 266,288 bytes
    assert fits(24, 20000, 4000, 20, 12) == (1, 0)  # FP32 alpha sweep: 324,832 bytes
    assert fits(36, 16000, 2000, 8, 4) == (1, 0)
    assert fits(32, 2000, 16000, 0, 8) == (1, 0)  # the beta sweep
    assert fits(24, 30000, 100, 20, 2) == (0, 0)


def test_last_size_that_fits(fits):
    n = LIMIT // 16  # rows of a sweep without singles, and the zero row
    assert fits(20, n - 1, 50, 0, 0) == (1, 1) and fits(20, n, 50, 0, 0) == (1, 0)
    assert fits(20, 50, n - 1, 0, 0) == (1, 1) and fits(20, 50, n, 0, 0) == (1, 0)
    assert fits(20, n - 212, 50, 1, 0) == (1, 1) and fits(20, n - 211, 50, 1, 0) == (1, 0)  # 211 Coulomb rows
    m = (LIMIT - 16 * (1 + 2 * 211)) // 20
    assert fits(20, 50, m, 1, 1) == (1, 1) and fits(20, 50, m + 1, 1, 1) == (1, 0)
