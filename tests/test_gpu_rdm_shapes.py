"""The density-matrix kernels of rdm.cu at the edges of their splits: warps of 32
spectators, chunks of alpha singles and lists of beta singles by orbital pair, spins
without singles, more than 32 orbitals, rows (and beta singles) of more than a CTA's
shared memory, and vectors whose products fixed point cannot hold.

Tolerance: a spectator's product is rounded at 2^-58 of the largest of its 32 and
every sum is of FP64 terms, so an element is off by a few 1e-16 of the sum of its
terms' magnitudes, which the trace bounds; 1e-12 as for the other RDM tests.
"""
import numpy as np
import pytest

from oracle.oracle import Oracle
from sbd_gb300.engine import TPBProblem
from sbd_gb300.generators import make_problem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _close(x, ref):
    return np.abs(x - ref).max() <= 1e-12 * np.abs(ref).max()


# one string of a spin, 31 to 33 spectators, full spaces, more than 32 orbitals; then a
# row in shared memory but not the beta singles, and neither
SHAPES = [(12, 1, 1, 4), (12, 97, 1, 4), (12, 1, 70, 4), (10, 28, 31, 2), (10, 32, 33, 5), (12, 33, 65, 4),
          (40, 150, 61, 13), (20, 3, 9001, 8), (20, 2, 14700, 8)]


@pytest.mark.parametrize("norb,na,nb,nocc", SHAPES)
def test_rdms_against_oracle(engine, norb, na, nb, nocc):
    prob = make_problem(norb, nocc, nocc, na, nb, seed=na + nb)
    p = TPBProblem.from_problem(engine, prob)
    p.build_tables()
    W = np.random.default_rng(nb).uniform(-1, 1, prob.ndet) / np.sqrt(prob.ndet)
    one, two = p.rdm(W)
    ro, rt = Oracle.from_problem(prob).correlation(W)
    assert _close(one, ro) and _close(two, rt)
    only, none = p.rdm(W, two_body=False)
    assert none is None and _close(only, ro)
    # products above the exponents of fixed point: FP64 additions, the same sums
    big, big2 = p.rdm(np.ldexp(W, 450))
    assert _close(np.ldexp(big, -900), ro) and _close(np.ldexp(big2, -900), rt)
    W[prob.ndet // 2] = np.nan
    assert np.isnan(p.rdm(W)[0]).any()
    p.close()
