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
from sbd_gb300.engine import Engine
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


@pytest.mark.parametrize("decades", [0, 6, 12])
@pytest.mark.parametrize("norb,na,nb,nocc", [(12, 97, 150, 4), (40, 90, 61, 13)])
def test_elements_of_wide_vectors(engine, norb, na, nb, nocc, decades):
    """The sums of the same-spin singles over the spectators that have an orbital q,
    which are the whole of two[s, 1 - s][a, q, i, q]: each to the bound of its own k
    terms (2^-53 each in the products and in the sum, here and in the reference),
    with weights over that many decades on the strings of each spin."""
    prob = make_problem(norb, nocc, nocc, na, nb, seed=na + nb)
    o = Oracle.from_problem(prob)
    rng = np.random.default_rng(decades)
    W = (rng.normal(size=(na, nb)) * 10.0 ** rng.uniform(-decades, 0, (na, 1))
         * 10.0 ** rng.uniform(-decades, 0, (1, nb)))
    p = TPBProblem.from_problem(engine, prob)
    p.build_tables()
    one, two = p.rdm(W.ravel())
    ro, rt = o.correlation(W.ravel())
    L = norb
    one, ro = (np.asarray(x).reshape(2, L, L) for x in (one, ro))  # [s][a][i]
    two, rt = (np.asarray(x).reshape(4, L, L, L, L) for x in (two, rt))  # [s1 + 2 s2][d][c][b][a]
    bits = np.arange(L, dtype=np.uint64)
    for s, t, x, other in ((0, o.ta, np.abs(W), prob.bstr), (1, o.tb, np.abs(W).T, prob.astr)):
        occ = ((other.astype(np.uint64)[:, None] >> bits) & np.uint64(1)).astype(float)
        n = int(t.off_s[-1])
        bra = np.repeat(np.arange(len(x)), np.diff(t.off_s[:len(x) + 1].astype(np.int64)))
        ket, move = t.ket_s[:n].astype(np.int64), np.asarray(t.cran_s[:2 * n]).reshape(-1, 2) // 2
        size, count = np.zeros((L, L, L)), np.zeros((L, L))  # [i][a][q], [i][a]
        for b, k, (i, a) in zip(bra, ket, move):
            size[i, a] += (x[b] * x[k]) @ occ
            count[i, a] += len(occ)
        i, a, q = np.nonzero(size)
        for blk, got in ((s + 2 * (1 - s), lambda y: y[q, i, q, a]), ((1 - s) + 2 * s, lambda y: y[i, q, a, q])):
            err = np.abs(got(two[blk]) - got(rt[blk]))
            assert (err <= 4 * (count[i, a] + 4) * 2.0 ** -53 * size[i, a, q]).all()
        i, a = np.nonzero(count)
        total = np.zeros((L, L))
        for b, k, (ii, aa) in zip(bra, ket, move):
            total[ii, aa] += x[b] @ x[k]
        assert (np.abs(one[s, a, i] - ro[s, a, i]) <= 4 * (count[i, a] + 4) * 2.0 ** -53 * total[i, a]).all()
    p.close()


def test_density_matrices_within_a_budget():
    """The sorted singles, which the earlier kernels did without, take no room of a
    budget that has none left."""
    prob = make_problem(16, 5, 5, 1500, 30, seed=7)
    W = np.random.default_rng(0).normal(size=prob.ndet)
    e = Engine(0)
    p = TPBProblem.from_problem(e, prob)
    p.build_tables()
    one, two = p.rdm(W)
    used = e.bytes_in_use
    singles = sum(p.table_counts(s)[0] for s in (0, 1))
    p.close()
    e.close()
    e = Engine(0, hbm_budget=used - 4 * singles)
    p = TPBProblem.from_problem(e, prob)
    p.build_tables()
    for _ in range(2):
        a, b = p.rdm(W)
        assert _close(a, one) and _close(b, two)
    assert e.bytes_in_use <= used - 4 * singles
    p.close()
    e.close()
