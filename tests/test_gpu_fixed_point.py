"""The sigma kernels of sigma_slab.cu, which the engine takes by itself according to
the number of nonzeros and strings (sigma.cu:slab_pays): edges of their
slices of 32 rows, groups of 1, 2 and 4 columns and batches of ket rows, and the
vectors that fixed point cannot hold.

Tolerance: an element's error is at most 2^-55 times the number of its terms
times the largest |v| and |x| of its sums (below 2^-46 of the largest sigma for
the shapes here), plus a few FP64 roundings; 1e-13 of the largest sigma bounds
both.  Double-float results hold 48 bits (1e-12); FP32 sums of up to a few hundred
terms are held to the 5e-6 of the other FP32 kernels' tests.
"""
import numpy as np
import pytest

from golden_io import max_rel
from oracle.oracle import Oracle
from sbd_gb300.engine import TPBProblem
from sbd_gb300.engine import MIXED, Engine
from sbd_gb300.generators import make_problem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SLAB = "slab"


def _sigma(p, c, base=None):
    s = torch.full_like(c, float("nan")) if base is None else base.clone()
    p.sigma_device(c.data_ptr(), s.data_ptr(), accumulate=base is not None,
                   stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return s


def _problem(engine, *args, **kw):
    prob = make_problem(*args, **kw)
    p = TPBProblem.from_problem(engine, prob)
    p.diag_terms()
    return prob, p


# (norb, na, nb, occupied): one slice and one column group, a slice's edges, odd
# lengths on either side, two and four columns a group, one and both spins with
# few electrons; the last has under 8 alpha x beta pairs a determinant (FP64
# multiply-adds there), the one before it more than a batch of ket rows holds
SHAPES = [(12, 300, 1, 4), (8, 28, 28, 2), (10, 33, 32, 5), (12, 32, 97, 4), (12, 495, 70, 4), (12, 100, 495, 4),
          (16, 801, 799, 5), (16, 1500, 1237, 5), (24, 700, 733, 8), (36, 1401, 1333, 12)]


@pytest.mark.parametrize("norb,na,nb,nocc", SHAPES)
def test_products_against_oracle(engine, norb, na, nb, nocc):
    prob, p = _problem(engine, norb, nocc, nocc, na, nb, seed=na + nb)
    rng = np.random.default_rng(na)
    # a weight for each string over six orders of magnitude, as in a solution
    C = rng.normal(size=(na, nb)) * 10.0 ** rng.uniform(-3, 0, (na, 1)) * 10.0 ** rng.uniform(-3, 0, (1, nb))
    ref = Oracle.from_problem(prob).mult(C.ravel())
    c = torch.tensor(C.ravel(), device="cuda")
    s = _sigma(p, c)
    assert p.tuning(0)["beta_shape"] == SLAB
    assert max_rel(s.cpu().numpy(), ref) <= 1e-13
    assert torch.equal(_sigma(p, c), s)  # the same bits every time
    base = torch.tensor(rng.uniform(-1, 1, C.size), device="cuda")
    assert max_rel((_sigma(p, c, base) - base).cpu().numpy(), ref) <= 1e-13 * (1 + 1 / np.abs(ref).max())
    # double-float (48 bits in, 48 out) and FP32, one vector and blocks
    st = torch.cuda.current_stream().cuda_stream
    hi = c.float()
    x = torch.stack([hi, (c - hi.double()).float()], dim=-1).contiguous()
    y = torch.full_like(x, float("nan"))
    p.sigma_df_device(x.data_ptr(), y.data_ptr(), stream=st)
    torch.cuda.synchronize()
    assert p.tuning(2)["beta_shape"] == SLAB
    assert max_rel(y.double().sum(-1).cpu().numpy(), ref) <= 1e-12
    y = torch.stack([base.float(), (base - base.float().double()).float()], dim=-1).contiguous()
    p.sigma_df_device(x.data_ptr(), y.data_ptr(), accumulate=True, stream=st)
    torch.cuda.synchronize()
    assert max_rel((y.double().sum(-1) - base).cpu().numpy(), ref) <= 1e-12 * (1 + 1 / np.abs(ref).max())
    f = torch.stack([hi, -2 * hi, hi.flip(0), hi + 1]).contiguous()
    one = torch.full_like(f, float("nan"))
    for j in range(4):
        p.sigma_mixed_device(f[j].data_ptr(), one[j].data_ptr(), stream=st)
    torch.cuda.synchronize()
    assert p.tuning(1)["beta_shape"] == SLAB
    assert max_rel(one[0].double().cpu().numpy(), ref) <= 5e-6
    for nvec in (2, 3, 4):
        many = torch.full_like(f, float("nan"))
        p.sigma_mixed_block_device(f.data_ptr(), many.data_ptr(), nvec, stream=st)
        torch.cuda.synchronize()
        assert torch.equal(many[:nvec], one[:nvec])
    p.close()


@pytest.mark.parametrize("norb,na,nb,nocc", [(8, 28, 28, 2), (16, 801, 799, 5), (36, 1401, 1333, 12)])
def test_vectors_out_of_range(engine, norb, na, nb, nocc):
    """Infinities and NaN reach the same elements as in the FP64 kernels, and the
    others are as without them; zero, tiny and huge vectors keep their scale."""
    prob, p = _problem(engine, norb, nocc, nocc, na, nb, seed=5)
    q = TPBProblem.from_problem(engine, prob)
    q.diag_terms()
    q.set_tuning(0, 1, 1)  # the FP64 sweeps
    rng = np.random.default_rng(1)
    x = torch.tensor(rng.uniform(-1, 1, prob.ndet), device="cuda")
    _sigma(p, x)
    assert p.tuning(0)["beta_shape"] == SLAB
    for where in ([0], [prob.ndet // 2, 7], [prob.ndet - 1]):
        for v in (float("nan"), float("inf"), -float("inf"), 1e305):
            y = x.clone()
            y[where] = v
            s, r = _sigma(p, y), _sigma(q, y)
            assert torch.equal(torch.isnan(s), torch.isnan(r)) and torch.equal(torch.isinf(s), torch.isinf(r))
            ok = torch.isfinite(r)
            assert torch.equal(s[~ok & ~torch.isnan(r)], r[~ok & ~torch.isnan(r)])
            for part in (ok, ok & (r.abs() < 1e10)):
                assert max_rel(s[part].cpu().numpy(), r[part].cpu().numpy()) <= 1e-13
    assert not _sigma(p, torch.zeros_like(x)).any()
    for scale in (1e-300, 1e-200, 1e200):
        assert max_rel((_sigma(p, x * scale) / scale).cpu().numpy(), _sigma(q, x).cpu().numpy()) <= 1e-13
    y = x.clone()  # a row and a column far from the others
    y.reshape(na, nb)[na // 3] *= 1e-290
    y.reshape(na, nb)[:, nb // 3] = 0.0
    assert max_rel(_sigma(p, y).cpu().numpy(), _sigma(q, y).cpu().numpy()) <= 1e-13
    p.close()
    q.close()


def test_solver_products_and_fp64_sweeps_agree(engine):
    """The block-ordering product (the solvers') through a solve: energies as from
    the FP64 sweeps."""
    prob, p = _problem(engine, 16, 5, 5, 300, 280, seed=11)
    q = TPBProblem.from_problem(engine, prob)
    q.set_tuning(3, 1, 1)
    kw = dict(nroots=2, max_nb=16, eps=1e-9, max_it=40, init=1, want_vectors=False)
    a, b = p.davidson(**kw), q.davidson(**kw)
    assert p.tuning(3)["beta_shape"] == SLAB and q.tuning(3)["beta_shape"] != SLAB
    assert a.report["converged"] and np.abs(a.energies - b.energies).max() <= 1e-10
    p.close()
    q.close()


def test_unit_vector_starts_keep_the_fp64_sweeps(engine):
    """A stopped FP64 solve from init 0 goes by the FP64 sweeps (davidson.cu,
    Solver::ordered), with the same bits before and after a solve that does not."""
    prob, p = _problem(engine, 16, 5, 5, 300, 280, seed=11)
    kw = dict(nroots=2, max_nb=16, eps=1e-9)
    a = p.davidson(max_it=1, init=0, **kw)
    assert p.tuning(3)["beta_shape"] is None
    b = p.davidson(max_it=40, init=1, **kw)
    assert p.tuning(3)["beta_shape"] == SLAB and b.report["converged"]
    c = p.davidson(max_it=1, init=0, **kw)
    assert np.array_equal(a.vectors, c.vectors) and np.array_equal(a.energies, c.energies)
    p.close()


# alpha sweep, beta sweep, alpha x beta of FP32: the longest list that its shared
# memory holds, and one more string (the 8-byte forms go on to twice that)
@pytest.mark.parametrize("na,nb,seed,fits", [(14252, 12, 1, True), (14253, 12, 1, False), (1, 14252, 1, True),
                                             (1, 14253, 1, False), (12, 11232, 5, True), (12, 11233, 5, False)])
def test_fp32_at_its_shared_memory_limit(engine, na, nb, seed, fits):
    prob, p = _problem(engine, 20, 8, 8, na, nb, seed=seed)
    q = TPBProblem.from_problem(engine, prob)
    q.diag_terms()
    q.set_tuning(0, 1, 1)  # the FP64 sweeps
    st = torch.cuda.current_stream().cuda_stream
    f = torch.tensor(np.random.default_rng(nb).normal(size=(3, prob.ndet)), device="cuda").float()
    many, one = torch.full_like(f, float("nan")), torch.full_like(f, float("nan"))
    for j in range(3):
        p.sigma_mixed_device(f[j].data_ptr(), one[j].data_ptr(), stream=st)
    p.sigma_mixed_block_device(f.data_ptr(), many.data_ptr(), 3, stream=st)
    torch.cuda.synchronize()
    assert (p.tuning(1)["beta_shape"] == SLAB) == fits
    for j in range(3):
        ref = _sigma(q, f[j].double()).cpu().numpy()
        assert max_rel(one[j].double().cpu().numpy(), ref) <= 5e-6
        assert max_rel(many[j].double().cpu().numpy(), ref) <= 5e-6
    assert max_rel(_sigma(p, f[0].double()).cpu().numpy(), _sigma(q, f[0].double()).cpu().numpy()) <= 1e-13
    assert p.tuning(0)["beta_shape"] == SLAB
    if not fits:
        kw = dict(nroots=1, max_nb=16, eps=1e-7, max_it=40, init=1, want_vectors=False)
        a, b = p.davidson(precision=MIXED, **kw), q.davidson(**kw)
        assert a.report["converged"] and b.report["converged"]
        assert abs(a.energies[0] - b.energies[0]) <= 1e-8
    p.close()
    q.close()


@pytest.mark.parametrize("norb,na,nb,nocc,slab", [(40, 900, 700, 13, False), (16, 300, 280, 5, True)])
def test_one_choice_of_sweeps_a_problem(engine, norb, na, nb, nocc, slab):
    """A stopped solve returns the same vectors before and after calls that are not
    its own, and on a new problem of the same sizes, whether the other products go
    by the sweeps or by the fixed-point kernels; the shapes can be read."""
    kw = dict(nroots=2, max_nb=16, eps=1e-9)
    first = None
    for order in ("solve first", "solve last"):
        prob, p = _problem(engine, norb, nocc, nocc, na, nb, seed=3)
        if order == "solve first":
            first = p.davidson(max_it=1, init=0, **kw)
            assert (p.tuning(3)["beta_shape"] is None) == slab
        p.davidson(max_it=2, init=1, **kw)
        assert (p.tuning(3)["beta_shape"] == SLAB) == slab
        again = p.davidson(max_it=1, init=0, **kw)
        sweeps = p.tuning(6 if slab else 3)["beta_shape"]
        assert sweeps not in (None, SLAB) and (p.tuning(6)["beta_shape"] is None) == (not slab)
        assert np.array_equal(first.vectors, again.vectors) and np.array_equal(first.energies, again.energies)
        p.close()


def test_split_choice_is_kept(engine):
    """set_split on a precision that has taken the fixed-point kernels: 1 is what they
    do, 0 leads to the sweeps with the pairs inside."""
    prob, p = _problem(engine, 16, 5, 5, 300, 280, seed=11)
    x = torch.tensor(np.random.default_rng(0).normal(size=prob.ndet), device="cuda")
    a = _sigma(p, x)
    p.set_split(0, 1)
    assert p.tuning(0)["beta_shape"] == SLAB and torch.equal(_sigma(p, x), a)
    p.set_split(0, 0)
    b = _sigma(p, x)
    t = p.tuning(0)
    assert t["beta_shape"] not in (None, SLAB) and t["alpha_beta"]["split"] == 0
    assert max_rel(b.cpu().numpy(), a.cpu().numpy()) <= 1e-13
    p.close()


def test_fp32_list_sums_join_in_float_float(engine):
    """A beta single's term of 2^24 |V| that the diagonal's cancels, and doubles of
    order 1 beside it: what the doubles add survives.  The two products share every
    rounding of a table value, so their difference at the bra is the doubles' FP32
    sum, off by its own roundings and one rounding of each result."""
    prob, p = _problem(engine, 16, 5, 5, 300, 280, seed=11)
    o = Oracle.from_problem(prob)
    b = prob.bstr.astype(np.uint64)
    nb, ia = b.size, 7
    found = False
    for ib in range(nb):
        dist = np.array([bin(int(x)).count("1") for x in b ^ b[ib]])
        singles, doubles = np.nonzero(dist == 2)[0], np.nonzero(dist == 4)[0]
        if len(singles) == 0 or len(doubles) < 20:
            continue
        e = np.zeros(prob.ndet)
        e[ia * nb + singles[0]] = 1.0
        v, h = o.mult(e)[ia * nb + ib], o.hii()[ia * nb + ib]
        if abs(v) > 1e-3:
            found = True
            break
    assert found
    c = np.zeros(prob.ndet, dtype=np.float32)
    c[ia * nb + singles[0]] = 2.0 ** 24
    c[ia * nb + ib] = -v * 2.0 ** 24 / h
    d = c.copy()
    d[ia * nb + doubles] = np.random.default_rng(0).uniform(0.5, 1.0, len(doubles)).astype(np.float32)
    only = np.where(d != c, d, 0).astype(np.float64)
    want, size = o.mult(only)[ia * nb + ib], 0.0
    for k in doubles:
        e[:] = 0.0
        e[ia * nb + k] = d[ia * nb + k]
        size += abs(o.mult(e)[ia * nb + ib])
    out = []
    for x in (c, d):
        f = torch.tensor(x, device="cuda")
        s = torch.empty_like(f)
        p.sigma_mixed_device(f.data_ptr(), s.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        out.append(float(s[ia * nb + ib]))
    assert p.tuning(1)["beta_shape"] == SLAB
    bound = 2.0 ** -24 * (len(doubles) * size + abs(out[0]) + abs(out[1]))
    assert bound < 0.05 * abs(want)
    assert abs(out[1] - out[0] - want) <= 2 * bound
    p.close()


# weights over `decades` orders of magnitude on the strings of each spin; every fourth
# alpha string's at the size of rounding noise; one beta string's
@pytest.mark.parametrize("kind", ["3 decades", "6 decades", "12 decades", "noise", "one string"])
@pytest.mark.parametrize("norb,na,nb,nocc", [(12, 161, 187, 4), (24, 300, 280, 8), (16, 60, 300, 5)])
def test_elements_of_wide_vectors(engine, norb, na, nb, nocc, kind):
    """Every element of sigma to the bound of its own terms, k terms of relative
    error 2^-53 (2^-46 in double-float), whatever else its vector holds; twice
    that, for the reference's sums have it too."""
    prob, p = _problem(engine, norb, nocc, nocc, na, nb, seed=na + nb)
    H = Oracle.from_problem(prob).hamiltonian()
    rng = np.random.default_rng(nb)
    d = int(kind.split()[0]) if "decades" in kind else 2
    C = rng.normal(size=(na, nb)) * 10.0 ** rng.uniform(-d, 0, (na, 1)) * 10.0 ** rng.uniform(-d, 0, (1, nb))
    if kind == "noise":
        C[::4] *= 1e-17
    elif kind == "one string":
        C[:, nb // 2] *= 1e-17
    x = C.ravel()
    ref, size, k = H @ x, abs(H) @ np.abs(x), np.diff(H.indptr).max() + 8
    c = torch.tensor(x, device="cuda")
    s = _sigma(p, c)
    assert p.tuning(0)["beta_shape"] == SLAB
    assert (np.abs(s.cpu().numpy() - ref) <= 2 * k * 2.0 ** -53 * size).all()
    assert torch.equal(_sigma(p, c), s)
    hi = c.float()
    pair = torch.stack([hi, (c - hi.double()).float()], dim=-1).contiguous()
    y = torch.empty_like(pair)
    p.sigma_df_device(pair.data_ptr(), y.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert p.tuning(2)["beta_shape"] == SLAB
    # (FP32's exponents: below 1e-25 a value's low part, or a product's, is subnormal)
    err = np.abs(y.double().sum(-1).cpu().numpy() - ref) / (size + 1e-25)
    assert err.max() <= 2 * k * 2.0 ** -46
    p.close()


@pytest.mark.parametrize("norb,na,nb,nocc", [(16, 300, 280, 5), (24, 300, 280, 8)])
def test_a_budget_holds_what_it_held_without_the_tables(norb, na, nb, nocc):
    """Products and solves within a budget that the sweeps need: what they hold at the
    end of the same calls, and the vector that choosing their shapes takes."""
    prob = make_problem(norb, nocc, nocc, na, nb, seed=11)
    kw = dict(nroots=2, max_nb=16, eps=1e-9, max_it=1, want_vectors=False)

    def calls(e, sweeps):
        p = TPBProblem.from_problem(e, prob)
        p.diag_terms()
        if sweeps:
            p.set_tuning(0, 1, 1)
            p.set_tuning(3, 1, 1)
        x = torch.ones(prob.ndet, dtype=torch.float64, device="cuda")
        _sigma(p, x)
        for init in (0, 1):
            p.davidson(init=init, **kw)
        used, shape = e.bytes_in_use, p.tuning(0)["beta_shape"]
        p.close()
        return used, shape

    e = Engine(0)
    used, _ = calls(e, True)
    e.close()
    e = Engine(0, hbm_budget=used + 8 * prob.ndet + 4096)
    calls(e, False)
    e.close()
    e = Engine(0, hbm_budget=1 << 36)  # with room for the tables
    assert calls(e, False)[1] == SLAB
    e.close()


@pytest.mark.parametrize("norb,na,nb,nocc", [(24, 300, 280, 8), (16, 60, 300, 5)])
def test_ket_rows_of_different_scales(engine, norb, na, nb, nocc):
    """Every other alpha string 2^-35 below its neighbours, on the beta strings that
    those do not have, so that each row and column holds one scale and the rows of an
    alpha x beta batch two.  Every element to its terms' FP64 roundings (as above) and
    those of the matrix elements, at most 2^-45 of the largest (2^-39 in double-float)
    of each kind, whose scale may be eight times the largest off the diagonal."""
    prob, p = _problem(engine, norb, nocc, nocc, na, nb, seed=na + nb)
    H = Oracle.from_problem(prob).hamiltonian()
    off = H.copy()
    off.setdiag(0.0)
    C = np.random.default_rng(nb).uniform(0.5, 1.0, (na, nb))
    C[::2, 1::2] = 0.0
    C[1::2, ::2] = 0.0
    C[1::2] *= 2.0 ** -35
    x = C.ravel()
    ref, size, k = H @ x, abs(H) @ np.abs(x), np.diff(H.indptr).max() + 8
    table = 8 * np.abs(off.data).max() * ((off != 0) @ np.abs(x))
    c = torch.tensor(x, device="cuda")
    s = _sigma(p, c)
    assert p.tuning(0)["beta_shape"] == SLAB
    assert (np.abs(s.cpu().numpy() - ref) <= 2 * k * 2.0 ** -53 * size + 2.0 ** -45 * table).all()
    hi = c.float()
    pair = torch.stack([hi, (c - hi.double()).float()], dim=-1).contiguous()
    y = torch.empty_like(pair)
    p.sigma_df_device(pair.data_ptr(), y.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    err = np.abs(y.double().sum(-1).cpu().numpy() - ref)
    assert (err <= 2 * k * 2.0 ** -46 * size + 2.0 ** -39 * table + 1e-38).all()
    p.close()
