"""Fast paths of assembly and products against the oracle, at the sizes where
their index arithmetic and rounding are at their edges."""
import numpy as np
import pytest

from conftest import SPHERE, TORUS

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-12


@pytest.fixture(scope="module")
def ctx():
    import bembel_gb300 as bg
    return bg.Context(0)


def _operator(ctx, geo, M, P, kind, kappa=0.0, np_=6, **kw):
    import bembel_gb300 as bg
    lin = [bg.LaplaceSingleLayerOperator, bg.HelmholtzSingleLayerOperator, bg.MaxwellSingleLayerOperator][kind]()
    if kind:
        lin.set_wavenumber(kappa)
    d = bg.DiscreteOperator(bg.AnsatzSpace(bg.Geometry(geo, ctx), M, P), lin, n_p=np_, **kw)
    d.compute()
    return d


@pytest.mark.parametrize("geo,M,P,kind,kappa", [(SPHERE, 1, 1, 0, 0.0), (SPHERE, 0, 2, 0, 0.0), (TORUS, 0, 1, 1, 1.5),
                                                (TORUS, 1, 2, 1, 2.0), (SPHERE, 1, 3, 0, 0.0)])
def test_mirrored_element_pairs(ctx, oracle, geo, M, P, kind, kappa):
    """Blocks of swapped element pairs are transposed copies: both the block
    of a dense leaf and that of the swapped leaf match the oracle, which
    integrates every pair by itself (1e-12, the parity bound: its blocks are
    symmetric to a few 1e-15)."""
    d = _operator(ctx, geo, M, P, kind, kappa)
    o = oracle.Problem(geo, M, P, kind, kappa=kappa, np_=6)
    dense = [i for i, lv in enumerate(d.leaves()) if lv[0] == 2]
    assert dense
    for li in dense:
        a, b = d.leaf_block(li), o.leaf_matrix(li)
        assert np.linalg.norm(a - b) <= FP64_TOL * np.linalg.norm(b), li


def _fp64_dense(d):
    """The H2 matrix of an operator without far field (M = 1), from its FP64 leaf blocks and T."""
    ptr, idx, val = d.transform_csr()
    T = np.zeros((d.S, d.N))
    for r in range(d.S):
        T[r, idx[ptr[r]:ptr[r + 1]]] += val[ptr[r]:ptr[r + 1]]
    lv = d.leaves()
    ncl = d.S // d.leaf_block(0).shape[0] if d.lin_op.kind != 2 else 0
    n = d.S // ncl
    A = np.zeros((d.S, d.S), dtype=d.leaf_block(0).dtype)
    for i in range(len(lv)):
        r, c = lv[i][2], lv[i][3]
        A[r * n:(r + 1) * n, c * n:(c + 1) * n] = d.leaf_block(i)
    return T, A


@pytest.mark.parametrize("geo,P,kind", [(SPHERE, 0, 0), (SPHERE, 1, 0), (SPHERE, 2, 0), (SPHERE, 3, 0),
                                        (SPHERE, 1, 1), (TORUS, 2, 1)])
def test_digit_near_field_products(ctx, geo, P, kind):
    """Tensor-core products on digit bytes (leaf blocks of 4, 16, 36 and 64
    rows, real and complex) against FP64 sums of the same leaf blocks, for
    column counts around the 16- and 32-column passes, a zero column and
    columns 1e-150 and 1e+150 times the others. Bound per column: 2^-52 of
    sum |A| |x| for the product's digits and fixed point, plus the reference's
    own rounding, below 1e-14 of the column's norm."""
    d = _operator(ctx, geo, 1, P, kind, 2.0)
    assert d.n_lowrank == 0
    T, A = _fp64_dense(d)
    H = d.get_discrete_operator()
    rng = np.random.default_rng(5)
    for nrhs in (3, 15, 16, 17, 31, 32, 33, 45):
        x = rng.normal(size=(d.N, nrhs)) + (1j * rng.normal(size=(d.N, nrhs)) if kind else 0)
        x[:, 0] = 0.0
        x[:, 1] *= 1e-150
        x[:, 2] *= 1e150
        ref = T.T @ (A @ (T @ x))
        for prec in ("fp64", "mixed"):
            y = H.matvec(x, precision=prec)
            assert not y[:, 0].any()
            err = np.linalg.norm(y - ref, axis=0)[1:] / np.linalg.norm(ref, axis=0)[1:]
            assert err.max() < 1e-14, (nrhs, prec, err.max())


@pytest.mark.parametrize("np_", [4, 6, 7, 8, 9, 10, 11, 12])
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_digit_far_field_products(ctx, oracle, np_, kind):
    """FP64 products through the far field's digits for every interpolation
    degree (blocks of n_p^2 rows with 0, 1 or 4 columns in the last group of
    8; n_p = 12 keeps the double-float pairs) match the oracle to 1e-12, with
    one column, a part of a pass and more than one pass."""
    d = _operator(ctx, SPHERE, 2, 1, kind, 2.0, np_)
    o = oracle.Problem(SPHERE, 2, 1, kind, kappa=2.0 if kind else 0.0, np_=np_)
    rng = np.random.default_rng(6)
    x = rng.normal(size=(d.N, 35)) + (1j * rng.normal(size=(d.N, 35)) if kind else 0)
    ref = o.matvec(x)
    A = d.get_discrete_operator()
    for n in (1, 7, 20, 35):
        y = A.matvec(x[:, :n])
        assert np.linalg.norm(y - ref[:, :n]) < FP64_TOL * np.linalg.norm(ref[:, :n]), n


@pytest.mark.parametrize("kind", [0, 1])
def test_digit_products_keep_infinities_apart(ctx, kind):
    """A column with Inf or NaN does not touch the others, and stays Inf or
    NaN itself."""
    d = _operator(ctx, SPHERE, 2, 2, kind, 2.0, 9)
    A = d.get_discrete_operator()
    rng = np.random.default_rng(8)
    x = rng.normal(size=(d.N, 6)) + (1j * rng.normal(size=(d.N, 6)) if kind else 0)
    clean = A.matvec(x)
    x[3, 2], x[d.N // 2, 4] = np.inf, np.nan
    y = A.matvec(x)
    assert not np.isfinite(y[:, [2, 4]]).all(axis=0).any()
    assert np.isnan(y[:, 4]).any() and np.array_equal(y[:, [0, 1, 3, 5]], clean[:, [0, 1, 3, 5]])


@pytest.mark.parametrize("P,np_", [(1, 6), (2, 6), (1, 7), (2, 8), (2, 9), (1, 10), (1, 11)])
@pytest.mark.parametrize("kind", [0, 1])
def test_fused_transforms_for_few_columns(ctx, P, np_, kind):
    """The fused FP64 transforms pack the columns there are into a warp (1, 2,
    4, .. 32 lanes a row): the product of any number of columns equals the
    same columns of a 33-column product to rounding (1e-13, the transforms'
    sums are the same ones), and the batched-GEMM transforms to 1e-12."""
    d = _operator(ctx, SPHERE, 3, P, kind, 2.0, np_)
    A = d.get_discrete_operator()
    rng = np.random.default_rng(10)
    x = rng.normal(size=(d.N, 33)) + (1j * rng.normal(size=(d.N, 33)) if kind else 0)
    full = A.matvec(x)
    for n in (1, 2, 3, 5, 9, 16, 17, 32):
        y = A.matvec(x[:, :n])
        assert np.linalg.norm(y - full[:, :n]) < 1e-13 * np.linalg.norm(full[:, :n]), n
        d.set_plan(n, "fp64", transforms=1)
        z = A.matvec(x[:, :n])
        d.set_plan(n, "fp64")
        assert np.linalg.norm(z - y) < 1e-12 * np.linalg.norm(y), n


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("nrhs", [1, 3, 33, 100, 256])
def test_solver_sums_for_any_number_of_columns(ctx, kind, nrhs):
    """The Krylov sums share a CTA among the columns (256 / columns chains each,
    whole groups of 32 threads): every column of a batched solve meets the
    tolerance it was asked for in an FP64 product's residual."""
    d = _operator(ctx, SPHERE, 2, 1, kind, 1.0, 6)
    A = d.get_discrete_operator()
    rng = np.random.default_rng(11)
    b = rng.normal(size=(d.N, nrhs)) + (1j * rng.normal(size=(d.N, nrhs)) if kind else 0)
    x, _ = A.solve(b, tol=1e-9, inner="fp64")
    r = np.linalg.norm(A.matvec(x) - b, axis=0) / np.linalg.norm(b, axis=0)
    assert r.max() < 2e-9


@pytest.mark.parametrize("kind,P", [(0, 0), (0, 2), (1, 1), (1, 3)])
@pytest.mark.parametrize("npts,nrhs", [(64, 2), (8, 8), (33, 16), (100, 32), (31, 40), (700, 17)])
def test_potential_of_many_columns(ctx, kind, P, npts, nrhs):
    """The potential with lanes as points and all columns at once: the same
    sums as one column at a time up to their order (1e-13 of the largest)."""
    d = _operator(ctx, SPHERE, 1, P, kind, 1.3)
    rng = np.random.default_rng(12)
    rho = rng.normal(size=(d.N, nrhs)) + (1j * rng.normal(size=(d.N, nrhs)) if kind else 0)
    pts = rng.uniform(-0.4, 0.4, (npts, 3))
    y = d.potential(rho, pts)
    z = np.stack([np.asarray(d.potential(rho[:, c:c + 1], pts)).reshape(npts) for c in range(nrhs)], 1)
    assert np.abs(np.asarray(y).reshape(npts, nrhs) - z).max() < 1e-13 * np.abs(z).max()


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("kind,nrhs", [(0, 1), (0, 33), (1, 1), (1, 5), (2, 3)])
def test_near_field_beside_the_far_field(ctx, kind, nrhs, precision):
    """From the second product of a shape on, the near field is a branch of a
    graph beside the transforms and the far field: the same bits as the first
    product's launches in a row, also after another shape in between."""
    d = _operator(ctx, SPHERE, 3, 1, kind, 1.1)
    A = d.get_discrete_operator()
    rng = np.random.default_rng(13)
    x = rng.normal(size=(d.N, nrhs)) + (1j * rng.normal(size=(d.N, nrhs)) if kind else 0)
    y = A.matvec(x, precision=precision)
    for _ in range(3):
        assert np.array_equal(A.matvec(x, precision=precision), y)
        A.matvec(x[:, :1], precision="fp64")


@pytest.mark.parametrize("P,np_,mcl", [(2, 6, 2), (2, 9, 2), (3, 11, 2), (1, 11, 3), (3, 12, 1)])
@pytest.mark.parametrize("kind", [0, 1])
def test_transforms_of_large_panels(ctx, oracle, P, np_, mcl, kind):
    """Leaf clusters of 16 and 64 elements and the largest interpolation
    degree, whose transform panels pass the shared memory of a block at some
    number of columns, are served at every number of columns and precision
    (FP64 and the FP64-accurate near field against the oracle to 1e-12; the
    FP32 far field and near field to 1e-4, their rounding of 6e-8 times the
    condition of the interpolation). n_p = 12 has no FP32 far field at any
    size, so FP64 only there."""
    M = 3 if mcl < 3 else 4
    d = _operator(ctx, SPHERE, M, P, kind, 1.2, np_, min_cluster_level=mcl)
    assert d.n_lowrank > 0
    o = oracle.Problem(SPHERE, M, P, kind, kappa=1.2 if kind else 0.0, np_=np_, mcl=mcl)
    rng = np.random.default_rng(14)
    x = rng.normal(size=(d.N, 33)) + (1j * rng.normal(size=(d.N, 33)) if kind else 0)
    ref = o.matvec(x)
    A = d.get_discrete_operator()
    for n in (1, 8, 9, 16, 17, 33):
        for prec, tol in (("fp64", FP64_TOL), ("mixed", 1e-4), ("fp32", 1e-4))[:1 if np_ == 12 else 3]:
            y = A.matvec(x[:, :n], precision=prec)
            assert np.linalg.norm(y - ref[:, :n]) < tol * np.linalg.norm(ref[:, :n]), (n, prec)


def _spread_columns(d, T, rng, cplx):
    """Columns whose entries differ widely: single unknowns, magnitudes from 1
    to 1e-20 at random and by position, beside a normal one."""
    N = d.N
    x = np.zeros((N, 8), dtype=complex if cplx else float)
    for c, j in enumerate((0, N // 3, N - 1)):
        x[j, c] = 1.0
    x[:, 3] = rng.normal(size=N) * 10.0 ** (-20 * rng.uniform(size=N))
    x[:, 4] = rng.normal(size=N) * 10.0 ** (-20 * np.arange(N) / N)
    x[:, 5] = rng.normal(size=N) * np.where(np.arange(N) < N // 6, 1.0, 1e-18)
    x[:, 6] = rng.normal(size=N) * np.where(np.arange(N) == N // 2, 1e30, 1.0)
    x[:, 7] = rng.normal(size=N)
    if cplx:
        x[:, 3:] *= np.exp(1j * rng.uniform(0, 2 * np.pi, (N, 5)))
    return x


@pytest.mark.parametrize("geo,P,kind,kappa", [(SPHERE, 0, 0, 0), (SPHERE, 1, 0, 0), (SPHERE, 2, 0, 0), (SPHERE, 1, 1, 2.0),
                                              (SPHERE, 1, 1, 2.0 - 30.0j), (TORUS, 2, 1, 1.0 - 20.0j)])
def test_digit_near_field_keeps_every_entry(ctx, geo, P, kind, kappa):
    """Entry by entry the FP64 product is as good as plain FP64 sums, whatever
    the sizes of x in one column and of the blocks in one row (a damped kernel
    decays by up to e^-120 over the surface): the error of each entry is below
    the bound of such sums, (n + 20) 2^-53 times |T^t| |A| |T| |x| for rows of
    n = S terms (complex: 2 n, and twice that for the two parts), against sums
    in extended precision. The 20 covers T and T^t (at most 16 terms a row)."""
    d = _operator(ctx, geo, 1, P, kind, kappa)
    assert d.n_lowrank == 0
    T, A = _fp64_dense(d)
    x = _spread_columns(d, T, np.random.default_rng(15), bool(kind))
    wide = np.clongdouble if kind else np.longdouble
    Tw = T.astype(np.longdouble)
    ref = Tw.T @ (A.astype(wide) @ (Tw @ x.astype(wide)))
    bound = np.abs(T).T @ (np.abs(A) @ (np.abs(T) @ np.abs(x)))
    n = d.S * (2 if kind else 1)
    for prec in ("fp64", "mixed") if kind else ("fp64",):  # the real mixed product promises less
        y = d.get_discrete_operator().matvec(x, precision=prec)
        err = np.abs(y - ref).astype(float)
        assert (err <= (2 if kind else 1) * (n + 20) * 2.0 ** -53 * bound).all(), \
            (prec, (err / np.maximum(bound, 1e-300)).max(axis=0))


@pytest.mark.parametrize("M,P,kind,kappa,np_", [(2, 1, 0, 0, 6), (3, 1, 0, 0, 9), (2, 2, 1, 2.0, 9), (2, 1, 1, 2.0 - 1.0j, 7)])
def test_digit_far_field_keeps_every_entry(ctx, oracle, M, P, kind, kappa, np_):
    """With a far field, entry by entry the FP64 product stays within n 2^-48
    |T^t| |A| |T| |x| (n = S, the bound of double-float sums over a row; A the
    dense matrix) of the oracle's FP64 product of the same H2 matrix, for
    columns of widely different sizes."""
    d = _operator(ctx, SPHERE, M, P, kind, kappa, np_)
    assert d.n_lowrank > 0
    o = oracle.Problem(SPHERE, M, P, kind, kappa=kappa, np_=np_)
    T = o.transform_dense()
    x = _spread_columns(d, T, np.random.default_rng(18), bool(kind))
    bound = np.abs(T).T @ (np.abs(o.dense_ss()) @ (np.abs(T) @ np.abs(x)))
    err = np.abs(d.get_discrete_operator().matvec(x) - o.matvec(x))
    assert (err <= d.S * 2.0 ** -48 * bound).all(), (err / bound).max(axis=0)


@pytest.mark.parametrize("np_", [6, 9])
@pytest.mark.parametrize("batched", [False, True])
def test_far_field_of_a_damped_kernel(ctx, oracle, np_, batched):
    """A column that lives on one side of the surface, with a kernel that
    decays by e^-28 to the other side: the values there, 1e-8 to 1e-12 of the
    largest, match the oracle to 1e-10 of themselves, by itself and as one of
    two batched wavenumbers (the other without damping)."""
    kappa = 1.5 - 14.0j
    d = _operator(ctx, SPHERE, 3, 1, 1, 1.5, np_)
    if batched:
        d.prepare_wavenumbers([1.5, kappa])
        d.assemble_wavenumbers()
    else:
        d.get_discrete_operator().matvec(np.ones(d.N))  # work vectors of the undamped operator
        d.lin_op.set_wavenumber(kappa)
        d.compute()
    o = oracle.Problem(SPHERE, 3, 1, 1, kappa=kappa, np_=np_)
    rng = np.random.default_rng(16)
    x = np.zeros((d.N, 4), dtype=complex)
    x[:d.N // 24] = rng.uniform(0.5, 1.0, (d.N // 24, 4))
    ref = o.matvec(x)
    y = d.get_discrete_operator().matvec(np.hstack([x, x]) if batched else x)[:, -4:]
    size = np.linalg.norm(ref, axis=1)
    low = size < 1e-8 * size.max()
    assert low.sum() > d.N // 20
    assert (np.linalg.norm(y - ref, axis=1)[low] < 1e-10 * size[low]).all()


DEGENERATE_DAT = """# nurbs mesh v.2.1
# screen
# a square whose upper side is shrunk to nearly a point
#
2 3 1 0 0
PATCH 0
1 1
2 2
0 0 1 1
0 0 1 1
0 1 0 0.000001
0 0 1 1
0 0 0 0
1 1 1 1
"""


def test_far_field_of_a_shrunk_patch(ctx, oracle, tmp_path):
    """Couplings of one row that differ by the surface measure of a nearly
    singular patch (1e-6 at the shrunk side) are kept as FP32 pairs instead of
    digits: unit vectors there and normal columns match the oracle, 1e-12 of
    the column, for one column and several, also after another assembly."""
    geo = str(tmp_path / "shrunk.dat")
    with open(geo, "w") as f:
        f.write(DEGENERATE_DAT)
    d = _operator(ctx, geo, 4, 1, 0, 0.0, 9)
    assert d.n_lowrank > 0
    o = oracle.Problem(geo, 4, 1, 0, np_=9)
    rng = np.random.default_rng(17)
    x = rng.normal(size=(d.N, 33))
    x[:, 0] = 0.0
    x[-1, 0] = 1.0
    ref = o.matvec(x)
    A = d.get_discrete_operator()
    for _ in range(2):
        for n in (1, 5, 33):
            y = A.matvec(x[:, :n])
            assert (np.linalg.norm(y - ref[:, :n], axis=0) < FP64_TOL * np.linalg.norm(ref[:, :n], axis=0)).all(), n
        d.compute()


LARGE_DAT = """# nurbs mesh v.2.1
# screen
# a square of side 1e150, whose surface measure is beyond FP64
#
2 3 1 0 0
PATCH 0
1 1
2 2
0 0 1 1
0 0 1 1
0 1e150 0 1e150
0 0 1e150 1e150
0 0 0 0
1 1 1 1
"""


@pytest.mark.parametrize("geo,M,kind,kappa,np_", [
    (None, 1, 0, 0.0, 6), (SPHERE, 1, 1, np.nan, 6), (SPHERE, 1, 1, 1.0 + 800.0j, 6), (SPHERE, 3, 1, np.nan, 6),
    (SPHERE, 3, 1, 1.0 + 60.0j, 9), (SPHERE, 3, 1, 1.0 + 800.0j, 7), (SPHERE, 2, 2, np.nan, 6)])
def test_operators_with_infinities(ctx, tmp_path, geo, M, kind, kappa, np_):
    """Where every row of the couplings has Inf or NaN (a surface measure or a
    growing kernel beyond FP64, a wavenumber that is NaN), no entry of the
    product is finite, at any number of columns. Growth by e^120 leaves FP64
    couplings finite but passes the range of the FP32 pairs that complex far
    fields are kept as: not finite there either. With a finite wavenumber again
    the operator is the one it was before (1e-13)."""
    if geo is None:
        geo = str(tmp_path / "large.dat")
        with open(geo, "w") as f:
            f.write(LARGE_DAT)
    d = _operator(ctx, geo, M, 1, kind, 2.0, np_)
    rng = np.random.default_rng(19)
    x = rng.normal(size=(d.N, 17)) + (1j * rng.normal(size=(d.N, 17)) if kind else 0)
    if kind:
        clean = d.get_discrete_operator().matvec(x)
        d.lin_op.set_wavenumber(kappa)
        d.compute()
    A = d.get_discrete_operator()
    near = d.n_lowrank == 0 or np.isnan(kappa)  # the near field, which "mixed" keeps in FP64, has them too
    for n in (1, 2, 3, 5, 17):
        for prec in ("fp64", "mixed") if near else ("fp64",):
            assert not np.isfinite(A.matvec(x[:, :n], precision=prec)).any(), (n, prec)
    if kind:
        d.lin_op.set_wavenumber(2.0)
        d.compute()
        y = d.get_discrete_operator().matvec(x)
        assert np.linalg.norm(y - clean) < 1e-13 * np.linalg.norm(clean)


@pytest.mark.parametrize("kind", [0, 1])
def test_digit_panels_come_with_the_products_that_read_them(ctx, kind):
    """The digit panels of x are allocated by the first product that reads them
    (near field: mixed and FP64, far field: FP64), so that the first product of
    another kind does not wait for them; whatever the order of the precisions
    and column counts, also over graphs that the growing panels make stale,
    results have the bits of an operator that starts with the largest."""
    import ctypes
    from bembel_gb300 import _lib

    def allocated(d):
        a, e = ctypes.c_size_t(), ctypes.c_size_t()
        ctx.check(_lib.load().bg_operator_memory(d.h, ctypes.byref(a), ctypes.byref(e)))
        return a.value

    d, whole = (_operator(ctx, SPHERE, 2, 1, kind, 1.3) for _ in range(2))
    assert d.n_lowrank > 0
    rng = np.random.default_rng(21)
    x = rng.normal(size=(d.N, 70)) + (1j * rng.normal(size=(d.N, 70)) if kind else 0)
    ref = {n: whole.get_discrete_operator().matvec(x[:, :n]) for n in (70, 40, 5)}
    mixed = whole.get_discrete_operator().matvec(x[:, :5], precision="mixed")
    A = d.get_discrete_operator()
    A.matvec(x[:, :5], precision="fp32")
    m = [allocated(d)]
    for prec in ("mixed", "fp64"):
        for _ in range(3):
            assert np.array_equal(A.matvec(x[:, :5], precision=prec), mixed if prec == "mixed" else ref[5])
        m.append(allocated(d))
    assert m[0] < m[1] < m[2]
    for n in (40, 5, 70, 40):
        for _ in range(2):
            assert np.array_equal(A.matvec(x[:, :n]), ref[n]), n
    assert np.array_equal(A.matvec(x[:, :5], precision="mixed"), mixed)


@pytest.mark.parametrize("mcl", [0, 2])
@pytest.mark.parametrize("geo,M,P,kind", [(SPHERE, 2, 1, 0), (TORUS, 2, 1, 1), (SPHERE, 2, 2, 1)])
@pytest.mark.parametrize("prepared", [False, True])
def test_mirrored_element_pairs_of_other_leaves(ctx, oracle, geo, M, P, kind, mcl, prepared):
    """The copies of swapped pairs with one element and with 16 per leaf
    cluster (pairs across leaves only, and mostly within one), assembled for
    one wavenumber and prepared with a second one: every leaf block matches
    the oracle to 1e-12, the parity bound."""
    if prepared and not kind:
        pytest.skip("no wavenumber to prepare")
    d = _operator(ctx, geo, M, P, kind, 1.4, min_cluster_level=mcl)
    if prepared:
        d.prepare_wavenumbers([0.6, 2.2])
        d.lin_op.set_wavenumber(2.2)
        d.compute()
    o = oracle.Problem(geo, M, P, kind, kappa=(2.2 if prepared else 1.4) if kind else 0.0, np_=6, mcl=mcl)
    dense = [i for i, lv in enumerate(d.leaves()) if lv[0] == 2]
    assert dense
    for li in dense:
        a, b = d.leaf_block(li), o.leaf_matrix(li)
        assert np.linalg.norm(a - b) <= FP64_TOL * np.linalg.norm(b), li


@pytest.mark.parametrize("P,np_", [(1, 7), (2, 9)])
@pytest.mark.parametrize("nr", [1, 2, 3, 17])
def test_batched_wavenumber_products_of_few_columns(ctx, P, np_, nr):
    """Products of three batched wavenumbers, whose digit products read and
    write a column block of wider rows, equal each wavenumber's own operator's
    around the column counts at which the near field changes its kernel and a
    pass is full (1e-13 for FP64, 1e-12 for mixed, as for other counts)."""
    ks = [0.7, 2.0, 3.5 - 0.2j]
    d = _operator(ctx, SPHERE, 2, P, 1, ks[0], np_)
    d.prepare_wavenumbers(ks)
    d.assemble_wavenumbers()
    rng = np.random.default_rng(20)
    x = rng.normal(size=(d.N, 3 * nr)) + 1j * rng.normal(size=(d.N, 3 * nr))
    y = {prec: d.get_discrete_operator().matvec(x, precision=prec) for prec in ("fp64", "mixed")}
    for q, k in enumerate(ks):
        A = _operator(ctx, SPHERE, 2, P, 1, k, np_).get_discrete_operator()
        cols = slice(q * nr, (q + 1) * nr)
        for prec, tol in (("fp64", 1e-13), ("mixed", 1e-12)):
            ref = A.matvec(x[:, cols], precision=prec)
            assert np.linalg.norm(y[prec][:, cols] - ref) < tol * np.linalg.norm(ref), (prec, q)


@pytest.mark.parametrize("kind,kappa", [(0, 0), (1, 2.0), (1, 2.0 - 30.0j)])
def test_digit_near_field_of_large_blocks_keeps_every_entry(ctx, kind, kappa):
    """Leaf blocks of 64 rows, whose floors are kept by two groups of rows:
    entry by entry the bound of plain FP64 sums, as for smaller blocks."""
    d = _operator(ctx, SPHERE, 1, 3, kind, kappa)
    assert d.n_lowrank == 0
    T, A = _fp64_dense(d)
    x = _spread_columns(d, T, np.random.default_rng(21), bool(kind))
    wide = np.clongdouble if kind else np.longdouble
    Tw = T.astype(np.longdouble)
    ref = Tw.T @ (A.astype(wide) @ (Tw @ x.astype(wide)))
    bound = np.abs(T).T @ (np.abs(A) @ (np.abs(T) @ np.abs(x)))
    n = d.S * (2 if kind else 1)
    err = np.abs(d.get_discrete_operator().matvec(x) - ref).astype(float)
    assert (err <= (2 if kind else 1) * (n + 20) * 2.0 ** -53 * bound).all(), \
        (err / np.maximum(bound, 1e-300)).max(axis=0)
