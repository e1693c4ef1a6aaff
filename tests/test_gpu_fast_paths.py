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
                                                (TORUS, 1, 2, 1, 2.0), (SPHERE, 1, 3, 0, 0.0), (SPHERE, 1, 1, 2, 2.0)])
def test_mirrored_element_pairs(ctx, oracle, geo, M, P, kind, kappa):
    """Blocks of swapped element pairs are transposed copies: both the block
    of a dense leaf and that of the swapped leaf match the oracle, which
    integrates every pair by itself (1e-12, the parity bound: its blocks are
    symmetric to a few 1e-15)."""
    d = _operator(ctx, geo, M, P, kind, kappa)
    o = oracle.Problem(geo, M, P, kind, kappa=kappa, np_=6)
    comps = [(0, 0), (0, 1), (1, 0), (1, 1)] if kind == 2 else [(0, 0)]
    dense = [i for i, lv in enumerate(d.leaves()) if lv[0] == 2]
    assert dense
    for li in dense:
        for rc, cc in comps:
            a, b = d.leaf_block(li, rc, cc), o.leaf_matrix(li, rc, cc)
            assert np.linalg.norm(a - b) <= FP64_TOL * max(np.linalg.norm(b), 1e-300), (li, rc, cc)
