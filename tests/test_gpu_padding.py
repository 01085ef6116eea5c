"""The node columns past nlat/2 of the folded coefficients (their stride is
nlat/2 rounded up to 4) hold whatever an earlier call left there: a call's
results may not depend on them.  A plan that has transformed infinite and
undefined values gives, for finite input, the values of a fresh plan."""
import numpy as np
import pytest

from oracle import oracle as O
from tests._helpers import random_spec

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def analyse(S, G, grids):
    q, s, t = (G.new_spec() for _ in range(3))
    S.fftp2d_vec_to_qst(G, *grids, q, s, t)
    a = G.new_spec()
    S.fftp2d_real_to_complex_xy(G, grids[0], a)
    return [x.cpu().numpy() for x in (a, q, s, t)]


# nlat / 2 = 5, 6, 7 (3, 2, 1 columns past it) and 130
@pytest.mark.parametrize("lmax,nlat,nphi", [(3, 10, 12), (3, 12, 24), (7, 14, 26), (40, 260, 96)])
def test_finite_after_undefined(lmax, nlat, nphi):
    from redondito_b200 import sphp as S
    P = O.Plan(lmax, 9, nlat=nlat, nphi=nphi)
    rng = np.random.default_rng(nlat)
    ref = [dev(r) for r in P.qst_synthesis(*(random_spec(P, rng, radial=False) for _ in range(3)))]
    fresh = S.Plan(lmax, 9, nlat=nlat, nphi=nphi)
    used = S.Plan(lmax, 9, nlat=nlat, nphi=nphi)
    bad = [used.new_spec() for _ in range(3)]
    for x in bad:
        x.fill_(float("inf"))
    S.fftp2d_qst_to_vec(used, *bad, *(used.new_grid() for _ in range(3)))
    for k, (x, y) in enumerate(zip(analyse(S, used, ref), analyse(S, fresh, ref))):
        assert np.isfinite(y).all()
        np.testing.assert_array_equal(x, y, err_msg=f"output {k}")
    fresh.close()
    used.close()
