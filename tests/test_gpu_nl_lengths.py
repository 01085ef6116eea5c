"""The nonlinear step at general radial lengths (and nz 512, which has no
two-step kernel) against the CPU oracle."""
import numpy as np
import pytest

from oracle import extended as X
from oracle import oracle as O
from tests._helpers import check, random_spec, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-12  # the FP64 bound of the transform tests
TOL_MIXED, TOL_NL = 1e-6, 1e-5  # the mixed bounds: transforms, right-hand sides


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def radial_error(P, a):
    """The oracle's own error in the radial derivative and in D_l of a, and
    what becomes in them of a rounding of a (the fields they act on come from
    angular transforms)."""
    x1, x2 = (X.derivr_rows(P, a, o) for o in (1, 2))
    x2 = x2 - (P.ell * (P.ell + 1.0))[None, :] / np.asarray(P.z, dtype=X.L)[:, None] ** 2 * np.asarray(a, np.clongdouble)
    b = a * (1.0 + 2.0 ** -52 * np.random.default_rng(0).uniform(-1, 1, a.shape))
    return max(X.rel_l2(f(y), x) for f, x in ((lambda y: P.derivr(y, 1), x1), (P.dlr, x2)) for y in (a, b))


# 36, 90 = 10 9 (register radices), 58 = 2 29 (a prime alone), 99 = 9 11
# (odd), 81 (one buffer on a mixed plan); 2 and 16 lm columns per CTA
LENGTHS = [(36, 0), (58, 0), (58, 2), (81, 0), (90, 16), (99, 0), (121, 0)]


# nz 512 in FP64 only: its derivatives amplify the fp32 rounding of a mixed
# plan's planes past TOL_NL
@pytest.mark.parametrize("nz,cols,mixed", [(n, c, m) for n, c in LENGTHS for m in (False, True)] + [(512, 0, False)])
def test_nl_lengths(nz, cols, mixed):
    from redondito_b200 import sphp as S
    lmax, nlat, nphi = (3, 12, 24) if nz == 512 else (7, 24, 48)
    P = O.Plan(lmax, nz, nlat=nlat, nphi=nphi, C=25, d=5, rint=0.5, rext=1.5)
    G = S.Plan(lmax, nz, nlat=nlat, nphi=nphi, Cz=25, oz=5, rint=0.5, rext=1.5,
               precision=S.SPH_MIXED if mixed else S.SPH_FP64)
    S.set_tiles(G, z_cols=cols)
    S.setup_bc(G)
    rng = np.random.default_rng(nz)
    Z, W = (random_spec(P, rng, power=3.0) for _ in range(2))
    phi = P.dlr(W)
    steps = nz <= 121  # the oracle's boundary tables, and the boundary solve, end below 512
    if steps:
        P.bc_setup(("noslip", "noslip"), tables=X.bc_tables(P, ("noslip", "noslip")))
        Z, phi, W = P.imposebc(Z, phi)
    # FP64: both sides round their radial derivatives like the oracle's own,
    # ten at most in a right-hand side
    tol = TOL_NL if mixed else max(TOL, 10 * max(radial_error(P, a) for a in (Z, W, phi)))
    tol_e = TOL_MIXED if mixed else max(TOL, tol)
    rz_ref, rf_ref, e_ref = P.nl_rhs(Z, W, phi, 1e-3)
    rz, rf = G.new_spec(), G.new_spec()
    e = S.nl_rhs(G, dev(Z), dev(W), dev(phi), 1e-3, rz, rf)
    check(abs(e - e_ref) / e_ref, tol_e, f"nz {nz} energy")
    check(rel_l2(rz.cpu().numpy(), rz_ref), tol, f"nz {nz} rhs_z")
    check(rel_l2(rf.cpu().numpy(), rf_ref), tol, f"nz {nz} rhs_phi")
    if steps:
        ref = P.rk3_step(Z, W, phi, 1e-3, 1e-4)
        state = [dev(x) for x in (Z, W, phi)]
        e = S.rk3_step(G, *state, 1e-3, 1e-4)
        check(abs(e - ref[3]) / ref[3], tol_e, f"nz {nz} rk3 energy")
        for x, r, name in zip(state, ref, "ZWF"):
            check(rel_l2(x.cpu().numpy(), r), tol, f"nz {nz} rk3 {name}")
    S.plan_status(G)
    G.close()
