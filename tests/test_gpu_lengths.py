"""The general-length FFTs (fft_gen.cuh) against the CPU oracle: radial and
azimuthal lengths of every kind of factor -- one pass, several register
radices, a prime above the largest register radix alone, first, last and
twice, no register radix at all -- with part-full tiles of ring pairs and of
lm columns."""
import numpy as np
import pytest

from oracle import oracle as O
from tests._helpers import check, check_derivative, random_spec, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-12  # the FP64 bound of the transform tests


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


# nphi: 10 and 13 (one pass), 26, 74 = 2 37, 289 = 17 17, 323 = 17 19 (primes
# only), 520 = 8 5 13, 1100 and 1924 = 4 13 37 (2 and 1 ring pairs per tile);
# nlat / 2 = 3, 5, 13, ... leave the last tile of ring pairs part full
@pytest.mark.parametrize("lmax,nlat,nphi", [(3, 6, 10), (4, 10, 13), (7, 14, 26), (9, 26, 74), (9, 22, 289),
                                            (11, 18, 323), (15, 34, 520), (7, 10, 1100), (5, 10, 1924)])
@pytest.mark.parametrize("pairs", [0, 1])
def test_phi_lengths(lmax, nlat, nphi, pairs):
    from redondito_b200 import sphp as S
    P = O.Plan(lmax, 3, nlat=nlat, nphi=nphi)
    G = S.Plan(lmax, 3, nlat=nlat, nphi=nphi)
    S.set_tiles(G, ring_pairs=pairs)
    rng = np.random.default_rng(nphi)
    q, s, t = (random_spec(P, rng, radial=False) for _ in range(3))
    ref = P.qst_synthesis(q, s, t)
    g = [G.new_grid() for _ in range(3)]
    S.fftp2d_qst_to_vec(G, dev(q), dev(s), dev(t), *g)
    for x, r in zip(g, ref):
        check(rel_l2(x.cpu().numpy(), r), TOL, f"nphi {nphi} synthesis")
    c = [G.new_spec() for _ in range(3)]
    S.fftp2d_vec_to_qst(G, *(dev(r) for r in ref), *c)
    for x, r in zip(c, P.qst_analysis(*ref)):
        check(rel_l2(x.cpu().numpy(), r), TOL, f"nphi {nphi} analysis")
    G.close()


# nz: 31, 37 (one prime pass), 34 = 2 17, 39 = 13 3, 58 = 2 29, 90 = 10 9,
# 289 = 17 17, 323 = 17 19, 1024 (no continuation: too long for the oracle's
# derivative reference to stay within its bound); 10, 36 and 528 lm columns
@pytest.mark.parametrize("lmax,nz", [(3, 31), (7, 34), (7, 37), (31, 39), (31, 58), (7, 90), (3, 289), (3, 323),
                                     (7, 1024)])
@pytest.mark.parametrize("cols", [0, 2])
def test_z_lengths(lmax, nz, cols):
    from redondito_b200 import sphp as S
    nlat, nphi = O.nlat_for(lmax), 2 * O.nlat_for(lmax)
    C, d = (25, 5) if nz < 200 else (0, 0)
    P = O.Plan(lmax, nz, nlat=nlat, nphi=nphi, C=C, d=d)
    G = S.Plan(lmax, nz, nlat=nlat, nphi=nphi, Cz=C, oz=d)
    S.set_tiles(G, z_cols=cols)
    a = random_spec(P, np.random.default_rng(nz))
    x = dev(a)
    S.fftp1d_real_to_complex_z(G, x)
    f = P.z_forward(a)
    check(rel_l2(x.cpu().numpy(), f), TOL, f"nz {nz} forward")
    x = dev(f)
    S.fftp1d_complex_to_real_z(G, x)
    check(rel_l2(x.cpu().numpy(), P.z_inverse(f)), TOL, f"nz {nz} inverse")
    if C:
        b = G.new_spec()
        for order in (1, "dlr"):
            (S.dlr(G, dev(a), b) if order == "dlr" else S.derivr(G, dev(a), b, order, "r"))
            check_derivative(b.cpu().numpy(), P, a, order, f"nz {nz}")
        x = dev(a)
        S.fc_filter(G, x, "r")
        check(rel_l2(x.cpu().numpy(), P.fc_filter(a, "r")), 1e-11, f"nz {nz} filter")
    G.close()


# A mixed plan's radial transforms of FP64 arrays (the passes of
# fft_engine.cuh, odd primes one output per thread): 31 (one prime pass),
# 39 = 3 13, 58 = 2 29, 81 = 3^4 (one buffer), 90 = 2 9 5, 289 = 17 17
@pytest.mark.parametrize("nz", [31, 39, 58, 81, 90, 289])
@pytest.mark.parametrize("cols", [0, 2])
def test_z_lengths_mixed(nz, cols):
    from redondito_b200 import sphp as S
    lmax, nlat, nphi = 7, 24, 48
    C, d = (25, 5) if nz < 200 else (0, 0)
    P = O.Plan(lmax, nz, nlat=nlat, nphi=nphi, C=C, d=d)
    G = S.Plan(lmax, nz, nlat=nlat, nphi=nphi, Cz=C, oz=d, precision=S.SPH_MIXED)
    S.set_tiles(G, z_cols=cols)
    a = random_spec(P, np.random.default_rng(nz))
    x = dev(a)
    S.fftp1d_real_to_complex_z(G, x)
    f = P.z_forward(a)
    check(rel_l2(x.cpu().numpy(), f), TOL, f"nz {nz} forward")
    x = dev(f)
    S.fftp1d_complex_to_real_z(G, x)
    check(rel_l2(x.cpu().numpy(), P.z_inverse(f)), TOL, f"nz {nz} inverse")
    if C:
        b = G.new_spec()
        for order in (1, "dlr"):
            (S.dlr(G, dev(a), b) if order == "dlr" else S.derivr(G, dev(a), b, order, "r"))
            check_derivative(b.cpu().numpy(), P, a, order, f"nz {nz}")
    G.close()
