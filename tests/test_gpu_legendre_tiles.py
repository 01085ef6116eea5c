"""The FP64 Legendre kernels at the edges of their tiles, against the CPU
oracle: rows of 128 l, 64 and 32 nodes, groups of 8 planes in blocks of 16 and
32, K tiles of 16 nodes or degrees -- just under, at and past each."""
import numpy as np
import pytest

from oracle import oracle as O
from tests._helpers import check, random_spec, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-12  # the FP64 bound of the transform tests


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


# lmax + 1 = 2 degrees, 16 and 17 (a K tile), 63 to 65, 128 to 130 (row blocks,
# with nlat / 2 at, under and past 16, 32 and 64 nodes); planes 2, 7, 8, 9,
# 16, 17, 33 (groups and blocks of planes)
@pytest.mark.parametrize("lmax,nlat,nz", [(1, 4, 8), (3, 6, 9), (15, 32, 7), (16, 36, 17), (31, 64, 16),
                                          (62, 98, 2), (63, 128, 3), (64, 130, 33), (127, 192, 2), (128, 198, 2),
                                          (129, 200, 2)])
def test_legendre_tile_edges(lmax, nlat, nz):
    from redondito_b200 import sphp as S
    nphi = max(8, 2 * nlat)
    P = O.Plan(lmax, nz, nlat=nlat, nphi=nphi)
    G = S.Plan(lmax, nz, nlat=nlat, nphi=nphi)
    rng = np.random.default_rng(lmax + 31 * nz)
    q, s, t = (random_spec(P, rng, radial=False) for _ in range(3))
    s[:, 0] = t[:, 0] = 0.0
    ref = P.qst_synthesis(q, s, t)
    g = [G.new_grid() for _ in range(3)]
    S.fftp2d_qst_to_vec(G, dev(q), dev(s), dev(t), *g)
    for k, (x, r) in enumerate(zip(g, ref)):
        if np.linalg.norm(r):
            check(rel_l2(x.cpu().numpy(), r), TOL, f"lmax {lmax} synthesis {k}")
        else:
            assert not x.any()
    c = [G.new_spec() for _ in range(3)]
    S.fftp2d_vec_to_qst(G, *(dev(r) for r in ref), *c)
    for k, (x, r) in enumerate(zip(c, P.qst_analysis(*ref))):
        if np.linalg.norm(r):
            check(rel_l2(x.cpu().numpy(), r), TOL, f"lmax {lmax} analysis {k}")
        else:
            assert not x.any()
    G.close()
