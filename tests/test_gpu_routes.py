"""Routes that a rule on sizes chooses: each against the oracle or, where the
arithmetic is the same, bit for bit against the route beside it."""
import numpy as np
import pytest

from oracle import oracle as O
from tests._helpers import check, random_spec, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-12  # the FP64 bound of the transform tests


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


# The inverse phi transforms with 2 ring pairs per tile on grids past the L2
# cache (40 planes: 286 MB of FP64 grids, 143 MB of float ones; nphi 384 at 80
# planes the same), where their launches hold fewer CTAs per SM: every plane
# as a call of 10 planes, far below it, gives it.
@pytest.mark.parametrize("form", ["fp64", "mixed", "f32"])
@pytest.mark.parametrize("nlat,nphi,nz", [(388, 768, 40), (388, 384, 80)])
def test_inverse_phi_past_l2(form, nlat, nphi, nz):
    from redondito_b200 import sphp as S
    lmax, few = 20, 10
    prec = S.SPH_FP64 if form == "fp64" else S.SPH_MIXED
    many, part = (S.Plan(lmax, n, nlat=nlat, nphi=nphi, precision=prec) for n in (nz, few))
    gen = torch.Generator(device="cuda").manual_seed(nphi)
    f32 = form == "f32"
    spec = [torch.randn((nz, many.nlm), generator=gen, device="cuda", dtype=torch.complex128) for _ in range(3)]
    if f32:
        spec = [x.to(torch.complex64) for x in spec]
    call = S.fftp2d_qst_to_vec_f32 if f32 else S.fftp2d_qst_to_vec
    g, h = ([P.new_grid32() if f32 else P.new_grid() for _ in range(3)] for P in (many, part))
    call(many, *spec, *g)
    for k in range(0, nz, few):
        call(part, *(x[k:k + few].contiguous() for x in spec), *h)
        for x, y in zip(g, h):
            assert torch.equal(x[k:k + few], y), f"planes {k}.."
    many.close()
    part.close()


# Tuned widths of the general radial lengths past the shared memory of two
# CTAs per SM: cut to it (58 at 64 columns, 400 at 8, 120 at 32), or, for 1024
# and 2048, the in-place passes at the full width.
@pytest.mark.parametrize("nz,cols", [(58, 64), (120, 32), (400, 8), (1024, 4), (2048, 2)])
@pytest.mark.parametrize("form", ["fp64", "mixed", "f32"])
def test_wide_slabs(nz, cols, form):
    from redondito_b200 import sphp as S
    lmax, nlat, nphi = 7, 24, 48
    P = O.Plan(lmax, nz, nlat=nlat, nphi=nphi)
    G, H, M = (S.Plan(lmax, nz, nlat=nlat, nphi=nphi, precision=p)
               for p in ((S.SPH_FP64, S.SPH_FP64, S.SPH_MIXED) if form == "fp64" else (S.SPH_MIXED,) * 3))
    S.set_tiles(G, z_cols=cols)
    a = random_spec(P, np.random.default_rng(nz))
    f32 = form == "f32"
    x, b, c = (dev(a.astype(np.complex64 if f32 else np.complex128)) for _ in range(3))
    tol = 1e-6 if f32 else TOL  # float arrays round to 6e-8
    call = lambda name: getattr(S, name + ("_f32" if f32 else ""))
    ref = P.z_forward(x.cpu().numpy().astype(np.complex128))
    call("fftp1d_real_to_complex_z")(G, x)
    check(rel_l2(x.cpu().numpy(), ref), tol, f"nz {nz} forward")
    ref = P.z_inverse(x.cpu().numpy().astype(np.complex128))
    call("fftp1d_complex_to_real_z")(G, x)
    check(rel_l2(x.cpu().numpy(), ref), tol, f"nz {nz} inverse")
    # the operators against the default width, whose engine is the same but
    # for the in-place derivatives: those are a mixed plan's, of FP64 arrays
    inplace = nz >= 1024 and form != "mixed"
    for name, args, plan in (("derivr", (2, "r"), M if inplace else H), ("dlr", (), H)):
        if inplace and f32 and name == "derivr":
            continue
        call(name)(G, b, x, *args)
        call(name)(plan, b, c, *args)
        assert torch.equal(x, c), name
    for plan in (G, H, M):
        plan.close()


# Azimuthal lengths past those that fit two ring pairs: 2048 and 4096 (the
# in-place engine where two buffers leave one ring pair), 4608 and 6400 (the
# longest) out of place, 6500 and 8192 whose two buffers do not fit; pairs 1 at
# 2048 goes out of place; nlat / 2 = 5 and 6 (1 and 2 ring pairs in place)
@pytest.mark.parametrize("nphi", [2048, 4096, 4608, 6400, 6500, 8192])
@pytest.mark.parametrize("nlat,pairs", [(10, 0), (12, 0), (12, 1)])
def test_long_phi_lengths(nphi, nlat, pairs):
    from redondito_b200 import sphp as S
    P = O.Plan(5, 2, nlat=nlat, nphi=nphi)
    G = S.Plan(5, 2, nlat=nlat, nphi=nphi)
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
