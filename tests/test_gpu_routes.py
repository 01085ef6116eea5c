"""Routes that a rule on sizes chooses: each against the oracle or, where the
arithmetic is the same, bit for bit against the route beside it."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


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
