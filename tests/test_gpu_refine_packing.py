"""The refinement kernels pack the quads of a CTA's FP64 work: a quad's
results do not depend on how many others share its CTA."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _inputs(n, seed=7):
    g = torch.Generator(device="cpu").manual_seed(seed)
    img = torch.rand((203, 317), generator=g).cuda()
    centre = torch.rand((n, 1, 2), generator=g) * torch.tensor([280.0, 170.0]) + 15.0
    square = torch.tensor([[-1.0, -1.0], [1.0, -1.0], [1.0, 1.0], [-1.0, 1.0]])
    corners = centre + square * (4.0 + 10.0 * torch.rand((n, 1, 1), generator=g)) + torch.rand((n, 4, 2), generator=g)
    return img, corners.cuda(), torch.randn((n, 4, 2), generator=g).cuda(), torch.randn((n, 4), generator=g).cuda()


# below, at and above one quad per CTA (four CTAs per SM), a last CTA that is
# part full, and the most quads a CTA takes
@pytest.mark.parametrize("n", [1, 607, 1217, 4863, 5003])
def test_results_do_not_depend_on_the_packing(n):
    from atag import refine
    img, corners, g_ref, g_res = _inputs(n)
    whole = refine.refine_forward(img, corners) + refine.refine_backward(img, corners, g_ref, g_res)[:2]
    parts = []
    for i in range(0, n, 500):  # one quad per CTA
        c = corners[i:i + 500]
        parts.append(refine.refine_forward(img, c) +
                     refine.refine_backward(img, c, g_ref[i:i + 500], g_res[i:i + 500])[:2])
    for k, name in enumerate(("refined", "residual", "samples", "grad corners", "grad samples")):
        assert torch.equal(whole[k], torch.cat([p[k] for p in parts])), name
    none_res = refine.refine_backward(img, corners, g_ref, None)[0]
    zero_res = refine.refine_backward(img, corners, g_ref, torch.zeros_like(g_res))[0]
    assert torch.equal(none_res, zero_res)
