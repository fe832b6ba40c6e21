"""facet2facet on inputs of at most four channels (its own fp32 kernels) against the fp64 formula: every channel count, basis
counts that are no multiple of four, output counts around the kernels' groups, faces without samples and face counts around a tile."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,cin,cout,F", [(4096, 3, 32, 16), (4097, 1, 4, 1), (4159, 2, 16, 9), (4223, 3, 33, 25), (4351, 4, 28, 32),
                                            (4353, 3, 48, 16), (5000, 3, 100, 9), (4500, 1, 130, 25), (4200, 3, 7, 7), (8193, 3, 64, 25),
                                            (90000, 3, 32, 16), (4099, 3, 16, 8), (4101, 3, 33, 8), (4096, 3, 32, 12), (4200, 3, 64, 12),
                                            (4111, 3, 12, 4), (4111, 3, 11, 16), (4105, 3, 33, 16)])
def test_small_inputs(nf, cin, cout, F):
    from picassoplus_b200.mesh.pi_modules import conv3d
    g = torch.Generator(device="cuda").manual_seed(nf + F)
    counts = torch.randint(0, 5, (nf,), device="cuda", generator=g)
    cum = counts.cumsum(0).to(torch.int32)
    n = int(cum[-1])
    x = torch.randn(n, cin, device="cuda", generator=g)
    b = torch.randn(n, F, device="cuda", generator=g)
    w = torch.randn(cout, cin, F, device="cuda", generator=g)
    go = torch.randn(nf, cout, device="cuda", generator=g)
    owner = torch.repeat_interleave(torch.arange(nf, device="cuda"), counts)
    A = torch.zeros(nf, F, cin, dtype=torch.float64, device="cuda").index_add_(0, owner, b.double()[:, :, None] * x.double()[:, None, :])
    A /= counts.clamp(min=1).double()[:, None, None]
    want = torch.einsum("fdc,ocd->fo", A, w.double())
    out = conv3d.facet2facet_forward(x, w, b, cum)
    assert rel_err(out, want) <= 1e-5
    gin, gf = conv3d.facet2facet_backward(go, x, w, b, cum)
    assert rel_err(gf, torch.einsum("fo,fdc->ocd", go.double(), A)) <= (1e-5 if cin * cout * F <= 3600 else 2e-5)
    again = conv3d.facet2facet_backward(go, x, w, b, cum)
    assert torch.equal(gf, again[1]) and torch.equal(out, conv3d.facet2facet_forward(x, w, b, cum))
