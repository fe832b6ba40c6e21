"""F2FConv3d on colours (three channels, bases in quads: its own kernels with the layer's epilogue and prologue) against the same layer in
fp64: output counts around a warp and two outputs per lane, faces without samples and with more than are loaded ahead, face counts
around a batch of eight, with and without normalisation and activation, samples that need a gradient (the separate kernels) and
weights that lie off 16 bytes."""
import pytest
import torch

from picassoplus_b200.mesh.layers import F2FConv3d

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = a.detach(), b.detach()
    return float((a.double() - b.double()).norm() / (b.double().norm() + 1e-30))


@pytest.mark.parametrize("nf,cout,L,with_bn,act", [(4096, 32, 3, True, True), (4097, 16, 3, True, True), (4103, 33, 3, True, True),
                                                   (5001, 17, 3, True, False), (4104, 48, 3, False, True), (4100, 64, 3, True, True),
                                                   (4099, 70, 3, False, False), (6007, 32, 1, True, True), (4110, 65, 1, True, True),
                                                   (50001, 32, 3, True, True), (4101, 3, 3, True, True)])
@pytest.mark.parametrize("grad_in,offset", [(False, 0), (True, 0), (False, 1)])
def test_layer(nf, cout, L, with_bn, act, grad_in, offset):
    g = torch.Generator(device="cuda").manual_seed(nf + cout)
    torch.manual_seed(nf)
    F = (L + 1) ** 2
    counts = torch.randint(0, 4, (nf,), device="cuda", generator=g)
    counts[torch.randint(0, nf, (nf // 50,), device="cuda", generator=g)] = 9
    counts = counts.int()
    n = int(counts.sum())
    x = torch.rand(n, 3, device="cuda", generator=g).requires_grad_(grad_in)
    bary = torch.randn(n * F + offset, device="cuda", generator=g)[offset:].view(n, F)
    up = torch.randn(nf, cout, device="cuda", generator=g)
    conv = F2FConv3d(3, cout, L, activation_fn=torch.nn.ReLU() if act else None, with_bn=with_bn).cuda().train()
    params = list(conv.parameters())
    for p in params:
        p.data += 0.1 * torch.randn(p.shape, device="cuda", generator=g)
    out = conv(x, bary, counts)
    grads = torch.autograd.grad(out, params + ([x] if grad_in else []), up)

    # the layer in fp64: named parameters by shape, filter first
    ref = {k: v.detach().double().requires_grad_() for k, v in conv.named_parameters()}
    xd = x.detach().double().requires_grad_()
    owner = torch.repeat_interleave(torch.arange(nf, device="cuda"), counts.long())
    A = torch.zeros(nf, F, 3, dtype=torch.float64, device="cuda").index_add(0, owner, bary.double()[:, :, None] * xd[:, None, :])
    A = A / counts.clamp(min=1).double()[:, None, None]
    y = torch.einsum("fdc,ocd->fo", A, ref["weights"]) + ref["biases"].reshape(-1)
    if act:
        y = torch.relu(y)
    if with_bn:
        bn = next(k[:-len(".weight")] for k in ref if k.endswith(".weight"))
        y = torch.nn.functional.batch_norm(y, None, None, ref[bn + ".weight"], ref[bn + ".bias"], True, 0.0, conv.get_submodule(bn).eps)
    want = torch.autograd.grad(y, list(ref.values()) + ([xd] if grad_in else []), up.double())
    # a pre-activation within 1e-6 of zero may fall on either side: about that share of entries, its square root in the gradients
    assert rel(out, y) <= 1e-5
    for (k, _), a, b in zip(list(conv.named_parameters()) + [("x", None)], grads, want):
        if k == "biases" and with_bn and not act:
            # the batch's mean takes a bias out again: zero, up to the rounding of nf terms of unit size
            assert float(a.abs().max()) <= nf * 2.0 ** -24
        else:
            assert rel(a, b) <= 3e-3, k
    again = torch.autograd.grad(conv(x, bary, counts), params + ([x] if grad_in else []), up)
    assert all(torch.equal(a, b) for a, b in zip(grads, again))
