"""F2FConv3d on colours (three channels, 4 or 16 bases: its own kernels with the layer's epilogue and prologue) against the same layer in
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
            # without the activation there is nothing to fall on another side: sums of nf terms in fp32
            assert rel(a, b) <= (3e-3 if act else 1e-5), k
    again = torch.autograd.grad(conv(x, bary, counts), params + ([x] if grad_in else []), up)
    assert all(torch.equal(a, b) for a, b in zip(grads, again))


@pytest.mark.parametrize("F", [4, 8, 12, 16])
@pytest.mark.parametrize("cout", [3, 4, 16, 33, 68, 75])
def test_layer_entries(F, cout):
    """The layer's C entries: bias, ReLU and statistics of the forward pass, the bias gradient of the fused gradient, on either side of
    the sizes that have kernels of their own."""
    import ctypes
    from picassoplus_b200 import _lib
    from picassoplus_b200.topology import ptr, stream_ptr
    nf, fp32 = 4099, _lib.PREC_FP32
    g = torch.Generator(device="cuda").manual_seed(F + cout)
    counts = torch.randint(0, 4, (nf,), device="cuda", generator=g)
    cum = counts.cumsum(0).int()
    n = int(cum[-1])
    x, b = torch.rand(n, 3, device="cuda", generator=g), torch.randn(n, F, device="cuda", generator=g)
    w, bias = torch.randn(cout, 3, F, device="cuda", generator=g), torch.randn(cout, device="cuda", generator=g)
    owner = torch.repeat_interleave(torch.arange(nf, device="cuda"), counts)
    A = torch.zeros(nf, F, 3, dtype=torch.float64, device="cuda").index_add(0, owner, b.double()[:, :, None] * x.double()[:, None, :])
    A = A / counts.clamp(min=1).double()[:, None, None]
    want = torch.relu(torch.einsum("fdc,ocd->fo", A, w.double()) + bias.double())
    need = _lib.query("pb200_facet2facet_forward_workspace_bytes", nf, n, 3, cout, F, fp32)
    ws, act = torch.empty(need, dtype=torch.uint8, device="cuda"), torch.empty(nf, cout, device="cuda")
    partial = torch.empty(_lib.query("pb200_norm_parts", nf, cout), 3, cout, device="cuda")
    parts = ctypes.c_int(0)
    s = stream_ptr(x.device)
    _lib.call("pb200_facet2facet_layer_forward", nf, n, 3, cout, F, ptr(x), ptr(w), ptr(b), ptr(cum), ptr(bias), 1, ptr(act), ptr(partial),
              ctypes.addressof(parts), fp32, ptr(ws), need, s)
    assert rel(act, want) <= 1e-5 and 0 < parts.value <= partial.shape[0]
    count, mean, m2 = partial[:parts.value].double().unbind(1)
    assert bool((count.sum(0) == nf).all())
    whole = (count * mean).sum(0) / nf
    assert rel(whole, want.mean(0)) <= 1e-5 and rel(m2.sum(0) + (count * (mean - whole) ** 2).sum(0), want.var(0, correction=0) * nf) <= 1e-5
    fused = _lib.query("pb200_facet2facet_layer_gradient_fused", nf, n, 3, cout, F, ptr(b), fp32)
    assert fused == (F in (4, 16) and cout != 3 and cout != 68)
    if fused:
        go = torch.randn(nf, cout, device="cuda", generator=g)
        need = _lib.query("pb200_facet2facet_layer_filter_gradient_workspace_bytes", nf, cout, F)
        ws, gf, gb = torch.empty(need, dtype=torch.uint8, device="cuda"), torch.empty_like(w), torch.empty_like(bias)
        _lib.call("pb200_facet2facet_layer_filter_gradient", nf, n, 3, cout, F, ptr(go), ptr(act), 1, None, ptr(x), ptr(b), ptr(cum), ptr(gf),
                  ptr(gb), fp32, ptr(ws), need, s)
        masked = go.double() * (act > 0)                        # by the activations that it is given
        assert rel(gf, torch.einsum("fo,fdc->ocd", masked, A)) <= 1e-5 and rel(gb, masked.sum(0)) <= 1e-5
