"""Layers and operators under what torch wraps around calls: tracing, forward mode, hooks on saved tensors, checkpointing, functional
transforms.  The result is right or the call is refused; a native node is never silently outside."""
import pytest
import torch
import torch.autograd.forward_ad as fwd
import torch.nn as nn
from torch.utils.checkpoint import checkpoint

from cases import conv_inputs, pcloud_inputs

pytestmark = [pytest.mark.gpu, pytest.mark.filterwarnings("ignore")]       # the tracer's warnings: sizes are constants to it
KINDS = ["rows", "mesh", "facet", "point", "block", "shared", "pool_max", "pool_avg", "unpool", "mean"]


class Call(nn.Module):
    """One call as a module of its feature rows, everything else fixed."""

    def __init__(self, kind):
        super().__init__()
        from picassoplus_b200 import topology
        from picassoplus_b200.math_utils import sph_harm_coeff
        from picassoplus_b200.mesh import utils as mesh_utils
        from picassoplus_b200.mesh.layers import F2FConv3d, PerItemConv3d, V2VConv3d
        from picassoplus_b200.point.layers import PCloudConv3d
        torch.manual_seed(5)
        on = lambda d: {k: (v.cuda() if isinstance(v, torch.Tensor) else v) for k, v in d.items()}      # noqa: E731
        self.kind = kind
        d = self.d = on(conv_inputs("ico2x3", 32, 1, 16, 24, seed=13, zero_sample_faces=False))
        nv = d["x_v"].shape[0]
        self.vt = torch.arange(nv, dtype=torch.int32, device="cuda")
        self.nfc = mesh_utils.count_vertex_adjface(d["face"], self.vt, d["vertex"])
        self.x = d["x_v"]
        if kind == "rows":
            self.m = PerItemConv3d(32, 24)
        elif kind == "mesh":
            self.m = V2VConv3d(32, [40, 24], 3, [1, 1])
        elif kind == "facet":
            self.m, self.x = F2FConv3d(32, 24, 3), d["tex"]
        elif kind == "point":
            self.q = on(pcloud_inputs(500, 300, 12, 17, 16, 1, 3, seed=23))
            self.m, self.x = PCloudConv3d(16, 24, 17), self.q["x"]
        elif kind == "block":
            self.w = nn.ParameterList([nn.Parameter(torch.randn(*s) * 0.1) for s in ((16, 32), (64, 32, 16), (16, 64, 1))])
            self.eye = sph_harm_coeff(3, torch.eye(3, device="cuda"))
        elif kind == "shared":
            self.x = d["x_f"]
        if kind in ("block", "shared"):
            self.means = topology.face_means(d["bary"], d["cum"])
        # clusters of up to three vertices in a row
        first = torch.arange(0, nv, 3, dtype=torch.int32, device="cuda")
        self.rep = -(self.vt // 3 * 3)
        self.rep[first.long()] = torch.minimum(first + 2, torch.tensor(nv - 1, device="cuda", dtype=torch.int32)) - first
        self.map = torch.full_like(self.vt, -1)
        self.map[first.long()] = torch.arange(first.shape[0], dtype=torch.int32, device="cuda")
        self.coarse = torch.zeros(first.shape[0], 3, device="cuda")
        if kind == "unpool":
            self.x = torch.randn(first.shape[0], 8, device="cuda")
        self.rep[0] = 0                       # (vertex 0 cannot be a representative: -0 is 0)
        self.rep[1] = self.rep[2] = 0
        self.counts = torch.tensor([nv - 10, 10], dtype=torch.int32, device="cuda")
        self.cuda().eval()

    def forward(self, x):
        from picassoplus_b200.block import conv_block, facet2facet_shared_rows
        from picassoplus_b200.mesh.layers import GlobalPool3d, Pool3d, Unpool3d
        d, kind = self.d, self.kind
        if kind == "rows":
            return self.m(x)
        if kind == "mesh":
            return self.m(x, d["face"], self.nfc, self.vt, d["coeff"])
        if kind == "facet":
            return self.m(x, d["bary"], d["counts"])
        if kind == "point":
            return self.m(x, *(self.q[k] for k in ("nn_count", "nn_index", "bin_index", "bin_coeff")))
        if kind == "block":
            return conv_block(x, *self.w, d["face"], d["cum"], self.means, d["coeff"], self.nfc, self.vt, self.eye)
        if kind == "shared":
            return facet2facet_shared_rows(x, d["filt_f2f"], self.means, d["cum"])
        if kind == "unpool":
            return Unpool3d()(x, self.rep, self.map)
        if kind == "mean":
            return GlobalPool3d("avg")(x, self.counts)
        return Pool3d(kind[5:])(x, self.rep, self.map, self.coarse)


def close(a, b):
    return float((a - b).norm() / b.norm()) <= 5e-5         # products of bf16 hi + lo pairs in one, fp32 in the other


@pytest.mark.parametrize("kind", KINDS)
def test_tracing(kind):
    """The traced call computes from its argument, it does not return what it returned while it was traced."""
    from picassoplus_b200 import math_utils
    math_utils._corners.clear()
    call = Call(kind)
    with torch.no_grad():
        traced = torch.jit.trace(call, (call.x,), check_trace=False)
        other = torch.randn_like(call.x)
        assert close(traced(other), call(other)) and not close(traced(other), call(call.x))


@pytest.mark.parametrize("kind", KINDS)
def test_forward_mode(kind):
    """A tangent goes through (as a difference quotient has it) or the call is refused; it is never dropped."""
    call = Call(kind)
    x, t = call.x, torch.randn_like(call.x)
    with torch.no_grad():
        quotient = (call(x + 1e-2 * t) - call(x - 1e-2 * t)) / 2e-2
    with fwd.dual_level():
        try:
            tangent = fwd.unpack_dual(call(fwd.make_dual(x, t))).tangent
        except (RuntimeError, NotImplementedError):
            return
        assert tangent is not None and float((tangent.detach() - quotient).norm() / quotient.norm()) <= 0.1       # (ReLU kinks)
    assert kind in ("rows", "mean")


@pytest.mark.parametrize("kind", KINDS)
def test_functional_transforms_are_refused(kind):
    if kind == "mean":
        return                                              # torch's own operator there
    call = Call(kind)
    with pytest.raises(RuntimeError):
        torch.func.vmap(call)(torch.stack([call.x, call.x]))
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda x: call(x).sum())(call.x)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("train", [False, True])
def test_saved_tensors_elsewhere(kind, train):
    """Saved tensors kept on the host, forward passes repeated for the backward pass: gradients bit for bit."""
    call = Call(kind).train(train)
    x = call.x.clone().requires_grad_()
    leaves = [x, *call.parameters()]
    out = call(x)
    g = torch.randn_like(out)
    want = torch.autograd.grad(out, leaves, g)
    with torch.autograd.graph.save_on_cpu():
        out = call(x)
    for a, b in zip(torch.autograd.grad(out, leaves, g), want):
        assert torch.equal(a, b)
    for a, b in zip(torch.autograd.grad(checkpoint(call, x, use_reentrant=False), leaves, g), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("kind", ["facet", "point"])
def test_hooks_on_the_activation_run(kind):
    """Facet and point layers call their activation module; with a hook on it, or on all modules, they still do."""
    call = Call(kind)
    call.m.activation_fn = nn.ReLU()
    with torch.no_grad():
        want, seen = call(call.x), []
        handle = call.m.activation_fn.register_forward_hook(lambda module, args, out: seen.append(out))
        out = call(call.x)
        handle.remove()
        assert len(seen) == 1 and close(out, want) and bool((seen[0] >= 0).all())
        handle = nn.modules.module.register_module_forward_hook(lambda module, args, out: seen.append(type(module)))
        call(call.x)
        handle.remove()
        assert nn.ReLU in seen and nn.BatchNorm1d in seen
        n = len(seen)
        assert torch.equal(call(call.x), want) and len(seen) == n


@pytest.mark.parametrize("kind", ["rows", "mesh", "facet", "point"])
@pytest.mark.parametrize("train", [False, True])
def test_widths_of_bias_and_batch_norm(kind, train):
    """A batch norm or a bias of another width is refused, as the separate operators refuse it; one value of the bias stands for all."""
    call = Call(kind).train(train)
    layer = call.m.V2F_conv3d if kind == "mesh" else call.m
    bias, norm = layer.biases, layer.BatchNorm
    with torch.no_grad():
        bias.fill_(0.25)
        want = call(call.x)
        for width in (bias.shape[1] - 8, bias.shape[1] + 8):
            layer.BatchNorm = nn.BatchNorm1d(width).cuda().train(train)
            with pytest.raises(RuntimeError):
                call(call.x)
            layer.BatchNorm = norm
            layer.biases = nn.Parameter(torch.zeros(1, width, device="cuda"))
            with pytest.raises(RuntimeError):
                call(call.x)
            layer.biases = bias
    layer.biases = nn.Parameter(torch.full((1, 1), 0.25, device="cuda"))
    if not train:
        with torch.no_grad():
            assert torch.equal(call(call.x), want)
    out = call(call.x)
    g = torch.randn_like(out)
    got, = torch.autograd.grad(out, [layer.biases], g)
    layer.biases = bias
    each, = torch.autograd.grad(call(call.x), [bias], g)
    assert got.shape == (1, 1) and abs(float(got - each.sum())) <= 1e-3 * float(each.abs().sum())


@pytest.mark.parametrize("kind,name", [("mesh", "spatial_weights"), ("point", "depth_weights")])
def test_strided_weights(kind, name):
    """Weights that go into a torch product may have any strides (a transposed parameter, a slice of a larger one)."""
    call = Call(kind)
    layer = call.m.V2F_conv3d if kind == "mesh" else call.m
    w = getattr(layer, name)
    out = call(call.x)
    g = torch.randn_like(out)
    want, = torch.autograd.grad(out, [w], g)
    other = nn.Parameter(w.detach().t().contiguous().t())
    assert not other.is_contiguous()
    setattr(layer, name, other)
    got = call(call.x)
    assert close(got.detach(), out.detach()) and close(torch.autograd.grad(got, [other], g)[0], want)
