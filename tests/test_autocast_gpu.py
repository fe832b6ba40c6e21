"""The native layers under torch.autocast: autocast rounds torch's products to half precision, the kernels take none of it, so that
outputs and gradients are those without it, bit for bit, whichever of the two passes runs inside the region."""
import pytest
import torch

from cases import conv_inputs, pcloud_inputs

pytestmark = pytest.mark.gpu


def _mesh():
    d = conv_inputs("ico2x3", 32, 1, 16, 64, seed=13, zero_sample_faces=False)
    c = {k: (v.cuda() if isinstance(v, torch.Tensor) else v) for k, v in d.items()}
    nv = c["x_v"].shape[0]
    c["vt"] = torch.arange(nv, dtype=torch.int32, device="cuda")
    from picassoplus_b200.mesh import utils as mesh_utils
    c["nfc"] = mesh_utils.count_vertex_adjface(c["face"], c["vt"], c["vertex"])
    return c


def _case(kind):
    from picassoplus_b200.block import conv_block
    from picassoplus_b200.math_utils import sph_harm_coeff
    from picassoplus_b200.mesh.layers import F2FConv3d, PerItemConv3d, V2VConv3d
    from picassoplus_b200.point.layers import PCloudConv3d
    torch.manual_seed(5)
    if kind == "point":
        d = {k: (v.cuda() if isinstance(v, torch.Tensor) else v) for k, v in pcloud_inputs(500, 300, 12, 17, 16, 1, 3, seed=23).items()}
        m = PCloudConv3d(16, 24, 17).cuda()
        x = d["x"].requires_grad_()
        return lambda: m(x, d["nn_count"], d["nn_index"], d["bin_index"], d["bin_coeff"]), [x, *m.parameters()]
    c = _mesh()
    x = c["x_v"].requires_grad_()
    if kind == "rows":
        m = PerItemConv3d(32, 24).cuda()
        return lambda: m(x), [x, *m.parameters()]
    if kind == "mesh":
        m = V2VConv3d(32, [40, 24], 3, [1, 1]).cuda()
        return lambda: m(x, c["face"], c["nfc"], c["vt"], c["coeff"]), [x, *m.parameters()]
    if kind == "facet":
        m = F2FConv3d(3, 24, 3).cuda()
        counts = torch.diff(c["cum"], prepend=c["cum"].new_zeros(1))
        rgb = torch.rand(c["bary"].shape[0], 3, device="cuda")
        return lambda: m(rgb, c["bary"], counts), list(m.parameters())
    w = [(torch.randn(*s, device="cuda") * 0.1).requires_grad_() for s in ((16, 32), (64, 32, 16), (16, 64, 1))]
    eye = sph_harm_coeff(3, torch.eye(3, device="cuda"))
    return lambda: conv_block(x, *w, c["face"], c["cum"], c["bary"], c["coeff"], c["nfc"], c["vt"], eye), [x, *w]


@pytest.mark.parametrize("kind", ["point", "rows", "mesh", "facet", "block"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_same_under_autocast(kind, dtype):
    run, leaves = _case(kind)
    want = run()
    upstream = torch.randn_like(want)
    want_grads = torch.autograd.grad(want, leaves, upstream)
    for backward_inside in (False, True):
        with torch.autocast("cuda", dtype=dtype):
            out = run()
            if backward_inside:
                grads = torch.autograd.grad(out, leaves, upstream)
        if not backward_inside:
            grads = torch.autograd.grad(out, leaves, upstream)
        assert out.dtype == torch.float32 and torch.equal(out, want)
        assert all(torch.equal(a, b) for a, b in zip(grads, want_grads))


def test_foreign_tensors_are_refused():
    """Tensors of another type or on the host do not reach a kernel."""
    from picassoplus_b200 import _lib
    x, w = torch.randn(8, 16, device="cuda"), torch.randn(16, 8, device="cuda")
    norm = (0, None, None, None, None, None, 0.0, 0.0)
    _lib.ops.rows_layer(x, w, torch.zeros(1, 8, device="cuda"), True, *norm, 0)
    for bias in (torch.zeros(1, 8), torch.zeros(1, 8, device="cuda", dtype=torch.float16)):
        with pytest.raises(RuntimeError):
            _lib.ops.rows_layer(x, w, bias, True, *norm, 0)
