"""Point-cloud depthwise convolution (hard and fuzzy bins), called through the C ABI (via the
operator API that mirrors picasso/point/pi_modules/conv3d.py), against the fp64 oracle and the
reference's own CUDA kernels on identical seeded inputs; gate 1e-4 relative per tensor."""
import os

import numpy as np
import pytest
import torch

from cases import PCLOUD_GOLDEN_CASES, pcloud_inputs
from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-4

CASES = [
    # Np, Mp, knn, F, C, r, T (0 = hard bins), shuffle
    (200, 60, 12, 9, 6, 2, 0, False),
    (150, 80, 10, 17, 8, 1, 3, False),
    (3000, 1000, 24, 33, 64, 1, 3, True),
    (4000, 4000, 16, 17, 128, 1, 0, False),
    (64, 16, 40, 5, 3, 3, 2, True),
    (2500, 700, 20, 51, 32, 1, 3, True),       # eight lanes per point: four points to a warp
    (900, 300, 37, 25, 12, 1, 0, True),        # four channels per lane without the warp-cooperative walk
    (700, 200, 70, 140, 128, 1, 3, False),     # runs longer than a warp; a filter table the cooperative kernels decline
]


def _dev(d):
    return {k: (v.cuda() if isinstance(v, torch.Tensor) else v) for k, v in d.items()}


@pytest.mark.parametrize("Np,Mp,knn,F,C,r,T,shuffle", CASES)
def test_matches_oracle_and_reference(Np, Mp, knn, F, C, r, T, shuffle):
    from oracle import mesh_oracle as mo, ref_cuda as ref
    from picassoplus_b200.point.pi_modules import conv3d
    d = pcloud_inputs(Np, Mp, knn, F, C, r, T, seed=19, shuffle=shuffle)
    c = _dev(d)
    dbl = lambda t: None if t is None else t.double()                               # noqa: E731
    want = mo.pcloud_conv3d_forward(d["x"].double(), d["filt"].double(), d["nn_count"], d["nn_index"], d["bin_index"],
                                    dbl(d["bin_coeff"]))
    wgin, wgf = mo.pcloud_conv3d_backward(d["g_out"].double(), d["x"].double(), d["filt"].double(), d["nn_count"],
                                          d["nn_index"], d["bin_index"], dbl(d["bin_coeff"]))
    if T == 0:
        out = conv3d.SPH3D_forward(c["x"], c["filt"], c["nn_count"], c["nn_index"], c["bin_index"])
        gin, gf = conv3d.SPH3D_backward(c["g_out"], c["x"], c["filt"], c["nn_count"], c["nn_index"], c["bin_index"])
    else:
        out = conv3d.fuzzySPH3D_forward(c["x"], c["filt"], c["nn_count"], c["nn_index"], c["bin_index"], c["bin_coeff"])
        gin, gf = conv3d.fuzzySPH3D_backward(c["g_out"], c["x"], c["filt"], c["nn_count"], c["nn_index"], c["bin_index"],
                                             c["bin_coeff"])
    assert rel_err(out, want) <= TOL and rel_err(gin, wgin) <= TOL and rel_err(gf, wgf) <= TOL
    no_pairs = torch.bincount(d["nn_index"][:, 0].long(), minlength=Mp) == 0
    assert torch.all(out[no_pairs.cuda()] == 0)                  # output points without a neighbour stay exactly 0
    again = conv3d._backward(c["g_out"], c["x"], c["filt"], c["nn_count"], c["nn_index"], c["bin_index"], c["bin_coeff"])
    assert torch.equal(again[0], gin) and torch.equal(again[1], gf)                  # run to run identical
    if ref.available():
        r_out = ref.pcloud_forward(c["x"], c["filt"], c["nn_count"], c["nn_index"], c["bin_index"], c["bin_coeff"])
        r_gin, r_gf = ref.pcloud_backward(c["g_out"], c["x"], c["filt"], c["nn_count"], c["nn_index"], c["bin_index"],
                                          c["bin_coeff"])
        assert rel_err(out, r_out) <= TOL and rel_err(gin, r_gin) <= TOL and rel_err(gf, r_gf) <= TOL


@pytest.mark.parametrize("F,C,T", [
    (33, 256, 3), (33, 256, 0),          # vector kernels, a filter table of 34 KB beside the staged pairs
    (65, 128, 0), (65, 128, 3),          # cooperative kernels, 33 KB
    (12, 1024, 0),                       # the largest table and the widest rows: 48 KB, one group of lanes per block
    (17, 64, 3), (17, 64, 0), (9, 32, 2), (9, 48, 3),
    (9, 128, 5), (9, 20, 4),             # more bins than are staged
])
def test_input_points_with_many_pairs(F, C, T):
    """Padded neighbour lists name a few input points over and over: rows of 64 (walked with the others), 65, 256, 257, 300 and
    thousands of pairs, several of them in one block's range of points, one in another's."""
    from oracle import mesh_oracle as mo
    from picassoplus_b200.point.pi_modules import conv3d
    d = pcloud_inputs(2500, 600, 16, F, C, 1, T, seed=29, shuffle=True)
    n = d["nn_index"].shape[0]
    at = 0
    for point, pairs in ((0, 1500), (7, 64), (8, 65), (9, 256), (10, 257), (1023, 300), (2047, 100), (2499, 700)):
        d["nn_index"][:, 1][d["nn_index"][:, 1] == point] = 3
        d["nn_index"][at:at + pairs, 1] = point
        at += pairs
    assert at < n
    dbl = lambda t: None if t is None else t.double()                               # noqa: E731
    want_in, want_filter = mo.pcloud_conv3d_backward(d["g_out"].double(), d["x"].double(), d["filt"].double(), d["nn_count"],
                                                     d["nn_index"], d["bin_index"], dbl(d["bin_coeff"]))
    c = _dev(d)
    args = [c[k] for k in ("g_out", "x", "filt", "nn_count", "nn_index", "bin_index", "bin_coeff")]
    gin, gf = conv3d._backward(*args)
    assert rel_err(gin, want_in) <= 1e-5 and rel_err(gf, want_filter) <= 1e-5
    for point in (0, 8, 257, 2499):
        assert rel_err(gin[point], want_in[point]) <= 1e-4
    again = conv3d._backward(*args)
    assert torch.equal(again[0], gin) and torch.equal(again[1], gf)


def test_a_bad_index_that_only_the_backward_pass_looks_up():
    """An input point or vertex outside the range contributes nothing to a forward pass, under autograd or not; the backward pass, which
    sorts by it, refuses it."""
    from picassoplus_b200.mesh.layers import V2FConv3d
    from picassoplus_b200.mesh.pi_modules import conv3d as mesh_conv
    from picassoplus_b200.point.layers import PCloudConv3d
    from picassoplus_b200.point.pi_modules import conv3d
    d = _dev(pcloud_inputs(200, 60, 12, 9, 8, 1, 0, seed=3))
    layer, x, w = PCloudConv3d(8, 16, 9).cuda().eval(), d["x"].requires_grad_(), torch.randn(9, 8, 1, device="cuda", requires_grad=True)
    d["nn_index"][5, 1] = 200
    pairs = d["nn_count"], d["nn_index"], d["bin_index"]
    face = torch.randint(0, 200, (50, 3), dtype=torch.int32, device="cuda")
    face[7, 2] = 200
    faces, f = V2FConv3d(8, 16, 2).cuda().eval(), torch.randn(3, 8, 1, device="cuda", requires_grad=True)
    for call in (lambda: layer(x, *pairs), lambda: conv3d.conv3d(x, w, *pairs), lambda: faces(x, face), lambda: mesh_conv.vertex2facet(x, f, face)):
        with torch.no_grad():
            want = call()
        out = call()
        assert rel_err(out, want) <= 1e-5
        with pytest.raises(RuntimeError, match="outside"):
            torch.autograd.grad(out, [x], torch.ones_like(out))
    for m, rest in ((layer, pairs), (faces, (face,))):        # also where only the layer's weights have a gradient
        with pytest.raises(RuntimeError, match="outside"):
            torch.autograd.grad(m(x.detach(), *rest).sum(), [m.depth_weights])


def test_pairs_and_faces_of_another_width_are_refused():
    """Rows of one or three indices are told before the grouping reads them as rows of two, faces of two or four before the adjacency
    reads them as triangles."""
    from picassoplus_b200.mesh.layers import F2VConv3d, V2FConv3d
    from picassoplus_b200.mesh.pi_modules import conv3d as mesh_conv
    from picassoplus_b200.point.layers import PCloudConv3d
    d = _dev(pcloud_inputs(200, 60, 12, 9, 8, 1, 0, seed=3))
    layer = PCloudConv3d(8, 16, 9).cuda()
    for index in (d["nn_index"][:, :1].contiguous(), torch.cat([d["nn_index"], d["nn_index"][:, :1]], 1)):
        with pytest.raises(RuntimeError, match="pairs, 2"):
            layer(d["x"], d["nn_count"], index, d["bin_index"])
    x, ones = torch.randn(30, 8, device="cuda"), torch.ones(30, dtype=torch.int32, device="cuda")
    for width in (2, 4):
        face = torch.zeros(20, width, dtype=torch.int32, device="cuda")
        rows, coeff = torch.randn(20, 8, device="cuda"), torch.rand(20, 9, device="cuda")
        for call in (lambda: V2FConv3d(8, 16, 2).cuda()(x, face), lambda: F2VConv3d(8, 16, 2).cuda()(rows, face, ones, ones * 0, coeff),
                     lambda: mesh_conv.vertex2facet(x.requires_grad_(), torch.randn(3, 8, 1, device="cuda"), face),
                     lambda: mesh_conv.facet2vertex(rows, torch.randn(9, 8, 1, device="cuda"), coeff, face, ones, ones * 0)):
            with pytest.raises(RuntimeError, match="NfIn, 3"):
                call()


@pytest.mark.parametrize("C", [32, 64, 128, 48])
@pytest.mark.parametrize("T", [0, 3])
def test_nan_reaches_every_bin_of_its_pairs(C, T):
    """A NaN row of the upstream gradient is in the filter gradient of all bins that its pairs name, those of weight 0 among them, and
    in no other; bins outside the table take no part."""
    from picassoplus_b200.point.pi_modules import conv3d
    d = pcloud_inputs(400, 200, 12, 17, C, 1, T, seed=31)
    if T:
        d["bin_coeff"][::2, 1] = 0
    d["bin_index"].view(-1)[::7] = 17
    d["bin_index"].view(-1)[3::7] = -1
    row = int(d["nn_index"][40, 0])
    d["g_out"][row] = float("nan")
    named = d["bin_index"][d["nn_index"][:, 0] == row].flatten()
    named = set(int(b) for b in named if 0 <= b < 17)
    c = _dev(d)
    _, gf = conv3d._backward(*[c[k] for k in ("g_out", "x", "filt", "nn_count", "nn_index", "bin_index", "bin_coeff")])
    assert len(named) < 17 and set(torch.isnan(gf).flatten(1).any(1).nonzero().flatten().tolist()) == named


@pytest.mark.parametrize("name", sorted(PCLOUD_GOLDEN_CASES))
def test_against_committed_reference_fixtures(name):
    from picassoplus_b200.point.pi_modules import conv3d
    z = np.load(os.path.join(os.path.dirname(__file__), "golden", name + ".npz"))
    c = _dev(pcloud_inputs(*PCLOUD_GOLDEN_CASES[name]))
    out = conv3d._forward(c["x"], c["filt"], c["nn_count"], c["nn_index"], c["bin_index"], c["bin_coeff"])
    gin, gf = conv3d._backward(c["g_out"], c["x"], c["filt"], c["nn_count"], c["nn_index"], c["bin_index"], c["bin_coeff"])
    assert rel_err(out, z["ref_out"]) <= TOL and rel_err(gin, z["ref_gin"]) <= TOL and rel_err(gf, z["ref_gf"]) <= TOL


def test_module_and_autograd():
    """PCloudConv3d (fuzzy bins) through torch autograd against the oracle composition in fp64."""
    from oracle import mesh_oracle as mo
    from picassoplus_b200.point.layers import PCloudConv3d
    d = pcloud_inputs(500, 300, 12, 17, 16, 2, 3, seed=23)
    c = _dev(d)
    torch.manual_seed(0)
    mod = PCloudConv3d(16, 24, 17, depth_multiplier=2, with_bn=False).cuda()
    x = c["x"].clone().requires_grad_()
    y = mod(x, c["nn_count"], c["nn_index"], c["bin_index"], c["bin_coeff"])
    G = torch.randn_like(y)
    (y * G).sum().backward()
    P = lambda t: t.detach().cpu().double()                                          # noqa: E731
    xo, sw = P(d["x"]).requires_grad_(), P(mod.spatial_weights).requires_grad_()
    f = mo.pcloud_conv3d_forward(xo, sw, d["nn_count"], d["nn_index"], d["bin_index"], d["bin_coeff"].double())
    yo = torch.relu(f @ P(mod.depth_weights) + P(mod.biases))
    (yo * P(G)).sum().backward()
    assert rel_err(y, yo) <= TOL and rel_err(x.grad, xo.grad) <= TOL and rel_err(mod.spatial_weights.grad, sw.grad) <= TOL
