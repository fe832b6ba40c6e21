"""torch.inference_mode.  Training on meshes that an evaluation under it has seen first: what is kept between calls (adjacency,
clusters, groupings, per-face means, basis tables) is made of ordinary tensors and can be saved for a backward pass.  Index tensors
made under it count no versions: their structures are made anew on every call."""
import pytest
import torch

from cases import pcloud_inputs
from picassoplus_b200 import synth

pytestmark = pytest.mark.gpu


def test_training_after_an_evaluation():
    from picassoplus_b200 import math_utils, topology
    from picassoplus_b200.block import conv_block
    from picassoplus_b200.math_utils import sph_harm_coeff
    from picassoplus_b200.mesh.layers import GlobalPool3d, Pool3d, Unpool3d, V2VConv3d
    from picassoplus_b200.mesh.utils import MeshHierarchy
    from picassoplus_b200.point.layers import PCloudConv3d
    torch.manual_seed(1)
    v, f = synth.icosphere(2)
    vertex, face = torch.from_numpy(v).float().cuda(), torch.from_numpy(f).int().cuda()
    nv, mf = (torch.tensor([n], dtype=torch.int32, device="cuda") for n in (len(v), len(f)))
    counts = torch.randint(1, 4, (len(f),), device="cuda", dtype=torch.int32)
    cum = counts.cumsum(0, dtype=torch.int32)
    bary = torch.randn(int(cum[-1]), 9, device="cuda")
    vt_map = torch.arange(len(v), dtype=torch.int32, device="cuda")
    prep = topology.prepare_level(vertex, face, vt_map, len(v), 2)
    levels = MeshHierarchy([4], [8], True, 1.0)(vertex, face, nv, mf)
    eye = sph_harm_coeff(2, torch.eye(3, device="cuda"))
    conv = V2VConv3d(16, [16, 16], 2, [1, 1]).cuda().eval()
    w = [torch.randn(*s, device="cuda", requires_grad=True) for s in ((9, 16), (16, 16, 9), (9, 16, 1))]
    x = torch.randn(len(v), 16, device="cuda", requires_grad=True)
    d = {k: (t.cuda() if isinstance(t, torch.Tensor) else t) for k, t in pcloud_inputs(500, 300, 12, 17, 16, 1, 3, seed=23).items()}
    points = PCloudConv3d(16, 24, 17).cuda().eval()

    def run():
        y = conv(x, face, prep["nf_count"], vt_map, prep["coeff"])
        y = conv_block(y, *w, face, cum, bary, prep["coeff"], prep["nf_count"], vt_map, eye)
        coarse = Pool3d("max")(y, levels[1][5], levels[1][6], levels[1][0]) + Pool3d("avg")(y, levels[1][5], levels[1][6], levels[1][0])
        y = y + Unpool3d()(coarse, levels[1][5], levels[1][6])
        z = points(d["x"], d["nn_count"], d["nn_index"], d["bin_index"], d["bin_coeff"])
        return GlobalPool3d("avg")(y, nv).sum() + z.sum()
    leaves = [x, *w, *conv.parameters(), *points.parameters()]
    d["x"].requires_grad_()

    topology.clear_cache()
    math_utils._corners.clear()
    with torch.inference_mode():
        seen = run()
    got = torch.autograd.grad(run(), leaves + [d["x"]])
    topology.clear_cache()
    math_utils._corners.clear()
    loss = run()
    want = torch.autograd.grad(loss, leaves + [d["x"]])
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert abs(float(seen) - float(loss.detach())) <= 1e-4 * abs(float(seen)) + 1e-2      # running statistics inside or behind the kernel


def test_counts_made_under_inference_mode():
    from picassoplus_b200 import topology
    from picassoplus_b200.mesh.layers import GlobalPool3d
    pool, x = GlobalPool3d("avg"), torch.randn(10, 8, device="cuda")
    topology.clear_cache()
    with torch.inference_mode():
        nv = torch.tensor([4, 6], device="cuda", dtype=torch.int32)
        first = pool(x, nv)
        nv.copy_(torch.tensor([3, 7], dtype=torch.int32))
        second = pool(x, nv)
    for got, n in ((first, 4), (second, 3), (pool(x, nv), 3)):
        assert torch.allclose(got, torch.stack([x[:n].mean(0), x[n:].mean(0)]), atol=1e-6)
    assert topology.cache_stats()["slots"] == 0
