"""Batch normalisation inside the native layers and the per-sample mean, against torch in fp64 at the sizes where their
kernels' work split changes (one row per block, remainders of the unrolled loops, channels that are no multiple of four,
more than one chunk of 32 thread columns)."""
import pytest
import torch
import torch.nn as nn

from conftest import rel_err

pytestmark = pytest.mark.gpu


def norm_err(a, b):
    a, b = a.detach().double(), b.detach().double()
    return float((a - b).norm() / b.norm())


@pytest.mark.parametrize("rows,C", [(2, 8), (33, 5), (1000, 32), (4097, 100), (70001, 128), (513, 260)])
@pytest.mark.parametrize("relu", [True, False])
def test_rows_layer_with_batch_norm(rows, C, relu):
    """PerItemConv3d in training (two steps: running statistics), then in inference, forward and backward."""
    from picassoplus_b200.mesh.layers import PerItemConv3d
    torch.manual_seed(rows + C)
    m = PerItemConv3d(16, C, activation_fn=nn.ReLU() if relu else None).cuda().train()
    with torch.no_grad():
        m.biases.normal_(0, 0.3)
        m.BatchNorm.weight.uniform_(0.5, 1.5)
        m.BatchNorm.bias.normal_()
    bn = nn.BatchNorm1d(C, eps=1e-3).cuda().double().train()
    bn.load_state_dict(m.BatchNorm.state_dict())
    for step in range(2):
        x = (torch.randn(rows, 16, device="cuda") * 0.5 + 1.0).requires_grad_()
        g = torch.randn(rows, C, device="cuda")
        y = m(x)
        got = torch.autograd.grad(y, [x, m.weights, m.biases, m.BatchNorm.weight, m.BatchNorm.bias], g)
        xd = x.detach().double().requires_grad_()
        p = [t.detach().double().requires_grad_() for t in (m.weights, m.biases)]
        z = xd @ p[0] + p[1]
        # a pre-activation within rounding of zero may fall on either side of the ReLU: gradients get more room with it
        act = torch.relu(z) if relu else z
        want_y = bn(act)
        want = torch.autograd.grad(want_y, [xd, p[0], p[1], bn.weight, bn.bias], g.double())
        assert rel_err(y, want_y) <= 2e-4
        for i, (a, b) in enumerate(zip(got, want)):
            if rows > 2 and (relu or i != 2):       # two rows normalise to +-1: rounding noise; without ReLU the bias has no gradient
                assert norm_err(a, b) <= (2e-2 if relu else 1e-3)
    assert rel_err(m.BatchNorm.running_mean, bn.running_mean) <= 1e-4
    assert rel_err(m.BatchNorm.running_var, bn.running_var) <= 1e-4
    assert int(m.BatchNorm.num_batches_tracked) == 2
    m.eval(), bn.eval()
    x = torch.randn(rows, 16, device="cuda")
    z = x.double() @ m.weights.double() + m.biases.double()
    want = bn(torch.relu(z) if relu else z)
    with torch.no_grad():
        assert rel_err(m(x), want) <= 2e-4          # running statistics inside the kernel
    assert rel_err(m(x), want) <= 2e-4              # under autograd: the torch module behind the kernel


@pytest.mark.parametrize("rows,C", [(2, 3), (777, 12), (50000, 32)])
def test_facet_layer_statistics(rows, C):
    """F2FConv3d: bias, ReLU and statistics in one pass, running and batch statistics, data without gradient."""
    from picassoplus_b200.mesh.layers import F2FConv3d
    torch.manual_seed(rows)
    m = F2FConv3d(3, C, 2).cuda().train()
    counts = torch.randint(1, 4, (rows,), device="cuda", dtype=torch.int32)
    n = int(counts.sum())
    tex, bary = torch.rand(n, 3, device="cuda"), torch.randn(n, 9, device="cuda")
    seg = torch.repeat_interleave(torch.arange(rows, device="cuda"), counts)
    A = torch.zeros(rows, 9, 3, device="cuda", dtype=torch.float64).index_add_(0, seg, bary.double()[:, :, None] * tex.double()[:, None])
    z = torch.einsum("fdc,ocd->fo", A / counts[:, None, None], m.weights.double()) + m.biases.double()
    bn = nn.BatchNorm1d(C, eps=1e-3).cuda().double().train()
    want = bn(torch.relu(z))
    got = m(tex, bary, counts)
    assert rel_err(got, want) <= 1e-3 if rows == 2 else rel_err(got, want) <= 2e-4
    assert rel_err(m.BatchNorm.running_var, bn.running_var) <= 1e-4
    g = torch.randn(rows, C, device="cuda")
    gw, = torch.autograd.grad(got, [m.weights], g)
    if rows > 2:
        gw_want, = torch.autograd.grad(want, [m.weights], g.double())
        assert norm_err(gw, gw_want) <= 2e-2
    m.eval(), bn.eval()
    with torch.no_grad():
        assert rel_err(m(tex, bary, counts), bn(torch.relu(z))) <= 2e-4


@pytest.mark.parametrize("lengths,C", [([1], 1), ([5, 1, 1000, 3], 40), ([512, 512, 511, 513], 128), ([100] * 130, 33), ([70000], 4)])
def test_global_mean(lengths, C):
    from picassoplus_b200.mesh.layers import GlobalPool3d
    x = torch.randn(sum(lengths), C, device="cuda").requires_grad_()
    nv = torch.tensor(lengths, device="cuda", dtype=torch.int32)
    out = GlobalPool3d("avg")(x, nv)
    g = torch.randn_like(out)
    gx, = torch.autograd.grad(out, x, g)
    parts = torch.split(x.detach().double(), lengths)
    assert rel_err(out, torch.stack([p.mean(0) for p in parts])) <= 1e-5
    assert rel_err(gx, torch.repeat_interleave(g / nv[:, None], nv.long(), 0)) <= 1e-6
    with pytest.raises(RuntimeError):
        GlobalPool3d("avg")(x, nv + 1)
    with pytest.raises(RuntimeError):
        GlobalPool3d("avg")(x[:0], nv[:0])                  # no samples at all: torch's operator refuses them


@pytest.mark.parametrize("lengths", [[300, 900, 1200], [100, -4000, 500], [5000000, 1, 1], [-5, 1000, 5]])
def test_global_mean_of_wrong_counts_with_deferred_validation(lengths):
    """Counts that do not add up to the rows are reported at the next check; until then nothing behind the rows is read.
    (Samples in front of the first wrong row keep their mean while the totals rise; a negative count makes the search over them
    meaningless.)"""
    from picassoplus_b200 import topology
    from picassoplus_b200.mesh.layers import GlobalPool3d
    x = torch.randn(1000, 40, device="cuda").requires_grad_()
    nv = torch.tensor(lengths, device="cuda", dtype=torch.int32)
    topology.set_validation("deferred")
    try:
        out = GlobalPool3d("avg")(x, nv)
        torch.autograd.grad(out, x, torch.ones_like(out))
        if 0 < lengths[0] < 1000 and min(lengths) >= 0:
            assert rel_err(out[0], x[:lengths[0]].double().mean(0)) <= 1e-5
        with pytest.raises(RuntimeError, match="add up"):
            topology.check_deferred()
    finally:
        topology.set_validation("sync")


def test_global_mean_of_two_views_of_one_count_table():
    """Row and column of a table share address, length and storage; so do two types' views of one buffer."""
    from picassoplus_b200.mesh.layers import GlobalPool3d
    pool = GlobalPool3d("avg")
    x = torch.randn(10, 8, device="cuda")

    def want(lengths):
        return torch.stack([p.mean(0) for p in torch.split(x.double(), lengths)])
    table = torch.tensor([[3, 5, 2], [2, 1, 1], [5, 1, 1]], device="cuda", dtype=torch.int32)
    assert rel_err(pool(x, table[0]), want([3, 5, 2])) <= 1e-6
    assert rel_err(pool(x, table[:, 0]), want([3, 2, 5])) <= 1e-6
    table = torch.tensor([[3, 5, 2], [2, 1, 1], [4, 1, 1]], device="cuda", dtype=torch.int32)
    pool(x, table[0])
    with pytest.raises(RuntimeError, match="add up"):
        pool(x, table[:, 0])
    counts = torch.tensor([10, 0, 0], device="cuda", dtype=torch.int64)
    assert rel_err(pool(x, counts[:1]), want([10])) <= 1e-6
    assert rel_err(pool(x, counts.view(torch.int32)[:1]), want([10])) <= 1e-6
    ones = torch.full((5,), 2, device="cuda", dtype=torch.int32)
    assert rel_err(pool(x, ones), want([2] * 5)) <= 1e-6
    with pytest.raises(RuntimeError, match="add up"):
        pool(x, ones.view(torch.float32))


@pytest.mark.parametrize("frozen", [True, False])
@pytest.mark.parametrize("kind", ["rows", "facet", "mesh", "point"])
def test_inference_statistics_under_autograd(kind, frozen):
    """eval() with gradients on, the layer's own weights frozen or not: weight and bias of the batch norm have their gradients."""
    from cases import conv_inputs, pcloud_inputs
    from picassoplus_b200.mesh.layers import F2FConv3d, PerItemConv3d, V2FConv3d
    from picassoplus_b200.point.layers import PCloudConv3d
    torch.manual_seed(3)
    on = lambda d: {k: (v.cuda() if isinstance(v, torch.Tensor) else v) for k, v in d.items()}      # noqa: E731
    d = on(conv_inputs("ico2x3", 16, 1, 16, 24, seed=13))
    q = on(pcloud_inputs(500, 300, 12, 17, 16, 1, 3, seed=23))
    m, args = {"rows": (PerItemConv3d(16, 24), (d["x_v"],)), "facet": (F2FConv3d(16, 24, 3), (d["tex"], d["bary"], d["counts"])),
               "mesh": (V2FConv3d(16, 24, 3), (d["x_v"], d["face"])),
               "point": (PCloudConv3d(16, 24, 17), (q["x"], q["nn_count"], q["nn_index"], q["bin_index"], q["bin_coeff"]))}[kind]
    m = m.cuda()
    for _ in range(2):
        m(*args)                                            # running statistics
    m.eval()
    own = [p for n, p in m.named_parameters() if not n.startswith("BatchNorm")]
    for p in own:
        p.requires_grad_(not frozen)
    bn = m.BatchNorm
    out = m(*args)
    g = torch.randn_like(out)
    grads = torch.autograd.grad(out, [bn.weight, bn.bias] + ([] if frozen else own), g)
    with torch.no_grad():
        whole = m(*args)
    xhat = (out - bn.bias) / bn.weight
    assert rel_err(whole, out) <= 1e-5
    assert rel_err(grads[0], (g * xhat).sum(0)) <= 1e-4 and rel_err(grads[1], g.sum(0)) <= 1e-5
    assert all(bool(t.abs().sum() > 0) for t in grads)


@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("with_bn", [True, False])
@pytest.mark.parametrize("kind", ["facet", "point"])
def test_nan_and_infinity_spread_as_in_torch(kind, with_bn, value):
    """One bad value in the input: the native layer's outputs and gradients are NaN, infinite or finite where those of the separate
    operators are (ReLU lets a NaN through in both directions)."""
    from cases import conv_inputs, pcloud_inputs
    from picassoplus_b200.mesh import layers
    from picassoplus_b200.point.layers import PCloudConv3d
    torch.manual_seed(3)
    on = lambda d: {k: (v.cuda() if isinstance(v, torch.Tensor) else v) for k, v in d.items()}      # noqa: E731
    if kind == "facet":
        d = on(conv_inputs("ico2x3", 16, 1, 16, 24, seed=13))
        x = d["tex"]
        m, args = layers.F2FConv3d(16, 24, 3, with_bn=with_bn), (d["bary"], d["counts"])
    else:
        d = on(pcloud_inputs(500, 300, 12, 17, 16, 1, 3, seed=23))
        x = d["x"]
        m, args = PCloudConv3d(16, 24, 17, with_bn=with_bn), tuple(d[k] for k in ("nn_count", "nn_index", "bin_index", "bin_coeff"))
    m = m.cuda()
    x[7, 3] = value
    upstream = torch.randn(args[1 if kind == "facet" else 0].shape[0], 24, device="cuda")    # (of a constant one a batch norm keeps only noise)
    results = []
    for native in (True, False):
        layers.set_fusion(native)
        try:
            out = m(x, *args)
            results.append([out, *torch.autograd.grad(out, [m.biases], upstream)])
        finally:
            layers.set_fusion(True)
    for a, b in zip(*results):
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isposinf(a), torch.isposinf(b))
        ok = torch.isfinite(b)
        assert rel_err(a[ok], b[ok]) <= 1e-4
    if with_bn:
        assert bool(torch.isnan(results[0][0]).any())
