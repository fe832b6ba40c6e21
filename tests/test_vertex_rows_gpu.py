"""The kernels that walk the faces of a vertex (vertex2facet backward, facet2vertex forward) and vertex2facet forward against the fp64
formulas where the work is split: vertices with no face, with as many as a batch holds (5 to 9), with more (17, 33, 70), odd numbers of
faces, and every number of lanes per row."""
import pytest
import torch

from conftest import rel_err
from picassoplus_b200.mesh.pi_modules import conv3d

pytestmark = pytest.mark.gpu

DEGREES = [0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 12, 13, 16, 17, 33, 70]


def _faces(copies, seed):
    """Faces whose vertex v has exactly DEGREES[v % 16] corners, in random order and corner position (one corner more where needed)."""
    ids = torch.cat([torch.full((d,), v + 16 * c) for c in range(copies) for v, d in enumerate(DEGREES)])
    g = torch.Generator().manual_seed(seed)
    ids = ids[torch.randperm(ids.numel(), generator=g)]
    ids = ids[:ids.numel() // 3 * 3]
    return ids.view(-1, 3).int().cuda(), 16 * copies


@pytest.mark.parametrize("C", [4, 8, 12, 16, 32, 64, 100, 128, 132])
@pytest.mark.parametrize("copies,odd", [(1, False), (1, True), (40, False), (300, True)])
def test_rows(copies, odd, C):
    face, nv = _faces(copies, C + copies)
    if (face.shape[0] % 2 == 1) != odd:
        face = face[:-1].contiguous()
    nf, g = face.shape[0], torch.Generator(device="cuda").manual_seed(C)
    x, w = torch.randn(nv, C, device="cuda", generator=g), torch.randn(3, C, 1, device="cuda", generator=g)
    go = torch.randn(nf, C, device="cuda", generator=g)
    vid = face.long()
    picked = x.double()[vid]                                                      # (nf, 3, C)
    out = conv3d.vertex2facet_forward(x, w, face)
    assert rel_err(out, (picked * w.double()[None, :, :, 0]).sum(1)) <= 1e-6
    gin, gw = conv3d.vertex2facet_backward(go, x, w, face)
    want = torch.zeros(nv, C, dtype=torch.float64, device="cuda")
    want.index_add_(0, vid.reshape(-1), (go.double()[:, None] * w.double()[None, :, :, 0]).reshape(-1, C))
    # sums of up to 70 terms of unit size: 70 * 2^-24 of the largest
    assert rel_err(gin, want) <= 5e-6 and rel_err(gw[:, :, 0], (go.double()[:, None] * picked).sum(0)) <= 5e-6
    K = 9
    coeff, filt = torch.randn(nf, K, device="cuda", generator=g), torch.randn(K, C, 1, device="cuda", generator=g)
    vt = torch.arange(nv, dtype=torch.int32, device="cuda")
    count = torch.bincount(vid.reshape(-1), minlength=nv).int()
    rows = conv3d.facet2vertex_forward(go, filt, coeff, face, count, vt)
    want = torch.zeros(nv, C, dtype=torch.float64, device="cuda")
    prod = (coeff.double() @ filt.double()[:, :, 0]) * go.double()
    want.index_add_(0, vid.reshape(-1), prod.repeat_interleave(3, 0))
    assert rel_err(rows, want / count.clamp(min=1).double()[:, None]) <= 5e-6
    again = conv3d.vertex2facet_backward(go, x, w, face)
    assert torch.equal(gin, again[0]) and torch.equal(gw, again[1])


@pytest.mark.parametrize("train", [False, True])
@pytest.mark.parametrize("rows", [99999, 100000, 100003])
@pytest.mark.parametrize("C,cout", [(8, 72), (64, 128), (136, 136)])
def test_layers_where_the_gather_leaves_the_product(C, cout, rows, train):
    """Layers over 100 000 rows and more gather in a kernel of their own: the bits of the fused kernel, which takes each part of a call
    that is split in two, with and without the features kept for a backward pass."""
    from picassoplus_b200 import _lib
    from picassoplus_b200.mesh.pi_modules import fused
    g = torch.Generator(device="cuda").manual_seed(rows + C)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    half = 50000
    weights, bias, filt = randn(C, cout), randn(1, cout), randn(3, C, 1)
    x = randn(4000, C)
    face = torch.randint(4000, (rows, 3), device="cuda", generator=g).int()
    whole = fused.vertex2facet_pointwise(x, filt, face, weights.requires_grad_(train), bias, True)
    with torch.no_grad():
        parts = [fused.vertex2facet_pointwise(x, filt, f.contiguous(), weights, bias, True) for f in (face[:half], face[half:])]
    assert torch.equal(whole, torch.cat(parts))
    if train:
        go = randn(rows, cout)
        grad, = torch.autograd.grad(whole, weights, go)
        rows64 = (x.double()[face.long()] * filt.double()[:, :, 0]).sum(1)
        # operands of a bf16 high and low part: 2^-16 of each product
        assert rel_err(grad, rows64.t() @ (go.double() * (whole > 0))) <= 1e-4
    # vertices: the first have no faces, the last have many
    degree = torch.arange(rows, device="cuda") % 11
    rowptr = torch.cat([degree.new_zeros(1), degree.cumsum(0)]).int()
    nf, K = 30000, 9
    entries = (torch.randint(nf, (int(rowptr[-1]),), device="cuda", generator=g) * 4).int()
    xf, coeff, wf = randn(nf, C), randn(nf, K), randn(K, C, 1)
    fake = torch.zeros(nf, 3, dtype=torch.int32, device="cuda")
    tail = (1, *fused._NO_NORM)

    def layer(lo, hi):
        return _lib.ops.f2v_layer(xf, fake, degree[lo:hi].int(), torch.zeros(hi - lo, dtype=torch.int32, device="cuda"),
                                  rowptr[lo:hi + 1].clone(), entries, coeff, wf, weights, bias, *tail, fused._precision)
    whole = layer(0, rows)
    with torch.no_grad():
        assert torch.equal(whole, torch.cat([layer(0, half), layer(half, rows)]))


BAD = [-1, -2 ** 31, 2 ** 31 - 1]                  # and the number of vertices


@pytest.mark.parametrize("C,r", [(4, 1), (12, 1), (64, 1), (132, 1), (5, 1), (8, 2)])
@pytest.mark.parametrize("nf", [1, 2, 7, 5001])
def test_corner_outside_the_vertices(nf, C, r):
    """It contributes nothing to vertex2facet, not even its product with an infinite filter value."""
    g = torch.Generator(device="cuda").manual_seed(nf + C)
    nv = 60
    x, w = torch.randn(nv, C, device="cuda", generator=g), torch.randn(3, C, r, device="cuda", generator=g)
    face = torch.randint(nv, (nf, 3), device="cuda", generator=g).int()
    for i, bad in enumerate(BAD + [nv]):
        face[i % nf, i % 3] = bad
    w[0, 0, 0] = float("inf")                       # of a corner that the first face does not have
    good = (face >= 0) & (face < nv)
    picked = x.double()[face.long().clamp(0, nv - 1)].repeat_interleave(r, 2)                    # (nf, 3, C * r)
    want = torch.where(good[:, :, None], picked * w.double().view(1, 3, C * r), 0.0).sum(1)
    out = conv3d.vertex2facet_forward(x, w, face).double()
    assert bool(out[0].isfinite().all()) and torch.equal(out.isfinite(), want.isfinite())
    # three products of unit size, each rounded once
    assert rel_err(out.nan_to_num(0, 0, 0), want.nan_to_num(0, 0, 0)) <= 1e-6


@pytest.mark.parametrize("C,cout", [(8, 24), (64, 136)])
def test_layer_over_a_corner_outside_the_vertices(C, cout):
    """The vertex2facet layer tolerates one forward at any size, under autograd or not, with the same result; its backward pass refuses it."""
    from picassoplus_b200.mesh.layers import V2FConv3d
    g = torch.Generator(device="cuda").manual_seed(C)
    rows, half, nv = 100003, 50000, 4000
    layer, x = V2FConv3d(C, cout, 2).cuda().eval(), torch.randn(nv, C, device="cuda", generator=g).requires_grad_()
    face = torch.randint(nv, (rows, 3), device="cuda", generator=g).int()
    for i, bad in enumerate(BAD + [nv]):
        face[i::20000, i % 3] = bad
    with torch.no_grad():
        want = torch.cat([layer(x, f.contiguous()) for f in (face[:half], face[half:])])         # gathered inside the product
        assert torch.equal(layer(x, face), want)
    out = layer(x, face)
    assert rel_err(out, want) <= 1e-5               # normalised by a kernel of its own
    with pytest.raises(RuntimeError, match="outside"):
        torch.autograd.grad(out, [x], torch.ones_like(out))


@pytest.mark.parametrize("C", [4, 8, 64, 100, 132, 6])
def test_rows_that_take_no_part(C):
    """An infinite row of a vertex without faces, or in the corner numbers that a vertex is not, stays out of the filter gradient, and an
    infinite filter value out of the input gradient of the vertices that it does not meet."""
    inf, nan = float("inf"), float("nan")
    g = torch.Generator(device="cuda").manual_seed(C)
    # 0: no face; 1: corner 0 of every face and nothing else; 2 to 9: corners 1 and 2
    face = torch.randint(2, 10, (40, 3), device="cuda", generator=g).int()
    face[:, 0] = 1
    x, w = torch.randn(10, C, device="cuda", generator=g), torch.randn(3, C, 1, device="cuda", generator=g)
    go = torch.randn(40, C, device="cuda", generator=g)
    x[0], x[1, 0] = nan, inf
    w[0, 1], w[2, 2] = inf, nan
    gin, gw = conv3d.vertex2facet_backward(go, x, w, face)
    assert bool((gin[0] == 0).all())                                              # no face
    assert bool(gin[2:, 1].isfinite().all()) and bool(gin[1, 2].isfinite())       # filters of corners that these vertices are not
    assert not bool(gin[1, 1].isfinite()) and bool(gin[face[0, 2].long(), 2].isnan())
    want = (go.double()[:, None] * x.double()[face.long()]).sum(0)                # (3, C)
    assert not bool(want[0, 0].isfinite()) and bool(gw[1:, 0].isfinite().all()) and not bool(gw[0, 0].isfinite())
    assert rel_err(gw[:, 1:, 0], want[:, 1:]) <= 5e-6


def test_inference_takes_no_room_that_is_not_there():
    """Gathered rows that a layer could do without are not asked for where they do not fit: no failed allocation, which would cost the
    process its cached memory call after call, and the same results."""
    from picassoplus_b200.mesh.layers import V2FConv3d
    g = torch.Generator(device="cuda").manual_seed(0)
    rows, nv, C = 400000, 20000, 256
    layer, x = V2FConv3d(C, 128, 2).cuda().eval(), torch.randn(nv, C, device="cuda", generator=g)
    face = torch.randint(nv, (rows, 3), device="cuda", generator=g).int()
    scratch = 4 * rows * C
    with torch.no_grad():
        torch.cuda.reset_peak_memory_stats()
        want = layer(x, face)
        assert torch.cuda.max_memory_allocated() - torch.cuda.memory_allocated() > scratch          # the sizes do ask for them
        torch.cuda.empty_cache()
        figures = lambda: [torch.cuda.memory_stats()[k] for k in ("num_ooms", "num_alloc_retries")]
        counts, total = figures(), torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + want.numel() * 4 + scratch // 2) / total)
        try:
            for _ in range(3):
                assert torch.equal(layer(x, face), want)
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
        assert figures() == counts


def test_inference_over_many_rows_is_captured():
    """The question for room and the rows themselves inside a graph capture: the replay has the results of the plain call."""
    from picassoplus_b200.mesh.layers import V2FConv3d
    g = torch.Generator(device="cuda").manual_seed(1)
    rows, nv, C = 200000, 20000, 64
    layer, x = V2FConv3d(C, 128, 2).cuda().eval(), torch.randn(nv, C, device="cuda", generator=g)
    face = torch.randint(nv, (rows, 3), device="cuda", generator=g).int()
    with torch.no_grad():
        want = layer(x, face)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()                    # nothing at hand: the device is asked
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = layer(x, face)
        out.zero_()
        graph.replay()
        assert torch.equal(out, want)
