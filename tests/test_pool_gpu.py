"""Mesh pooling / unpooling kernels, called through the C ABI (via the operator API that mirrors
picasso/mesh/pi_modules/pool3d.py and unpool3d.py), against the oracle and the reference's own
CUDA kernels on identical seeded inputs.  Gates: values selected or copied (max pool, its backward,
average-pool backward, unpool forward) bit-exact, max indices bit-exact, sums (average pool
forward, unpool backward) <= 1e-6 relative (the reference adds with float atomics)."""
import numpy as np
import pytest
import torch

from cases import POOL_GOLDEN_CASES, cluster_inputs
from conftest import max_abs, rel_err

pytestmark = pytest.mark.gpu

CASES = [
    # NvIn, NvOut, C, ties
    (300, 90, 8, False),
    (257, 64, 5, False),          # scalar path (C not a multiple of 4)
    (64, 64, 4, False),           # every vertex its own cluster
    (5000, 700, 128, False),
    (20000, 5000, 64, True),      # equal maxima inside clusters
    (40, 1, 12, False),           # one cluster
]


def _dev(d):
    return {k: (v.cuda() if isinstance(v, torch.Tensor) else v) for k, v in d.items()}


@pytest.fixture(scope="module")
def mods():
    from picassoplus_b200.mesh.pi_modules import pool3d, unpool3d
    from oracle import mesh_oracle, ref_cuda
    return pool3d, unpool3d, mesh_oracle, ref_cuda


@pytest.mark.parametrize("nv_in,nv_out,C,ties", CASES)
def test_pool_and_unpool_match_oracle_and_reference(mods, nv_in, nv_out, C, ties):
    pool3d, unpool3d, mo, ref = mods
    d = cluster_inputs(nv_in, nv_out, C, seed=17, ties=ties)
    c = _dev(d)
    vt_out = torch.zeros(nv_out, 3, device="cuda")
    out, idx = pool3d.max_forward(c["x"], c["vt_replace"], c["vt_map"], vt_out)
    w_out, w_idx = mo.mesh_max_pool_forward(d["x"], d["vt_replace"], d["vt_map"], nv_out)
    assert torch.equal(out.cpu(), w_out) and torch.equal(idx.cpu(), w_idx)
    gin = pool3d.max_backward(c["g_coarse"], c["x"], idx)
    assert torch.equal(gin.cpu(), mo.mesh_max_pool_backward(d["g_coarse"], nv_in, w_idx))
    _, _, clusters = pool3d.max_forward(c["x"], c["vt_replace"], c["vt_map"], vt_out, return_clusters=True)
    assert torch.equal(pool3d.max_backward(c["g_coarse"], c["x"], idx, clusters), gin)     # the gather form
    avg = pool3d.avg_forward(c["x"], c["vt_replace"], c["vt_map"], vt_out)
    assert rel_err(avg, mo.mesh_avg_pool_forward(d["x"].double(), d["vt_replace"], d["vt_map"], nv_out)) <= 1e-6
    avg_b = pool3d.avg_backward(c["g_coarse"], c["x"], c["vt_replace"], c["vt_map"])
    assert torch.equal(avg_b.cpu(), mo.mesh_avg_pool_backward(d["g_coarse"], d["vt_replace"], d["vt_map"]))
    up = unpool3d.forward(c["x_coarse"], c["vt_replace"], c["vt_map"])
    assert torch.equal(up.cpu(), mo.mesh_unpool_forward(d["x_coarse"], d["vt_replace"], d["vt_map"]))
    up_b = unpool3d.backward(c["g_fine"], c["x_coarse"], c["vt_replace"], c["vt_map"])
    assert rel_err(up_b, mo.mesh_unpool_backward(d["g_fine"].double(), nv_out, d["vt_replace"], d["vt_map"])) <= 1e-6
    # run to run identical
    assert torch.equal(avg, pool3d.avg_forward(c["x"], c["vt_replace"], c["vt_map"], vt_out))
    assert torch.equal(up_b, unpool3d.backward(c["g_fine"], c["x_coarse"], c["vt_replace"], c["vt_map"]))
    if ref.available():
        r_out, r_idx = ref.max_pool_forward(c["x"], c["vt_replace"], c["vt_map"], nv_out)
        assert torch.equal(out, r_out)
        if not ties:
            assert torch.equal(idx, r_idx)
            assert torch.equal(gin, ref.max_pool_backward(c["g_coarse"], nv_in, r_idx))
        else:       # the reference's index among equal maxima depends on its thread order: any attaining member is right
            picked = torch.gather(c["x"], 0, r_idx.long())
            assert torch.equal(picked, r_out)
        assert rel_err(avg, ref.avg_pool_forward(c["x"], c["vt_replace"], c["vt_map"], nv_out)) <= 1e-6
        assert torch.equal(avg_b, ref.avg_pool_backward(c["g_coarse"], c["vt_replace"], c["vt_map"]))
        assert torch.equal(up, ref.unpool_forward(c["x_coarse"], c["vt_replace"], c["vt_map"]))
        assert rel_err(up_b, ref.unpool_backward(c["g_fine"], nv_out, c["vt_replace"], c["vt_map"])) <= 1e-6


@pytest.mark.parametrize("name", sorted(POOL_GOLDEN_CASES))
def test_against_committed_reference_fixtures(mods, name):
    import os
    pool3d, unpool3d, _, _ = mods
    path = os.path.join(os.path.dirname(__file__), "golden", name + ".npz")
    z = np.load(path)
    nv_in, nv_out, C, seed = POOL_GOLDEN_CASES[name]
    c = _dev(cluster_inputs(nv_in, nv_out, C, seed))
    vt_out = torch.zeros(nv_out, 3, device="cuda")
    out, idx = pool3d.max_forward(c["x"], c["vt_replace"], c["vt_map"], vt_out)
    assert max_abs(out, z["ref_max_out"]) == 0.0 and np.array_equal(idx.cpu().numpy(), z["ref_max_index"])
    assert max_abs(pool3d.max_backward(c["g_coarse"], c["x"], idx), z["ref_max_gin"]) == 0.0
    assert rel_err(pool3d.avg_forward(c["x"], c["vt_replace"], c["vt_map"], vt_out), z["ref_avg_out"]) <= 1e-6
    assert max_abs(pool3d.avg_backward(c["g_coarse"], c["x"], c["vt_replace"], c["vt_map"]), z["ref_avg_gin"]) == 0.0
    assert max_abs(unpool3d.forward(c["x_coarse"], c["vt_replace"], c["vt_map"]), z["ref_unpool_out"]) == 0.0
    assert rel_err(unpool3d.backward(c["g_fine"], c["x_coarse"], c["vt_replace"], c["vt_map"]), z["ref_unpool_gin"]) <= 1e-6


def test_autograd_through_pool_layers(mods):
    """Pool3d / Unpool3d modules: gradients of max, avg and unpool through torch autograd against the
    oracle's explicit backward formulas."""
    from picassoplus_b200.mesh.layers import Pool3d, Unpool3d
    _, _, mo, _ = mods
    d = cluster_inputs(900, 250, 16, seed=23)
    c = _dev(d)
    vt_out = torch.zeros(250, 3, device="cuda")
    for method in ("max", "avg"):
        x = c["x"].clone().requires_grad_()
        y = Pool3d(method)(x, c["vt_replace"], c["vt_map"], vt_out)
        y.backward(c["g_coarse"])
        if method == "max":
            _, idx = mo.mesh_max_pool_forward(d["x"], d["vt_replace"], d["vt_map"], 250)
            want = mo.mesh_max_pool_backward(d["g_coarse"], 900, idx)
        else:
            want = mo.mesh_avg_pool_backward(d["g_coarse"], d["vt_replace"], d["vt_map"])
        assert torch.equal(x.grad.cpu(), want)
    xc = c["x_coarse"].clone().requires_grad_()
    Unpool3d()(xc, c["vt_replace"], c["vt_map"]).backward(c["g_fine"])
    assert rel_err(xc.grad, mo.mesh_unpool_backward(d["g_fine"].double(), 250, d["vt_replace"], d["vt_map"])) <= 1e-6


def test_max_pool_gradient_with_memberless_coarse_vertices(mods):
    """More output rows than clusters: the extra coarse vertices have no members, record index 0 and hand their
    gradient to vertex 0 (picasso/mesh/pi_modules/source/mesh_pool3d_gpu.cu:93-105); the gather form does the same.
    Vertex 0 belongs to no cluster here, so no two writers meet there."""
    pool3d, _, mo, _ = mods
    d = cluster_inputs(400, 120, 8, seed=7)
    assert int(d["vt_map"][0]) < 0 and int(d["vt_replace"][0]) == 0       # this seed leaves vertex 0 outside every cluster
    c = _dev(d)
    nv_out = 121
    vt_out = torch.zeros(nv_out, 3, device="cuda")
    g = torch.randn(nv_out, 8, device="cuda")
    out, idx, clusters = pool3d.max_forward(c["x"], c["vt_replace"], c["vt_map"], vt_out, return_clusters=True)
    assert torch.all(out[120] == 0) and torch.all(idx[120] == 0)
    scatter = pool3d.max_backward(g, c["x"], idx)
    gather = pool3d.max_backward(g, c["x"], idx, clusters)
    assert torch.equal(scatter, gather) and torch.equal(gather[0], g[120])
    assert torch.equal(gather.cpu(), mo.mesh_max_pool_backward(g.cpu(), 400, idx.cpu()))


def test_bad_cluster_indices_are_reported(mods):
    pool3d, _, _, _ = mods
    c = _dev(cluster_inputs(100, 30, 4, seed=1))
    bad = c["vt_replace"].clone()
    bad[5] = -10 ** 6
    with pytest.raises(RuntimeError):
        pool3d.avg_forward(c["x"], bad, c["vt_map"], torch.zeros(30, 3, device="cuda"))
    assert torch.isfinite(pool3d.avg_forward(c["x"], c["vt_replace"], c["vt_map"], torch.zeros(30, 3, device="cuda"))).all()


@pytest.mark.parametrize("kind,L,orient", [("grid17x2", 4, False), ("grid17x2+drop", 3, True), ("ico2x3", 2, True),
                                           ("tet+iso", 5, True)])
def test_level_prepare_matches_the_separate_calls(kind, L, orient):
    """pb200_level_prepare (one fused pass per mesh level) against the separate entry points, the
    oracle, and the CSR built by pb200_build_vertex_csr: geometry and basis bit-identical to the
    separate kernels, nfCount and CSR bit-exact."""
    from cases import conv_inputs
    from oracle import mesh_oracle as mo
    from picassoplus_b200 import topology
    from picassoplus_b200.math_utils import sph_harm_coeff
    from picassoplus_b200.mesh.pi_modules import decimate
    d = conv_inputs(kind, 4, 1, 4, 2, seed=33)
    vertex = (d["vertex"] - 0.5).cuda()             # centre the meshes on the origin so both orientations occur
    face, vt_map = d["face"].cuda(), d["vt_map"].cuda()
    topology.clear_cache()
    got = topology.prepare_level(vertex, face, vt_map, d["nv_out"], L, orient=orient, want_normals=True)
    geo = decimate.compute_triangle_geometry_(vertex, face)
    assert torch.equal(got["geometry"], geo)
    want_n = mo.oriented_normals(geo.cpu(), vertex.cpu(), d["face"]) if orient else geo[:, :3].cpu()
    assert torch.equal(got["normals"].cpu(), want_n)
    if orient:
        assert (want_n != geo[:, :3].cpu()).any()            # the case does flip some normals
    assert torch.equal(got["coeff"], sph_harm_coeff(L, got["normals"]))
    assert max_abs(got["coeff"], mo.sph_harm_coeff(L, want_n)) <= 2e-6
    assert torch.equal(got["nf_count"].cpu(), mo.count_vertex_adjface(d["face"], d["vt_map"], d["nv_out"]))
    ref_csr = topology.build_vertex_csr(face, vt_map, d["vt_map"].shape[0], d["nv_out"])
    assert torch.equal(got["csr"].rowptr, ref_csr.rowptr)
    n = int(ref_csr.rowptr[-1])
    assert torch.equal(got["csr"].entries[:n], ref_csr.entries[:n])
    assert topology.vertex_csr(face, vt_map, d["vt_map"].shape[0], d["nv_out"]) is got["csr"]     # served from the cache


@pytest.mark.parametrize("C", [5, 64])
def test_average_gradient_keeps_the_sign_of_zero(C):
    """A gradient of -0 over any member count is -0, as the division gives it."""
    from picassoplus_b200.mesh.pi_modules import pool3d
    d = _dev(cluster_inputs(300, 90, C, seed=3, ties=False))
    got = pool3d.avg_backward(torch.full((90, C), -0.0, device="cuda"), d["x"], d["vt_replace"], d["vt_map"])
    assert torch.signbit(got[d["vt_map"] >= 0]).all()


SPECIAL = [0.0, 2.0 ** -149, 2.0 ** -126, 2.0 ** -127, 2.0 ** -61, float(np.nextafter(np.float32(2.0 ** -60), np.float32(0))), 2.0 ** -60,
           float(np.nextafter(np.float32(2.0 ** -60), np.float32(1))), 2.0 ** -36, 1.0, 3.0, float(np.finfo(np.float32).max), float("inf"), float("nan")]


def _quotients(x, count, pool3d):
    """x / count by average pooling's gradient and forward pass: every vertex a cluster of its own that claims `count` members."""
    nv = x.shape[0]
    rep = torch.full((nv,), count - 1, dtype=torch.int32, device="cuda")
    key = torch.arange(nv, dtype=torch.int32, device="cuda")
    return pool3d.avg_backward(x, x, rep, key), pool3d.avg_forward(x, rep, key, torch.zeros(nv, 3, device="cuda"))


def _same_bits(a, b):
    number = ~a.isnan()
    return torch.equal(number, ~b.isnan()) and torch.equal(a.view(torch.int32)[number], b.view(torch.int32)[number])


@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 6, 7, 9, 10, 11, 13, 15, 17, 23, 31, 49, 63, 97, 255, 1021, 4095, 12288, 65537, 8388607,
                                   16777215, 16777216, 16777218, 2147483647])
def test_quotients_have_the_bits_of_the_division(count):
    """Every mantissa, at exponents all over the range, for a member count; and the values around the edges of the short form."""
    from picassoplus_b200.mesh.pi_modules import pool3d
    g = torch.Generator(device="cuda").manual_seed(count % 1000)
    mantissa = torch.arange(1 << 23, dtype=torch.int32, device="cuda")
    exponent = torch.randint(1, 255, mantissa.shape, dtype=torch.int32, device="cuda", generator=g)
    sign = torch.randint(0, 2, mantissa.shape, dtype=torch.int32, device="cuda", generator=g)
    edges = torch.tensor(SPECIAL + [-v for v in SPECIAL], device="cuda").repeat(256, 1)[:, :28].contiguous()
    divisor = torch.tensor(float(count), device="cuda")
    for x in (((exponent << 23) | mantissa | (sign << 31)).view(torch.float32).view(-1, 64), ((127 << 23) | mantissa).view(torch.float32).view(-1, 64),
              edges, edges[:, :27].contiguous()):
        want = x / divisor
        back, forward = _quotients(x, count, pool3d)
        assert _same_bits(back, want) and _same_bits(forward, want + 0.0)       # a sum from +0 has no -0
    few = x[:100]
    assert _same_bits(_quotients(few, count, pool3d)[1], few / divisor + 0.0)


@pytest.mark.parametrize("C", [4, 48, 64, 100, 9])
def test_average_of_many_and_of_few_clusters(C):
    """Either side of the line between a thread per quad and teams gives the same bits, for clusters of no, one, four, five and forty members."""
    from picassoplus_b200.mesh.pi_modules import pool3d
    sizes = torch.tensor([0, 1, 4, 5, 40], device="cuda").repeat(3000)
    key = torch.repeat_interleave(torch.arange(sizes.numel(), device="cuda"), sizes)
    first = torch.cumsum(sizes, 0) - sizes
    lead = torch.arange(key.numel(), device="cuda") == first[key]
    # the first vertex cannot be pointed at (its negative is no index): it stands alone
    rep = torch.where(lead, sizes[key] - 1, -first[key]).int()
    key = torch.where(lead, key, -1).int()
    x = torch.relu(torch.randn(key.numel(), C, device="cuda", generator=torch.Generator(device="cuda").manual_seed(C)))
    whole = pool3d.avg_forward(x, rep, key, torch.zeros(sizes.numel(), 3, device="cuda"))
    part, rows = 500, int(sizes[:500].sum())                    # 15 000 clusters against 500 of them
    few = pool3d.avg_forward(x[:rows].contiguous(), rep[:rows].contiguous(), key[:rows].contiguous(), torch.zeros(part, 3, device="cuda"))
    assert torch.equal(whole[:part], few) and bool((whole[::5] == 0).all())
    want = torch.zeros(sizes.numel(), C, dtype=torch.float64, device="cuda")
    owner = torch.repeat_interleave(torch.arange(sizes.numel(), device="cuda"), sizes)
    want.index_add_(0, owner, x.double())
    assert rel_err(whole, want / sizes.clamp(min=1).double()[:, None]) <= 1e-6
