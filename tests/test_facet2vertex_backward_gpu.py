"""facet2vertex backward against the fp64 formula where its kernel splits the work anew: 4 to 32 lanes per face, chunks behind 128
channels, coefficient counts that leave warps to share faces (K <= 16) or none, the general kernel (K > 32), and face counts
around a tile."""
import pytest
import torch

from conftest import rel_err
from picassoplus_b200 import _lib
from picassoplus_b200.topology import ptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [4, 16, 24, 32, 48, 64, 100, 128, 132, 136, 200, 256])
@pytest.mark.parametrize("nf,K", [(1, 1), (31, 9), (129, 4), (257, 16), (1025, 17), (3000, 25), (700, 32), (333, 36)])
def test_facet2vertex_backward(nf, K, C):
    g = torch.Generator(device="cuda").manual_seed(nf * 1000 + C)
    nv = nf // 2 + 3
    face = torch.randint(0, nv, (nf, 3), dtype=torch.int32, device="cuda", generator=g)
    vt_map = torch.randint(-1, nv, (nv,), dtype=torch.int32, device="cuda", generator=g)
    nf_count = torch.randint(1, 9, (nv,), dtype=torch.int32, device="cuda", generator=g)
    x, go = torch.randn(nf, C, device="cuda", generator=g), torch.randn(nv, C, device="cuda", generator=g)
    filt, coeff = torch.randn(K, C, device="cuda", generator=g), torch.randn(nf, K, device="cuda", generator=g)
    gin, gf = torch.empty_like(x), torch.empty_like(filt)
    need = _lib.query("pb200_facet2vertex_backward_workspace_bytes", nf, C, 1, K)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")

    def run():
        _lib.call("pb200_facet2vertex_backward", nf, nv, nv, C, 1, K, ptr(go), ptr(x), ptr(filt), ptr(coeff), ptr(face), ptr(nf_count),
                  ptr(vt_map), ptr(gin), ptr(gf), ptr(ws), need, stream_ptr(x.device))
        return gin.clone(), gf.clone()

    got, again = run(), run()
    vo = vt_map[face.long()].long()
    gt = torch.where((vo >= 0)[..., None], go.double()[vo] / nf_count[vo].double()[..., None], 0.).sum(1)
    assert rel_err(got[0], gt * (coeff.double() @ filt.double())) <= 1e-5
    assert rel_err(got[1], coeff.double().T @ (x.double() * gt)) <= 1e-5
    assert torch.equal(got[0], again[0]) and torch.equal(got[1], again[1])


@pytest.mark.parametrize("C,K,r", [(4, 9, 1), (64, 16, 1), (100, 25, 1), (64, 36, 1), (5, 9, 1), (8, 9, 2)])
def test_indices_out_of_range(C, K, r):
    """With deferred validation the backward passes run on indices that are looked at later: corners outside the vertices, and output
    vertices outside theirs, have no part in either operator's gradients."""
    from picassoplus_b200 import topology
    from picassoplus_b200.mesh.pi_modules import conv3d
    g = torch.Generator(device="cuda").manual_seed(C + K)
    nv, nf = 70, 301
    face = torch.randint(nv, (nf, 3), device="cuda", generator=g).int()
    vt_map = torch.randint(-1, nv, (nv,), device="cuda", generator=g).int()
    for i, bad in enumerate((-1, nv, 2 ** 31 - 1, -2 ** 31)):
        face[i::50, i % 3] = bad
        vt_map[i] = bad
    count = torch.randint(1, 9, (nv,), device="cuda", generator=g).int()
    x, xv = torch.randn(nf, C, device="cuda", generator=g), torch.randn(nv, C, device="cuda", generator=g)
    coeff, w = torch.randn(nf, K, device="cuda", generator=g), torch.randn(K, C, r, device="cuda", generator=g)
    w3, gv, gf = (torch.randn(*s, device="cuda", generator=g) for s in ((3, C, r), (nv, C * r), (nf, C * r)))
    there = (face >= 0) & (face < nv)
    vid = face.long().clamp(0, nv - 1)
    out = vt_map.long()[vid]
    there_out = there & (out >= 0) & (out < nv)
    topology.set_validation("deferred")
    try:
        gin, gw = conv3d.facet2vertex_backward(gv, x, w, coeff, face, count, vt_map)
        gx, gw3 = conv3d.vertex2facet_backward(gf, xv, w3, face)
        with pytest.raises(RuntimeError, match="outside"):
            topology.check_deferred()
    finally:
        topology._deferred.clear()
        topology.set_validation("sync")
    rows = (gv.double() / count.double()[:, None])[out.clamp(0, nv - 1)] * there_out[:, :, None]           # (nf, 3, C * r)
    gt = rows.sum(1).view(nf, C, r)
    mult = torch.einsum("fk,kcr->fcr", coeff.double(), w.double())
    assert rel_err(gin, (gt * mult).sum(2)) <= 1e-5
    assert rel_err(gw, torch.einsum("fk,fc,fcr->kcr", coeff.double(), x.double(), gt)) <= 1e-5
    per = gf.double().view(nf, 1, C, r) * there[:, :, None, None]                                          # (nf, 3, C, r)
    want = torch.zeros(nv, C, dtype=torch.float64, device="cuda").index_add_(0, vid.reshape(-1), (per * w3.double()).sum(3).reshape(-1, C))
    assert rel_err(gx, want) <= 1e-5
    assert rel_err(gw3, torch.einsum("fkcr,fkc->kcr", per, xv.double()[vid])) <= 1e-5
