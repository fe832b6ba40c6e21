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
