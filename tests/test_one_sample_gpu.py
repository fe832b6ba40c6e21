"""Backward pass of facet2facet with one sample per face (its own kernels for the input and the filter gradient) against the
fp64 formula, where their work splits change: less than a tile of faces, one face more than a stage or a tile, channel counts
that fill no tile or take several blocks, more than 256 contracted channels, fewer tiles than SMs, and enough faces for
the filter gradient's accumulators to be read out on the way."""
import pytest
import torch

from conftest import rel_err
from picassoplus_b200 import _lib
from picassoplus_b200.topology import ptr, stream_ptr

pytestmark = pytest.mark.gpu


def one_sample_backward(go, x, filt, w, precision):
    nf, cin = x.shape
    cout, _, F = filt.shape
    wp = torch.nn.functional.pad(w, (0, -F % 4)).contiguous()
    one_each = torch.arange(1, nf + 1, dtype=torch.int32, device="cuda")
    gin, gf = torch.empty_like(x), torch.empty_like(filt)
    need = _lib.query("pb200_facet2facet_backward_workspace_bytes", nf, nf, cin, cout, F, precision)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    _lib.call("pb200_facet2facet_one_sample_backward", nf, cin, cout, F, ptr(go), ptr(x), ptr(filt), ptr(w), ptr(wp), ptr(one_each),
              ptr(gin), ptr(gf), precision, ptr(ws), need, stream_ptr(x.device))
    return gin, gf


@pytest.mark.parametrize("nf,cin,cout,F", [(1, 16, 16, 4), (15, 64, 64, 16), (17, 32, 128, 9), (128, 100, 48, 25), (129, 128, 100, 16),
                                            (4097, 24, 96, 25), (1000, 260, 300, 9), (9000, 16, 64, 25), (777, 4, 8, 4),
                                            (650, 48, 40, 7), (140001, 64, 128, 25)])
@pytest.mark.parametrize("precision,gate", [(_lib.PREC_FP32, 2e-5), (_lib.PREC_BF16, 2e-2)])
def test_one_sample_backward(nf, cin, cout, F, precision, gate):
    g = torch.Generator(device="cuda").manual_seed(nf + cin)
    x = torch.randn(nf, cin, device="cuda", generator=g)
    go = torch.randn(nf, cout, device="cuda", generator=g)
    w = torch.rand(nf, F, device="cuda", generator=g)
    filt = torch.randn(cout, cin, F, device="cuda", generator=g) / (cin * F) ** 0.5
    gin, gf = one_sample_backward(go, x, filt, w, precision)
    again = one_sample_backward(go, x, filt, w, precision)
    want_gf = torch.zeros(cout, cin * F, device="cuda", dtype=torch.float64)
    want_gin = []
    for o in range(0, nf, 20000):
        s = slice(o, o + 20000)
        wd, xd, gd = w[s].double(), x[s].double(), go[s].double()
        want_gf += gd.T @ (xd[:, :, None] * wd[:, None, :]).reshape(xd.shape[0], -1)
        want_gin.append(((gd @ filt.double().reshape(cout, -1)).reshape(-1, cin, F) * wd[:, None, :]).sum(2))
    assert rel_err(gin, torch.cat(want_gin)) <= gate
    assert rel_err(gf, want_gf.reshape(cout, cin, F)) <= gate
    assert torch.equal(gin, again[0]) and torch.equal(gf, again[1])
    assert _lib.query("pb200_async_error") == 0


@pytest.mark.parametrize("nf", [1, 127, 128, 129, 255, 256, 257, 511, 40001])
@pytest.mark.parametrize("cin,cout,F", [(100, 20, 4), (128, 48, 9), (100, 128, 16), (260, 36, 25), (64, 64, 16), (512, 12, 9),
                                          (192, 48, 25), (256, 40, 9), (252, 132, 4), (160, 36, 16), (220, 20, 9)])
@pytest.mark.parametrize("precision,gate", [(_lib.PREC_FP32, 2e-5), (_lib.PREC_BF16, 2e-2)])
def test_one_sample_forward(nf, cin, cout, F, precision, gate):
    """Around the 128 rows of a tile and the 256 of a pair of CTAs (from 97 contracted channels on), contracted channels that fill no
    K-block, more than one launch holds or, in bf16, take rows through stages (from 161 on), and rows behind the last face."""
    g = torch.Generator(device="cuda").manual_seed(nf + cin)
    x = torch.randn(nf, cin, device="cuda", generator=g)
    w = torch.rand(nf, F, device="cuda", generator=g)
    filt = torch.randn(cout, cin, F, device="cuda", generator=g) / (cin * F) ** 0.5
    wp = torch.nn.functional.pad(w, (0, -F % 4)).contiguous()
    need = _lib.query("pb200_facet2facet_one_sample_forward_workspace_bytes", nf, cin, cout, F, precision)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    out = torch.full((nf + 1, cout), 7., device="cuda")

    def run():
        _lib.call("pb200_facet2facet_one_sample_forward", nf, cin, cout, F, ptr(x), ptr(filt), ptr(w), ptr(wp), ptr(out), precision, ptr(ws),
                  need, stream_ptr(x.device))
        return out.clone()

    got = run()
    want = ((x.double() @ filt.double().transpose(1, 2).reshape(cout, F, cin).reshape(-1, cin).T).reshape(nf, cout, F) * w.double()[:, None]).sum(2)
    assert rel_err(got[:nf], want) <= gate
    assert torch.equal(got, run()) and bool((got[nf] == 7).all())
    assert _lib.query("pb200_async_error") == 0


@pytest.mark.parametrize("precision,F,cin,names", [
    (_lib.PREC_FP32, 16, 64, {"f2f_bwd_gin_one_tc", "f2f_bwd_gfilter_one_tc", "f2f_bwd_gfilter_one_reduce"}),
    (_lib.PREC_BF16, 25, 128, {"f2f_bwd_gin_one_tc", "f2f_bwd_gfilter_one_tc", "f2f_bwd_gfilter_one_reduce"}),
    (_lib.PREC_FP32, 7, 48, {"f2f_gA_sgemm", "f2f_bwd_gfilter_one_tc"}),            # a basis count the product kernels are not built for
    (_lib.PREC_TF32, 16, 64, {"f2f_bwd_gin_tc", "f2f_bwd_gfilter_tc"}),            # tf32 operands: the general kernels
])
def test_which_kernels_run(precision, F, cin, names):
    x, go = torch.randn(300, cin, device="cuda"), torch.randn(300, 64, device="cuda")
    w, filt = torch.rand(300, F, device="cuda"), torch.randn(64, cin, F, device="cuda")
    _lib.prof_reset()
    _lib.prof_enable(True)
    try:
        one_sample_backward(go, x, filt, w, precision)
        torch.cuda.synchronize()
    finally:
        _lib.prof_enable(False)
    ran = {n for n, _, _ in _lib.prof_read(64)}
    _lib.prof_reset()
    others = {"f2f_bwd_gin_tc", "f2f_bwd_gin_one_tc", "f2f_bwd_gfilter_tc", "f2f_bwd_gfilter_one_tc"} - names
    assert names <= ran and not others & ran, ran
