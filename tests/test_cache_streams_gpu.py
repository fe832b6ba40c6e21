"""The structure cache between streams and graph captures: what one stream is still making is waited for by the others, and what a
capture makes stays inside it."""
import pytest
import torch

from cases import conv_inputs

pytestmark = pytest.mark.gpu
SLEEP = 200_000_000          # clocks: about a tenth of a second


@pytest.fixture
def deferred():
    """Validation without synchronisations, which would order the streams by themselves."""
    from picassoplus_b200 import topology
    topology.set_validation("deferred")
    topology.clear_cache()
    yield topology
    topology.check_deferred()
    topology.set_validation("sync")
    topology.clear_cache()


def mesh():
    d = conv_inputs("ico2x3", 8, 1, 16, 8, seed=3, zero_sample_faces=False)
    face, cum, bary = d["face"].cuda(), d["cum"].cuda(), d["bary"].cuda()
    nv = d["x_v"].shape[0]
    want = torch.cat([torch.zeros(1, dtype=torch.int64), torch.bincount(d["face"].flatten().long(), minlength=nv).cumsum(0)])
    return face, nv, cum, bary, want.to(torch.int32)


def test_a_second_stream_waits(deferred):
    face, nv, cum, bary, want = mesh()
    fresh = deferred.face_means(bary, cum).rows.clone()
    deferred.clear_cache()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(SLEEP)
        deferred.vertex_csr(face, None, nv, nv)
        deferred.face_means(bary, cum)
    csr, means = deferred.vertex_csr(face, None, nv, nv), deferred.face_means(bary, cum)
    got = csr.rowptr.clone(), means.rows.clone()
    torch.cuda.synchronize()
    assert deferred.cache_stats()["slots"] == 2
    assert torch.equal(got[0].cpu(), want) and torch.equal(got[1], fresh)


def test_made_inside_a_capture(deferred):
    face, nv, _, _, want = mesh()
    deferred.vertex_csr(face, None, nv, nv)                  # first launches of the kernels, allocations
    deferred.clear_cache()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        inside = deferred.vertex_csr(face, None, nv, nv)
        assert deferred.vertex_csr(face, None, nv, nv) is inside
    outside = deferred.vertex_csr(face, None, nv, nv)        # the graph has not run yet
    assert outside is not inside and torch.equal(outside.rowptr.cpu(), want)
    assert deferred.vertex_csr(face, None, nv, nv) is outside
    deferred._deferred.clear()                               # the graph's status words have no value yet
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(inside.rowptr, outside.rowptr) and torch.equal(inside.entries, outside.entries)


def test_a_capture_waits_for_what_another_stream_makes(deferred):
    face, nv, _, _, want = mesh()
    deferred.vertex_csr(face, None, nv, nv)
    deferred.clear_cache()
    side, out = torch.cuda.Stream(), torch.empty(nv + 1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        with torch.cuda.stream(side):                        # not part of the capture
            torch.cuda._sleep(SLEEP)
            deferred.vertex_csr(face, None, nv, nv)
        out.copy_(deferred.vertex_csr(face, None, nv, nv).rowptr)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out.cpu(), want)
