"""What mesh_decimation and MeshHierarchy take as the samples' sizes and targets, and what they refuse before any kernel sees it."""
import numpy as np
import pytest
import torch

from picassoplus_b200 import synth
from picassoplus_b200.mesh.pi_modules import decimate as dm
from picassoplus_b200.mesh.utils import MeshHierarchy


def host_batch():
    """Two icospheres of 42 vertices and 80 faces."""
    v, f = synth.icosphere(1)
    v, f = np.concatenate([v, v + 3]).astype(np.float32), np.concatenate([f, f + len(v)]).astype(np.int32)
    vertex, face = torch.from_numpy(v), torch.from_numpy(f)
    return vertex, face, torch.zeros(160, 5), torch.tensor([42, 42], dtype=torch.int32), torch.tensor([80, 80], dtype=torch.int32)


def target(*n):
    return torch.tensor(n, dtype=torch.int32)


@pytest.mark.parametrize("change,why", [
    (dict(nvOut=target(20, 20, 20)), "one entry per sample"), (dict(nvOut=target()), "one entry per sample"),
    (dict(nvOut=target(20, 20)[None]), "dimension of 1"),
    (dict(nvIn=target(42, 21, 21)), "one entry per sample"), (dict(nvIn=target(42, 42)[None]), "dimension of 1"),
    (dict(mfIn=target(160)), "one entry per sample"), (dict(mfIn=target(80, 40, 40)), "one entry per sample"),
    (dict(nvIn=target(85, -1)), "negative"), (dict(mfIn=target(161, -1)), "negative"),
    (dict(), "CUDA"),                                             # everything in order, but on the host
])
def test_refused_on_the_host(change, why):
    vertex, face, geometry, nv, mf = host_batch()
    args = dict(vertexIn=vertex, faceIn=face, geometryIn=geometry, nvIn=nv, mfIn=mf, nvOut=target(20, 20))
    args.update(change)
    with pytest.raises(RuntimeError, match=why):
        dm.mesh_decimation_(**args)


def test_nothing_to_remove():
    """No vertex above the target: the inputs come back, whatever they are."""
    vertex, face, geometry, nv, mf = host_batch()
    out = dm.mesh_decimation_(vertex, face, geometry, nv, mf, target(42, 50))
    assert all(a is b or torch.equal(a, b) for a, b in zip(out[:5], (vertex, face, geometry, nv, mf)))
    assert torch.equal(out[5], torch.zeros(84, dtype=torch.int32)) and torch.equal(out[6], torch.arange(84, dtype=torch.int32))


@pytest.mark.gpu
def test_refused_on_the_gpu():
    """Meshes on the GPU with sizes that are on the host, or do not belong to them."""
    vertex, face, geometry, nv, mf = host_batch()
    v, f = vertex.cuda(), face.cuda()
    g = dm.compute_triangle_geometry_(v, f)
    cn, cm, ct = nv.cuda(), mf.cuda(), target(20, 20).cuda()
    for args in ((v, f, g, nv, mf, target(20, 20)), (v, f, g, cn, mf, ct), (v, f, g, nv, cm, target(20, 20)), (v, f, g, cn, cm, target(20, 20)),
                 (v, face, g, cn, cm, ct), (v, f, geometry, cn, cm, ct), (v, f, g, cn, target(160).cuda(), ct), (v, f, g, cn, cm, ct[:0]),
                 (v, f, g, target(85, -1).cuda(), cm, ct), (v, f, g, cn, cm, target(20, 20, 20).cuda()), (v.double(), f, g, cn, cm, ct)):
        with pytest.raises(RuntimeError):
            dm.mesh_decimation_(*args)
    for build in (MeshHierarchy([4], [4], True, 1.0), MeshHierarchy([target(20, 20)], True, 1.0)):
        with pytest.raises(RuntimeError):
            build(v, f, nv, mf)
        with pytest.raises(RuntimeError):
            build(v, f, cn, target(160).cuda())
    with pytest.raises(RuntimeError):
        MeshHierarchy([target(20, 20, 20)], True, 1.0)(v, f, cn, cm)


@pytest.mark.gpu
def test_forms_of_the_target():
    """One number per sample, one for all (a tensor of one element, without dimension, or a plain number), fractions, 64-bit sizes."""
    vertex, face, _, nv, mf = host_batch()
    v, f, cn, cm = vertex.cuda(), face.cuda(), nv.cuda(), mf.cuda()
    g = dm.compute_triangle_geometry_(v, f)
    want = dm.mesh_decimation_(v, f, g, cn, cm, target(20, 20).cuda())
    for t in (target(20).cuda(), target(20).cuda()[0], target(20)[0], 20, 19.5, torch.tensor([19.25, 20.], device="cuda"),
              torch.tensor([20, 20], device="cuda")):
        for sizes in ((cn, cm), (cn.long(), cm.long())):
            got = dm.mesh_decimation_(v, f, g, *sizes, t)
            assert all(torch.equal(a, b) for a, b in zip(got, want))
    want = dm.mesh_decimation_(v, f, g, cn, cm, 20, True, 5.0)
    for t in (target(20), target(20)[0], torch.tensor([19.5, 20.]), target(20, 20).cuda()):
        got = MeshHierarchy([t], True, 5.0)(v, f, cn, cm)[1]
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.gpu
@pytest.mark.parametrize("stride", [1.1, 1.5, 2, 2.7, 3, 4, 5, 7, 10, 41, 47, 55, 61, 83])
def test_vertices_kept_per_stride(stride):
    """The whole range of counts: those of tensor / stride on the GPU, to the vertex."""
    n = torch.arange(0, 300001, dtype=torch.int32, device="cuda")
    want = torch.clip((n.to(torch.float) / float(stride)).to(torch.int), min=4).tolist()
    assert MeshHierarchy([stride], [4], True, 1.0)._target(0, n.tolist()) == want


@pytest.mark.gpu
def test_meshes_without_faces():
    """A vertex without a face is dropped: a batch, or a sample of it, that has none comes out empty."""
    vertex, face, _, _, _ = host_batch()
    v, f = vertex.cuda(), face[:80].cuda()
    none = torch.zeros(0, 3, dtype=torch.int32, device="cuda")
    out = dm.mesh_decimation_(v, none, torch.zeros(0, 5, device="cuda"), target(42, 42).cuda(), target(0, 0).cuda(), target(20, 20).cuda())
    assert [tuple(t.shape) for t in out[:3]] == [(0, 3), (0, 3), (0, 5)]
    assert out[3].tolist() == [0, 0] and out[4].tolist() == [0, 0] and out[6].tolist() == [-1] * 84
    out = dm.mesh_decimation_(v, f, dm.compute_triangle_geometry_(v, f), target(42, 42).cuda(), target(80, 0).cuda(), target(20, 20).cuda())
    w = v[:42].contiguous()
    alone = dm.mesh_decimation_(w, f, dm.compute_triangle_geometry_(w, f), target(42).cuda(), target(80).cuda(), target(20).cuda())
    assert out[3].tolist() == [int(alone[3]), 0] and all(torch.equal(a, b) for a, b in zip(out[:3], alone[:3]))
    levels = MeshHierarchy([4], [4], True, 1.0)(v, none, target(42, 42).cuda(), target(0, 0).cuda())
    assert levels[1][0].shape == (0, 3)
