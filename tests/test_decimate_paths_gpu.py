"""The clustering's two forms (a block per sample, the whole grid) and the long-row path of the edge kernel against the
sequential restatement, bit for bit, where the choice between them and the selection of the early stop can go wrong."""
import numpy as np
import pytest
import torch

from oracle import c_oracle
from picassoplus_b200 import synth
from test_decimate_gpu import check_against_oracle, dm, on, oracle_decimation, planar_grid

pytestmark = pytest.mark.gpu


def batch(meshes):
    v = np.concatenate([m[0] for m in meshes]).astype(np.float32)
    off = np.cumsum([0] + [m[0].shape[0] for m in meshes[:-1]])
    f = np.concatenate([m[1] + o for m, o in zip(meshes, off)]).astype(np.int32)
    nv, mf = (np.array([m[i].shape[0] for m in meshes], np.int32) for i in (0, 1))
    return v, f, c_oracle.triangle_geometry(v, f), nv, mf


def fan(n):
    """n triangles round one hub (long vertex rows), the rim closed."""
    a = np.linspace(0, 2 * np.pi, n, endpoint=False)
    v = np.concatenate([[[0, 0, 0.3]], np.stack([np.cos(a), np.sin(a), 0.1 * np.sin(5 * a)], 1)])
    i = np.arange(n)
    return v, np.stack([np.zeros(n, np.int64), 1 + i, 1 + (i + 1) % n], 1)


def book(n):
    """n pages that share one edge: with few vertices to keep, all of them join the cluster of its two ends."""
    a = np.linspace(0, 2 * np.pi, n, endpoint=False)
    v = np.concatenate([[[0, 0, 0], [0, 0, 1]], np.stack([np.cos(a), np.sin(a), np.full(n, 0.5)], 1)])
    i = np.arange(n)
    return v, np.stack([np.zeros(n, np.int64), np.ones(n, np.int64), 2 + i], 1)


# 96 x 96: 16 245 faces, one block's sample at most; 98 x 98: the grid
@pytest.mark.parametrize("sizes", [(96, 20, 33), (98, 20, 33), (130, 120, 8)])
@pytest.mark.parametrize("frac", [0.05, 0.3, 0.45, 0.75])
def test_samples_and_grid(sizes, frac):
    meshes = [synth.heightfield(n, seed=n) for n in sizes] + [planar_grid(17)]
    v, f, geo, nv, mf = batch(meshes)
    remove = np.floor(nv * frac).astype(np.int32)
    remove[1] = 0
    check_against_oracle(torch.device("cuda"), [v, f, geo, np.cumsum(nv).astype(np.int32), np.cumsum(mf).astype(np.int32), remove],
                         True, 5.0)


@pytest.mark.parametrize("n", [15, 16, 17, 33, 500, 2500])
@pytest.mark.parametrize("frac", [0.2, 0.8])
def test_hub_vertices(n, frac):
    v, f, geo, nv, mf = batch([fan(n), fan(7), synth.icosphere(1)])
    remove = np.floor(nv * frac).astype(np.int32)
    check_against_oracle(torch.device("cuda"), [v, f, geo, np.cumsum(nv).astype(np.int32), np.cumsum(mf).astype(np.int32), remove],
                         False, 1.0)


@pytest.mark.parametrize("n,D", [(16, 3), (17, 3), (18, 40), (33, 3), (300, 5), (2000, 3), (20000, 3)])
def test_large_clusters(n, D):
    """Clusters around and above what a thread sorts by itself, several of them, rows wider than a warp."""
    v, f, geo, nv, mf = batch([book(n), synth.icosphere(1), book(n + 40), fan(30), book(19)])
    if D > 3:
        v = np.concatenate([v, np.random.default_rng(n).standard_normal((v.shape[0], D - 3))], 1).astype(np.float32)
    remove = (nv - 3).astype(np.int32)
    got, _ = check_against_oracle(torch.device("cuda"), [v, f, geo, np.cumsum(nv).astype(np.int32), np.cumsum(mf).astype(np.int32),
                                                         remove], False, 1.0)
    assert int(got["vtReplace"].max()) >= n - 3


@pytest.mark.parametrize("mesh,keep", [(book, 3), (fan, 100000)])
def test_time_of_large_clusters_and_hubs_is_not_quadratic(mesh, keep):
    """200 000 pages of a book, a fan of 200 000 triangles: some 0.1 s where the work grows with the lists, minutes with their square."""
    import time
    dev = torch.device("cuda")
    for n in (2000, 200000):
        v, f, geo, nv, mf = batch([mesh(n)])
        args = [on(dev, a) for a in (v, f, geo, nv, mf, (nv - min(keep, n // 2)).astype(np.int32))]
        t0 = time.perf_counter()
        dm().simplify(*args, False, 1.0)
        torch.cuda.synchronize()
        assert time.perf_counter() - t0 < (0.25 if n == 2000 else 3)


@pytest.mark.parametrize("sizes,stride", [((40, 30), 4), ((110,), 16)])
def test_pass_loop(sizes, stride):
    """mesh_decimation_ (native loop) against the same loop over the restatement: meshes, sizes and clusters identical."""
    dev = torch.device("cuda")
    v, f, geo, nv, mf = batch([synth.heightfield(n, seed=n + 1) for n in sizes])
    target = np.maximum(nv // stride, 16).astype(np.int32)
    geo = dm().compute_triangle_geometry_(on(dev, v), on(dev, f)).cpu().numpy()
    d = dict(vertex=torch.from_numpy(v), face=torch.from_numpy(f), geometry=torch.from_numpy(geo), nv=torch.from_numpy(nv),
             mf=torch.from_numpy(mf))
    want = oracle_decimation(d, target, True, 1.0)
    got = dm().mesh_decimation_(on(dev, v), on(dev, f), on(dev, geo), on(dev, nv), on(dev, mf), on(dev, target), True, 1.0)
    got = [got[i].cpu().numpy() for i in (0, 1, 3, 4, 5, 6)]
    assert np.array_equal(got[2], want[2]) and np.array_equal(got[3], want[3])
    assert np.array_equal(got[1], want[1]) and np.array_equal(got[4], want[4]) and np.array_equal(got[5], want[5])
    assert np.array_equal(got[0].view(np.uint32), want[0].view(np.uint32))


def test_face_across_samples():
    v, f, geo, nv, mf = batch([synth.icosphere(1), synth.icosphere(1)])
    f[3, 1] = 60
    dev = torch.device("cuda")
    args = [on(dev, a) for a in (v, f, geo, np.cumsum(nv).astype(np.int32), np.cumsum(mf).astype(np.int32), nv // 2)]
    with pytest.raises(RuntimeError, match="two samples"):
        dm().simplify(*args, True, 1.0)


def test_other_threads_go_on_while_the_gpu_is_waited_for():
    """A loader thread prepares a batch behind a long kernel; the main thread's interpreter runs meanwhile."""
    import threading
    import time
    dev = torch.device("cuda")
    v, f, geo, nv, mf = batch([synth.icosphere(3)])
    args = [on(dev, a) for a in (v, f, geo, nv, mf, nv // 4)]
    want = dm().mesh_decimation_(*args)
    got, ticks = [], 0
    torch.cuda.synchronize()

    def load():
        torch.cuda._sleep(600_000_000)                       # some 0.3 s
        got.extend(dm().mesh_decimation_(*args))
    loader = threading.Thread(target=load)
    loader.start()
    while loader.is_alive():
        time.sleep(0.001)
        ticks += 1
    loader.join()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert ticks >= 50
