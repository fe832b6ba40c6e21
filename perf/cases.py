"""The work that the framework's performance is measured on.

Six kinds of it, each through the public entry points and each over a range of sizes:

  block      one training step (forward + backward) of the V2F -> F2F -> F2V block, block.conv_block
  texture    the texture entry of a scene network: SH basis of the sample positions, F2FConv3d on RGB samples, training
  encoder    training step of an encoder: per mesh level a V2VConv3d module and a max pool, then one row per mesh
  segment    inference of an encoder-decoder: V2VConv3d and average pool down, unpool and PerItemConv3d up
  hierarchy  what a network does with a new batch before its first convolution: MeshHierarchy, then prepare_level per level
  points     training step of the point-cloud convolution, fuzzy or hard bins

Meshes are either batches of icospheres with radial noise ("ico", size = subdivision level: shape analysis) or batches
of height fields with a tenth of the faces missing ("grid", size = vertices along an edge: scenes).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from picassoplus_b200 import synth, topology
from picassoplus_b200.block import conv_block
from picassoplus_b200.math_utils import sph_harm_coeff
from picassoplus_b200.mesh.layers import F2FConv3d, GlobalPool3d, PerItemConv3d, Pool3d, SphHarmCoeff, Unpool3d, V2VConv3d
from picassoplus_b200.mesh.pi_modules import conv3d, fused
from picassoplus_b200.mesh.utils import MeshHierarchy
from picassoplus_b200.point.layers import PCloudConv3d

DEV = "cuda"


# ---------------------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # a single small shape: the step is launches and host work
        dict(name="block_one_shape", kind="block", mesh="ico", size=3, batch=1, cin=32, cout=64, L=3, precision="fp32"),
        # a shape-analysis batch (64 meshes of 642 vertices)
        dict(name="block_shapes", kind="block", mesh="ico", size=3, batch=64, cin=64, cout=128, L=3, precision="fp32"),
        # two scenes of 700 x 700 vertices
        dict(name="block_scenes", kind="block", mesh="grid", size=700, batch=2, cin=64, cout=64, L=3, precision="fp32"),
        # the multi-GPU configuration's whole batch on one GPU: the largest case
        dict(name="block_batch", kind="block", mesh="grid", size=360, batch=32, cin=128, cout=128, L=4, precision="fp32"),
        # an eighth of that batch (its shard on eight GPUs) with bf16 operands
        dict(name="block_shard_bf16", kind="block", mesh="grid", size=360, batch=4, cin=128, cout=128, L=4, precision="bf16"),
        # RGB texture samples of two scenes, one to four per facet
        dict(name="texture_scenes", kind="texture", mesh="grid", size=700, batch=2, cin=3, cout=32, L=3),
        # the encoder stack of the scene configuration, and one for a batch of shapes
        dict(name="encoder_scenes", kind="encoder", mesh="grid", size=700, batch=2, c0=64, c1=128, c2=256, c3=384, L=3),
        dict(name="encoder_shapes", kind="encoder", mesh="ico", size=3, batch=64, c0=32, c1=64, c2=96, c3=128, L=3),
        # one scene of odd size at inference
        dict(name="segment_scene", kind="segment", mesh="grid", size=351, batch=1, c0=32, c1=64, c2=128, L=3),
        # preparation of new batches: scenes, shapes
        dict(name="hierarchy_scenes", kind="hierarchy", mesh="grid", size=700, batch=2, levels=3, L=3),
        dict(name="hierarchy_shapes", kind="hierarchy", mesh="ico", size=3, batch=64, levels=2, L=3),
        # a cloud of a quarter million points, up to 16 neighbours, three fuzzy bins per pair
        dict(name="points_scene", kind="points", np=262144, mp=65537, knn=16, bins=17, fuzzy=3, cin=64, cout=64),
    ]


def _between(rng, lo, hi):
    """A whole number of [lo, hi], even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng, most_vertices):
    """A mesh kind, size and batch of at most about `most_vertices` vertices."""
    if rng.random() < 0.4:
        size = rng.randint(2, 4)
        return dict(mesh="ico", size=size, batch=_between(rng, 1, min(128, most_vertices // (10 * 4 ** size + 2))))
    size = _between(rng, 24, min(700, int(math.sqrt(most_vertices))))
    return dict(mesh="grid", size=size, batch=_between(rng, 1, max(1, min(32, most_vertices // size ** 2))))


def draw(rng):
    kind = rng.choice(["block", "block", "block", "texture", "encoder", "segment", "hierarchy", "points"])
    if kind == "block":
        widths = [16, 24, 32, 48, 64, 96, 100, 128]
        return dict(kind=kind, **_mesh(rng, 32 * 360 ** 2), cin=rng.choice(widths), cout=rng.choice(widths),
                    L=rng.randint(2, 4), precision=rng.choice(["fp32", "fp32", "fp32", "bf16"]))
    if kind == "texture":
        return dict(kind=kind, **_mesh(rng, 2 * 700 ** 2), cin=3, cout=rng.choice([16, 32, 48, 64]), L=rng.randint(2, 4))
    if kind == "encoder":
        a = rng.choice([16, 32, 48, 64])
        return dict(kind=kind, **_mesh(rng, 2 * 700 ** 2), c0=a, c1=2 * a, c2=rng.choice([2 * a, 3 * a, 4 * a]),
                    c3=rng.choice([3 * a, 4 * a, 6 * a]), L=rng.randint(2, 3))
    if kind == "segment":
        a = rng.choice([16, 32, 48, 64])
        return dict(kind=kind, **_mesh(rng, 2 * 700 ** 2), c0=a, c1=rng.choice([a, 2 * a]), c2=rng.choice([2 * a, 4 * a]),
                    L=rng.randint(2, 3))
    if kind == "hierarchy":
        return dict(kind=kind, **_mesh(rng, 32 * 360 ** 2), levels=rng.randint(1, 3), L=rng.randint(2, 3))
    mp = _between(rng, 500, 262144)
    return dict(kind=kind, np=mp * rng.choice([1, 2, 4]) + rng.randint(0, 3), mp=mp, knn=rng.choice([8, 16, 24]),
                bins=rng.choice([9, 17, 33]), fuzzy=rng.choice([0, 0, 3]), cin=rng.choice([16, 32, 48, 64, 128]),
                cout=rng.choice([32, 64, 128]))


# --------------------------------------------------------------------------------------------------------------- inputs
def _rng(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _normal(g, *shape):
    return torch.randn(*shape, device=DEV, generator=g)


@functools.lru_cache(maxsize=8)
def _icosphere(level):
    v, f = synth.icosphere(level)
    return torch.from_numpy(v.astype(np.float32)).to(DEV), torch.from_numpy(f.astype(np.int32)).to(DEV)


def _ico_batch(level, batch, g):
    """`batch` icospheres with radial noise of +-10 %."""
    v0, f0 = _icosphere(level)
    radius = 0.9 + 0.2 * torch.rand(batch, v0.shape[0], 1, device=DEV, generator=g)
    first = torch.arange(batch, dtype=torch.int32, device=DEV).mul_(v0.shape[0]).view(-1, 1, 1)
    return (v0 * radius).reshape(-1, 3), (f0 + first).reshape(-1, 3), [v0.shape[0]] * batch, [f0.shape[0]] * batch


def _grid_faces(n):
    return 2 * (n - 1) ** 2 - (n - 1) ** 2 // 5


def _grid_batch(n, batch, g):
    """`batch` height fields of n x n vertices on the unit square: four octaves of noise, a tenth of the faces missing."""
    z = torch.zeros(batch, 1, n, n, device=DEV)
    for octave in range(4):
        cells = 4 << octave
        lattice = torch.rand(batch, 1, cells + 1, cells + 1, device=DEV, generator=g) * 2 - 1
        z += 0.5 ** (octave + 1) * torch.nn.functional.interpolate(lattice, size=(n, n), mode="bicubic", align_corners=True)
    line = torch.linspace(0, 1, n, device=DEV)
    xy = torch.stack(torch.meshgrid(line, line, indexing="xy"), -1).expand(batch, n, n, 2)
    vertex = torch.cat([xy, z.view(batch, n, n, 1)], -1).reshape(-1, 3).contiguous()
    at = torch.arange(n * n, dtype=torch.int32, device=DEV).view(n, n)
    a, b, c, d = at[:-1, :-1].flatten(), at[:-1, 1:].flatten(), at[1:, :-1].flatten(), at[1:, 1:].flatten()
    one = torch.stack([torch.stack([a, b, c], 1), torch.stack([b, d, c], 1)], 1).reshape(-1, 3)
    first = torch.arange(batch, dtype=torch.int32, device=DEV).mul_(n * n).view(-1, 1, 1)
    # a fifth of the lower triangles goes; the upper ones and the last one stay, so that every vertex keeps a face
    order = torch.rand(batch, (n - 1) ** 2 - 1, device=DEV, generator=g).argsort(1)
    keep = torch.ones(batch, (n - 1) ** 2, 2, dtype=torch.bool, device=DEV)
    keep[:, :, 1].scatter_(1, order[:, :(n - 1) ** 2 // 5], False)
    return vertex, (one + first)[keep.view(batch, -1)], [n * n] * batch, [_grid_faces(n)] * batch


def _batch(case, g):
    make = _ico_batch if case["mesh"] == "ico" else _grid_batch
    return make(case["size"], case["batch"], g)


def _level(vertex, face, L):
    """A mesh level as the convolutions take it."""
    nv = vertex.shape[0]
    vt_map = torch.arange(nv, dtype=torch.int32, device=DEV)
    prep = topology.prepare_level(vertex, face, vt_map, nv, L, want_geometry=False)
    return dict(vertex=vertex, face=face, vt_map=vt_map, nf_count=prep["nf_count"], coeff=prep["coeff"])


def _samples(nf, g):
    """One to four texture samples per face: (nf,) counts and (samples, 3) barycentric coordinates."""
    counts = torch.randint(1, 5, (nf,), dtype=torch.int32, device=DEV, generator=g)
    e = -torch.log(torch.rand(int(counts.sum()), 3, device=DEV, generator=g) + 1e-9)
    return counts, (e / e.sum(1, keepdim=True)).contiguous()


def _stack(case, g, levels, train):
    """A hierarchy (a quarter of the vertices per level) and one V2VConv3d module per level."""
    vertex, face, nv, mf = _batch(case, g)
    sizes = [torch.tensor(s, dtype=torch.int32, device=DEV) for s in (nv, mf)]
    hier = MeshHierarchy([4] * levels, [16] * levels, True, 1.0)(vertex, face, *sizes)
    ch = [case["c%d" % i] for i in range(levels + 1)]
    convs = [V2VConv3d(ch[i], [ch[i + 1], ch[i + 1]], case["L"], [1, 1]).to(DEV).train(train) for i in range(levels)]
    return dict(levels=[_level(h[0][:, :3].contiguous(), h[1].contiguous(), case["L"]) for h in hier],
                clusters=[(h[5], h[6]) for h in hier[1:]], coarsest=hier[-1][3], convs=convs, channels=ch,
                x=_normal(g, vertex.shape[0], ch[0]))


def prepare(case, seed):
    g = _rng(seed)
    torch.manual_seed(int(seed))                            # the layers draw their weights from the global generator
    s = dict(case)
    kind = case["kind"]
    if kind == "block":
        vertex, face, _, _ = _batch(case, g)
        s.update(_level(vertex, face, case["L"]))
        counts, bary = _samples(face.shape[0], g)
        s["cum"] = torch.cumsum(counts, 0, dtype=torch.int32)
        s["means"] = topology.face_means_sph_harm(case["L"], bary, s["cum"])
        s["sh_eye"] = sph_harm_coeff(case["L"], torch.eye(3, device=DEV))
        K, cin, cout = (case["L"] + 1) ** 2, case["cin"], case["cout"]
        s["x"] = _normal(g, vertex.shape[0], cin).requires_grad_()
        s["weights"] = [_normal(g, K, cin).mul_((2 / (K + cin)) ** 0.5).requires_grad_(),
                        _normal(g, cout, cin, K).mul_((2 / (K * (cin + cout))) ** 0.5).requires_grad_(),
                        _normal(g, K, cout, 1).mul_((2 / (K + cout)) ** 0.5).requires_grad_()]
        s["upstream"] = _normal(g, vertex.shape[0], cout)
    elif kind == "texture":
        _, face, _, _ = _batch(case, g)
        s["counts"], s["bary"] = _samples(face.shape[0], g)
        s["rgb"] = torch.rand(s["bary"].shape[0], case["cin"], device=DEV, generator=g)
        s["basis"] = SphHarmCoeff(case["L"])
        s["conv"] = F2FConv3d(case["cin"], case["cout"], case["L"]).to(DEV).train()
        s["upstream"] = _normal(g, face.shape[0], case["cout"])
    elif kind == "encoder":
        s.update(_stack(case, g, 3, True), pool=Pool3d("max"), last=GlobalPool3d("avg"))
        s["x"].requires_grad_()
        s["weights"] = [p for c in s["convs"] for p in c.parameters()]
        s["state"] = [b for c in s["convs"] for n, b in c.named_buffers() if n.endswith(("running_mean", "running_var"))]
        s["upstream"] = _normal(g, case["batch"], case["c3"])
    elif kind == "segment":
        s.update(_stack(case, g, 2, False), pool=Pool3d("avg"), unpool=Unpool3d())
        ch = s["channels"]
        s["heads"] = [PerItemConv3d(ch[2] + ch[1], ch[1]).to(DEV).eval(), PerItemConv3d(ch[1] + ch[0], ch[0]).to(DEV).eval()]
    elif kind == "hierarchy":
        s["vertex"], s["face"], nv, mf = _batch(case, g)
        s["nv"], s["mf"] = (torch.tensor(t, dtype=torch.int32, device=DEV) for t in (nv, mf))
        s["build"] = MeshHierarchy([4] * case["levels"], [16] * case["levels"], True, 1.0)
        # the levels go into fixed buffers behind one another, as a loader hands them on: how many faces a coarse level
        # has (and how many vertices, where a cluster has lost all its faces) is known only once it is there
        nv, nf, K = s["vertex"].shape[0], s["face"].shape[0], (case["L"] + 1) ** 2
        s["packed"] = {k: torch.zeros(2 * rows * w, dtype=t, device=DEV) for k, rows, w, t in
                       (("vertex", nv, 3, torch.float32), ("replace", nv, 1, torch.int32), ("map", nv, 1, torch.int32),
                        ("nf_count", nv, 1, torch.int32), ("rowptr", nv, 1, torch.int32), ("face", nf, 3, torch.int32),
                        ("geometry", nf, 5, torch.float32), ("normals", nf, 3, torch.float32),
                        ("coeff", nf, K, torch.float32), ("entries", nf, 3, torch.int32))}
    else:
        npts, mp, knn, T = case["np"], case["mp"], case["knn"], case["fuzzy"]
        # pairs as a radius search emits them: grouped by output point, neighbours near it in the ordering of the cloud
        counts = torch.randint(knn // 2, knn + 1, (mp,), device=DEV, generator=g)
        centre = torch.repeat_interleave(torch.arange(mp, device=DEV), counts)
        near = centre * (npts // mp) + torch.randint(-1024, 1025, centre.shape, device=DEV, generator=g)
        s["nn_index"] = torch.stack([centre, near.clamp_(0, npts - 1)], 1).to(torch.int32).contiguous()
        s["nn_count"] = counts.to(torch.int32)
        s["bin_index"] = torch.randint(0, case["bins"], centre.shape + ((T,) if T else ()), dtype=torch.int32, device=DEV,
                                       generator=g)
        s["bin_coeff"] = None
        if T:
            w = torch.rand(centre.shape[0], T, device=DEV, generator=g) + 0.05
            s["bin_coeff"] = (w / w.sum(1, keepdim=True)).contiguous()
        s["conv"] = PCloudConv3d(case["cin"], case["cout"], case["bins"]).to(DEV).train()
        s["x"] = _normal(g, npts, case["cin"]).requires_grad_()
        s["upstream"] = _normal(g, mp, case["cout"])
    return s


# ----------------------------------------------------------------------------------------------------------------- pass
def _run_block(s):
    conv3d.set_f2f_precision(s["precision"])
    out = conv_block(s["x"], *s["weights"], s["face"], s["cum"], s["means"], s["coeff"], s["nf_count"], s["vt_map"],
                     s["sh_eye"])
    return out, torch.autograd.grad(out, [s["x"]] + s["weights"], s["upstream"])


def _run_texture(s):
    conv3d.set_f2f_precision("fp32")
    conv = s["conv"]
    out = conv(s["rgb"], s["basis"](s["bary"]), s["counts"])             # the samples themselves are data: no gradient
    return out, torch.autograd.grad(out, list(conv.parameters()), s["upstream"])


def _run_encoder(s):
    fused.set_pointwise_precision("fp32")
    x = s["x"]
    for i, conv in enumerate(s["convs"]):
        lv = s["levels"][i]
        x = conv(x, lv["face"], lv["nf_count"], lv["vt_map"], lv["coeff"])
        x = s["pool"](x, *s["clusters"][i], s["levels"][i + 1]["vertex"])
    x = s["last"](x, s["coarsest"])
    return x, torch.autograd.grad(x, [s["x"]] + s["weights"], s["upstream"]), s["state"]


def _run_segment(s):
    fused.set_pointwise_precision("fp32")
    with torch.no_grad():
        x, skips = s["x"], []
        for i, conv in enumerate(s["convs"]):
            lv = s["levels"][i]
            skips.append(x)
            x = conv(x, lv["face"], lv["nf_count"], lv["vt_map"], lv["coeff"])
            x = s["pool"](x, *s["clusters"][i], s["levels"][i + 1]["vertex"])
        for head, clusters, skip in zip(s["heads"], reversed(s["clusters"]), reversed(skips)):
            x = head(torch.cat([s["unpool"](x, *clusters), skip], 1))
    return x


def _run_hierarchy(s):
    counts, levels = [], {k: [] for k in s["packed"]}
    for vertex, face, geometry, nv, mf, replace, vmap in s["build"](s["vertex"], s["face"], s["nv"], s["mf"]):
        vt_map = torch.arange(vertex.shape[0], dtype=torch.int32, device=DEV)
        prep = topology.prepare_level(vertex, face, vt_map, vertex.shape[0], s["L"], orient=True, want_geometry=False,
                                      want_normals=True)
        counts.append((nv, mf))
        for k, t in dict(vertex=vertex, replace=replace, map=vmap, nf_count=prep["nf_count"], rowptr=prep["csr"].rowptr,
                         face=face, geometry=geometry, normals=prep["normals"], coeff=prep["coeff"],
                         entries=prep["csr"].entries).items():
            if t is not None:                               # the first level has no clusters
                levels[k].append(t.reshape(-1))
    for k, parts in levels.items():
        torch.cat(parts, out=s["packed"][k][:sum(p.shape[0] for p in parts)])
    return counts, s["packed"]


def _run_points(s):
    conv = s["conv"]
    out = conv(s["x"], s["nn_count"], s["nn_index"], s["bin_index"], s["bin_coeff"])
    return out, torch.autograd.grad(out, [s["x"]] + list(conv.parameters()), s["upstream"])


_RUN = dict(block=_run_block, texture=_run_texture, encoder=_run_encoder, segment=_run_segment, hierarchy=_run_hierarchy,
            points=_run_points)


def run(state):
    return _RUN[state["kind"]](state)


# ---------------------------------------------------------------------------------------------------- work and tolerance
def _sizes(case):
    """Vertices and faces of the case's meshes."""
    if case["mesh"] == "ico":
        return case["batch"] * (10 * 4 ** case["size"] + 2), case["batch"] * 20 * 4 ** case["size"]
    return case["batch"] * case["size"] ** 2, case["batch"] * _grid_faces(case["size"])


def work(case):
    kind = case["kind"]
    if kind == "points":
        pairs, ci, co = 0.75 * case["knn"] * case["mp"], case["cin"], case["cout"]
        bins = 8 * case["fuzzy"] if case["fuzzy"] else 4
        return dict(bytes=8 * ci * case["np"] + 8 * co * case["mp"] + pairs * (8 + bins),
                    flops=6 * case["mp"] * ci * co + 6 * pairs * ci * (1 + case["fuzzy"]))
    nv, nf = _sizes(case)
    K = (case["L"] + 1) ** 2
    if kind == "block":
        ci, co = case["cin"], case["cout"]
        return dict(bytes=8 * (ci + co) * nv + nf * (12 + 8 * K) + 8 * K * ci * co,
                    flops=6 * nf * (K * ci * co + 3 * ci + K * co + 3 * co))
    if kind == "texture":
        ci, co, ns = case["cin"], case["cout"], 2.5 * nf
        return dict(bytes=4 * ns * (ci + 3) + 4 * nf * (1 + 2 * co), flops=4 * nf * K * ci * co + 4 * ns * K * ci)
    if kind == "hierarchy":
        b = f = 0
        for i in range(case["levels"] + 1):
            v, t = nv / 4 ** i, nf / 4 ** i
            b += v * 12 + t * 12 + (8 * 4 * v if i else 0)                 # vertices, faces, clusters over the level before
            b += t * (20 + 12 + 4 * K + 12) + 8 * v                        # geometry, normals, basis, adjacency
            f += t * (150 + 10 * K)
        return dict(bytes=b, flops=f)
    levels, times = (3, 3) if kind == "encoder" else (2, 1)                # training: forward and two products backward
    ch = [case["c%d" % i] for i in range(levels + 1)]
    b = 4 * nv * ch[0] * (2 if times == 3 else 1) + 8 * case["batch"] * ch[levels] * (times - 1)
    f = 0
    for i in range(levels):
        v, t = nv / 4 ** i, nf / 4 ** i
        b += t * (12 + 4 * K) + 24 * v
        f += 2 * times * (t * (3 * ch[i] + ch[i] * ch[i + 1] + K * ch[i + 1] + 3 * ch[i + 1]) + v * ch[i + 1] ** 2)
    if kind == "segment":
        b += 4 * nv * ch[0]
        f += 2 * (nv / 4 * (ch[2] + ch[1]) * ch[1] + nv * (ch[1] + ch[0]) * ch[0])
    return dict(bytes=b, flops=f)


def tolerance(case):
    if case["kind"] == "block" and case["precision"] == "bf16":
        return {"rel": 1e-2}
    if case["kind"] == "hierarchy":
        return {"rel": 2e-6, "differ": 0.0}
    if case["kind"] in ("block", "segment"):
        return {"rel": 5e-5}                                # products of bf16 hi + lo pairs: 16 bits of every operand
    # training through ReLU (and max pooling): a pre-activation within rounding error of zero, or two candidates of a
    # maximum that close, may fall on either side in a correct implementation.  A share p of flipped entries moves the
    # gradients by sqrt(p) in the 2-norm, and p is about the 1e-5 of the activations' own error.
    return {"rel": 1e-2}
