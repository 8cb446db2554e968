"""The work a user of the codec has it do, as cases that can be timed and compared.

Every family goes through the public Python host (csvb200) over the C ABI.  The volumes are the benchmark's
seeded generators (smooth Voronoi cells, neurite-like tubes over them, dense thin tubes) at the benchmark's own
sizes or smaller, with their cell and tube counts scaled with the volume:

  decode   brick requests -> labels on the device: a captured graph of a whole data set, or one batch call
  encode   device volume -> .csbd image on the device, brick edge 16, 32 or 64
  image    host .csbd bytes -> host labels (parse, copy, seek index, decode, copy back)
  serve    frames of the viewer's loop along an orbit: plan, cache, on-demand decode, 1080p ray march
  select   an encode with a mode and table per brick: from the network, or from the exhaustive search
  train    one training step of the selector network: forward, backward, Adam

listed() names one case per kind of use; draw() gives others of the same ranges.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "fast-compressed-segmentation_b200"))

FOV = math.pi / 3
MLP = (("W1", 256, 64), ("b1", 256, 1), ("W2", 256, 256), ("b2", 256, 1), ("W3", 32, 256), ("b3", 32, 1))


def listed():
    return [
        # what one frame of a moving viewer asks for: a few blocks of one data set at the LODs their distance needs
        dict(name="decode_blocks", op="decode", x=320, y=256, z=200, fill="neurite", brick=64, left=0, blocks=24,
             lod=-1, graph=False),
        # a whole data set of dense thin tubes at full resolution, its edges padded to whole bricks; palettes of
        # several hundred labels, streams up to about 100 KB
        dict(name="decode_dense", op="decode", x=500, y=470, z=333, fill="dense", brick=64, left=0, blocks=0, lod=6,
             graph=False),
        # the benchmark's uneven batch: the x < 512 half in 32^3 bricks, the rest in 64^3, one graph replay
        dict(name="decode_mixed1024", op="decode", x=1024, y=1024, z=1024, fill="mixed", brick=64, left=32, blocks=0,
             lod=6, graph=True),
        # the smallest encodes: a cut-out of a few bricks, no edge a multiple of the brick
        dict(name="encode_cutout", op="encode", x=150, y=97, z=70, fill="neurite", brick=32),
        # the benchmark's encode, a neurite-like 512^3 volume in 64^3 bricks
        dict(name="encode_neurite512", op="encode", x=512, y=512, z=512, fill="neurite", brick=64),
        # many small bricks: smooth cells in 32^3 bricks
        dict(name="encode_cells32", op="encode", x=1024, y=512, z=500, fill="voronoi", brick=32),
        # a file from elsewhere opened for a preview: no index in it, coarse labels to the host
        dict(name="image_preview", op="image", x=512, y=512, z=256, fill="neurite", brick=64, lod=3),
        # the viewer's loop: label and depth frames along an orbit, blocks decoded as they come into view
        dict(name="serve_orbit", op="serve", x=768, y=768, z=768, fill="neurite", width=1920, height=1080, frames=6,
             rgba=False),
        # the same as the viewer shows it: transfer function, shading, shadow rays
        dict(name="serve_rgba", op="serve", x=512, y=512, z=512, fill="neurite", width=1920, height=1080, frames=2,
             rgba=True),
        # an encode that lets the network choose mode and table of each brick
        dict(name="select_learned", op="select", x=512, y=512, z=320, fill="neurite", brick=64, how="network"),
        # the search it replaces, which also labels its training data
        dict(name="select_search", op="select", x=384, y=320, z=300, fill="neurite", brick=64, how="search"),
        # a step of its training at the benchmark's batch
        dict(name="train_step", op="train", rows=2048),
    ]


def draw(rng):
    op = rng.choice(["decode", "decode", "decode", "encode", "encode", "encode", "image", "serve", "select", "train"])

    def sides(lo, hi, least=40, most=1024):
        """Three edges of about equal length whose product is spread over [lo, hi] in its logarithm."""
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        e = n ** (1 / 3)
        a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
        return [int(min(most, max(least, round(v)))) for v in (e * a, e * b, e / (a * b))]

    if op == "decode":
        fill = rng.choice(["neurite", "dense", "mixed", "voronoi"])
        x, y, z = sides(1 << 19, 1 << 29)
        left = 32 if fill == "mixed" else 0
        if left:  # the two brick sizes meet in the middle, on a border of both
            x = max(128, x // 128 * 128)
        brick = 64 if left else rng.choice([32, 64, 64])
        top = brick.bit_length() - 1
        blocks = rng.choice([0, 0, rng.randint(1, 200)])
        return dict(op=op, x=x, y=y, z=z, fill=fill, brick=brick, left=left, blocks=blocks,
                    lod=rng.choice([top, top, rng.randint(2, top), -1]), graph=rng.random() < 0.5)
    if op == "encode":
        x, y, z = sides(1 << 18, 1 << 28)
        return dict(op=op, x=x, y=y, z=z, fill=rng.choice(["neurite", "dense", "voronoi"]),
                    brick=rng.choice([16, 32, 64, 64]))
    if op == "image":
        x, y, z = sides(1 << 18, 1 << 26)
        brick = rng.choice([32, 64])
        return dict(op=op, x=x, y=y, z=z, fill=rng.choice(["neurite", "dense", "voronoi"]), brick=brick,
                    lod=rng.randint(1, brick.bit_length() - 1))
    if op == "serve":
        x, y, z = sides(1 << 22, 1 << 28)
        w, h = rng.choice([(1920, 1080), (1280, 720), (rng.randint(320, 1600), rng.randint(240, 900))])
        rgba = rng.random() < 0.4
        return dict(op=op, x=x, y=y, z=z, fill="neurite", width=w, height=h,
                    frames=rng.randint(1, 2) if rgba else rng.randint(1, 6), rgba=rgba)
    if op == "select":
        how = rng.choice(["network", "search"])
        x, y, z = sides(1 << 19, 1 << (27 if how == "network" else 25), least=64)
        return dict(op=op, x=x, y=y, z=z, fill=rng.choice(["neurite", "dense"]), brick=rng.choice([32, 64]), how=how)
    return dict(op="train", rows=int(math.exp(rng.uniform(math.log(100), math.log(20000)))))


# ---------------------------------------------------------------- inputs
_codec = None


def codec():
    """The program's one context."""
    global _codec
    if _codec is None:
        from csvb200 import Codec
        _codec = Codec(0)
    return _codec


def volume(c, seed):
    """The case's label volume, (z, y, x) int64 on the device, from the benchmark's generators."""
    W, H, D = c["x"], c["y"], c["z"]
    vol = torch.empty((D, H, W), dtype=torch.int64, device="cuda")
    n = W * H * D

    def of(per, cube):  # `per` things in a volume of cube^3 voxels
        return max(2, round(per * n / cube ** 3))

    kind, cells, tubes, r0, r1, zero = {
        "neurite": (1, of(3000, 512), of(400, 512), 2.0, 12.0, 0.15),
        "dense": (1, of(2000, 1024), of(80000, 1024), 0.5, 1.5, 0.0),
        "voronoi": (0, of(2000, 1024), 0, 0.0, 0.0, 0.1),
        "mixed": (2, of(2000, 1024), of(5000, 1024), 1.0, 4.0, 0.0),
    }[c["fill"]]
    codec().synth_volume(vol, kind, cells, tubes, r0, r1, zero, 1 + seed % (1 << 40))
    return vol


def prepare(case, seed):
    return globals()["prepare_" + case["op"]](case, seed)


def run(state):
    return globals()["run_" + state["op"]](state)


# ---------------------------------------------------------------- decode
def prepare_decode(c, seed):
    from csvb200 import DecodeConfig, requests, requests_tensor
    k, b, rng = codec(), c["brick"], np.random.default_rng(1)  # (which blocks, at which LOD: the case's, not the data's)
    vol, parts = volume(c, seed), []
    for lo, hi, edge in ([(0, c["x"] // 2, c["left"]), (c["x"] // 2, c["x"], b)] if c["left"] else [(0, c["x"], b)]):
        k.encode_device(vol[:, :, lo:hi].contiguous(), edge)
        parts.append(k.open_encoded())
    del vol
    ds = k.concat(parts) if len(parts) > 1 else parts[0]
    top = np.concatenate([[p.brick_size.bit_length() - 1] * p.num_bricks for p in parts])
    bricks = np.arange(len(top))
    if c["blocks"]:  # this many of them, in the order in which a viewer came to want them
        bricks = rng.permutation(len(top))[:c["blocks"]]
    lods = rng.integers(2, top[bricks] + 1) if c["lod"] < 0 else np.minimum(top[bricks], c["lod"])
    sizes = 8 ** lods.astype(np.uint64)
    dst = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.uint64)
    s = dict(op="decode", ds=ds, parts=parts, reqs=requests_tensor(requests(bricks, lods, dst)),
             out=torch.empty(int(sizes.sum()), dtype=torch.int64, device="cuda"),
             status=torch.empty(len(bricks), dtype=torch.int32, device="cuda"), graph=None)
    if c["graph"]:  # the configuration the autotuner settles on for uneven batches: all that fit, staged, longest first
        s["graph"] = k.decode_graph(ds, s["reqs"], s["out"], s["status"], DecodeConfig(0, 1, 1, 0))
    return s


def run_decode(s):
    if s["graph"] is not None:
        s["graph"].launch()
    else:
        codec().decode_batch(s["ds"], s["reqs"], s["out"], s["status"])
    return s["out"], s["status"]


# ---------------------------------------------------------------- encode
def image_buffer(vol):
    """Where the program keeps an encoded image (the context's own copy lives until its next encode)."""
    return torch.zeros(vol.numel() + (1 << 16), dtype=torch.uint8, device="cuda")


def keep_image(buf):
    img = codec().encoded_image_tensor()
    buf[:img.numel()].copy_(img)
    return img.numel(), buf


def prepare_encode(c, seed):
    vol = volume(c, seed)
    return dict(op="encode", vol=vol, brick=c["brick"], image=image_buffer(vol))


def run_encode(s):
    codec().encode_device(s["vol"], s["brick"])
    return keep_image(s["image"])


# ---------------------------------------------------------------- image
def prepare_image(c, seed):
    codec().encode_device(volume(c, seed), c["brick"])
    return dict(op="image", img=bytes(codec().encoded_image_tensor().cpu().numpy()), lod=c["lod"])


def run_image(s):
    return codec().decode_image(s["img"], s["lod"])


# ---------------------------------------------------------------- serve
def prepare_serve(c, seed):
    from csvb200 import Server
    from csvb200.camera import orbit
    k, rng = codec(), np.random.default_rng(seed)
    k.encode_device(volume(c, seed), 64)
    ds = k.open_encoded()
    nb = ds.num_bricks
    srv = Server(k, ds, c["width"], c["height"], FOV, cache_bytes=2 * 8 * nb * 64 ** 3 + (1 << 20))
    # the benchmark's orbit: two turns in 600 frames at 1600 to 3600 voxels from a 2048^3 volume
    size = (c["x"] * c["y"] * c["z"]) ** (1 / 3)
    centre, yaw0 = [c["x"] / 2, c["y"] / 2, c["z"] / 2], rng.uniform(0, 2 * math.pi)
    pitch, radius = rng.uniform(-0.35, 0.35), size / 2048 * rng.uniform(1600, 3600)
    views, bufs, n = [], [], c["width"] * c["height"]
    for f in range(c["frames"]):
        views.append(orbit(centre, radius, yaw0 + 4 * math.pi * f / 600, pitch))
        kinds = [torch.int32] if c["rgba"] else [torch.int64, torch.float32]
        bufs.append([torch.empty(n, dtype=t, device="cuda") for t in kinds])
    return dict(op="serve", srv=srv, ds=ds, views=views, bufs=bufs, rgba=c["rgba"])


def run_serve(s):
    srv = s["srv"]
    for (pos, d), b in zip(s["views"], s["bufs"]):
        (srv.submit_rgba if s["rgba"] else srv.submit)(0, pos, d, *b)
        srv.step()
        srv.poll(wait=False, max_frames=8)
    return s["bufs"]


# ---------------------------------------------------------------- select
def prepare_select(c, seed):
    from csvb200 import SelectorNet
    from csvb200.selector import build_model
    vol, b = volume(c, seed), c["brick"]
    # 16 shared tables around the op statistics of encoded volumes: many Rp and neighbour ops, few palette ops
    rng = np.random.default_rng(seed)
    base = np.array([30, 60, 6, 20, 6, 20, 6, 20, 1, 2, 3, 8, 2, 5, 1, 1], float)
    tables = np.stack([build_model(1e5 * base * rng.gamma(2.0, 0.5, 16)) for _ in range(16)])
    nb = math.prod(-(-n // b) for n in vol.shape)
    return dict(op="select", vol=vol, brick=b, tables=tables, how=c["how"], image=image_buffer(vol),
                net=SelectorNet(codec(), SelectorNet.init_params(seed % (1 << 30))),
                hist=torch.empty((nb, 12, 16), dtype=torch.int32, device="cuda"),
                sel=torch.empty(nb, dtype=torch.uint8, device="cuda"))


def run_select(s):
    k = codec()
    if s["how"] == "network":
        k.encode_learned(s["vol"], s["brick"], s["net"], s["tables"])
        return keep_image(s["image"])
    k.encode_stats(s["vol"], s["brick"], s["hist"])
    k.select_exhaustive(s["hist"], s["tables"], s["sel"])
    k.encode_device_sel(s["vol"], s["brick"], s["tables"], s["sel"])
    return s["hist"], s["sel"], keep_image(s["image"])


# ---------------------------------------------------------------- train
def batch(c, seed):
    """Feature rows as brick statistics are (shares in [0, 1], groups that sum to one), labels a function of them."""
    rng = np.random.default_rng(seed)
    n = c["rows"]
    f = rng.random((n, 32))
    f[:, 8:15] = rng.dirichlet(np.full(7, 0.7), n)
    f[:, 16:32] = rng.dirichlet(np.full(16, 0.5), n)
    f = f.astype(np.float32)
    w = rng.normal(size=(32, 28))
    z = f.astype(np.float64) @ w
    return f, (z[:, :12].argmax(1) | (z[:, 12:].argmax(1) << 4)).astype(np.uint8)


def params(seed):
    """He-uniform weights, small biases, in csv_mlp_create's order; what the network does not use is zero."""
    rng, p = np.random.default_rng(seed + 1), []
    for name, r, k in MLP:
        w = rng.uniform(-1, 1, (r, k)) * (0.05 if name[0] == "b" else math.sqrt(6.0 / (32 if name == "W1" else 256)))
        if name == "W1":
            w[:, 32:] = 0
        if name[1] == "3":
            w[28:] = 0
        p.append(w.ravel())
    return np.concatenate(p).astype(np.float32)


def prepare_train(c, seed):
    from csvb200 import SelectorNet
    f, y = batch(c, seed)
    return dict(op="train", net=SelectorNet(codec(), params(seed)), f=torch.from_numpy(f).cuda(),
                y=torch.from_numpy(y).cuda())


def run_train(s):
    loss = s["net"].grad(s["f"], s["y"])
    s["net"].adam(2e-3)
    p, g = s["net"].params(grads=True)
    return {"loss": loss, "params": p, "grads": g}


def exact_train(c, seed):
    f, y = batch(c, seed)
    p, at, w = torch.from_numpy(params(seed)).double(), 0, {}
    for name, r, k in MLP:
        w[name] = p[at:at + r * k].clone().view(r, k).requires_grad_()
        at += r * k
    y = torch.from_numpy(y.astype(np.int64))
    h = torch.relu(torch.from_numpy(f).double() @ w["W1"][:, :32].T + w["b1"].T)
    h = torch.relu(h @ w["W2"].T + w["b2"].T)
    z = h @ w["W3"].T + w["b3"].T
    ce = torch.nn.functional.cross_entropy
    loss = ce(z[:, :12], y & 15) + ce(z[:, 12:28], y >> 4)
    loss.backward()
    # (a first Adam step moves every weight by its gradient's sign: near zero that has no exact value)
    return {"loss": float(loss), "params": None, "grads": torch.cat([w[n].grad.reshape(-1) for n, _, _ in MLP])}


def exact(case, seed):
    """The training step in 64 bits; everything else is whole numbers."""
    return exact_train(case, seed) if case["op"] == "train" else None


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    c = dict(case)
    if c["op"] == "train":
        m = 64 * 256 + 256 * 256 + 256 * 32
        return {"bytes": c["rows"] * (32 * 4 + 1) + 4 * 6 * m, "flops": 3 * 2.0 * c["rows"] * m}
    if c["op"] == "serve":
        return {"bytes": c["frames"] * c["width"] * c["height"] * (4 if c["rgba"] else 12), "flops": 0}

    def bricks(x, b):
        return math.prod(-(-n // b) for n in (x, c["y"], c["z"]))

    voxels = c["x"] * c["y"] * c["z"]
    if c["op"] in ("encode", "select"):  # the volume read once; the image is a few percent of it
        return {"bytes": 8 * voxels, "flops": 0}
    # labels written once (a mixed-LOD request by the mean of its LODs); the streams are a few percent of them
    def labels(n, b, lod):
        top = b.bit_length() - 1
        return n * (sum(8 ** k for k in range(2, top + 1)) / (top - 1) if lod < 0 else 8 ** min(lod, top))

    if c["op"] == "image":
        return {"bytes": 8 * labels(bricks(c["x"], c["brick"]), c["brick"], c["lod"]) + voxels // 20, "flops": 0}
    halves = [(c["x"] // 2, c["left"]), (c["x"] - c["x"] // 2, c["brick"])] if c["left"] else [(c["x"], c["brick"])]
    every = [(bricks(x, b), b) for x, b in halves]
    n = sum(k for k, _ in every)
    share = min(1.0, c["blocks"] / n) if c["blocks"] else 1.0
    return {"bytes": 8 * share * sum(labels(k, b, c["lod"]) for k, b in every) + 16 * share * n, "flops": 0}
