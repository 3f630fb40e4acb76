"""Workloads of the geodesic distance transform, as a program that uses this package meets them.

Each case is a dict of plain values.  ``prepare`` makes what the program holds before the call (device tensors,
a batch plan, pinned host buffers, a running server), ``run`` is one pass through the public entry points,
``work`` the bytes and operations a pass cannot do without, ``exact`` the same maps in 64-bit arithmetic.

Kinds of case (``kind``) and the use each stands for:

* ``call``: one image in device memory, ``geodesic_distance_transform``.  ``content`` is the picture: ``blobs``
  (smooth gray with sensor noise, the usual photograph-like input), ``voronoi`` (piecewise constant rgb8 with
  noise) or ``maze`` (narrow winding corridors, the longest dependency chains a picture can have).  ``pitched``
  says whether rows start on 128-byte boundaries, as the package's own allocators lay them out, or the tensor is
  plainly contiguous, as most torch code has it.
* ``ref``: the reference's weight (8 neighbours, lambda blend), as a persistent run (``variant`` task) or in
  host-driven rounds (``variant`` blocks).
* ``batch``: a ragged batch of gray and rgb8 images in device memory, one call.
* ``plan``: the same as a prepared plan that a training or evaluation loop runs again and again.
* ``host``: a batch in pinned host memory, streamed through the device by the library.
* ``serve``: a burst of new images and then a burst of seed edits through the serving engine.
"""
import math

import numpy as np
import torch

import distance_transform_benchmarks_b200 as dtb
from distance_transform_benchmarks_b200 import workloads

GAMMA_GRAY = float(workloads.GAMMA_C0)


def listed():
    return [
        # The smallest call in use: a thumbnail or a crop with odd sides; launches and latency decide.
        dict(name="gray_97x61", kind="call", content="blobs", w=97, h=61, gamma=GAMMA_GRAY, seeds=3, pitched=True),
        # One ordinary small gray picture, the smallest benchmark configuration.
        dict(name="gray_512", kind="call", content="blobs", w=512, h=512, gamma=GAMMA_GRAY, seeds=5, pitched=True),
        # A photograph-sized rgb8 tensor as torch code holds it: contiguous, odd sides, rows off any alignment.
        dict(name="rgb_1333x1999", kind="call", content="voronoi", w=1333, h=1999, gamma=0.1, seeds=8, pitched=False),
        # The long-corridor configuration: one seed, serial fronts.
        dict(name="maze_4096", kind="call", content="maze", w=4096, h=4096, gamma=0.5, seeds=1, pitched=True),
        # The large single picture configuration.
        dict(name="rgb_8192", kind="call", content="voronoi", w=8192, h=8192, gamma=0.02, seeds=64, pitched=True),
        # The reference's benchmark shape through its task variant, and another blend and shape of it.
        dict(name="ref_3648x2432", kind="ref", variant="task", w=3648, h=2432, lam=0.5, seeds=5),
        dict(name="ref_1023x777_grad", kind="ref", variant="task", w=1023, h=777, lam=1.0, seeds=3),
        # The reference's blocks variant: rounds driven from the host.
        dict(name="ref_blocks_1500x1100", kind="ref", variant="blocks", w=1500, h=1100, lam=0.5, seeds=4),
        # A data loader's ragged device batch, one call with new buffers.
        dict(name="batch_48", kind="batch", n=48, smin=64, smax=1024, sizes=11),
        # The ragged batch configuration as a plan.
        dict(name="plan_512", kind="plan", n=512, smin=64, smax=2048, sizes=3),
        # The same kind of batch in pinned host memory.
        dict(name="host_64", kind="host", n=64, smin=64, smax=2048, sizes=7),
        # Interactive serving: pictures arrive together, then users add seeds to some of them.
        dict(name="serve_24_12", kind="serve", n=24, edits=12, smin=128, smax=1024, sizes=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "call", "call", "ref", "ref", "batch", "plan", "host", "serve"])
    if kind == "call":
        content = rng.choice(["blobs", "blobs", "voronoi", "voronoi", "maze"])
        if content == "maze":
            side = 32 * _log(rng, 8, 128)
            return dict(kind=kind, content=content, w=side, h=32 * _log(rng, 8, 128), gamma=rng.choice([0.1, 0.5]), seeds=1,
                        pitched=True)
        return dict(kind=kind, content=content, w=_log(rng, 64, 8192), h=_log(rng, 61, 8192),
                    gamma=rng.choice([0.01, 0.02, GAMMA_GRAY, 0.1, 1.0]), seeds=rng.randint(1, 64),
                    pitched=rng.random() < 0.6)
    if kind == "ref":
        variant = rng.choice(["task", "task", "blocks"])
        top = 3648 if variant == "task" else 1500
        return dict(kind=kind, variant=variant, w=_log(rng, 128, top), h=_log(rng, 128, top), lam=rng.choice([0.0, 0.1, 0.5, 0.9, 1.0]),
                    seeds=rng.randint(1, 12))
    smax = rng.choice([512, 1024, 2048])
    if kind == "serve":
        return dict(kind=kind, n=rng.randint(8, 24), edits=rng.randint(2, 16), smin=128, smax=min(smax, 1024),
                    sizes=rng.randrange(1 << 16))
    top = {"batch": 64, "plan": 400, "host": 64}[kind]
    return dict(kind=kind, n=_log(rng, 8, top), smin=64, smax=smax, sizes=rng.randrange(1 << 16))


# ------------------------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------------------------
def _specs(case):
    """(kind, w, h, gamma) of each image of a ragged case: sides log-uniform, gray and rgb8 in turn."""
    return [s[:4] for s in workloads.config3_specs(case["sizes"], case["n"], case["smin"], case["smax"])]


def _batch(case, seed):
    return [workloads.make_image(s + (workloads._seed_of(21, seed, i),)) for i, s in enumerate(_specs(case))]


def _picture(case, seed):
    """(img, mask) of a single-image case as numpy arrays."""
    w, h = case["w"], case["h"]
    rng = np.random.default_rng(workloads._seed_of(20, seed))
    content = case.get("content", "blobs")
    if content == "maze":
        img, (sx, sy) = workloads.maze_gray(workloads._seed_of(20, seed, 1), w, h)
        mask = np.zeros((h, w), np.uint8)
        mask[sy, sx] = 1
        return img, mask
    make = workloads.blobs_gray if content == "blobs" else workloads.voronoi_rgb
    return make(workloads._seed_of(20, seed, 1), w, h), workloads.random_disks(rng, w, h, case["seeds"], 2, 5)


def _flat_maps(shapes):
    """Distance maps of a batch with 128-byte rows in one device buffer (returned first)."""
    offs, off = [], 0
    for h, w in shapes:
        pitch = -(-w // 32) * 32
        offs.append((off, pitch))
        off += h * pitch
    flat = torch.zeros(off, dtype=torch.float32, device="cuda")
    return flat, [torch.as_strided(flat, (h, w), (p, 1), o) for (h, w), (o, p) in zip(shapes, offs)]


def _device(arr, pitched):
    return dtb.pitched_from(arr) if pitched else torch.from_numpy(arr).cuda()


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind in ("call", "ref"):
        img, mask = _picture(case, seed)
        pitched = case.get("pitched", True)
        st.update(img=_device(img, pitched), mask=_device(mask, pitched))
        h, w = mask.shape
        st["dist"] = dtb.pitched_empty(h, w, 1, torch.float32) if pitched else torch.empty((h, w), device="cuda")
        st.update({k: case[k] for k in ("gamma", "lam", "variant") if k in case})
        return st
    batch = _batch(case, seed)
    st["gammas"] = [b[2] for b in batch]
    if kind in ("batch", "plan"):
        st["imgs"] = [dtb.pitched_from(b[0]) for b in batch]
        st["masks"] = [dtb.pitched_from(b[1]) for b in batch]
        st["flat"], st["dists"] = _flat_maps([b[1].shape for b in batch])
        if kind == "plan":
            st["plan"] = dtb.BatchPlan(st["imgs"], st["masks"], st["gammas"], dists=st["dists"])
        return st
    if kind == "host":
        st["imgs"], st["masks"], st["dists"] = dtb.host_batch_arena([b[0] for b in batch], [b[1] for b in batch])
        st["n"] = len(batch)
        return st
    # serve: pinned inputs and outputs, as a front end that receives pictures has them
    st["imgs"], st["masks"], st["outs"] = dtb.host_batch_arena([b[0] for b in batch], [b[1] for b in batch])
    rng = np.random.default_rng(workloads._seed_of(22, seed))
    st["edits"] = []
    for j in range(min(case["edits"], len(batch))):
        h, w = batch[j][1].shape
        disks = [(int(rng.integers(0, w)), int(rng.integers(0, h)), int(rng.integers(2, 7))) for _ in range(int(rng.integers(1, 4)))]
        st["edits"].append((j, disks, torch.empty((h, w), dtype=torch.float32).pin_memory()))
    st["server"] = dtb.Server(1 << 29)
    st["next_id"] = 0  # each picture gets an id of its own; the server drops the least recently used ones
    return st


# ------------------------------------------------------------------------------------------------------
# One pass
# ------------------------------------------------------------------------------------------------------
def _answers(server, n):
    """Collects n completions, as a front end's event loop does."""
    while n > 0:
        for c in server.poll(64, wait_ms=1000):
            if c["status"] != 0:
                raise RuntimeError("request %d failed with status %d" % (c["request_id"], c["status"]))
            n -= 1


def run(st):
    kind = st["kind"]
    if kind == "call":
        return dtb.geodesic_distance_transform(st["img"], st["mask"], st["gamma"], dist=st["dist"])
    if kind == "ref":
        fn = dtb.generalised_distance_transform_task if st["variant"] == "task" else dtb.generalised_distance_transform_blocks
        return fn(st["img"], st["mask"], st["lam"], dist=st["dist"])
    if kind == "batch":
        dtb.geodesic_distance_transform_batch(st["imgs"], st["masks"], st["gammas"], dists=st["dists"])
        return st["flat"]
    if kind == "plan":
        st["plan"].run()
        return st["flat"]
    if kind == "host":
        return dtb.geodesic_distance_transform_batch(st["imgs"], st["masks"], st["gammas"], dists=st["dists"])
    srv, first = st["server"], st["next_id"]
    st["next_id"] += len(st["imgs"])
    for i, (img, mask) in enumerate(zip(st["imgs"], st["masks"])):
        srv.submit_image(first + i, img, mask, st["gammas"][i], st["outs"][i])
    _answers(srv, len(st["imgs"]))
    for j, disks, out in st["edits"]:
        srv.submit_edit(first + j, disks, out)
    _answers(srv, len(st["edits"]))
    return st["outs"] + [out for _, _, out in st["edits"]]


# ------------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ------------------------------------------------------------------------------------------------------
def work(case):
    """Each image and mask read once, each map written once (an edit also reads the map it starts from); one add
    and one comparison per directed edge (4 a pixel, 8 with the reference's neighbourhood)."""
    if case["kind"] in ("call", "ref"):
        px = case["w"] * case["h"]
        ch = 3 if case.get("content") == "voronoi" else 1
        return {"bytes": px * (ch + 1 + 4), "flops": px * (8 if case["kind"] == "call" else 16)}
    total = {"bytes": 0, "flops": 0}
    for i, (kind, w, h, _) in enumerate(_specs(case)):
        ch = 3 if kind == "rgb8" else 1
        total["bytes"] += w * h * (ch + 1 + 4)
        total["flops"] += w * h * 8
        if case["kind"] == "serve" and i < case["edits"]:
            total["bytes"] += w * h * (ch + 1 + 4 + 4)
            total["flops"] += w * h * 8
    return total


# ------------------------------------------------------------------------------------------------------
# The maps in 64-bit arithmetic
# ------------------------------------------------------------------------------------------------------
def _fixpoint(d, wh, wv, diag=None):
    """Shortest distances on the pixel grid: wh [H, W-1], wv [H-1, W] edge weights, diag = (down-right, down-left)
    weights [H-1, W-1].  Whole rows and columns are closed at once (prefix sums), until nothing falls any more."""
    sh = torch.nn.functional.pad(wh.cumsum(1), (1, 0))
    sv = torch.nn.functional.pad(wv.cumsum(0), (0, 0, 1, 0))

    def lower(d, new):
        return torch.where(new < d * (1 - 1e-13), new, d)

    while True:
        old = d
        for s, dim in ((sh, 1), (sv, 0)):
            d = lower(d, (d - s).cummin(dim).values + s)
            d = lower(d, (d + s).flip(dim).cummin(dim).values.flip(dim) - s)
        if diag is not None:
            for wd, a, b in ((diag[0], slice(None, -1), slice(1, None)), (diag[1], slice(1, None), slice(None, -1))):
                d = d.clone()
                d[1:, b] = torch.minimum(d[1:, b], d[:-1, a] + wd)
                d[:-1, a] = torch.minimum(d[:-1, a], d[1:, b] + wd)
        if torch.equal(d, old):
            return d


def exact(case, seed):
    # Only single pictures of up to a megapixel: the rest would take minutes.
    if case["kind"] not in ("call", "ref") or case["w"] * case["h"] > 1 << 20 or case.get("content") == "maze":
        return None
    img, mask = _picture(case, seed)
    x = torch.from_numpy(img).double().cuda()
    d = torch.where(torch.from_numpy(mask).cuda() != 0, 0.0, 1e10).double()
    if case["kind"] == "ref":
        lam = float(np.float32(case["lam"]))

        def edge(a, b, dist):
            return (1.0 - lam) * dist + lam * (a - b).abs()

        r2 = math.sqrt(2.0)
        return _fixpoint(d, edge(x[:, 1:], x[:, :-1], 1.0), edge(x[1:], x[:-1], 1.0),
                         (edge(x[1:, 1:], x[:-1, :-1], r2), edge(x[1:, :-1], x[:-1, 1:], r2)))
    g2 = float(np.float32(case["gamma"])) ** 2
    x = x if x.dim() == 3 else x.unsqueeze(2)

    def weight(a, b):
        return (1.0 + g2 * (a - b).square().sum(2)).sqrt()

    return _fixpoint(d, weight(x[:, 1:], x[:, :-1]), weight(x[1:], x[:-1]))
