"""Timed cases of the labeler's public entry points (labeling_b200).

Every case is one call, or one batch launch, as a user's program makes it, on seeded synthetic
images of the kinds the benchmark uses: Bernoulli noise (the dense noise of a threshold), a
one-pixel-wide spiral with random cuts (the deepest merge chains), filled disks over noise, and
thresholded Gaussian random fields (blobs, the usual content of volumes).  Sizes and densities are
those of the benchmark's configurations, of the batch (sides log-uniform in 64..2048) and of the
served mix (2D sides up to 8192, 3D sides 64..384, 512 for the plain volumes).  Tensors are dense
as torch gives them, so a width that is not a multiple of 16 gives rows of every alignment.

Kinds of a case:
  2d     label2d on a device image             3d     label3d on a device volume
  batch  Batch.run over uneven device images   host   Labeling.Label on a host image
`algo` names the form: auto (block equivalence), lbeq (pixel label equivalence, 4-connected),
runeq (run equivalence, 4-connected), iter (the iterative scan / analyze form).
"""
import functools
import math

import numpy as np
import torch

import labeling_b200 as be
from labeling_b200 import workloads

DEV = "cuda"
ALGO = {"auto": be.ALGO_AUTO, "lbeq": be.ALGO_PIXEL, "runeq": be.ALGO_RUNS, "iter": be.ALGO_ITER}


def listed():
    return [
        # The smallest call: one tile, the count read back -- launches and host latency.
        {"name": "2d-64-count", "kind": "2d", "h": 64, "w": 64, "family": "bern", "p": 0.5, "thr": 0, "algo": "auto", "count": True},
        # An ordinary image whose width is odd: every row starts at another alignment.
        {"name": "2d-1021x1787", "kind": "2d", "h": 1021, "w": 1787, "family": "bern", "p": 0.5, "thr": 8, "algo": "auto", "count": False},
        # The 2048 x 2048 configuration.
        {"name": "2d-2048", "kind": "2d", "h": 2048, "w": 2048, "family": "bern", "p": 0.5, "thr": 0, "algo": "auto", "count": False},
        # The 8192 x 8192 configuration: dense noise, and the deepest chains.
        {"name": "2d-8192-bern0.6", "kind": "2d", "h": 8192, "w": 8192, "family": "bern", "p": 0.6, "thr": 0, "algo": "auto", "count": False},
        {"name": "2d-8192-spiral", "kind": "2d", "h": 8192, "w": 8192, "family": "spiral", "p": 0.0, "thr": 0, "algo": "auto", "count": False},
        # A served volume: odd sides, blobs at the 60th percentile.
        {"name": "3d-191x223x157", "kind": "3d", "d0": 191, "d1": 223, "d2": 157, "family": "grf", "p": 0.4, "thr": 0, "algo": "auto", "count": True},
        # The 512^3 configuration: the noise with the most 26-connected links, and blobs.
        {"name": "3d-512-bern0.3", "kind": "3d", "d0": 512, "d1": 512, "d2": 512, "family": "bern", "p": 0.3, "thr": 0, "algo": "auto", "count": False},
        {"name": "3d-512-grf50", "kind": "3d", "d0": 512, "d1": 512, "d2": 512, "family": "grf", "p": 0.5, "thr": 0, "algo": "auto", "count": False},
        # The batch configuration: 4096 uneven images, densities U[0.2, 0.8], one graph launch.
        {"name": "batch-4096", "kind": "batch", "n": 4096, "lo": 64, "hi": 2048, "thr": 0},
        # The other forms of the algorithm selection, on the 2048 x 2048 configuration and twice that.
        {"name": "lbeq-2048", "kind": "2d", "h": 2048, "w": 2048, "family": "bern", "p": 0.5, "thr": 0, "algo": "lbeq", "count": False},
        {"name": "runeq-4096", "kind": "2d", "h": 4096, "w": 4096, "family": "bern", "p": 0.5, "thr": 0, "algo": "runeq", "count": False},
        # The drop-in labeler interface on a host frame (upload, label, download).
        {"name": "host-1080x1920", "kind": "host", "h": 1080, "w": 1920, "family": "bern", "p": 0.5, "thr": 8},
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def family(choices):
        f = rng.choice(choices)
        return f, round(rng.uniform(0.1, 0.9), 3) if f == "bern" else round(rng.uniform(0.2, 0.5), 3)

    kind = rng.choice(["2d", "2d", "2d", "2d", "3d", "3d", "3d", "batch", "batch", "form", "form", "host"])
    thr = rng.choice([0, 8, 128])
    if kind == "2d":
        f, p = family(["bern", "bern", "disks", "spiral"])
        return {"kind": "2d", "h": side(16, 8192), "w": side(16, 8192), "family": f, "p": p, "thr": thr, "algo": "auto", "count": rng.random() < 0.5}
    if kind == "form":
        f, p = family(["bern", "bern", "disks", "spiral"])
        return {"kind": "2d", "h": side(64, 4096), "w": side(64, 4096), "family": f, "p": p, "thr": thr, "algo": rng.choice(["lbeq", "runeq", "iter"]), "count": rng.random() < 0.5}
    if kind == "3d":
        f, p = family(["bern", "grf"])
        return {"kind": "3d", "d0": side(16, 512), "d1": side(16, 512), "d2": side(16, 512), "family": f, "p": p, "thr": thr, "algo": rng.choice(["auto", "auto", "auto", "lbeq"]),
                "count": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": "batch", "n": side(16, 2048), "lo": side(16, 128), "hi": side(256, 2048), "thr": thr}
    return {"kind": "host", "h": side(64, 2048), "w": side(64, 2048), "family": "bern", "p": round(rng.uniform(0.1, 0.9), 3), "thr": 8}


def _pixels(mask, thr, g):
    """Foreground mask -> uint8 pixels: 0 / 255 for threshold 0, gray values either side of it else."""
    if thr == 0:
        return mask.to(torch.uint8) * 255
    gray = torch.randint(0, 1 << 15, mask.shape, generator=g, device=DEV, dtype=torch.int16).to(torch.int32)
    return torch.where(mask, thr + 1 + gray % (255 - thr), gray % (thr + 1)).to(torch.uint8)


@functools.lru_cache(maxsize=2)
def _spiral(h, w):
    return torch.from_numpy(workloads.spiral(h, w)).to(DEV) != 0


def _mask(case, shape, seed, g):
    f, p = case["family"], case["p"]
    if f == "bern":
        return torch.rand(shape, generator=g, device=DEV) < p
    if f == "spiral":
        m = _spiral(*shape).clone()
        cuts = torch.randint(0, m.numel(), (128,), generator=g, device=DEV)
        m.view(-1)[cuts] = False
        return m
    if f == "disks":
        scale = max(shape)
        rmax = max(3.0, scale / 41)
        return torch.from_numpy(workloads.disks(shape[0], shape[1], 500, min(4, rmax / 2), rmax, 0.05, seed)).to(DEV) != 0
    # Gaussian random field of standard deviation 4 voxels, the fraction p of it foreground.
    spec = torch.fft.rfftn(torch.randn(shape, generator=g, device=DEV))
    for axis, n in enumerate(shape):
        fr = torch.fft.rfftfreq(n, device=DEV) if axis == len(shape) - 1 else torch.fft.fftfreq(n, device=DEV)
        spec *= torch.exp(-2 * math.pi ** 2 * 16.0 * fr * fr).reshape([-1 if i == axis else 1 for i in range(len(shape))])
    field = torch.fft.irfftn(spec, s=shape)
    del spec
    flat = field.reshape(-1)
    sample = flat[:: max(1, flat.numel() // 1000000)].sort().values
    return field > sample[min(sample.numel() - 1, int(sample.numel() * (1 - p)))]


@functools.lru_cache(maxsize=1)
def _context():
    return be.Context(0)


@functools.lru_cache(maxsize=1)
def _labeler():
    return be.make_labeler("bleq")


def _sides(case):
    """The images' sides of a batch: log-uniform, the same for every seed (the pixels are not)."""
    rng = np.random.default_rng(case["n"])
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    return np.exp(rng.uniform(lo, hi, (case["n"], 2))).round().astype(int).tolist()


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    if case["kind"] == "batch":
        sides = _sides(case)
        dens = np.random.default_rng(seed).uniform(0.2, 0.8, case["n"]).tolist()
        # Each image and label map starts 256-byte aligned, as the allocator gives tensors.
        at, total = [], 0
        for h, w in sides:
            at.append(total)
            total += (h * w + 255) // 256 * 256
        pix = torch.empty(total, dtype=torch.uint8, device=DEV)
        labels = torch.zeros(total, dtype=torch.int32, device=DEV)
        items = []
        for (h, w), p, o in zip(sides, dens, at):
            x, y = pix[o:o + h * w].view(h, w), labels[o:o + h * w].view(h, w)
            x.copy_(_pixels(torch.rand((h, w), generator=g, device=DEV) < p, case["thr"], g))
            items.append((x, y, case["thr"]))
        return {"case": case, "batch": be.Batch(_context(), items), "labels": labels}
    if case["kind"] == "host":
        img = _pixels(_mask(case, (case["h"], case["w"]), seed, g), case["thr"], g).cpu().numpy()
        return {"case": case, "labeler": _labeler(), "img": img}
    shape = (case["h"], case["w"]) if case["kind"] == "2d" else (case["d0"], case["d1"], case["d2"])
    img = _pixels(_mask(case, shape, seed, g), case["thr"], g)
    return {"case": case, "ctx": _context(), "img": img, "out": torch.empty(shape, dtype=torch.int32, device=DEV)}


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].run()
        return state["labels"]
    if case["kind"] == "host":
        labels, _ = state["labeler"].Label(state["img"])
        return labels
    label = be.label2d if case["kind"] == "2d" else be.label3d
    k = label(state["ctx"], state["img"], state["out"], threshold=case["thr"], algo=ALGO[case["algo"]], want_count=case["count"])
    return (state["out"], k) if case["count"] else state["out"]


def work(case):
    """One byte read and one int32 label written per pixel; labeling counts no floating operations."""
    if case["kind"] == "batch":
        px = sum(h * w for h, w in _sides(case))
    elif case["kind"] == "3d":
        px = case["d0"] * case["d1"] * case["d2"]
    else:
        px = case["h"] * case["w"]
    return {"bytes": 5.0 * px, "flops": 0.0}


def exact(case, seed):
    """Labels and counts are whole numbers: they are compared as they are."""
    return None
