"""Cases for timing the framework's public entry points.

Each case is one call (or the short sequence of calls) that a program using the package
makes, on synthetic volumes of the two kinds the workloads are quoted on: a sum of random
Gaussians plus a little noise, and a Gaussian random field with power spectrum k^-3
(zero mean, unit variance).  Both are made on the GPU from the seed.

Kinds of case:

  grad      lower_star_grad of a device volume (3D) or image (2D): the complete .grad
  host      steepest_lstar of a volume in pinned host memory: what the command line does
  batch     lower_star_grad_batch of volumes of uneven sizes
  labels    integrated_labels: both directions' destination labels of a volume and its .grad
  graph     ms_graph: the Morse-Smale complex nodes and arcs of a .grad (extractmsc's flags),
            put into the buffers of fixed capacity that the next stage reads
  conform   conforming_grad on a copy of the base .grad, from the final labels of both directions
  triage    triage_labels with the trained network
  train     one training pass of the triage network: forward, loss and every gradient
"""
import math

import numpy as np
import torch

import msceer_gb300 as msc
from msceer_gb300 import triage

DEV = "cuda"


# ---- volumes ------------------------------------------------------------------------------

def gaussian_sum(shape, n_gauss, seed, noise=1e-3):
    """Sum of n_gauss Gaussians (amplitudes U[-1,1], centres uniform, sigma U[3,10]) plus
    U[-noise,noise]; shape is (Z, Y, X)."""
    rng = np.random.default_rng(seed)
    axes = [torch.arange(n, dtype=torch.float64, device=DEV) for n in shape]
    out = torch.zeros(shape, dtype=torch.float64, device=DEV)
    for _ in range(n_gauss):
        a, s = float(rng.uniform(-1, 1)), float(rng.uniform(3, 10))
        e = [torch.exp(-(ax - float(rng.uniform(0, n))) ** 2 / (2 * s * s)) for ax, n in zip(axes, shape)]
        out += a * (e[0][:, None, None] * e[1][None, :, None] * e[2][None, None, :])
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    out += noise * (2 * torch.rand(shape, dtype=torch.float64, device=DEV, generator=gen) - 1)
    return out.float()


def power_law(shape, seed):
    """Gaussian random field with power spectrum k^-3; shape is (Z, Y, X) or (Y, X)."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    spec = torch.fft.rfftn(torch.randn(shape, dtype=torch.float32, device=DEV, generator=gen))
    k2 = torch.zeros(spec.shape, dtype=torch.float32, device=DEV)
    for a, n in enumerate(shape):
        k = torch.fft.rfftfreq(n, device=DEV) if a == len(shape) - 1 else torch.fft.fftfreq(n, device=DEV)
        k2 += (k * k).reshape([-1 if b == a else 1 for b in range(len(shape))])
    origin = (0,) * len(shape)
    k2[origin] = 1.0
    spec *= k2.pow_(-0.75)
    spec[origin] = 0.0
    f = torch.fft.irfftn(spec, s=shape).double()
    return ((f - f.mean()) / f.std()).float().contiguous()


def volume(case, seed):
    shape = (case["Z"], case["Y"], case["X"]) if "Z" in case else (case["Y"], case["X"])
    if case["field"] == "k3":
        return power_law(shape, seed)
    # as many Gaussians as keep the density of the 256^3 labeling workload, 16 at least
    return gaussian_sum(shape, max(16, min(64, round(64 * math.prod(shape) / 256**3))), seed)


def batch_shapes(case):
    """Edge lengths log-uniform in [lo, hi] per axis; the same for every seed of the inputs."""
    e = np.exp(np.random.default_rng(case["shapes"]).uniform(np.log(case["lo"]), np.log(case["hi"]), (case["n"], 3)))
    return [tuple(int(round(v)) for v in row) for row in e]


# ---- the cases ----------------------------------------------------------------------------

def vol(name, kind, field, x, y, z=None):
    c = {"name": name, "kind": kind, "field": field, "X": x, "Y": y}
    if z is not None:
        c["Z"] = z
    return c


def listed():
    return [
        # the small volume of the bit-exact check, one call: launches and synchronisations
        vol("grad_64", "grad", "gauss", 64, 64, 64),
        # the scale workload in 3D: a simulation snapshot resident on the device
        vol("grad_512", "grad", "k3", 512, 512, 512),
        # the scale workload in 2D
        vol("grad2d_8192", "grad", "k3", 8192, 8192),
        # the command line's path: an odd-sized scan in host memory, .grad back to the host
        vol("host_301x173x97", "host", "k3", 301, 173, 97),
        # an ensemble of uneven volumes in one call, buffers reused from frame to frame
        {"name": "batch_24", "kind": "batch", "n": 24, "lo": 32, "hi": 256, "shapes": 0},
        # labels of a small volume: latency of the whole labeling chain
        vol("labels_64", "labels", "gauss", 64, 64, 64),
        # the labeling workload: smooth features, long streamlines
        vol("labels_256", "labels", "gauss", 256, 256, 256),
        # labels at scale on a rough field: ten vertices a basin, the heaviest call
        vol("labels_512", "labels", "k3", 512, 512, 512),
        # the consumer of the .grad: nodes and arcs of the Morse-Smale complex
        vol("graph_256", "graph", "k3", 256, 256, 256),
        # the accurate 3-manifold .grad of an odd-sized volume
        vol("conform_223x187x241", "conform", "gauss", 223, 187, 241),
        # labels with the learned triage
        vol("triage_192", "triage", "k3", 192, 192, 192),
        # one training pass of the triage network at the size it is trained on
        {"name": "train_128", "kind": "train", "X": 128, "Y": 128, "Z": 128},
    ]


def _edges(rng, lo, hi, cap):
    """Three log-uniform edges in [lo, hi] with at most cap vertices."""
    while True:
        e = [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(3)]
        if math.prod(e) <= cap:
            return e


def draw(rng):
    kind = rng.choice(["grad", "grad2d", "host", "batch", "labels", "labels", "graph", "conform", "triage", "train"])
    field = rng.choice(["k3", "gauss"])
    if kind == "grad2d":
        x, y = (int(round(math.exp(rng.uniform(math.log(256), math.log(8192))))) for _ in range(2))
        return {"kind": "grad", "field": "k3", "X": x, "Y": y}
    if kind == "batch":
        return {"kind": "batch", "n": rng.randint(3, 24), "lo": 32, "hi": rng.randint(64, 256),
                "shapes": rng.randint(1, 1 << 20)}
    lo, hi, cap = {"grad": (32, 512, 512**3), "host": (48, 320, 160 * 160 * 256), "labels": (48, 400, 256**3),
                   "graph": (64, 320, 256**3), "conform": (64, 256, 256 * 192 * 192),
                   "triage": (48, 224, 192**3), "train": (48, 160, 128**3)}[kind]
    x, y, z = _edges(rng, lo, hi, cap)
    if kind == "train":
        return {"kind": kind, "X": x, "Y": y, "Z": z}
    return {"kind": kind, "field": field, "X": x, "Y": y, "Z": z}


# ---- inputs -------------------------------------------------------------------------------

def train_inputs(case, seed):
    """Features like the ones the labeling's first pass makes (10 of 16 channels: the value,
    the gradient magnitude, the unit flow direction, indicators of label boundaries, a
    fraction of neighbours and the neighbour's label), targets on ~9% of the vertices."""
    shape = (case["Z"], case["Y"], case["X"])
    f = power_law(shape, seed)
    gen = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
    g = torch.stack(torch.gradient(f), -1)
    mag = g.norm(dim=-1, keepdim=True)
    u = torch.rand(shape + (4,), device=DEV, generator=gen)
    feat = torch.zeros(shape + (16,), device=DEV)
    feat[..., 0] = f
    feat[..., 1:2] = mag / mag.mean()
    feat[..., 2:5] = g / mag.clamp_min(1e-12)
    feat[..., 5:8] = (u[..., :3] < torch.tensor([0.6, 0.3, 0.02], device=DEV)).float()
    feat[..., 8] = torch.round(6 * u[..., 3]) / 6
    feat[..., 9] = (u[..., 0] < 0.3).float()
    feat = feat.bfloat16()
    score = (feat[..., 5] * feat[..., 8]).float() + 0.5 * torch.rand(shape, device=DEV, generator=gen)
    tgt = (score > torch.quantile(score.reshape(-1)[:: max(1, f.numel() // 100000)], 0.91)).to(torch.uint8)
    return feat, torch.stack([tgt.reshape(-1)] * 2)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        feat, tgt = train_inputs(case, seed)
        rows = torch.stack([feat[..., :8], feat[..., 8:]], 2).contiguous().view(torch.int16).reshape(-1)
        return {"kind": kind, "shape": (case["Z"], case["Y"], case["X"]), "feat": rows, "tgt": tgt,
                "w": triage.TriageNet.load().weights, "pos": 10.0}
    if kind == "batch":
        vols = [power_law(s[::-1], seed * 1000 + i) for i, s in enumerate(batch_shapes(case))]
        outs = [torch.empty(msc.num_cells(v.shape[::-1]), dtype=torch.uint8, device=DEV) for v in vols]
        return {"kind": kind, "vols": vols, "outs": outs}
    f = volume(case, seed)
    if kind == "grad":
        return {"kind": kind, "f": f, "out": torch.empty(msc.num_cells(f.shape[::-1]), dtype=torch.uint8, device=DEV)}
    if kind == "host":
        out = torch.empty(msc.num_cells(f.shape[::-1]), dtype=torch.uint8, pin_memory=True)
        return {"kind": kind, "f": f.cpu().pin_memory().numpy(), "out": out.numpy()}
    s = {"kind": kind, "f": f, "g": msc.lower_star_grad(f)}
    if kind == "conform":
        lab = msc.integrated_labels(f, s["g"])
        s.update(asc=lab["asc"], dsc=lab["dsc"], out=torch.empty_like(s["g"]))
    elif kind == "triage":
        s["net"] = triage.TriageNet.load()
    elif kind == "graph":  # room for a node per vertex and two arcs (rough fields have 0.4 and 0.6)
        n = f.numel()
        s["buf"] = {"node_cell": torch.zeros(n, dtype=torch.int64, device=DEV),
                    "node_value": torch.zeros(n, dtype=torch.float32, device=DEV),
                    "node_dim": torch.zeros(n, dtype=torch.uint8, device=DEV),
                    "node_boundary": torch.zeros(n, dtype=torch.uint8, device=DEV),
                    "arc_lower": torch.zeros(2 * n, dtype=torch.int32, device=DEV),
                    "arc_upper": torch.zeros(2 * n, dtype=torch.int32, device=DEV),
                    "arc_persistence": torch.zeros(2 * n, dtype=torch.float32, device=DEV)}
    return s


# ---- one pass -----------------------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind == "grad":
        return msc.lower_star_grad(s["f"], s["out"])
    if kind == "host":
        return msc.steepest_lstar(s["f"], s["out"])
    if kind == "batch":
        return msc.lower_star_grad_batch(s["vols"], s["outs"])
    if kind == "labels":
        r = msc.integrated_labels(s["f"], s["g"])
        return {"asc": r["asc"], "dsc": r["dsc"]}
    if kind == "graph":
        for name, t in msc.ms_graph(s["g"], s["f"]).items():
            s["buf"][name][:t.numel()].copy_(t)
        return s["buf"]
    if kind == "conform":
        s["out"].copy_(s["g"])  # the call re-pairs the .grad in place; the base one is kept
        touched = msc.conforming_grad(s["f"], s["out"], s["asc"], s["dsc"])
        return {"grad": s["out"], "touched": touched}
    if kind == "triage":
        r = triage.triage_labels(s["f"], s["g"], s["net"])
        return {"asc": r["asc"], "dsc": r["dsc"]}
    a1, a2, logits = triage.forward(s["feat"], s["shape"], s["w"])
    loss, grads = triage.backward(s["feat"], a1, a2, logits, s["tgt"], s["shape"], s["w"], s["pos"])
    return {"logits": logits, "loss": loss, "grads": grads}


# ---- what a pass cannot do without ---------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "batch":
        v = [math.prod(s) for s in batch_shapes(case)]
        c = [math.prod(2 * n - 1 for n in s) for s in batch_shapes(case)]
        return {"bytes": 4 * sum(v) + sum(c), "flops": 0}
    e = [case[k] for k in "XYZ" if k in case]
    v, c = math.prod(e), math.prod(2 * n - 1 for n in e)
    if kind == "train":
        layer = 2 * 27 * 16 * 16 * v  # three forward, two input-gradient, three weight-gradient layers
        return {"bytes": (32 + 2 + 8) * v, "flops": 8 * layer}
    return {"bytes": {"grad": 4 * v + c, "host": 4 * v + c, "labels": 4 * v + c + 8 * v, "graph": 4 * v + c,
                      "conform": 12 * v + 2 * c, "triage": 4 * v + c + 8 * v}[kind], "flops": 0}


# ---- 64-bit values of the computed numbers -------------------------------------------------

def exact(case, seed):
    """The network's logits, loss and gradients in 64 bits; the other cases return bytes and
    labels, and a .grad's graph holds input values and their differences."""
    if case["kind"] != "train":
        return None
    feat, tgt = train_inputs(case, seed)
    w = triage.TriageNet.load().weights.double()
    nw = 27 * 256
    # [tap][cin][cout], tap = dx + 3 dy + 9 dz -> [cout][cin][dz][dy][dx]
    W = [w[i * nw:(i + 1) * nw].reshape(3, 3, 3, 16, 16).permute(4, 3, 0, 1, 2).contiguous().requires_grad_()
         for i in range(3)]
    b = [w[3 * nw + 16 * i:3 * nw + 16 * (i + 1)].clone().requires_grad_() for i in range(3)]

    def conv(x, k, bias):
        # one product per tap, so that no convolution library's choice of algorithm enters
        n, ci, Z, Y, X = x.shape
        p = torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1))
        out = bias[None, :, None, None, None].expand(n, -1, Z, Y, X)
        for t in range(27):
            dx, dy, dz = t % 3, t // 3 % 3, t // 9
            out = out + torch.einsum("nczyx,oc->nozyx", p[:, :, dz:dz + Z, dy:dy + Y, dx:dx + X], k[:, :, dz, dy, dx])
        return out

    x = feat.double().permute(3, 0, 1, 2)[None]
    h = torch.relu(conv(x, W[0], b[0]))
    h = torch.relu(conv(h, W[1], b[1]))
    z = conv(h, W[2][:2], b[2][:2])[0].reshape(2, -1)
    y = tgt.double()
    wt = torch.where(y > 0, 10.0, 1.0)
    loss = (wt * (torch.nn.functional.softplus(z) - y * z)).sum() / z.numel()
    loss.backward()
    flat = [k.grad.permute(2, 3, 4, 1, 0).reshape(-1) for k in W] + [t.grad for t in b]
    return {"logits": z.detach(), "loss": float(loss), "grads": torch.cat(flat)}
