"""The workloads whose speed this package answers for.

Each case is a dict of plain values.  ``kind`` names what a user's program calls:

``predict``   ``layer.compute_activation(x)`` on a device tensor: inference, and every layer below the one in training
``step``      ``compute_activation`` + ``train_step`` of a structural-plasticity layer on device tensors: the body of the
              unsupervised training loop, with a mask update for one hypercolumn after another where ``mask`` is set
``classify``  ``compute_activation`` + ``train_step`` of the dense output layer on one-hot labels
``host``      ``layer.step_host`` on numpy arrays: the same step for a program that keeps its batches in host memory
``fit``       ``Network.fit`` of a two-layer network on numpy arrays: two epochs of the hidden layer (the second one
              updates the mask), one of the classifier, dataset upload and shuffling included
``kernel``    ``kernels_b200.update_weights``, the drop-in for the reference's fused kernel, on numpy arrays

``n`` inputs feed ``hc`` hypercolumns of ``mc`` units, ``batch`` samples at a time.  Inputs are pixels, ``dark`` of them
zero, complementary-coded where ``coded`` is set.  The layers start from the traces of a layer that has already been trained (with the constructor's constant traces the mask score is 0/0).
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

from streambrain_b200 import kernels_b200
from streambrain_b200.backend.b200_backend import DenseLayer, Network, StructuralPlasticityLayer

# Hyper-parameters of the MNIST runs (trace constants are per batch of 128, scaled by sqrt(batch / 128)).
TAUPDT, PMIN, KHALF, TAUBDT, OUT_TAUPDT = 0.006908854922437549, 0.06195283356566607, -139.02586632856327, 0.02218100432360414, 0.0007449780036161324

CLASSES = 10
BATCHES = 4                # batches a state holds and takes in turn
BATCH_BYTES = 512 << 20    # ... as far as they fit this


def listed():
    return [
        # one sample through the MNIST hidden layer: a serving call, where launches and the host path are all there is
        dict(name="predict_one_f32", kind="predict", dtype="float32", n=1568, hc=30, mc=100, batch=1, density=0.1, dark=0.8, coded=True),
        # the training driver's MNIST network (784 raw pixels, 15 x 200 units) in its double mode, forward pass
        dict(name="predict_f64", kind="predict", dtype="float64", n=784, hc=15, mc=200, batch=128, density=0.1, dark=0.8, coded=False),
        # the output layer of every configuration: 3000 hidden units to 10 classes
        dict(name="classify_f32", kind="classify", dtype="float32", n=3000, hc=1, mc=CLASSES, batch=128),
        # the MNIST hidden layer in both precisions (complementary-coded pixels, 30 x 100 units)
        dict(name="step_mnist_f32", kind="step", dtype="float32", n=1568, hc=30, mc=100, batch=128, density=0.1, mask=True, dark=0.8, coded=True),
        dict(name="step_mnist_f64", kind="step", dtype="float64", n=1568, hc=30, mc=100, batch=128, density=0.1, mask=True, dark=0.8, coded=True),
        # odd sizes: a user's own features and hypercolumns, and the short last batch of an epoch
        dict(name="step_ragged_f32", kind="step", dtype="float32", n=1001, hc=13, mc=37, batch=97, density=0.2, mask=True, dark=0.8, coded=False),
        # the wide hidden layer (100 x 300 units) at batch 1024
        dict(name="step_wide_f32", kind="step", dtype="float32", n=1568, hc=100, mc=300, batch=1024, density=0.1, mask=True, dark=0.8, coded=True),
        # the STL-10 layer, whose traces and weights are 664 MB each: the benchmark's default workload
        dict(name="step_stl10_f32", kind="step", dtype="float32", n=55296, hc=30, mc=100, batch=256, density=0.568746541818903, mask=True, dark=0.0, coded=True),
        # the same layer at the large-batch configuration's batch of 8192, on one device
        dict(name="step_stl10_large_batch_f32", kind="step", dtype="float32", n=55296, hc=30, mc=100, batch=8192, density=0.568746541818903, mask=False, dark=0.0, coded=True),
        # the MNIST step for a program whose batches are numpy arrays
        dict(name="host_step_f32", kind="host", dtype="float32", n=1568, hc=30, mc=100, batch=128, density=0.1, mask=True, dark=0.8, coded=True),
        # the training driver on Fashion-MNIST-shaped data: 784 pixels, 30 x 100 units, a last batch of 8 samples
        dict(name="fit_fashion_f32", kind="fit", dtype="float32", n=784, hc=30, mc=100, batch=128, density=0.1, samples=5000, dark=0.8, coded=False),
        # the reference's kernel interface in its default precision, at the driver's layer
        dict(name="kernel_weights_f64", kind="kernel", dtype="float64", n=784, hc=15, mc=200, batch=128, dark=0.8, coded=False),
    ]


def draw(rng):
    """One more case of the same ranges: every kind, both precisions, sizes spread over their logarithm, about half of
    them with rows that start on 16-byte boundaries and half odd."""
    def size(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    largest = 8192 * 55296 * 3000
    while True:
        kind = rng.choice(["predict", "step", "step", "step", "classify", "host", "fit", "kernel"])
        c = dict(kind=kind, dtype="float32" if rng.random() < 0.7 else "float64", n=size(64, 55296), hc=size(1, 100), mc=size(2, 300), batch=size(1, 8192))
        even = rng.random() < 0.5
        if kind == "classify":
            c.update(hc=1, mc=CLASSES, n=size(64, 30000), batch=size(1, 1024))
        elif kind == "fit":
            c.update(n=size(64, 4096), hc=size(1, 30), batch=size(32, 512))
        elif kind in ("host", "kernel"):
            c.update(batch=size(1, 1024))
        if even:
            c["n"] = (c["n"] + 7) // 8 * 8
            if kind != "classify":
                c["mc"] = (c["mc"] + 3) // 4 * 4
        m = c["hc"] * c["mc"]
        if kind == "fit":
            # at least one batch per hypercolumn and one more: the mask schedule needs them
            c["samples"] = min(20000, c["batch"] * (c["hc"] + 1) + size(1, 8000))
            if -(-c["samples"] // c["batch"]) <= c["hc"]:
                continue
        if kind != "classify":
            c.update(dark=rng.choice([0.0, 0.8]), coded=c["n"] % 2 == 0 and rng.random() < 0.5)
        if kind != "classify" and kind != "kernel":
            c["density"] = round(rng.uniform(0.1, 0.6), 3)
        if kind in ("step", "host"):
            c["mask"] = rng.random() < 0.5
        # no dearer than the largest listed case: float64 and odd rows run at a fraction of the float32 tensor rate
        cost = c["batch"] * c["n"] * m * (8 if c["dtype"] == "float64" else 1 if even else 5)
        if kind == "fit":
            cost *= 3 * c["samples"] / c["batch"]
        limit = 16 << 20 if kind in ("host", "fit", "kernel") else 55296 * 3000 // (2 if c["dtype"] == "float64" else 1)
        if c["n"] * m <= limit and cost <= largest and c["batch"] * max(c["n"], m) <= 8192 * 55296:
            return c


class _Trained:
    """Skips the constructors' draw of an initial state on the host (seconds for the largest layers): the caller writes
    the state of a trained layer on the device instead."""

    def __init__(self, n, hc, mc, taupdt, dtype, **more):
        self.in_features, self.hypercolumns, self.minicolumns, self.out_features, self.taupdt = n, hc, mc, hc * mc, taupdt
        for k, v in more.items():
            setattr(self, k, v)
        self._create(dtype, {})


class _Hidden(_Trained, StructuralPlasticityLayer):
    use_mask_iterations = False


class _Output(_Trained, DenseLayer):
    pass


def _pixels(c, gen, rows):
    dt, k = getattr(torch, c["dtype"]), c["n"] // 2 if c["coded"] else c["n"]
    p = torch.rand((rows, k), generator=gen, device="cuda", dtype=dt)
    if c["dark"] > 0:
        p *= torch.rand((rows, k), generator=gen, device="cuda") >= c["dark"]
    return torch.stack((p, 1 - p), dim=2).reshape(rows, c["n"]) if c["coded"] else p


def _labels(c, gen, rows):
    t = torch.zeros((rows, CLASSES), device="cuda", dtype=getattr(torch, c["dtype"]))
    return t.scatter_(1, torch.randint(0, CLASSES, (rows, 1), generator=gen, device="cuda"), 1)


def _units(c, gen, rows, hc, mc):
    """Activations of a trained hidden layer: a softmax with a few strong units per hypercolumn."""
    a = torch.randn((rows, hc, mc), generator=gen, device="cuda", dtype=getattr(torch, c["dtype"]))
    return torch.softmax(a.mul_(3), dim=2).reshape(rows, hc * mc)


def _trained_traces(gen, ci, m, mc, spread, dt):
    """Ci, Cj and a joint trace whose ratio to the independent one is log-normal, below both marginals."""
    ci = ci.clamp(0.02, 0.98).to(dt)
    cj = (torch.rand(m, generator=gen, device="cuda", dtype=dt) * 0.4 + 0.8) / mc
    cij = torch.randn((ci.numel(), m), generator=gen, device="cuda", dtype=dt).mul_(spread).exp_()
    cij.mul_(ci[:, None]).mul_(cj[None, :])
    torch.minimum(cij, torch.minimum(ci[:, None], cj[None, :]).mul_(0.98), out=cij)
    return ci, cj, cij


def _fill(layer, gen, ci, density=None):
    """Writes a trained state: the log-ratio weights under a random mask, the bias of the marginals."""
    n, hc, mc, m = layer.in_features, layer.hypercolumns, layer.minicolumns, layer.out_features
    dt = torch.float32 if layer.dtype == np.float32 else torch.float64
    s = {k: layer.state_tensor(k) for k in layer._state_names}
    for view in s.values():
        view.layer = layer   # the views are of the layer's own memory: whoever holds one keeps the layer
    spread = min(0.5, 17 / math.sqrt(n * (density or 1)))   # the wider the layer, the weaker its single connections
    ci, cj, cij = _trained_traces(gen, ci, m, mc, spread, dt)
    s["Ci"].copy_(ci)
    s["Cj"].copy_(cj)
    s["Cij"].copy_(cij)
    s["bias"].copy_(cj.log())
    cij.div_(ci[:, None]).div_(cj[None, :]).log_()
    if density is not None:
        s["kbi"].fill_(1)
        s["wmask"].copy_(torch.rand((n, hc), generator=gen, device="cuda") < density)
        cij.view(n, hc, mc).mul_(s["wmask"][:, :, None])
    s["weights"].copy_(cij)
    return s


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind, n, hc, mc, b = c["kind"], c["n"], c["hc"], c["mc"], c["batch"]
    dt = getattr(np, c["dtype"])
    scale = math.sqrt(b / 128)
    s = SimpleNamespace(kind=kind, hc=hc, mask=c.get("mask", False), passes=0)
    if kind == "kernel":
        x, y = _pixels(c, gen, b), _units(c, gen, b, hc, mc)
        traces = _trained_traces(gen, x.mean(dim=0), hc * mc, mc, 0.5, x.dtype)
        s.args = [a.cpu().numpy() for a in (*traces, x, y)]
        s.weights = np.zeros((n, hc * mc), dtype=dt)
        s.taupdt = TAUPDT * scale
        return s
    if kind == "classify":
        s.layer = _Output(n, hc, mc, OUT_TAUPDT * scale, dt)
        units = [_units(c, gen, b, 1, n) if n < 100 else _units(c, gen, b, n // 100, 100) for _ in range(BATCHES)]
        s.x = [u if u.shape[1] == n else torch.nn.functional.pad(u, (0, n - u.shape[1])) for u in units]
        s.t = [_labels(c, gen, b) for _ in range(BATCHES)]
        s.state = _fill(s.layer, gen, s.x[0].mean(dim=0))
        return s
    hidden = _Hidden(n, hc, mc, TAUPDT * scale, dt, khalf=KHALF, pmin=PMIN, taubdt=TAUBDT, density=c["density"], mask_iterations=16)
    if kind == "fit":
        out = _Output(hc * mc, 1, CLASSES, OUT_TAUPDT * scale, dt)
        x = _pixels(c, gen, c["samples"])
        s.images, s.labels = x.cpu().numpy(), _labels(c, gen, c["samples"]).cpu().numpy()
        s.state = {"hidden": _fill(hidden, gen, x.mean(dim=0), c["density"]),
                   "out": _fill(out, gen, torch.full((hc * mc,), 1 / mc, device="cuda"))}
        s.net, s.batch, s.seed = Network(dt), b, seed
        s.net.verbose = False
        s.net.add_layer(hidden)
        s.net.add_layer(out)
        return s
    batches = max(1, min(BATCHES, BATCH_BYTES // (b * n * np.dtype(dt).itemsize)))
    s.layer, s.x = hidden, [_pixels(c, gen, b) for _ in range(batches)]
    s.state = _fill(hidden, gen, s.x[0].mean(dim=0), c["density"])
    if kind == "host":
        s.x = [x.cpu().numpy() for x in s.x]
    return s


def run(state):
    s = state
    i = s.passes
    s.passes = i + 1
    if s.kind == "predict":
        return s.layer.compute_activation(s.x[i % len(s.x)])
    if s.kind == "step":
        x = s.x[i % len(s.x)]
        y = s.layer.compute_activation(x)
        s.layer.train_step(x, y, i % s.hc if s.mask else None)
        return {"activation": y, "state": s.state}
    if s.kind == "classify":
        x = s.x[i % len(s.x)]
        y = s.layer.compute_activation(x)
        s.layer.train_step(x, s.t[i % len(s.t)])
        return {"activation": y, "state": s.state}
    if s.kind == "host":
        y = s.layer.step_host(s.x[i % len(s.x)], None, i % s.hc if s.mask else None)
        return {"activation": y, "state": s.state}
    if s.kind == "fit":
        np.random.seed((s.seed + i) % (1 << 32))   # the shuffles of a seeded run
        s.net.fit(s.images, s.labels, s.batch, [(0, 2), (1, 1)])
        return s.state
    return kernels_b200.update_weights(*s.args, s.taupdt, s.weights, s.taupdt / 2)


def work(case):
    c = case
    kind, n, b, e = c["kind"], c["n"], c["batch"], np.dtype(c["dtype"]).itemsize
    m = c["hc"] * c["mc"]

    def forward(rows, n, m):
        return (n * m + rows * (n + m) + m) * e, 2.0 * rows * n * m

    def train(rows, n, m):   # x and y are still at hand; Cij is read and written, the weights are written
        return (3 * n * m + 2 * (n + m)) * e, 2.0 * rows * n * m

    if kind == "predict":
        parts = [forward(b, n, m)]
    elif kind == "kernel":
        parts = [train(b, n, m), (b * (n + m) * e, 0)]
    elif kind == "classify":
        parts = [forward(b, n, m), train(b, n, m), (b * m * e, 0)]
    elif kind == "fit":
        k, last = divmod(c["samples"], b)
        parts = [(c["samples"] * (n + CLASSES) * e, 0)]
        for rows, times in ((b, k), (last, 1 if last else 0)):
            for by, fl in 3 * [forward(rows, n, m)] + 2 * [train(rows, n, m)] + [forward(rows, m, CLASSES), train(rows, m, CLASSES)]:
                parts.append((by * times, fl * times))
    else:
        parts = [forward(b, n, m), train(b, n, m)]
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


def tolerance(case):
    # A step: sums of up to 55296 float32 products, logarithms of their ratios.  A fit repeats it some hundred times on its own results.
    rel = 2e-5 if case["dtype"] == "float32" else 1e-12
    return {"rel": rel * (20 if case["kind"] == "fit" else 1), "differ": 1e-3}
