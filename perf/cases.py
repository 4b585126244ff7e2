"""Performance cases: what users of this package run, through its public entry
points, over the sizes, types and options they run it with.

  interp    smart_interpolation on host arrays, results back on the host
  batch     smart_interpolation_batch on a list of uneven volumes
  cleanfill postprocess.clean and postprocess.fill of one result volume
  geodesic  geodis.geodesic_segment_device
  acwe      active_contour.acwe_results (what smart_interpolation(acwe=True) adds)
  predict   surrogate.predict: the network's label probabilities of a whole crop
  train     one training step of the surrogate network

Contents are synthetic: label phases of ellipsoids and tubes, one grey value
per phase, Gaussian noise, labels kept on every n-th slice.
"""
import math
import random

import numpy as np
import torch

KINDS = ("interp", "batch", "cleanfill", "geodesic", "acwe", "predict", "train")


def listed():
    return [
        # a region of interest cut from a scan, for a quick look: latency and launches
        interp("interp_tiny", 40, 36, 33, "uint8", 2, 5),
        # the plain 128^3 job with every optional result a reviewer looks at
        interp("interp_plain", 128, 128, 128, "uint8", 2, 10, smooth=100, uncertainty=True),
        # a 16-bit scan of odd size, denoised: the float32 working image
        interp("interp_uint16", 117, 141, 133, "uint16", 5, 9, smooth=50, denoise=True),
        # labels on slices of all three axes, eight phases with soft interfaces
        interp("interp_allaxis", 176, 224, 208, "uint8", 8, 8, yx=16, blur=3, smooth=100),
        # a whole scan with two objects, labelled every 20th slice (the size of the published screw timing)
        interp("interp_screw", 419, 492, 462, "uint8", 2, 20),
        # a folder of small uneven 16-bit scans in one call
        {"name": "batch_uint16", "kind": "batch", "count": 6, "lo": 64, "hi": 144, "phases": 6, "sorw": 4000,
         "smooth": 50},
        # removing islands and filling holes of a noisy result
        {"name": "cleanfill_256", "kind": "cleanfill", "z": 256, "y": 256, "x": 256, "phases": 6, "speckle": 0.01},
        # geodesic interpolation of a 128^3-class scan, odd sizes
        {"name": "geodesic_128", "kind": "geodesic", "z": 120, "y": 131, "x": 125, "phases": 2, "every": 10},
        # active contour after an interpolation, both results
        {"name": "acwe_256", "kind": "acwe", "z": 192, "y": 256, "x": 250, "phases": 3},
        # the network on a whole scan
        {"name": "predict_200", "kind": "predict", "z": 200, "y": 192, "x": 216, "phases": 5, "every": 12},
        # a training step: 8 windows of 64^3
        {"name": "train_8x64", "kind": "train", "batch": 8, "patch": 64},
    ]


def interp(name, z, y, x, dtype, phases, every, yx=0, blur=0, nbrw=10, sorw=4000, smooth=0, uncertainty=False,
           denoise=False):
    return {"name": name, "kind": "interp", "z": z, "y": y, "x": x, "dtype": dtype, "phases": phases, "every": every,
            "yx": yx, "blur": blur, "nbrw": nbrw, "sorw": sorw, "smooth": smooth, "uncertainty": uncertainty,
            "denoise": denoise}


def draw(rng):
    kind = rng.choice(("interp",) * 6 + KINDS[1:])
    if kind == "interp":
        while True:
            base = math.exp(rng.uniform(math.log(32), math.log(420)))
            z, y, x = (max(24, int(base * rng.uniform(0.8, 1.25))) for _ in range(3))
            allaxis = rng.random() < 0.3
            c = interp("", z, y, x, rng.choice(("uint8", "uint8", "uint16", "float32")),
                       rng.randint(3, 8) if allaxis else rng.randint(2, 8), rng.randint(5, 20),
                       yx=rng.randint(9, 20) if allaxis else 0, blur=rng.choice((0, 3)),
                       nbrw=rng.choice((5, 10, 10, 20)), sorw=rng.choice((1000, 2500, 4000, 4000)),
                       smooth=rng.choice((0, 50, 100)), uncertainty=rng.random() < 0.5, denoise=rng.random() < 0.25)
            if _steps(c) <= 1.0e11 and z * y * x * (1 + c["phases"]) * (1 + c["smooth"]) <= 8e9:
                break
    elif kind == "batch":
        lo = rng.randint(40, 80)
        c = {"kind": kind, "count": rng.randint(2, 8), "lo": lo, "hi": rng.randint(lo + 16, 150),
             "phases": rng.randint(2, 8), "sorw": rng.choice((1000, 4000)), "smooth": rng.choice((0, 50))}
    else:
        lo, hi = {"cleanfill": (64, 300), "geodesic": (40, 180), "acwe": (48, 260), "predict": (48, 220),
                  "train": (0, 0)}[kind]
        c = {"kind": kind}
        if kind == "train":
            c.update(batch=rng.randint(1, 8), patch=rng.choice((40, 48, 56, 64)))
        else:
            base = math.exp(rng.uniform(math.log(lo), math.log(hi * 0.8)))
            c.update({a: max(lo * 3 // 4, int(base * rng.uniform(0.8, 1.25))) for a in "zyx"})
            c["phases"] = rng.randint(2, 6)
            if kind == "cleanfill":
                c["speckle"] = rng.choice((0.001, 0.01, 0.03))
            elif kind != "acwe":
                c["every"] = rng.randint(5, 15)
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _volume(seed, shape, phases, dtype="uint8", blur=0, sigma=12.0):
    """(image, truth) on the GPU: phase 1 is a tube through the whole volume,
    the others are ellipsoids and tubes; means spread over the grey range."""
    dev, rnd = _device(), random.Random(seed)
    g = torch.Generator(device=dev).manual_seed(seed)
    ax = [torch.arange(n, device=dev, dtype=torch.float32) for n in shape]
    Z, Y, X = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    truth = torch.zeros(shape, dtype=torch.uint8, device=dev)
    n = min(shape)
    for lab in range(phases, 0, -1):
        if lab == 1 or rnd.random() < 0.4:  # tube
            a, b = ([rnd.uniform(0.25, 0.75) * s for s in shape] for _ in range(2))
            if lab == 1:
                a[0], b[0] = -1.0, shape[0] + 1.0
            d = [q - p for p, q in zip(a, b)]
            t = ((Z - a[0]) * d[0] + (Y - a[1]) * d[1] + (X - a[2]) * d[2]) / max(sum(v * v for v in d), 1.0)
            t.clamp_(0.0, 1.0)
            inside = ((Z - a[0] - t * d[0]) ** 2 + (Y - a[1] - t * d[1]) ** 2 + (X - a[2] - t * d[2]) ** 2
                      <= (rnd.uniform(0.06, 0.14) * n) ** 2)
        else:
            c = [rnd.uniform(0.2, 0.8) * s for s in shape]
            s = [max(rnd.uniform(0.08, 0.25) * n, 2.0) for _ in range(3)]
            inside = ((Z - c[0]) / s[0]) ** 2 + ((Y - c[1]) / s[1]) ** 2 + ((X - c[2]) / s[2]) ** 2 <= 1.0
        truth[inside] = lab
    means = torch.linspace(60.0, 220.0, phases, device=dev) if phases > 1 else torch.tensor([160.0], device=dev)
    img = torch.cat([torch.tensor([20.0], device=dev), means])[truth.long()]
    for _ in range(2 if blur else 0):
        img = torch.nn.functional.avg_pool3d(img[None, None], blur, 1, blur // 2, count_include_pad=False)[0, 0]
    img = img + torch.randn(shape, generator=g, device=dev) * sigma
    if dtype == "uint8":
        img = img.round().clamp_(0, 255).to(torch.uint8)
    elif dtype == "uint16":
        img = (img * 200.0).round().clamp_(0, 65535).to(torch.int32)
    return img, truth


def _sparse(truth, every, yx=0):
    lab = torch.zeros(truth.shape, dtype=torch.int32, device=truth.device)
    lab[::every] = truth[::every].int()
    if yx:
        lab[:, ::yx] = truth[:, ::yx].int()
        lab[:, :, ::yx] = truth[:, :, ::yx].int()
    return lab


def _host(img, lab, dtype):
    return img.cpu().numpy().astype(dtype, copy=False), lab.cpu().numpy()


def _shape(case):
    return case["z"], case["y"], case["x"]


def _weights(seed):
    """Random weights of the default network (16 channels, dilations 1, 2, 4,
    8), in the layout of its checkpoints: [27][out][in] and a bias per output."""
    g = torch.Generator().manual_seed(seed)
    w = [torch.randn((27, 16, 16), generator=g) * math.sqrt(2.0 / (27 * 16)) * (0.5 if k else 1.0)
         for k in range(10)]
    b = [torch.randn(16, generator=g) * 0.01 for _ in range(10)]
    return w, b


def _net(seed):
    from biomedisa_gb300.surrogate import SurrogateNet

    net = SurrogateNet()
    w, b = _weights(seed)
    net.load_state_dict({"w": w, "b": b})
    return net


def _batch_shapes(case):
    rnd = random.Random(case["count"] * 1009 + case["lo"] * 31 + case["hi"])
    return [tuple(rnd.randint(case["lo"], case["hi"]) for _ in range(3)) + (rnd.randint(4, 20),)
            for _ in range(case["count"])]


def _training_batch(case, seed):
    """Windows as the training loop cuts them: 16 feature channels, soft
    targets over 13 label slots, weight 1."""
    N, p = case["batch"], case["patch"]
    dev = _device()
    feats, target = [], []
    for k in range(N):
        img, truth = _volume(seed * 64 + k, (p, p, p), 5)
        every = 6 + k
        f = torch.zeros((p, p, p, 16), device=dev)
        f[..., 0] = img.float() / 255.0
        z = torch.arange(p, device=dev)
        near = ((z + every // 2) // every * every).clamp(max=(p - 1) // every * every)
        f[..., 1] = ((z - near).float() / 16.0).clamp(-1, 1)[:, None, None]
        f[::every, ..., 2] = 1.0
        onehot = torch.nn.functional.one_hot(truth.long(), 13).float()
        f[..., 3:] = onehot[near]
        feats.append(f)
        target.append(0.9 * onehot + 0.1 * onehot[near])
    x = torch.stack(feats).to(torch.bfloat16).contiguous()
    t = torch.stack(target).contiguous()
    return x, t, torch.ones((N, p, p, p), device=dev)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "interp":
        img, truth = _volume(seed, _shape(case), case["phases"], case["dtype"], case["blur"])
        img, lab = _host(img, _sparse(truth, case["every"], case["yx"]), case["dtype"])
        return {"kind": kind, "img": img, "lab": lab, "kw": dict(
            nbrw=case["nbrw"], sorw=case["sorw"], allaxis=bool(case["yx"]), smooth=case["smooth"],
            uncertainty=case["uncertainty"], denoise=case["denoise"])}
    if kind == "batch":
        imgs, labs = [], []
        for k, (z, y, x, every) in enumerate(_batch_shapes(case)):
            img, truth = _volume(seed * 64 + k, (z, y, x), case["phases"], "uint16")
            img, lab = _host(img, _sparse(truth, every), "uint16")
            imgs.append(img)
            labs.append(lab)
        # fixed sort and sweep parameters: the tuner's timing runs are no part of the work
        return {"kind": kind, "imgs": imgs, "labs": labs,
                "kw": dict(sorw=case["sorw"], smooth=case["smooth"], autotune_params=False)}
    if kind == "cleanfill":
        _, truth = _volume(seed, _shape(case), case["phases"])
        g = torch.Generator(device=truth.device).manual_seed(seed + 1)
        flip = torch.rand(truth.shape, generator=g, device=truth.device) < case["speckle"]
        other = torch.randint(0, case["phases"] + 1, truth.shape, generator=g, device=truth.device).to(torch.uint8)
        return {"kind": kind, "lab": torch.where(flip, other, truth).contiguous()}
    if kind == "geodesic":
        img, truth = _volume(seed, _shape(case), case["phases"])
        return {"kind": kind, "img": img, "lab": _sparse(truth, case["every"])}
    if kind == "acwe":
        from biomedisa_gb300 import _native as nat
        from biomedisa_gb300.active_contour import Frame

        img, truth = _volume(seed, _shape(case), case["phases"])
        g = torch.Generator(device=truth.device).manual_seed(seed + 1)
        # a segmentation to be refined: the phases grown by a noisy rim
        grown = torch.nn.functional.max_pool3d(truth[None, None].float(), 3, 1, 1)[0, 0].to(torch.uint8)
        rim = torch.rand(truth.shape, generator=g, device=truth.device) < 0.5
        return {"kind": kind, "frame": Frame(img, nat.SI_U8, (1, 1, 1), _shape(case)),
                "lab": torch.where(rim, grown, truth).contiguous()}
    if kind == "predict":
        from biomedisa_gb300 import DeviceJob
        from biomedisa_gb300 import _native as nat

        img, truth = _volume(seed, _shape(case), case["phases"])
        job = DeviceJob(img, nat.SI_U8, _sparse(truth, case["every"]), nat.SI_I32)
        msg = job.analyze()
        if msg:
            raise ValueError(msg)
        job.prepare()
        return {"kind": kind, "net": _net(seed), "job": job}
    x, t, w = _training_batch(case, seed)
    return {"kind": kind, "net": _net(seed), "x": x, "t": t, "w": w}


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "interp":
        from biomedisa_gb300 import smart_interpolation

        return smart_interpolation(state["img"], state["lab"], **state["kw"])
    if kind == "batch":
        from biomedisa_gb300 import smart_interpolation_batch

        return smart_interpolation_batch(state["imgs"], state["labs"], **state["kw"])
    if kind == "cleanfill":
        from biomedisa_gb300.postprocess import clean, fill

        return {"cleaned": clean(state["lab"], 0.1), "filled": fill(state["lab"], 0.9)}
    if kind == "geodesic":
        from biomedisa_gb300 import _native as nat
        from biomedisa_gb300.geodis import geodesic_segment_device

        return geodesic_segment_device(state["img"], nat.SI_U8, state["lab"], nat.SI_I32)
    if kind == "acwe":
        from biomedisa_gb300.active_contour import acwe_results

        return acwe_results(state["frame"], state["lab"])
    if kind == "predict":
        from biomedisa_gb300.surrogate import predict

        return predict(state["net"], state["job"])
    net, w = state["net"], state["w"]
    logits = net.forward(state["x"], keep=True)
    loss, dlogits = net.loss_and_grad(logits, state["t"], w, 13, denom=w.numel())
    net.zero_grad()
    net.backward(dlogits)
    net.adamw(lr=1e-5)  # the first step of the training loop's warmup
    return {"loss": loss, "logits": logits, "gw": [c.gw for c in net.convs], "gb": [c.gb for c in net.convs]}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
STEP_FLOPS = 6 * 5 + 7       # six weights (difference, square, product, power, sum), the draw, the comparison
SMOOTH_FLOPS = 50            # curvature of one voxel from its 18 neighbours, and the update


def _seeds(z, y, x, every, yx=0):
    n = -(-z // every) * y * x
    return n + (-(-y // yx) * z * x + -(-x // yx) * z * y if yx else 0)


def _steps(case):
    return _seeds(*_shape(case), case["every"], case["yx"]) * case["nbrw"] * case["sorw"]


def work(case):
    kind = case["kind"]
    if kind in ("interp", "batch"):
        if kind == "interp":
            vols = [(_shape(case), case["every"], case["yx"])]
            size, nbrw, outs = np.dtype(case["dtype"]).itemsize, case["nbrw"], 1 + bool(case["smooth"]) + \
                case["uncertainty"]
        else:
            vols = [((z, y, x), every, 0) for z, y, x, every in _batch_shapes(case)]
            size, nbrw, outs = 2, 10, 1 + bool(case["smooth"])
        n = sum(math.prod(s) for s, _, _ in vols)
        steps = sum(_seeds(*s, e, yx) for s, e, yx in vols) * nbrw * case["sorw"]
        return {"bytes": n * (size + 4 + outs),
                "flops": steps * STEP_FLOPS + n * (case["phases"] + 1) * case["smooth"] * SMOOTH_FLOPS}
    if kind in ("predict", "train"):
        n = math.prod(_shape(case)) if kind == "predict" else case["batch"] * case["patch"] ** 3
        per = 10 * 27 * 16 * 16 * 2
        if kind == "predict":
            return {"bytes": n * (1 + 4 * (case["phases"] + 1)), "flops": n * per}
        return {"bytes": n * (32 + 13 * 4 + 4 + 64), "flops": n * per * 3}
    n = math.prod(_shape(case))
    if kind == "cleanfill":
        return {"bytes": n * 3, "flops": 0}
    if kind == "geodesic":  # 8 passes of 13 neighbours for each label
        return {"bytes": n * 6, "flops": n * (case["phases"] + 1) * 8 * 13 * 4}
    return {"bytes": n * 4, "flops": n * 100}


# ---------------------------------------------------------------------------
# The network's outputs in 64 bits (the other kinds return whole numbers)
# ---------------------------------------------------------------------------
DILATIONS = (1, 1, 1, 2, 2, 4, 4, 8, 8, 1)


def _taps(d):
    return [(k, d * (k // 9 - 1), d * (k // 3 % 3 - 1), d * (k % 3 - 1)) for k in range(27)]


def _shifted(x, dz, dy, dx, m):
    """x padded by m on D, H, W, read at an offset: x[.., p + d, ..], zero outside."""
    D, H, W = (s - 2 * m for s in x.shape[1:4])
    return x[:, m + dz:m + dz + D, m + dy:m + dy + H, m + dx:m + dx + W]


def _pad(x, m):
    return torch.nn.functional.pad(x, (0, 0, m, m, m, m, m, m))


def _conv(x, w, b, d):
    p = _pad(x, d)
    y = torch.zeros_like(x) + b
    for k, dz, dy, dx in _taps(d):
        y += _shifted(p, dz, dy, dx, d) @ w[k].T
    return y


def _forward(x, w, b):
    acts = [x, _conv(x, w[0], b[0], 1).relu_()]
    for i in range(4):
        t = _conv(acts[-1], w[1 + 2 * i], b[1 + 2 * i], DILATIONS[1 + 2 * i]).relu_()
        acts += [t, (_conv(t, w[2 + 2 * i], b[2 + 2 * i], DILATIONS[2 + 2 * i]) + acts[-1]).relu_()]
    return acts, _conv(acts[-1], w[9], b[9], 1)


def _conv_back(x, w, dy, d, need_dx=True):
    px, flat = _pad(x, d), dy.reshape(-1, 16)
    gw = torch.stack([flat.T @ _shifted(px, *o, d).reshape(-1, 16) for _, *o in _taps(d)])
    dx = None
    if need_dx:
        pd, dx = _pad(dy, d), torch.zeros_like(dy)
        for k, oz, oy, ox in _taps(d):
            dx += _shifted(pd, -oz, -oy, -ox, d) @ w[k]
    return gw, flat.sum(0), dx


def _double_weights(seed):
    dev = _device()
    w, b = _weights(seed)
    # the layers' working weights are bf16
    return [v.to(dev).to(torch.bfloat16).double() for v in w], [v.to(dev).double() for v in b]


def _exact_train(case, seed):
    x, t, wt = _training_batch(case, seed)
    w, b = _double_weights(seed)
    acts, logits = _forward(x.double(), w, b)
    logp = torch.log_softmax(logits[..., :13], -1)
    t, denom = t.double(), wt.numel()
    loss = -(t * logp).sum().reshape(1) / denom
    dy = torch.zeros_like(logits)
    dy[..., :13] = (logp.exp() * t.sum(-1, keepdim=True) - t) / denom
    gw, gb = [None] * 10, [None] * 10
    gw[9], gb[9], da = _conv_back(acts[-1], w[9], dy, 1)
    for i in reversed(range(4)):
        a, h, y = acts[1 + 2 * i:4 + 2 * i]
        da = da * (y > 0)
        gw[2 + 2 * i], gb[2 + 2 * i], dt = _conv_back(h, w[2 + 2 * i], da, DILATIONS[2 + 2 * i])
        dt = dt * (h > 0)
        gw[1 + 2 * i], gb[1 + 2 * i], dx = _conv_back(a, w[1 + 2 * i], dt, DILATIONS[1 + 2 * i])
        da = da + dx
    gw[0], gb[0], _ = _conv_back(acts[0], w[0], da * (acts[1] > 0), 1, False)
    return {"loss": loss, "logits": logits, "gw": gw, "gb": gb}


def _exact_predict(case, seed):
    img, truth = _volume(seed, _shape(case), case["phases"])
    lab = _sparse(truth, case["every"])
    pad = lambda v: torch.nn.functional.pad(v, (1,) * 6)  # noqa: E731
    img, lab = pad(img.double()), pad(lab)
    # the crop: the labels' bounding box grown by 100, cut at the padded frame
    at = torch.nonzero(lab)
    lo, hi = at.amin(0).tolist(), at.amax(0).tolist()
    box = tuple(slice(max(a - 100, 0), min(b + 100, s)) for a, b, s in zip(lo, hi, lab.shape))
    values = torch.unique(lab[lab >= 0])
    img, lab = img[box], lab[box]
    slices = sorted(set(torch.nonzero(lab.flatten(1).amax(1) > 0).flatten().tolist()))
    D, H, W = lab.shape
    slot = torch.full(lab.shape, -1, dtype=torch.int64, device=lab.device)
    for z in slices:
        if 0 < z < D - 1:
            slot[z, 1:-1, 1:-1] = torch.searchsorted(values, lab[z, 1:-1, 1:-1].contiguous())
    f = torch.zeros((1, D, H, W, 16), dtype=torch.float64, device=lab.device)
    f[0, ..., 0] = img / 255.0
    f[0, ..., 2] = (slot >= 0).double()
    for z in range(D):
        f[0, z, ..., 1] = max(-1.0, min(1.0, min((z - s for s in slices), key=abs) / 16.0))
        below, above = [s for s in slices if s <= z], [s for s in slices if s > z]
        if below and above and below[-1] != z:
            ends = ((below[-1], (above[0] - z) / (above[0] - below[-1])), (above[0], (z - below[-1]) /
                                                                           (above[0] - below[-1])))
        else:
            ends = ((below[-1], 1.0),) if below else ((above[0], 1.0),)
        for s, share in ends:
            for k in range(13):
                f[0, z, ..., 3 + k] += share * (slot[s] == k)
    _, logits = _forward(f, *_double_weights(seed))
    return torch.softmax(logits[0, ..., :len(values)], -1).permute(3, 0, 1, 2)


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "predict":
        return _exact_predict(case, seed)
    return None
