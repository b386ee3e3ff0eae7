"""The work that users of this package have it do, as cases that can be prepared, run and compared.

A case is a dict of plain values.  Its ``kind`` says which public entry points it goes through:

  layer     one masked convolution with its incremental activation, called as a module: ``layer([delta, None])``
  chain     strided convolution - sigmoid - convolution - tanh - x2 nearest upsample - skip sum, called as modules
  pointops  the reference-shaped native boundary: ``functional_conv_module`` with a [Cin,k,k,Cout] filter and a mask
  step      one incremental timestep of a network through ``IncrementalRunner.step`` (a captured graph by then)
  events    the same fed with raw events through ``IncrementalRunner.step_events``, recurrent state fed back
  refresh   the dense pass that refills every layer's state, ``IncrementalRunner.refresh``

Sizes are sensor sizes; the networks see them reflection-padded to the multiple they need, as the drivers pad.  The
weights are random with PyTorch's default bounds, the events come from drifting edges plus noise
(``synthetic.EdgeEventStream``) and the layer deltas from drifting blobs of active pixels.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from maskedincrementeval_b200 import _native as nat
from maskedincrementeval_b200 import fields as fl
from maskedincrementeval_b200.ext.pointops import pointops_functional as pf
from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr, E2VIDRecurrentIncr
from maskedincrementeval_b200.incr_modules.evflownet_incr import MultiResUNetRecurrentIncr
from maskedincrementeval_b200.incr_modules.fireflownet_incr import FireFlowNetIncr
from maskedincrementeval_b200.incr_modules.mask_incr_modules import nnReservedActivation
from maskedincrementeval_b200.runtime import IncrementalRunner
from maskedincrementeval_b200.synthetic import EdgeEventStream, reflection_pad_hw

DEV = "cuda"
FRAMES = 4          # inputs that a state's passes go round
BINS = 5            # voxel bins of the depth network; the flow networks read two count channels
NETS = {"e2depth": dict(multiple=8, channels=BINS), "fireflow": dict(multiple=1, channels=2), "evflow": dict(multiple=16, channels=2)}


def listed():
    return [
        # the smallest calls: one thin layer on a small ragged field, where launches and host time count
        dict(name="layer_16to24_97x131", kind="layer", n=1, cin=16, cout=24, k=3, stride=1, h=97, w=131, act="relu", frac=0.05, thr=0.0),
        # the single-layer workload: conv3x3 + ReLU on a sensor-sized field at 5 % active pixels
        dict(name="layer_32to32_260x346", kind="layer", n=1, cin=32, cout=32, k=3, stride=1, h=260, w=346, act="relu", frac=0.05, thr=0.0),
        # the layer-chain workload: batch 4, thresholded activations
        dict(name="chain_b4_260x346", kind="chain", n=4, h=260, w=346, frac=0.05, thr=1e-3),
        # a program written against the reference's extension functions
        dict(name="pointops_64to64_65x87_b2", kind="pointops", n=2, cin=64, cout=64, k=3, stride=1, h=65, w=87, frac=0.1),
        # one camera, lossless: the headline workload
        dict(name="e2depth_260x346", kind="step", net="e2depth", n=1, h=260, w=346, events=30000, thr=0.0),
        # one camera with an activation threshold: the deep layers fall silent
        dict(name="e2depth_260x346_thr", kind="step", net="e2depth", n=1, h=260, w=346, events=30000, thr=3e-4),
        # one camera from raw events, recurrent state fed back
        dict(name="e2depth_events_260x346", kind="events", net="e2depth", n=1, h=260, w=346, events=30000, thr=0.0),
        # a server that steps eight VGA streams together
        dict(name="e2depth_480x640_b8", kind="step", net="e2depth", n=8, h=480, w=640, events=80000, thr=0.0),
        # the dense pass at the start of a sequence and every few frames after
        dict(name="e2depth_refresh_260x346", kind="refresh", net="e2depth", n=1, h=260, w=346, events=30000, thr=0.0),
        dict(name="e2depth_refresh_480x640_b8", kind="refresh", net="e2depth", n=8, h=480, w=640, events=80000, thr=0.0),
        # the flow networks on two streams
        dict(name="fireflow_256x336_b2", kind="step", net="fireflow", n=2, h=256, w=336, events=20000, thr=0.0),
        dict(name="evflow_256x336_b2", kind="step", net="evflow", n=2, h=256, w=336, events=20000, thr=0.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dense_flops(c):
    return 2.0 * c["n"] * (c["h"] / c["stride"]) * (c["w"] / c["stride"]) * c["cin"] * c["cout"] * c["k"] ** 2


def draw(rng):
    kind = rng.choice(["layer", "layer", "chain", "pointops", "step", "step", "step", "events", "refresh"])
    frac = round(math.exp(rng.uniform(math.log(0.005), math.log(0.4))), 4)
    if kind == "layer":
        c = dict(kind=kind, n=_log_int(rng, 1, 8), cin=rng.choice([2, 8, 16, 32, 33, 64, 128, 256]), cout=rng.choice([1, 16, 24, 32, 64, 96, 128, 256]),
                 k=rng.choice([1, 3, 3, 3, 5, 7]), stride=rng.choice([1, 1, 2]), h=_log_int(rng, 33, 480), w=_log_int(rng, 44, 640),
                 act=rng.choice(["relu", "relu", "sigmoid", "tanh"]), frac=frac, thr=rng.choice([0.0, 0.0, 1e-3]))
        over = _dense_flops(c) / 5e11        # wide filters go with the smaller fields, as in a network
        if over > 1.0:
            c["n"] = 1
            over = _dense_flops(c) / 5e11
        if over > 1.0:
            c["h"], c["w"] = int(c["h"] / math.sqrt(over)), int(c["w"] / math.sqrt(over))
        return c
    if kind == "chain":
        # even extents: the x2 upsample of a stride-2 layer's output has to meet the skip
        return dict(kind=kind, n=_log_int(rng, 1, 8), h=2 * _log_int(rng, 24, 240), w=2 * _log_int(rng, 32, 320), frac=frac, thr=rng.choice([0.0, 1e-3]))
    if kind == "pointops":
        return dict(kind=kind, n=_log_int(rng, 1, 4), cin=rng.choice([5, 16, 32, 64, 128]), cout=rng.choice([8, 32, 64, 128]), k=rng.choice([1, 3, 3, 5, 7]),
                    stride=rng.choice([1, 1, 2]), h=_log_int(rng, 33, 264), w=_log_int(rng, 44, 352), frac=frac)
    net = "e2depth" if kind == "events" else rng.choice(["e2depth", "e2depth", "fireflow", "evflow"])
    thr = rng.choice([0.0, 0.0, 3e-4]) if kind == "step" and net == "e2depth" else 0.0
    h, w = _log_int(rng, 128, 480), _log_int(rng, 160, 640)
    return dict(kind=kind, net=net, n=_log_int(rng, 1, 8), h=h, w=w, events=int(h * w * rng.uniform(0.1, 0.4)), thr=thr)


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _randn(g, shape, scale=1.0):
    return (torch.randn(shape, generator=g, device=DEV) * scale).contiguous(memory_format=torch.channels_last)


def _fill_parameters(module, g):
    """U(-1/sqrt(fan_in), 1/sqrt(fan_in)) for every filter and its bias: PyTorch's default bounds for a convolution."""
    with torch.no_grad():
        for m in module.modules():
            w = getattr(m, "weight", None)
            if isinstance(w, torch.nn.Parameter):
                b = 1.0 / math.sqrt(w[0].numel())
                w.uniform_(-b, b, generator=g)
                if m.bias is not None:
                    m.bias.uniform_(-b, b, generator=g)
    return module


def _blob_deltas(g, n, c, h, w, frac, blobs=8, sigma=12.0, drift=3.0):
    """Two deltas whose active pixels (about ``frac`` of them, N(0, 0.5) on every channel) sit in drifting blobs, then
    their negatives: going round the four returns a layer to its state."""
    centre = torch.rand((n, blobs, 2), generator=g, device=DEV) * torch.tensor([h, w], device=DEV)
    heading = torch.rand((n, blobs), generator=g, device=DEV) * (2 * math.pi)
    step = drift * torch.stack([heading.sin(), heading.cos()], -1)
    ys, xs = torch.arange(h, device=DEV).view(1, 1, h, 1), torch.arange(w, device=DEV).view(1, 1, 1, w)
    out = []
    for _ in range(2):
        cy, cx = centre[..., 0].view(n, blobs, 1, 1), centre[..., 1].view(n, blobs, 1, 1)
        density = torch.exp(-((ys - cy) ** 2 + (xs - cx) ** 2) / (2 * sigma * sigma)).sum(1)
        p = (density * (frac * h * w / density.sum((1, 2), keepdim=True))).clamp_(max=1.0)
        p = (p * (frac * h * w / p.sum((1, 2), keepdim=True))).clamp_(max=1.0)
        active = torch.rand((n, h, w), generator=g, device=DEV) < p
        out.append(_randn(g, (n, c, h, w), 0.5) * active.unsqueeze(1))
        centre = (centre + step) % torch.tensor([h, w], device=DEV)
    return out + [-d for d in out]


def _voxel_grid(ev, h, w):
    """``synthetic.events_to_voxel_grid``'s arithmetic (bilinear in time, nearest in space), summed in a fixed order."""
    ts = (BINS - 1) * ev[:, 0]
    ti = ts.astype(np.int64)
    at = ti * (h * w) + ev[:, 2].astype(np.int64) * w + ev[:, 1].astype(np.int64)
    dt = ts - ti
    later = ti + 1 < BINS
    v = np.bincount(at, ev[:, 3] * (1.0 - dt), BINS * h * w) + np.bincount(at[later] + h * w, (ev[:, 3] * dt)[later], BINS * h * w)
    return v.reshape(BINS, h, w).astype(np.float32)


def _count_image(ev, h, w):
    at = (ev[:, 3] > 0).astype(np.int64) * (h * w) + ev[:, 2].astype(np.int64) * w + ev[:, 1].astype(np.int64)
    return np.bincount(at, minlength=2 * h * w).reshape(2, h, w).astype(np.float32)


def _windows(case, seed):
    """FRAMES windows of events of each stream: 10 drifting edges (15 for the larger sensors) and 5 % noise."""
    segments = 10 if case["h"] * case["w"] < 150000 else 15
    streams = [EdgeEventStream(case["h"], case["w"], case["events"], segments, seed * 1000 + s) for s in range(case["n"])]
    return [[s.window() for s in streams] for _ in range(FRAMES)]


def _frames(case, windows):
    h, w, spec = case["h"], case["w"], NETS[case["net"]]
    grid = _voxel_grid if spec["channels"] == BINS else _count_image
    pads = reflection_pad_hw(h, w, spec["multiple"])
    out = []
    for window in windows:
        x = torch.from_numpy(np.stack([grid(ev, h, w) for ev in window])).to(DEV)
        if any(pads):
            x = F.pad(x, pads, mode="reflect")
        out.append(x.contiguous(memory_format=torch.channels_last))
    return out


def _network(name, g):
    # built without storage, then filled: the flow networks' orthogonal gate initialisation would take seconds
    with torch.device("meta"):
        if name == "e2depth":
            net = E2VIDRecurrentIncr(dict(num_bins=BINS, skip_type="sum", recurrent_block_type="convlstm", num_encoders=3, base_num_channels=32,
                                          num_residual_blocks=2, norm=None, use_upsample_conv=True, compat="exact"))
        elif name == "fireflow":
            net = FireFlowNetIncr(dict(base_num_channels=32, kernel_size=3, mask_output=False), 2, compat="exact")
        else:
            net = MultiResUNetRecurrentIncr(compat="exact")
    return _fill_parameters(net.to_empty(device=DEV).eval(), g)


# ---------------------------------------------------------------------------------------------------------------
# states: what a program holds before the call
# ---------------------------------------------------------------------------------------------------------------
def _layer(cin, cout, k, stride, act, thr, g):
    layer = _fill_parameters(ConvLayerIncr(cin, cout, k, stride, k // 2, activation=act).to(DEV).eval(), g)
    layer.activation.threshold = thr
    return layer


def _reservoirs(net):
    """The persistent state that the pass updates: every activation's accumulated input."""
    return [m.in_res.reservoir for m in net.modules() if isinstance(m, nnReservedActivation) and m.in_res.reservoir is not None]


def prepare(case, seed):
    g = _generator(seed)
    s = {"kind": case["kind"], "at": 0}
    with torch.no_grad():
        if case["kind"] == "layer":
            s["net"] = _layer(case["cin"], case["cout"], case["k"], case["stride"], case["act"], case["thr"], g)
            s["net"].forward_refresh_reservoirs(_randn(g, (case["n"], case["cin"], case["h"], case["w"])))
            s["inputs"] = _blob_deltas(g, case["n"], case["cin"], case["h"], case["w"], case["frac"])
        elif case["kind"] == "chain":
            n, h, w = case["n"], case["h"], case["w"]
            s["first"], s["second"] = _layer(32, 64, 3, 2, "sigmoid", case["thr"], g), _layer(64, 64, 3, 1, "tanh", case["thr"], g)
            s["second"].forward_refresh_reservoirs(s["first"].forward_refresh_reservoirs(_randn(g, (n, 32, h, w))))
            s["inputs"] = list(zip(_blob_deltas(g, n, 32, h, w, case["frac"]), _blob_deltas(g, n, 64, h, w, case["frac"])))
            s["scratch"] = fl.Scratch()
        elif case["kind"] == "pointops":
            w = torch.empty((case["cin"], case["k"], case["k"], case["cout"]), device=DEV)
            b = 1.0 / math.sqrt(case["cin"] * case["k"] ** 2)
            s["filter"], s["stride"], s["pad"] = w.uniform_(-b, b, generator=g), case["stride"], case["k"] // 2
            s["inputs"] = [(d, d != 0) for d in _blob_deltas(g, case["n"], case["cin"], case["h"], case["w"], case["frac"])]
        else:
            fl.config.threshold = case["thr"]
            s["net"] = _network(case["net"], g)
            windows = _windows(case, seed)
            s["inputs"] = _frames(case, windows)
            s["runner"] = IncrementalRunner(s["net"], feedback=case["kind"] == "events")
            s["runner"].refresh(s["inputs"][0])
            if case["kind"] == "events":
                s["sensor"] = (case["h"], case["w"])
                s["inputs"] = [[torch.from_numpy(ev.astype(np.float32)).to(DEV) for ev in window] for window in windows]
            # a program in its loop: the runner has captured its step (it does so on the second one)
            if case["kind"] != "refresh":
                s["at"] = 1
                for _ in range(2):
                    run(s)
    return s


def run(s):
    x = s["inputs"][s["at"] % FRAMES]
    s["at"] += 1
    if s["kind"] == "step":
        y = s["runner"].step(x)
    elif s["kind"] == "events":
        y = s["runner"].step_events(x, s["sensor"])
    elif s["kind"] == "refresh":
        y = s["runner"].refresh(x)
    elif s["kind"] == "layer":
        with torch.no_grad():
            d, m = s["net"]([x, None])
        return {"delta": d, "mask": m.bits, "state": s["net"].activation.in_res.reservoir}
    elif s["kind"] == "chain":
        with torch.no_grad():
            dx, dskip = x
            y, m = s["second"](s["first"]([dx, None]))
            n, c, h, w = y.shape
            sc = s["scratch"]
            up = sc.get("up", (n, c, 2 * h, 2 * w), torch.float32, y.device, channels_last=True)
            mu = fl.upsample2x(y, m, None, None, up, sc.get("up.bits", (fl.n_tiles(n, 2 * h, 2 * w),), torch.int64, y.device), nat.UP_NEAREST)
            ds, ms = fl.resolve([dskip, None], sc, "skip")
            out = sc.get("out", tuple(ds.shape), torch.float32, y.device, channels_last=True)
            mo = fl.add(up, mu, ds, ms, out, sc.get("out.bits", (fl.n_tiles(n, 2 * h, 2 * w),), torch.int64, y.device))
        return {"delta": out, "mask": mo.bits, "state": [s["first"].activation.in_res.reservoir, s["second"].activation.in_res.reservoir]}
    else:
        d, mask = x
        return pf.functional_conv_module(d, s["filter"], mask=mask, stride=s["stride"], padding=s["pad"])[0]
    return {"out": y, "state": _reservoirs(s["net"])}


# ---------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far another correct implementation may be off
# ---------------------------------------------------------------------------------------------------------------
def _network_layers(case):
    """(cin, cout, k, output pixels, state floats per output pixel) of every convolution that a pass runs."""
    spec = NETS[case["net"]]
    left, right, top, bottom = reflection_pad_hw(case["h"], case["w"], spec["multiple"])
    px = case["n"] * (case["h"] + top + bottom) * (case["w"] + left + right)
    if case["net"] == "e2depth":
        out = [(BINS, 32, 5, px, 32)]
        for i in range(3):
            ci, co, p = 32 << i, 64 << i, px // 4 ** (i + 1)
            out += [(ci, co, 5, p, co), (co * (2 if case["kind"] == "events" else 1), 4 * co, 3, p, 5 * co)]
        out += [(256, 256, 3, px // 64, 256)] * 4
        out += [(256 >> i, 128 >> i, 5, px // 4 ** (2 - i), 128 >> i) for i in range(3)]
        return out + [(32, 1, 1, px, 2)]
    if case["net"] == "fireflow":
        return [(2, 32, 3, px, 32)] + [(32, 32, 3, px, 32)] * 6 + [(32, 2, 1, px, 4)]
    out = []
    for i in range(4):
        ci, co, p = 2 if i == 0 else 32 << i, 64 << i, px // 4 ** (i + 1)
        out += [(ci, co, 3, p, co), (co, co, 3, p, 2 * co), (co, co, 3, p, 2 * co)]
    out += [(512, 512, 3, px // 256, 512)] * 4
    for i in range(4):
        co, p = 256 >> i, px // 4 ** (3 - i)
        out += [((1024 >> i) + (2 if i else 0), co, 3, p, co), (co, 2, 1, p, 4)]
    return out


def work(case):
    """Bytes: inputs, filters, persistent state (read and written by a step, written by a refresh) and outputs, once
    each; nothing for what passes from layer to layer.  Operations: the multiplications and additions at the active
    pixels -- all of them in a lossless network after its first layers, about half with the threshold."""
    if case["kind"] in ("layer", "chain", "pointops"):
        px, frac = case["n"] * case["h"] * case["w"], case["frac"]
        if case["kind"] == "chain":
            near = min(1.0, 2 * frac)     # active pixels of a layer's output: those that the filter reaches
            return {"bytes": 4.0 * (px * (32 + 64) + near * px * (2 * 64 * 2 / 4 + 64) + 9 * 64 * 96),
                    "flops": 2.0 * 9 * px / 4 * (frac * 32 * 64 + near * 64 * 64)}
        k, cin, cout, outs = case["k"], case["cin"], case["cout"], px / case["stride"] ** 2
        flops = 2.0 * frac * outs * cin * cout * k * k
        if case["kind"] == "pointops":
            return {"bytes": 5.0 * px * cin + 4.0 * (outs * cout + cin * cout * k * k), "flops": flops}
        near = min(1.0, frac * (1 + (k - 1) / 2))
        return {"bytes": 4.0 * (px * cin + 3 * near * outs * cout + cin * cout * k * k), "flops": flops}
    layers = _network_layers(case)
    pixels = layers[-1][3]
    share = 0.5 if case["thr"] > 0 else 1.0
    moves = 1 if case["kind"] == "refresh" else 2 * share
    return {"bytes": 4.0 * (sum(ci * co * k * k + moves * p * st for ci, co, k, p, st in layers) + 3 * pixels * NETS[case["net"]]["channels"]),
            "flops": 2.0 * share * sum(ci * co * k * k * p for ci, co, k, p, _ in layers)}


def tolerance(case):
    if case["kind"] == "refresh" or case["kind"] == "pointops" or case.get("net") == "fireflow":
        # fp32 arithmetic; a step of the flow network without normalisation runs in split precision, which is as fine
        return {"rel": 2e-5}
    # TF32 inputs (2^-11 relative) with fp32 sums on the deltas.  With a threshold a change that lies at the threshold may
    # be sent by one implementation and held back by another; a mask bit flips where a change is near zero or the threshold.
    return {"rel": 3e-3 if case["thr"] > 0 else 1e-3, "max": 0.05, "differ": 0.005}
