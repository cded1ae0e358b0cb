"""The work that is timed for this framework: time steps of reaches (one at a time, in a
coupled loop, in the quasi-steady form and as ensembles) and the surrogate's passes, each
through the calls that a host program makes (hydist.lib, hydist.ensemble, hydist.surrogate).

A case is a dict of plain values; `kind` selects what it does:
  channel    the straight channel of the reference's channel test, FP64 hydraulics
  islands    a reach whose shelves wet and dry, several wet segments per line, sediment
  reach      a meandering reach, hydraulics + suspended sediment (+ the hourly bed update)
  coupled    the same reach with forcing in and levels out on the host in every step
  quasi      one bed period of the quasi-steady morphodynamic form
  ensemble   independent reaches of uneven sizes stepped side by side
  forward    the surrogate's forward pass
  train      a training pass of the surrogate: forward, loss, gradients
  layer      one convolution layer: forward, data gradient, weight and bias gradients
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "gpu-hydist_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from hydist import cases as C  # noqa: E402
from hydist import surrogate as S  # noqa: E402
from hydist.lib import Batch, Simulation, field_shape  # noqa: E402

# the band of config-5 crops that the surrogate is trained on
CROP_H, CROP_W = 1048, 89


def listed():
    return [
        # the smallest call: one step of the 400 x 60 channel test, waited for, as an
        # interactive host makes it (launch latency)
        {"name": "channel_400x60", "kind": "channel", "N": 400, "M": 60, "steps": 1},
        # an odd-sized reach with islands: many short segments per line, cells that open and
        # close in every step, sediment and the bed update every 10 s
        {"name": "islands_211x157", "kind": "islands", "N": 211, "M": 157, "steps": 10},
        # the ordinary run: the 1048 x 980 meander, hydraulics + sediment, FP64
        {"name": "reach_1048x980", "kind": "reach", "N": 1048, "M": 980, "dX": 5.0, "mixed": False, "steps": 20},
        # a coupled model: forcing sent in and the water level read back in every step
        {"name": "coupled_1048x980", "kind": "coupled", "N": 1048, "M": 980, "dX": 5.0, "mixed": False, "steps": 8},
        # the FP32-bulk form on a ragged grid
        {"name": "mixed_1531x777", "kind": "reach", "N": 1531, "M": 777, "dX": 5.0, "mixed": True, "steps": 20},
        # the largest single reach: 4096 x 2048 at 2.5 m, FP64
        {"name": "reach_4096x2048", "kind": "reach", "N": 4096, "M": 2048, "dX": 2.5, "mixed": False, "steps": 8},
        # morphodynamics: one bed period of the quasi-steady form (checkpoint, warm steps with
        # the steady residual after each, the bed update), mixed precision as its runs use
        {"name": "quasi_1048x980", "kind": "quasi", "N": 1048, "M": 980, "dX": 5.0, "mixed": True, "warm": 9},
        # an ensemble of reaches in the ensemble workload's size range, each on its own stream
        {"name": "ensemble_16", "kind": "ensemble", "n": 16, "lo": 128, "hi": 1024, "fused": False, "steps": 20},
        # and with every phase one launch for all reaches
        {"name": "ensemble_16_fused", "kind": "ensemble", "n": 16, "lo": 128, "hi": 1024, "fused": True, "steps": 20},
        # inference on a batch of channel-band crops
        {"name": "forward_16x1048x89", "kind": "forward", "B": 16, "H": CROP_H, "W": CROP_W},
        # a training pass at the training loop's batch of 8
        {"name": "train_8x1048x89", "kind": "train", "B": 8, "H": CROP_H, "W": CROP_W},
        # a single layer on odd sizes: the stride-2 one, whose data gradient is the
        # upsampling mapping
        {"name": "layer_down_4x517x83", "kind": "layer", "B": 4, "H": 517, "W": 83, "mode": "down", "cin": 48,
         "cout": 48},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["channel", "islands", "reach", "reach", "coupled", "quasi", "ensemble", "ensemble",
                       "forward", "train", "layer", "layer"])
    if kind == "channel":
        return {"kind": kind, "N": _log_int(rng, 60, 800), "M": rng.randint(24, 120), "steps": rng.randint(1, 4)}
    if kind == "islands":
        return {"kind": kind, "N": _log_int(rng, 48, 400), "M": _log_int(rng, 36, 300), "steps": rng.randint(2, 12)}
    if kind == "reach":
        # up to the large reach's cells; the 2.5 m grid only for the larger ones
        N = _log_int(rng, 128, 4096)
        M = _log_int(rng, 64, min(2048, 2 * N))
        return {"kind": kind, "N": N, "M": M, "dX": 2.5 if N * M > 2000000 else 5.0, "mixed": rng.random() < 0.4,
                "steps": rng.randint(2, 8) if N * M > 2000000 else rng.randint(4, 20)}
    if kind == "coupled":
        return {"kind": kind, "N": _log_int(rng, 128, 1600), "M": _log_int(rng, 64, 1000), "dX": 5.0,
                "mixed": rng.random() < 0.3, "steps": rng.randint(2, 8)}
    if kind == "quasi":
        return {"kind": kind, "N": _log_int(rng, 300, 1200), "M": _log_int(rng, 200, 1000), "dX": 5.0,
                "mixed": rng.random() < 0.7, "warm": rng.randint(4, 12)}
    if kind == "ensemble":
        lo = rng.randint(100, 300)
        return {"kind": kind, "n": rng.randint(3, 16), "lo": lo, "hi": rng.randint(lo, 1024),
                "fused": rng.random() < 0.5, "steps": rng.randint(4, 20)}
    if kind == "layer":
        mode = rng.choice(["same", "same", "down", "up"])
        cin, cout = rng.choice([(48, 48), (48, 48), (6, 48), (48, 3)]) if mode == "same" else (48, 48)
        return {"kind": kind, "B": rng.randint(1, 8), "H": _log_int(rng, 24, 1048), "W": _log_int(rng, 20, 160),
                "mode": mode, "cin": cin, "cout": cout}
    return {"kind": kind, "B": rng.randint(1, 16 if kind == "forward" else 8), "H": _log_int(rng, 48, CROP_H),
            "W": _log_int(rng, 20, 89)}


# ---- reaches ----------------------------------------------------------------------

def _geometry(c):
    """(channel width, depth, amplitude, wavelength) of a reach on N x M cells: the named
    workloads' meander, narrowed as the ensemble generator does where the grid is narrow."""
    k = 5.0 / c["dX"]  # the 2.5 m reach is the 5 m one scaled by 2
    span = c["M"] * c["dX"]
    width = min(150.0 * k, 0.35 * span)
    amp = min(120.0 * k, max(0.0, (span - width) / 2.0 - 6 * c["dX"]))
    return width, 4.0 + 4.0 * min(1.0, width / (150.0 * k)), amp, 1500.0 * k


def _reach(c, seed, hours=240.0, morpho=False):
    """The reach with a steady discharge after a one-hour ramp and a small slow tide: a run
    that can be continued for days (sediment from 0.25 h, bed change from 1 h)."""
    width, depth, amp, wavelength = _geometry(c)
    k = 5.0 / c["dX"]
    # the discharge per width of the 5 m reaches; the 2.5 m grid stays steady up to 800 m3/s
    q = (600.0 if k == 1.0 else 800.0) * width / (150.0 * k) * depth / 8.0
    m = C.meander_case(N=c["N"], M=c["M"], dX=c["dX"], dT=1.0, hours=hours, seed=seed, amp=amp,
                       wavelength=wavelength, width=width, depth=depth, noise_len=50.0 * k, Q0=q, Q1=q,
                       tide_amp=0.0 if morpho or k > 1.0 else 0.1, tide_period_h=12.42, spinup_h=1.0, tide_delay_h=1.0,
                       sediment_start=900.0, bed_change_start=3600.0,
                       end_cells=int(min(8 * k * k, c["N"] // 16)), name="reach")
    if morpho:
        C.with_feedback(m, morfac=1.0, bed_period=60.0)
    if c.get("mixed"):
        p = m.params.copy()
        p.precision_mode = 1
        m.params = p
    return m


@functools.lru_cache(maxsize=None)
def _wet(kind, N, M, dX):
    """Cells under water, roughly (for work())."""
    if kind == "channel":
        return N * (M - 10)
    if kind == "islands":
        return 0.55 * N * M
    return N * _geometry({"N": N, "M": M, "dX": dX})[0] / dX


class _Sim:
    """A stepping reach and the device tensors that its fields are read into."""

    def __init__(self, case, spin, fields):
        self.case = case
        self.sim = Simulation.from_case(case)
        if spin:
            self.sim.step(spin)
        self.fields = fields
        self.out = _buffers(self.sim, fields)

    def read(self):
        return {f: self.sim.get_device(f, self.out[f]) for f in self.fields}


def _buffers(sim, fields):
    return {f: torch.empty(field_shape(f, sim.N, sim.M)[0], dtype=torch.float64, device="cuda") for f in fields}


SPIN = 1800  # steps before the pass: half the ramp, sediment running


def _prepare_reach(c, seed):
    kind = c["kind"]
    if kind == "channel":
        # the channel test's discharge per width, varied with the seed
        r = np.random.default_rng(seed)
        case = C.channel_case(N=c["N"], M=c["M"], hours=300, Q=3.0 * (c["M"] - 10) * (0.9 + 0.2 * r.random()),
                              manning=0.02 + 0.01 * r.random())
        return _Sim(case, 200, ("z", "u", "v"))
    if kind == "islands":
        return _Sim(C.islands_case(N=c["N"], M=c["M"], seed=seed % 1000003, hours=300.0), 200,
                    ("z", "u", "v", "FS", "dH"))
    if kind == "quasi":
        return _Sim(_reach(c, seed, morpho=True), 3600, ("z", "u", "v", "FS", "dH", "h"))
    s = _Sim(_reach(c, seed), SPIN, ("z", "u", "v", "FS"))
    if kind == "coupled":
        s.sim.mirror_open("z")
        s.k = 0
    return s


class _View(np.ndarray):
    """A view of the library's host mirror that keeps the simulation owning it alive."""
    owner = None


def _run_coupled(s, steps):
    q, cc = s.case.tables, s.case.cc
    view = None
    for _ in range(steps):
        s.k += 1
        f = 1.0 + 0.01 * math.sin(0.05 * s.k)  # the coupled model's discharge
        s.sim.update_boundary([q[0], q[1], q[2] * f, q[3]], cc)
        s.sim.step(1, sync=False)
        view, _ = s.sim.mirror_update()
    s.sim.wait_fields()
    view = view.view(_View)
    view.owner = s
    return view


# ---- ensembles --------------------------------------------------------------------

class _Ensemble:
    def __init__(self, c, seed):
        # the sizes are the ensemble's own; the seed draws each reach's bed and roughness
        rng = np.random.default_rng(c["n"])
        lo, hi, reaches = c["lo"], c["hi"], []
        for k in range(c["n"]):
            # the ensemble workload's shapes: along 128-1024, across half of that
            N = int(round(math.exp(rng.uniform(math.log(lo), math.log(max(lo + 1, hi))))))
            M = int(round(math.exp(rng.uniform(math.log(lo / 2), math.log(max(lo / 2 + 1, hi / 2))))))
            reaches.append(_reach({"N": N, "M": M, "dX": 5.0}, seed + 1 + k, hours=120.0))
        self.batch = Batch(reaches)
        self.batch.set_fused(bool(c["fused"]))
        self.batch.step(SPIN)
        self.out = [_buffers(s, ("z", "u", "v", "FS")) for s in self.batch.members]


# ---- the surrogate ----------------------------------------------------------------

_MODES = {"same": S.CONV_SAME, "down": S.CONV_DOWN, "up": S.CONV_UP}


def _out_hw(c):
    H, W = c["H"], c["W"]
    return {"same": (H, W), "down": ((H + 1) // 2, (W + 1) // 2), "up": (2 * H, 2 * W - 1)}[c["mode"]]


def _smooth(g, *shape):
    """A field that varies slowly over the grid, of the size the features have."""
    a = torch.randn(shape[:1] + (12, 6) + shape[3:], generator=g, device="cuda")
    a = torch.nn.functional.interpolate(a.permute(0, 3, 1, 2), size=shape[1:3], mode="bilinear", align_corners=True)
    return a.permute(0, 2, 3, 1) + 0.1 * torch.randn(shape, generator=g, device="cuda")


def _net(c, seed):
    """The network and a batch of crops: bed, roughness, discharge, stage and the two
    coordinates in the first 6 of 16 channels; the targets and the wet mask for training."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, H, W = c["B"], c["H"], c["W"]
    net = S.Surrogate(device=0, seed=seed % 65537)
    for b in net.b:
        b.copy_(0.05 * torch.randn(b.shape, generator=g, device="cuda"))
    x = torch.zeros((B, H, W, S.CIN_PAD), dtype=torch.bfloat16, device="cuda")
    x[..., :2] = _smooth(g, B, H, W, 2).to(torch.bfloat16)
    x[..., 2:4] = torch.rand((B, 1, 1, 2), generator=g, device="cuda").to(torch.bfloat16)
    x[..., 4] = torch.linspace(0.0, 1.0, H, device="cuda")[:, None]
    x[..., 5] = torch.linspace(0.0, 1.0, W, device="cuda")[None, :]
    y = w = None
    if c["kind"] == "train":
        y = _smooth(g, B, H, W, S.OUT_CH).contiguous()
        w = (_smooth(g, B, H, W, 1)[..., 0] > 0).float().contiguous()
    return {"net": net, "x": x, "y": y, "w": w}


def _layer(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, H, W = c["B"], c["H"], c["W"]
    cinp, ncol = S.pad16(c["cin"]), S.pad16(c["cout"])
    Ho, Wo = _out_hw(c)
    net = S.Surrogate(device=0, seed=seed % 65537)
    x = torch.zeros((B, H, W, cinp), dtype=torch.bfloat16, device="cuda")
    x[..., :c["cin"]] = torch.relu(_smooth(g, B, H, W, c["cin"])).to(torch.bfloat16)
    dy = torch.zeros((B, Ho, Wo, ncol), dtype=torch.bfloat16, device="cuda")
    dy[..., :c["cout"]] = (1e-2 * torch.randn((B, Ho, Wo, c["cout"]), generator=g, device="cuda")).to(torch.bfloat16)
    w = torch.randn((c["cout"], 9, c["cin"]), generator=g, device="cuda") * math.sqrt(2.0 / (9 * c["cin"]))
    w = w.to(torch.bfloat16).float()
    b = 0.1 * torch.randn(c["cout"], generator=g, device="cuda")
    return {"net": net, "x": x, "dy": dy, "w": w, "b": b, "wpk": S.pack_weights(w, ncol, cinp),
            "wtpk": S.pack_weights(w.permute(2, 1, 0).contiguous(), cinp, ncol)}


def _run_layer(c, s):
    """What the network's forward and backward passes do for one layer (the data gradient
    masked by the ReLU of the layer's input)."""
    net, x, dy = s["net"], s["x"], s["dy"]
    B, H, W = c["B"], c["H"], c["W"]
    cin, cout = c["cin"], c["cout"]
    cinp, ncol = S.pad16(cin), S.pad16(cout)
    Ho, Wo = _out_hw(c)
    mode = _MODES[c["mode"]]
    y = net.conv(x, B, H, W, cinp, s["wpk"], s["b"], ncol, cout, mode, cout == 48, Ho, Wo, out_f32=cout != 48)
    dw = torch.zeros((cout, 9, cinp), device="cuda")
    db = torch.zeros(cout, device="cuda")
    st = net._stream()
    net._check(net.lib.hyd_conv_wgrad(x.data_ptr(), B, H, W, cinp, mode, dy.data_ptr(), Ho, Wo, ncol, cout,
                                      dw.data_ptr(), net.err.data_ptr(), st), "hyd_conv_wgrad")
    net._check(net.lib.hyd_bias_grad(dy.data_ptr(), B * Ho * Wo, ncol, cout, db.data_ptr(), st), "hyd_bias_grad")
    dx = None
    if cin == 48:
        dx = net.conv(dy, B, Ho, Wo, ncol, s["wtpk"], None, cinp, cin, S.ADJOINT[mode], False, H, W, mask=x)
    return {"y": y, "dw": dw, "db": db, "dx": dx}


# ---- the interface ----------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        state = _Ensemble(case, seed)
    elif kind in ("forward", "train"):
        state = _net(case, seed)
    elif kind == "layer":
        state = _layer(case, seed)
    else:
        state = _prepare_reach(case, seed)
    return case, state


def run(state):
    c, s = state
    kind = c["kind"]
    if kind in ("channel", "islands", "reach"):
        s.sim.step(c["steps"], sync=kind == "channel")
        return s.read()
    if kind == "coupled":
        return _run_coupled(s, c["steps"])
    if kind == "quasi":
        # the gate is wide here, so that every period is accepted at the same warm step and
        # a pass is the same work each time
        s.sim.quasi_steady_period(60.0, warm=2 * c["warm"], min_warm=c["warm"], gate=0.5)
        return s.read()
    if kind == "ensemble":
        s.batch.step(c["steps"], sync=False)
        return [{f: m.get_device(f, o[f]) for f in o} for m, o in zip(s.batch.members, s.out)]
    if kind == "layer":
        return _run_layer(c, s)
    net = s["net"]
    pred, saved = net.forward(s["x"])
    if kind == "forward":
        return pred
    loss, dy = net.loss_grad(pred, s["y"], s["w"])
    gw, gb = net.backward(saved, dy)
    return {"loss": loss, "gw": gw, "gb": gb}


def work(case):
    """A step's bytes: per wet cell the four state fields (z, u, v and the concentration)
    and five bed-derived ones read, the state written, FP64; then the fields handed over."""
    kind = case["kind"]
    if kind in ("channel", "islands", "reach", "coupled", "quasi"):
        wet = _wet(kind, case["N"], case["M"], case.get("dX", 5.0))
        cells = (case["N"] + 3) * (case["M"] + 3)
        per = 80 if kind == "channel" else 104
        steps = case["warm"] + 1 if kind == "quasi" else case["steps"]
        out = {"channel": 3, "islands": 5, "quasi": 6}.get(kind, 4) * 16 * cells
        return {"bytes": steps * per * wet + (0 if kind == "coupled" else out), "flops": steps * 400 * wet}
    if kind == "ensemble":
        size = math.exp(0.5 * (math.log(case["lo"]) + math.log(case["hi"])))  # a typical member
        N, M = int(size), int(size / 2)
        wet, cells = case["n"] * _wet("reach", N, M, 5.0), case["n"] * (N + 3) * (M + 3)
        return {"bytes": case["steps"] * 104 * wet + 64 * cells, "flops": case["steps"] * 400 * wet}
    if kind == "layer":
        n_in = case["B"] * case["H"] * case["W"]
        Ho, Wo = _out_hw(case)
        n_out = case["B"] * Ho * Wo
        pairs = 9 * (n_in / 4 if case["mode"] == "down" else n_in)  # (output pixel, tap) pairs with an input pixel
        cinp, ncol = S.pad16(case["cin"]), S.pad16(case["cout"])
        passes = 3 if case["cin"] == 48 else 2
        return {"bytes": 2 * n_in * cinp * (2 if passes == 3 else 1) + 2 * n_out * ncol * 2,
                "flops": passes * 2 * pairs * case["cin"] * case["cout"]}
    n = case["B"] * case["H"] * case["W"]
    macs = n * 9 * 48 * (6 + 48 / 4 + 48 / 4 + 48 / 4 + 48 + 3)
    if kind == "forward":
        return {"bytes": n * (S.CIN_PAD * 2 + S.OUT_CH * 4), "flops": 2 * macs}
    return {"bytes": n * (S.CIN_PAD * 2 + S.OUT_CH * 4 + 4), "flops": 6 * macs}


# ---- the same in 64 bits ------------------------------------------------------------

def _conv64(x, w, mode, out_hw):
    """x [B][C][H][W], w [n][9][C] with the layers' mappings."""
    F = torch.nn.functional
    k = w.reshape(w.shape[0], 3, 3, w.shape[2]).permute(0, 3, 1, 2)
    if mode == "same":
        return F.conv2d(x, k, padding=1)
    if mode == "down":
        return F.conv2d(x, k, stride=2, padding=1)
    H, W = x.shape[2:]
    return F.conv_transpose2d(x, k.transpose(0, 1), stride=2, padding=1,
                              output_padding=(out_hw[0] - (2 * H - 1), out_hw[1] - (2 * W - 1)))


def _exact_layer(c, s):
    x = s["x"][..., :c["cin"]].double().permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    w = s["w"].double().requires_grad_(True)
    b = s["b"].double().requires_grad_(True)
    dy = s["dy"][..., :c["cout"]].double().permute(0, 3, 1, 2)
    y = _conv64(x, w, c["mode"], _out_hw(c)) + b[:, None, None]
    dx, dw, db = torch.autograd.grad(y, (x, w, b), dy)
    out = y.detach().relu() if c["cout"] == 48 else y.detach()
    pad = torch.zeros((c["cout"], 9, S.pad16(c["cin"])), dtype=torch.float64, device="cuda")
    pad[..., :c["cin"]] = dw
    dx = (dx * (x.detach() > 0)).permute(0, 2, 3, 1).contiguous() if c["cin"] == 48 else None
    return {"y": out.permute(0, 2, 3, 1).contiguous(), "dw": pad, "db": db, "dx": dx}


def _exact_net(c, s):
    net = s["net"]
    w = [p.double().requires_grad_(True) for p in net.w]
    b = [p.double().requires_grad_(True) for p in net.b]
    cur = s["x"][..., :S.IN_CH].double().permute(0, 3, 1, 2).contiguous()
    names = {S.CONV_SAME: "same", S.CONV_DOWN: "down", S.CONV_UP: "up"}
    with torch.set_grad_enabled(c["kind"] == "train"):
        for l, (mode, _, _, relu) in enumerate(S.LAYERS):
            cur = _conv64(cur, w[l], names[mode], (c["H"], c["W"])) + b[l][:, None, None]
            cur = cur.relu() if relu else cur
        pred = cur.permute(0, 2, 3, 1).contiguous()
        if c["kind"] == "forward":
            return pred
        m = s["w"].double()
        loss = ((pred - s["y"].double()) ** 2 * m[..., None]).sum() / (m.sum() * S.OUT_CH)
        g = torch.autograd.grad(loss, w + b)
    return {"loss": loss.detach().reshape(1), "gw": list(g[:len(w)]), "gb": list(g[len(w):])}


def exact(case, seed):
    """What run() computes, from plain 64-bit arithmetic; None for the time steps, whose
    64-bit restatement on the host takes minutes."""
    if case["kind"] == "layer":
        return _exact_layer(case, _layer(case, seed))
    if case["kind"] in ("forward", "train"):
        return _exact_net(case, _net(case, seed))
    return None
