"""The work a user of this framework has it do, as cases that can be timed and compared.

``listed()`` gives the named cases, ``draw(rng)`` one more of the same ranges. ``prepare`` makes what
a program holds before the call (the engine, the inputs on the device), ``run`` is one pass through
the public Python API, ``work`` the bytes and operations a pass cannot do without, and ``exact`` the
same outputs in 64 bits without this repository's kernels, where they have such a value: a spiking
network has none (one rounding moves a spike, and the rasters part), the eye, the learning rules,
the readout and the surrogate have.

Kinds:
  frame      one frame of a batch of instances (BatchBrain.run_steps), with the frame's learning rule
             (BatchReward or BatchInstructDeep) where the case has one
  brain      one frame of a single instance through the NumPy-style ``Brain``
  eye        one game frame per instance through the motion eye
  rule       the deep instructed learning rule alone, on a frame's counts
  readout    the frame-end readout with its buttons and the closed-loop clamp
  mlp_train, mlp_forward   the learned surrogate: one training step, one screening pass
"""

from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.abspath("can-the-fly-play-f-zero-_b200")
if _PKG not in sys.path:
    sys.path.insert(1, _PKG)

from flyzero_b200 import connectome as cx  # noqa: E402
from flyzero_b200 import instruct as ins  # noqa: E402
from flyzero_b200 import workloads as wl  # noqa: E402
from flyzero_b200.batch import BatchReward  # noqa: E402
from flyzero_b200.brain import Brain, LIFParams  # noqa: E402
from flyzero_b200.gpu import BatchBrain  # noqa: E402
from flyzero_b200.learning import LearnParams  # noqa: E402
from flyzero_b200.motor import READOUT, BatchMotor, Clamp  # noqa: E402
from flyzero_b200.surrogate import MLP  # noqa: E402
from flyzero_b200.vision import BatchMotionEye, MotionParams  # noqa: E402

FULL = 138_639                  # neurons of the full-scale connectome
DT = 0.1                        # ms per step
FRAME = 166                     # steps of one game frame (16.64 ms)
WINDOW = FRAME * DT


def listed():
    return [
        # the benchmark's frame: 64 flies of the whole brain, their motor synapses plastic, the
        # reward rule at the frame's end (a training fleet)
        dict(name="fleet_frame", kind="frame", n=FULL, batch=64, steps=FRAME, plastic="motor", rule="reward",
             weights="counts", state="f32"),
        # one fly of the whole brain, one frame (playing or probing a single brain)
        dict(name="single_frame", kind="frame", n=FULL, batch=1, steps=FRAME, plastic="none", rule="none",
             weights="counts", state="f32"),
        # instructed training: every synapse onto the descending neurons and their inputs plastic
        dict(name="instructed_frame", kind="frame", n=FULL, batch=64, steps=FRAME, plastic="deep", rule="none",
             weights="counts", state="f32"),
        # a small network for a short window, as scripts and tests drive it: latency and launches
        dict(name="small_window", kind="frame", n=1000, batch=4, steps=100, plastic="none", rule="none",
             weights="counts", state="f32"),
        # a mid-size network with rescaled (non-integral) weights, an odd size and an odd batch
        dict(name="float_weights_frame", kind="frame", n=16_385, batch=13, steps=FRAME, plastic="motor", rule="none",
             weights="float", state="f32"),
        # the precision report's FP64 engine (two launches per step)
        dict(name="precision_f64_window", kind="frame", n=16_384, batch=16, steps=100, plastic="none", rule="none",
             weights="counts", state="f64"),
        # the single-instance NumPy-style API with the reference's random stream
        dict(name="numpy_brain_frame", kind="brain", n=16_384, steps=FRAME),
        # the motion eye of a fleet with the training channels
        dict(name="eye_fleet", kind="eye", batch=64, h=224, w=256, cell=4, cells=12_246, channels="training", flip=False),
        # the deep instructed rule at the frame's end, two slots per fly
        dict(name="instructed_rule", kind="rule", n=FULL, batch=64, slots=2),
        # the frame-end readout of 9 neuron groups with its buttons, and the clamp
        dict(name="readout_and_clamp", kind="readout", n=16_384, batch=64, size=4),
        # the surrogate's training step, and a screening pass over a generation of candidates
        dict(name="surrogate_train", kind="mlp_train", rows=4096),
        dict(name="surrogate_screen", kind="mlp_forward", rows=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 5 + ["brain", "eye", "eye", "rule", "readout", "mlp_train", "mlp_train", "mlp_forward"])
    if kind == "frame":
        n = _log(rng, 300, FULL)
        state = rng.choice(["f32"] * 5 + ["f64"])
        plastic = rng.choice(["none", "motor", "deep"]) if n >= 2000 else "none"
        return dict(kind=kind, n=n, batch=rng.randint(1, 64 if state == "f32" and n < 60_000 else 16),
                    steps=_log(rng, 10, FRAME), plastic=plastic,
                    rule="reward" if plastic == "motor" and rng.random() < 0.5 else "none",
                    weights=rng.choice(["counts", "counts", "float"]), state=state)
    if kind == "brain":
        return dict(kind=kind, n=_log(rng, 300, 30_000), steps=_log(rng, 10, FRAME))
    if kind == "eye":
        cell = rng.choice([2, 3, 4, 4, 4, 5, 8])
        return dict(kind=kind, batch=rng.randint(1, 64), h=rng.randint(60, 240), w=rng.randint(64, 256), cell=cell,
                    cells=_log(rng, 500, 13_000), channels=rng.choice(["training", "motion"]), flip=rng.random() < 0.3)
    if kind == "rule":
        return dict(kind=kind, n=_log(rng, 2000, 40_000), batch=rng.randint(1, 64), slots=rng.randint(1, 4))
    if kind == "readout":
        return dict(kind=kind, n=_log(rng, 1000, 40_000), batch=rng.randint(1, 64), size=rng.randint(1, 6))
    rows = _log(rng, 64, 4096)
    return dict(kind=kind, rows=rows // 8 * 8 if kind == "mlp_train" else rows)     # training takes whole groups of 8


# ---- what does not depend on the seed: the connectome and the sets of synapses and neurons in use --------

@functools.lru_cache(maxsize=4)
def _graph(n):
    """The full-scale stand-in, or a smaller graph of its statistics with 8 motor neurons."""
    if n == FULL:
        return cx.flywire_scale()
    return cx.synthetic(n, seed=0, mean_degree=min(cx.MEAN_DEGREE, n / 8), motor=min(8, n // 40),
                        motor_in=int(0.05 * n))


@functools.lru_cache(maxsize=4)
def _drive(n):
    conn = _graph(n)
    return wl.grating_drive(n, seed=0, n_inputs=max(16, int(0.0883 * n)), exclude=conn.motor)


@functools.lru_cache(maxsize=4)
def _plastic(n, which):
    conn = _graph(n)
    if which == "none":
        return None
    if which == "motor":
        return np.flatnonzero(np.isin(conn.weights.indices, conn.motor))
    dn = np.concatenate(_groups(n))
    dn_pos = np.flatnonzero(np.isin(conn.weights.indices, dn))
    return np.union1d(dn_pos, ins.deep_positions(conn.weights, dn_pos))


@functools.lru_cache(maxsize=4)
def _groups(n):
    """The 9 instructed groups: the motor neurons and one readout neuron."""
    conn = _graph(n)
    return tuple(np.array([m], np.int64) for m in [*conn.motor[:8], _drive(n).readout[9]])


@functools.lru_cache(maxsize=4)
def _scaled(n):
    """The graph with every weight rescaled (a fitted connectome: weights are not whole counts)."""
    w = _graph(n).weights.copy()
    w.data = (w.data * np.random.default_rng(5).uniform(0.7, 1.3, w.nnz)).astype(np.float32)
    return w


def _weights(case):
    return _scaled(case["n"]) if case.get("weights") == "float" else _graph(case["n"]).weights


def _flies(batch, slots):
    return np.arange(batch) // slots


# ---- prepare ---------------------------------------------------------------------------------------------

def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["go"](state)


def work(case):
    return globals()["_work_" + case["kind"]](case)


def exact(case, seed):
    f = globals().get("_exact_" + case["kind"])
    return f(case, seed) if f is not None else None


def _trained(gb, seed):
    """Plastic weights as a fleet in training has them: moved from the connectome's, one row per slot."""
    g = torch.Generator(device=gb.device).manual_seed(seed)
    w0 = torch.as_tensor(gb.w0, device=gb.device)
    gb.pw.copy_(w0 * (0.5 + torch.rand(gb.pw.shape, device=gb.device, generator=g)))


def _prepare_frame(case, seed):
    n, B = case["n"], case["batch"]
    drive = _drive(n)
    work_ = wl.BatchedWorkload.make(B, seed=seed)
    pos = _plastic(n, case["plastic"])
    gb = BatchBrain(_weights(case), LIFParams(dt=DT), batch=B, seed=seed, plastic_pos=pos, fp64=case["state"] == "f64")
    if pos is not None:
        _trained(gb, seed)
    gb.set_input(np.r_[drive.inputs, drive.tonic], work_.rates(drive, 0.0, work_.directions()))
    state = dict(go=_run_frame, gb=gb, steps=case["steps"], p=gb.p_ext.clone(), rule=None,
                 counts=torch.empty((B, n), dtype=torch.int32, device=gb.device))
    if case["rule"] == "reward":
        state["rule"] = BatchReward(gb, params=LearnParams(), fly_of_slot=_flies(B, 2), targets=_graph(n).motor)
        state["reward"] = np.random.default_rng(seed).standard_normal(B)
        state["learn"] = np.ones(B, bool)
    return state


def _run_frame(s):
    gb, rule = s["gb"], s["rule"]
    gb.p_ext.copy_(s["p"])                                  # the frame's rates
    counts = gb.run_steps(s["steps"], counts=s["counts"])
    out = dict(counts=counts, v=gb.v, g=gb.g, ref=gb.ref)
    if rule is not None:
        rule.step(counts, s["reward"], s["learn"], WINDOW)
        out.update(pw=gb.pw, elig=rule.elig, post_mean=rule.post_mean)
    return out


def _work_frame(case):
    # state read and written once, counts and the input probabilities, the connectome once; eight
    # operations per neuron and step
    n, B = case["n"], case["batch"]
    real, entry = (8, 6) if case["state"] == "f64" else (4, 6)
    if case["weights"] == "float":
        entry = 8
    nnz = n * min(cx.MEAN_DEGREE, n / 8)
    pl = {"none": 0.0, "motor": 0.053 * n, "deep": 5.7 * n}[case["plastic"]]
    return dict(bytes=B * n * (4 * real + 2 + 4) + B * 0.0883 * n * 4 + nnz * entry + B * pl * 4,
                flops=8.0 * B * n * case["steps"])


def _prepare_brain(case, seed):
    b = Brain(_graph(case["n"]).weights, LIFParams(dt=DT), seed=seed)
    drive = _drive(case["n"])
    idx = np.r_[drive.inputs[:512], drive.tonic]
    b.set_input(idx, np.random.default_rng(seed).uniform(40.0, 120.0, len(idx)).astype(np.float32))
    return dict(go=_run_brain, b=b, ms=case["steps"] * DT)


def _run_brain(s):
    counts = s["b"].run(s["ms"])
    return dict(counts=counts, v=s["b"].v, g=s["b"].g, ref=s["b"].ref)


def _work_brain(case):
    n = case["n"]
    return dict(bytes=n * 22.0 + 6.0 * n * min(cx.MEAN_DEGREE, n / 8), flops=8.0 * n * case["steps"])


# ---- the eye -------------------------------------------------------------------------------------------

def _eye_params(case):
    if case["channels"] == "training":
        return MotionParams(gain=10 ** 2.7, y_min=0.2, cell=case["cell"], transient_gain=4.0, sustained_gain=4.0,
                            chromatic_gain=1.0)
    return MotionParams(cell=case["cell"])


@functools.lru_cache(maxsize=8)
def _eye_layout(cells, h, w, cell, y_min, channels):
    drive = wl.grating_drive(16_384, seed=0, n_inputs=cells)
    lo = wl.eye_layout(drive, (h, w), cell, y_min)
    if channels == "motion":
        lo.chan = (lo.chan % 8).astype(np.uint8)
    return lo


def _eye_inputs(case, seed):
    """Two consecutive frames per instance: a drifting grating with noise (a cheap ``game_frames``)."""
    B, h, w = case["batch"], case["h"], case["w"]
    g = torch.Generator().manual_seed(seed)
    ang, speed = 2 * math.pi * torch.rand(B, 1, 1, generator=g), 1 + 5 * torch.rand(B, 1, 1, generator=g)
    yy, xx = torch.meshgrid(torch.arange(h), torch.arange(w), indexing="ij")
    noise = torch.randint(-12, 13, (B, h, w), generator=g)
    out = []
    for t in range(2):
        wave = 0.5 + 0.5 * torch.sin(2 * math.pi * (torch.cos(ang) * xx + torch.sin(ang) * yy + speed * t) / 19.0)
        img = torch.stack([wave * 180 + noise, wave * 120 + 40 + noise, 255 - wave * 200 - noise], -1)
        out.append(img.clamp(0, 255).to(torch.uint8))
    flip = (torch.rand(B, generator=g) < 0.5).numpy() if case["flip"] else None
    return out, flip


@functools.lru_cache(maxsize=1)
def _eye_graph():
    return cx.synthetic(16_384, seed=0, mean_degree=4)


def _prepare_eye(case, seed):
    p = _eye_params(case)
    lo = _eye_layout(case["cells"], case["h"], case["w"], case["cell"], p.y_min, case["channels"])
    gb = BatchBrain(_eye_graph().weights, LIFParams(dt=DT), batch=case["batch"], seed=seed)
    eye = BatchMotionEye(gb, None, (case["h"], case["w"]), p, eye_layout=lo)
    (first, second), flip = _eye_inputs(case, seed)
    eye.see(first.to(gb.device), flip)                      # the filters have seen a frame
    return dict(go=_run_eye, eye=eye, gb=gb, frame=second.to(gb.device), flip=flip)


def _run_eye(s):
    rates = s["eye"].see(s["frame"], s["flip"])
    return dict(rates=rates, p=s["gb"].p_ext)


def _work_eye(case):
    B, grid = case["batch"], (case["h"] // case["cell"]) * (case["w"] // case["cell"])
    return dict(bytes=B * (3.0 * case["h"] * case["w"] + 24.0 * grid + 8.0 * case["cells"]),
                flops=B * (4.0 * case["h"] * case["w"] + 40.0 * grid + 8.0 * case["cells"]))


def _exact_eye(case, seed):
    p = _eye_params(case)
    lo = _eye_layout(case["cells"], case["h"], case["w"], case["cell"], p.y_min, case["channels"])
    frames, flip = _eye_inputs(case, seed)
    c, gh, gw = p.cell, case["h"] // p.cell, case["w"] // p.cell
    gx, gy = torch.as_tensor(lo.gx), torch.as_tensor(lo.gy)
    lp = arms = sig = None
    for k, fr in enumerate(frames):
        if flip is not None:
            fr = torch.where(torch.as_tensor(flip)[:, None, None, None], fr.flip(2), fr)
        img = fr[:, :gh * c, :gw * c].double() / 255
        grid = img.reshape(-1, gh, c, gw, c, 3).mean((2, 4))
        lum = grid.mean(-1)
        lp = lum.clone() if lp is None else lp
        arms = [torch.zeros_like(lum), torch.zeros_like(lum)] if arms is None else [
            a + (s - a) / p.tau_delay for a, s in zip(arms, sig)]
        lp = lp + (lum - lp) / p.tau_hp
        sig = [(lum - lp).clamp(min=0), (lp - lum).clamp(min=0)]
    feat = torch.zeros((14, *lum.shape), dtype=torch.float64)
    for pol in range(2):
        s, d, k = sig[pol], arms[pol], p.shift
        feat[4 * pol, :, :, :-k] = d[:, :, :-k] * s[:, :, k:] - s[:, :, :-k] * d[:, :, k:]
        feat[4 * pol + 2, :, :-k] = d[:, :-k] * s[:, k:] - s[:, :-k] * d[:, k:]
        feat[4 * pol + 1], feat[4 * pol + 3] = -feat[4 * pol], -feat[4 * pol + 2]
        feat[8 + pol] = p.transient_gain * s / p.gain
    ii = torch.nn.functional.pad(lum, (1, 0, 1, 0)).cumsum(1).cumsum(2)
    y, x = torch.arange(gh), torch.arange(gw)
    y0, y1 = (y - p.surround).clamp(0, gh), (y + p.surround + 1).clamp(0, gh)
    x0, x1 = (x - p.surround).clamp(0, gw), (x + p.surround + 1).clamp(0, gw)
    box = ii[:, y1][:, :, x1] - ii[:, y0][:, :, x1] - ii[:, y1][:, :, x0] + ii[:, y0][:, :, x0]
    con = lum - box / ((y1 - y0)[:, None] * (x1 - x0)[None, :])
    feat[10], feat[11] = p.sustained_gain * con / p.gain, -p.sustained_gain * con / p.gain
    if p.chromatic_gain > 0:
        feat[12], feat[13] = p.chromatic_gain * grid[..., 2] / p.gain, p.chromatic_gain * grid[..., 1] / p.gain
    r = feat.clamp(min=0)[torch.as_tensor(lo.chan.astype(np.int64)), :, gy, gx].T
    rates = p.max_rate * (p.gain * r).clamp(0, 1) * torch.as_tensor(lo.visible)
    slot = np.argsort(np.argsort(lo.idx))                   # the eye's neurons take ext slots in index order
    p_ext = torch.empty_like(rates)
    p_ext[:, torch.as_tensor(slot)] = rates * DT / 1000.0
    return dict(rates=rates, p=p_ext)


# ---- the deep instructed rule --------------------------------------------------------------------------

def _rule_inputs(case, seed, n_pl):
    rng = np.random.default_rng(seed)
    B = case["batch"]
    intents = rng.uniform(-1, 1, (B, 5)) * np.array([1, 1, 0.5, 0.5, 0.5]) + np.array([0, 0, 0.5, 0.5, 0.5])
    tgt = np.array([ins.targets(x, ins.InstructParams()) for x in intents], np.float32)
    counts = rng.poisson(0.16, (B, case["n"])).astype(np.int32)          # ~10 Hz over a frame
    learn = rng.random(B) < 0.9
    learn[0] = True
    scale = np.random.default_rng(seed + 1).random((B, 1), np.float32) + np.float32(0.5)
    return tgt, counts, learn, scale


def _prepare_rule(case, seed):
    n, B = case["n"], case["batch"]
    pos = _plastic(n, "deep")
    gb = BatchBrain(_graph(n).weights, LIFParams(dt=DT), batch=B, seed=seed, plastic_pos=pos)
    rule = ins.BatchInstructDeep(gb, dict(zip(ins.GROUPS, _groups(n))), fly_of_slot=_flies(B, case["slots"]))
    tgt, counts, learn, scale = _rule_inputs(case, seed, len(pos))
    gb.pw.mul_(torch.as_tensor(scale[_flies(B, case["slots"])], device=gb.device))
    return dict(go=_run_rule, gb=gb, rule=rule, counts=torch.as_tensor(counts, device=gb.device), tgt=tgt, learn=learn)


def _run_rule(s):
    err = s["rule"].step(s["counts"], s["tgt"], s["learn"], WINDOW)
    r = s["rule"]
    return dict(err=err, pw=s["gb"].pw, trace=r.trace, rate=r.rate, delta=r.delta)


def _work_rule(case):
    n, B = case["n"], case["batch"]
    deg = min(cx.MEAN_DEGREE, n / 8)
    pl = min(5.7 * n, 9 * deg * deg * 2)
    return dict(bytes=B * (8.0 * pl + 4 * n + 16.0 * 0.3 * n) + 12.0 * pl, flops=6.0 * B * pl)


def _exact_rule(case, seed):
    n, B = case["n"], case["batch"]
    conn, pos, p = _graph(n), _plastic(n, "deep"), ins.InstructParams()
    w = conn.weights.tocsr()
    rows = np.repeat(np.arange(n), np.diff(w.indptr))
    pre, post = rows[pos], w.indices[pos]
    w_syn = LIFParams().w_syn
    w0 = (w.data[pos].astype(np.float32) * np.float32(w_syn)).astype(np.float64)
    tgt, counts, learn, scale = _rule_inputs(case, seed, len(pos))
    fly = _flies(B, case["slots"])
    pw = (w0.astype(np.float32)[None, :] * scale[fly]).astype(np.float64)
    upre, pk = np.unique(pre, return_inverse=True)
    upost, qk = np.unique(post, return_inverse=True)
    a_pre, a_rate = 1 - math.exp(-WINDOW / p.tau_pre_ms), 1 - math.exp(-WINDOW / p.tau_rate_ms)
    hz = 1000.0 / WINDOW
    trace = a_pre * counts[:, upre] * hz * p.tau_pre_ms / 1000.0
    rate = a_rate * counts[:, upost] * hz
    group = np.full(n, -1)
    for k, g in enumerate(_groups(n)):
        group[g] = k
    gk = group[upost]
    err = np.where(gk >= 0, tgt[:, np.maximum(gk, 0)].astype(np.float64) - rate, 0.0)
    dn = np.flatnonzero(group[post] >= 0)
    l1 = np.unique(pre[dn])
    at = np.full(n, -1)
    at[l1] = np.arange(len(l1))
    delta = np.zeros((B, len(l1)))
    for b in range(B):
        np.add.at(delta[b], at[pre[dn]], pw[b, dn] / w_syn * err[b, qk[dn]])
    wmax, sign = p.cap * np.maximum(np.abs(w0), w_syn), np.sign(w0)
    active = np.bincount(fly, weights=learn)
    deep = np.flatnonzero((at[post] >= 0) & (group[post] < 0))
    for sel, x, eta in ((dn, err[:, qk[dn]], p.eta), (deep, delta[:, np.maximum(at[post[deep]], 0)], 1e-6)):
        for f in range(fly[-1] + 1):
            own = np.flatnonzero(fly == f)
            on = own[learn[own]]
            d = sum((eta / active[f] * trace[b, pk[sel]] * x[b] for b in on), np.zeros(len(sel)))
            for b in own:
                moved = sign[sel] * np.clip(sign[sel] * (pw[b, sel] + d), 0, wmax[sel])
                pw[b, sel] = np.where(d == 0.0, pw[b, sel], moved)
    mean = np.zeros(B)
    for k in range(len(ins.GROUPS)):
        mem = np.flatnonzero(gk == k)
        if len(mem):
            mean += np.abs(tgt[:, k] - rate[:, mem].mean(1))
    return dict(err=np.where(learn, mean / len(ins.GROUPS), 0.0), pw=pw, trace=trace, rate=rate, delta=delta)


# ---- the frame-end readout and the clamp -----------------------------------------------------------------

def _readout_inputs(case, seed):
    rng = np.random.default_rng(seed)
    B, size = case["batch"], case["size"]
    idx = rng.choice(case["n"], len(READOUT) * size, replace=False).astype(np.int64).reshape(len(READOUT), size)
    counts = rng.poisson(0.4, (B, case["n"])).astype(np.int32)
    target = rng.uniform(0, 60, (B, 2)).astype(np.float32)
    return idx, counts, target, rng.random(B) < 0.8


def _prepare_readout(case, seed):
    idx, counts, target, active = _readout_inputs(case, seed)
    gb = BatchBrain(cx.synthetic(case["n"], seed=0, mean_degree=4).weights, LIFParams(dt=DT), batch=case["batch"], seed=seed)
    motor = BatchMotor(gb, dict(zip(READOUT, idx)))
    clamp = Clamp(gb, [idx[0], idx[6]])
    return dict(go=_run_readout, gb=gb, motor=motor, clamp=clamp, counts=torch.as_tensor(counts, device=gb.device),
                target=target, active=active)


def _run_readout(s):
    buttons = s["motor"].update(s["counts"], WINDOW)
    s["clamp"].step(s["counts"], s["target"], s["active"], WINDOW)
    return dict(rates=s["motor"].rates_dev, u=s["clamp"].u, rate=s["clamp"].rate, bias=s["gb"].bias_ext,
                pressed=np.array([[b[k] for k in sorted(b)] for b in buttons], np.int32))


def _work_readout(case):
    k = case["batch"] * len(READOUT)
    return dict(bytes=k * (4.0 * case["size"] + 12.0), flops=k * (case["size"] + 6.0))


def _exact_readout(case, seed):
    idx, counts, target, active = _readout_inputs(case, seed)
    a, hz = 1 - math.exp(-WINDOW / 80.0), 1000.0 / WINDOW
    inst = counts[:, idx].mean(2) * hz
    rate = a * inst[:, [0, 6]]
    on = active[:, None].astype(np.float64)
    u = np.clip(0.02 * (target - rate) * on, -20.0, 20.0) * on
    neurons = np.concatenate([idx[0], idx[6]])
    bias = np.zeros((case["batch"], len(neurons)))
    bias[:, np.argsort(np.argsort(neurons))] = np.repeat(u, case["size"], axis=1)
    return dict(rates=a * inst, u=u, rate=rate, bias=bias, pressed=None)


# ---- the learned surrogate ------------------------------------------------------------------------------

def _mlp_inputs(case, seed):
    """Features as the Featurizer makes them (log1p of counts, a projection) and DN counts."""
    g = torch.Generator().manual_seed(seed)
    M = case["rows"]
    patches = torch.log1p(torch.rand((M, 1024), generator=g) * 24.0)
    proj = torch.randn((M, 256), generator=g)
    Y = torch.poisson(torch.rand((M, 10), generator=g) * 3.0, generator=g)
    return torch.cat([patches, proj], 1), Y


def _mlp_moments(net, seed):
    """Adam's moments in the middle of training (a first step's would be the gradient's signs)."""
    g = torch.Generator(device=net.dev).manual_seed(seed)
    for li in range(len(net.W)):
        for t, (m, v) in enumerate(zip(net.m[li], net.v[li])):
            m.normal_(0.0, 1e-3, generator=g)
            v.uniform_(1e-5, 4e-5, generator=g)
    net.t = 200


def _prepare_mlp_train(case, seed):
    net = MLP(seed=seed)
    _mlp_moments(net, seed)
    X, Y = _mlp_inputs(case, seed)
    return dict(go=_run_mlp_train, net=net, X=X.to(net.dev), Y=Y.to(net.dev))


def _run_mlp_train(s):
    net = s["net"]
    loss = net.train_step(s["X"], s["Y"])
    return dict(loss=loss, grads=[list(t) for t in net.grads], W=net.W, b=net.b)


def _prepare_mlp_forward(case, seed):
    net = MLP(seed=seed)
    return dict(go=_run_mlp_forward, net=net, X=_mlp_inputs(case, seed)[0].to(net.dev))


def _run_mlp_forward(s):
    return dict(z=s["net"].forward(s["X"]))


def _mlp_sizes():
    d = (1280, 512, 512, 10)
    return d, sum(a * b + b for a, b in zip(d[:-1], d[1:]))


def _work_mlp_train(case):
    (d, params), M = _mlp_sizes(), case["rows"]
    mac = sum(a * b for a, b in zip(d[:-1], d[1:]))
    # forward and weight gradients of every layer, input gradients of all but the first
    return dict(bytes=4.0 * M * (d[0] + d[-1]) + params * (4.0 * 6 + 4), flops=2.0 * M * (3 * mac - d[0] * d[1]))


def _work_mlp_forward(case):
    (d, params), M = _mlp_sizes(), case["rows"]
    return dict(bytes=4.0 * M * (d[0] + d[-1]) + 2.0 * params, flops=2.0 * M * sum(a * b for a, b in zip(d[:-1], d[1:])))


def _mlp_start(seed, moments=False):
    """A new surrogate's parameters (and mid-training moments), in 64 bits."""
    net = MLP(seed=seed)
    if moments:
        _mlp_moments(net, seed)
    f = lambda t: t.double()  # noqa: E731
    return ([(f(W), f(b)) for W, b in zip(net.W, net.b)], [tuple(map(f, t)) for t in net.m],
            [tuple(map(f, t)) for t in net.v], net)


def _exact_mlp_forward(case, seed):
    params, _, _, net = _mlp_start(seed)
    h = _mlp_inputs(case, seed)[0].to(net.dev).double()
    for li, (W, b) in enumerate(params):
        h = h @ W.T + b
        if li < len(params) - 1:
            h = torch.nn.functional.gelu(h)
    return dict(z=h)


def _exact_mlp_train(case, seed):
    params, m0, v0, net = _mlp_start(seed, moments=True)
    X, Y = (t.to(net.dev).double() for t in _mlp_inputs(case, seed))
    leaf = [(W.clone().requires_grad_(True), b.clone().requires_grad_(True)) for W, b in params]
    h = X
    for li, (W, b) in enumerate(leaf):
        h = h @ W.T + b
        if li < len(leaf) - 1:
            h = torch.nn.functional.gelu(h)
    loss = (h.exp() - Y * h).sum() / X.shape[0]
    loss.backward()
    (b1, b2), t = net.betas, net.t + 1
    new, grads = [], []
    for pair, m, v in zip(leaf, m0, v0):
        out = []
        for w, mm, vv in zip(pair, m, v):
            g = w.grad
            mm, vv = b1 * mm + (1 - b1) * g, b2 * vv + (1 - b2) * g * g
            out.append(w.detach() - net.lr * (mm / (1 - b1 ** t)) / ((vv / (1 - b2 ** t)).sqrt() + net.eps))
        new.append(out)
        grads.append([w.grad for w in pair])
    return dict(loss=loss.detach().reshape(1), grads=grads, W=[x[0] for x in new], b=[x[1] for x in new])
