"""Cases of the framework's work, through its public entry points.

A case's ``kind`` is the entry point that a program calls:

  host      simulateRIR: numpy in, numpy out (gpuRIR's own call)
  device    Simulator.simulate_rir_device: positions and RIRs stay on the GPU
  plan      batch.BatchPlan.launch: a batch of rooms planned once, replayed
  batch     batch.simulate_batch: a batch of rooms that is new on every call
  step      autograd.TorchBatch.l2_step: one fused training step
  grad      autograd.TorchBatch with PyTorch's loss and backward
  filter    simulateTrajectory: numpy signal and RIRs of a moving source
  traj      trajectory.simulate_trajectory_torch, forward and backward

Input values: rooms, positions and orientations uniform inside the given sizes,
wall coefficients from the Sabine fit of a reverberation time, white-noise
signals, exponentially decaying RIRs for the filtering cases.
"""
import math

import numpy as np
import torch

import gpurir_gb300 as gpurir
from gpurir_gb300 import autograd, batch, trajectory

PATTERNS = ["omni", "homni", "card", "hypcard", "subcard", "bidir"]


def listed():
    return [
        # one source, two receivers, every sample from the image sources: the first
        # example of gpuRIR's users, where latency and launches are the time
        dict(name="plain_room_call", kind="host", room="3x4x2.5", t60=0.5, nb="11x9x13", tdiff=0.5,
             tmax=0.5, fs=16000, n_src=1, n_rcv=2, spkr="omni", mic="omni", mode="f32", noise="logistic"),
        # 64 sources x 32 microphones, the drop-in call: 131 MB of RIRs to host memory
        dict(name="mic_array_call", kind="host", room="6x5x3", t60=1.0, nb="12x14x24", tdiff=0.3,
             tmax=1.0, fs=16000, n_src=64, n_rcv=32, spkr="omni", mic="card", mode="f32", noise="gaussian"),
        # the same work kept on the GPU for what follows there (filtering, training)
        dict(name="mic_array_device", kind="device", room="6x5x3", t60=1.0, nb="12x14x24", tdiff=0.3,
             tmax=1.0, fs=16000, n_src=64, n_rcv=32, spkr="omni", mic="card", mode="f32", noise="gaussian"),
        # 48 kHz, directional source and microphones, few pairs, live diffuse tail
        dict(name="studio_48k_device", kind="device", room="7.3x5.1x2.9", t60=0.45, nb="12x17x30",
             tdiff=0.123, tmax=0.45, fs=48000, n_src=3, n_rcv=5, spkr="subcard", mic="card", mode="f32",
             noise="logistic"),
        # one pair in a small hard room, image sources up to one second (t2n(1.0))
        dict(name="dense_room_device", kind="device", room="4x3x2.5", t60=2.0, nb="172x229x275", tdiff=1.0,
             tmax=1.0, fs=16000, n_src=1, n_rcv=1, spkr="omni", mic="omni", mode="f32", noise="logistic"),
        # gpuRIR's default evaluation, its lookup table, on an array of ordinary size
        dict(name="lookup_array_device", kind="device", room="5.2x4.4x2.7", t60=0.6, nb="16x19x31", tdiff=0.24,
             tmax=0.6, fs=16000, n_src=11, n_rcv=8, spkr="omni", mic="hypcard", mode="lut", noise="logistic"),
        # uneven rooms planned once, sources and receivers moved between replays
        dict(name="rooms_plan", kind="plan", rooms=128, t_lo=0.12, t_hi=0.36, fs=16000, max_src=4, max_rcv=8,
             tail=False),
        # new random rooms with diffuse tails on every call: data augmentation
        dict(name="rooms_call", kind="batch", rooms=24, t_lo=0.2, t_hi=0.9, fs=16000, max_src=3, max_rcv=6,
             tail=True),
        # walls, sources and receivers fitted to measured RIRs: 16 rooms, 4 x 8 pairs
        dict(name="fit_rooms_step", kind="step", rooms=16, room="5x4x3", nb="9x11x13", tmax=0.4, fs=16000,
             n_src=4, n_rcv=8, mic="hypcard"),
        # the same through autograd, fewer and odd pairs
        dict(name="fit_rooms_autograd", kind="grad", rooms=7, room="4.3x6.1x2.8", nb="14x10x21", tmax=0.21, fs=16000,
             n_src=3, n_rcv=5, mic="card"),
        # a moving source, custom time stamps, numpy signal and RIRs
        dict(name="walk_filter_call", kind="filter", points=37, n_rcv=2, rir_len=9602, signal=48011, fs=16000,
             stamps=True),
        # the full trajectory filtered and differentiated on the GPU
        dict(name="walk_train", kind="traj", points=400, n_rcv=8, rir_len=12800, signal=160000, fs=16000,
             stamps=False),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _logint(rng, lo, hi):
    return max(lo, min(hi, int(round(_log(rng, lo, hi)))))


def _sizes(room):
    return [float(v) for v in room.split("x")]


def _counts(t, room, c=343.0):
    return [int(math.ceil(2 * t * c / d)) for d in room]


def draw(rng):
    kind = rng.choice(["host", "device", "device", "device", "plan", "batch", "step", "grad", "filter", "traj"])
    if kind in ("host", "device"):
        while True:
            room = [round(rng.uniform(2.6, 9.0), 2), round(rng.uniform(2.4, 7.0), 2), round(rng.uniform(2.3, 4.2), 2)]
            fs = rng.choice([8000, 16000, 16000, 22050, 44100, 48000])
            t60 = round(rng.uniform(0.2, 1.2), 3)
            tmax = round(t60 * rng.uniform(0.5, 1.0), 4)
            tdiff = tmax if rng.random() < 0.3 else round(tmax * rng.uniform(0.15, 0.6), 4)
            nb = _counts(tdiff * rng.uniform(0.5, 1.0), room)
            n_src, n_rcv = _logint(rng, 1, 64), _logint(rng, 1, 32)
            images = n_src * n_rcv * nb[0] * nb[1] * nb[2]
            cost = images * (0.008 * fs + 40)
            if nb[0] * nb[1] * nb[2] < 1 << 24 and cost < 2.5e9 and n_src * n_rcv * tmax * fs < 3e7:
                break
        mode = rng.choice(["f32", "f32", "f32", "f32", "lut", "mp"]) if kind == "device" else "f32"
        return dict(kind=kind, room="x".join(str(v) for v in room), t60=t60, nb="x".join(str(v) for v in nb),
                    tdiff=tdiff, tmax=tmax, fs=fs, n_src=n_src, n_rcv=n_rcv,
                    spkr=rng.choice(["omni", "omni", "omni", "card", "subcard"]), mic=rng.choice(PATTERNS), mode=mode,
                    noise=rng.choice(["logistic", "gaussian"]))
    if kind == "plan":
        return dict(kind=kind, rooms=_logint(rng, 4, 128), t_lo=0.12, t_hi=round(rng.uniform(0.2, 0.36), 3),
                    fs=rng.choice([8000, 16000]), max_src=rng.randint(1, 4), max_rcv=rng.randint(2, 8), tail=False)
    if kind == "batch":
        return dict(kind=kind, rooms=_logint(rng, 2, 32), t_lo=0.2, t_hi=round(rng.uniform(0.4, 0.9), 3),
                    fs=rng.choice([8000, 16000, 16000, 24000]), max_src=rng.randint(1, 3), max_rcv=rng.randint(2, 6),
                    tail=True)
    if kind in ("step", "grad"):
        room = [round(rng.uniform(3.0, 7.0), 2), round(rng.uniform(3.0, 6.0), 2), round(rng.uniform(2.4, 3.6), 2)]
        return dict(kind=kind, rooms=_logint(rng, 1, 16), room="x".join(str(v) for v in room),
                    nb="x".join(str(rng.randint(5, 17)) for _ in range(3)), tmax=round(rng.uniform(0.1, 0.4), 4),
                    fs=rng.choice([8000, 16000, 16000, 44100]), n_src=rng.randint(1, 4), n_rcv=rng.randint(1, 8),
                    mic=rng.choice(["omni", "card", "hypcard", "subcard", "bidir"]))
    big = kind == "traj"
    points = _logint(rng, 5, 400 if big else 60)
    return dict(kind=kind, points=points, n_rcv=rng.randint(1, 8 if big else 3),
                rir_len=2 * _logint(rng, 700, 6400), signal=points * rng.randint(200, 450) + rng.randint(0, points - 1),
                fs=16000, stamps=rng.random() < 0.5)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _inside(rng, n, room, margin=0.3):
    room = np.asarray(room)
    return (margin + rng.random((n, 3)) * (room - 2 * margin)).astype(np.float32)


def _unit(rng, n):
    v = rng.standard_normal((n, 3))
    return (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)


def _scene(case, seed):
    """Numpy inputs of a single-room case."""
    rng = np.random.default_rng(seed)
    room = _sizes(case["room"])
    return dict(room_sz=room, beta=gpurir.beta_sabine_closed_form(room, case["t60"]),
                pos_src=_inside(rng, case["n_src"], room), pos_rcv=_inside(rng, case["n_rcv"], room),
                orV_src=_unit(rng, case["n_src"]) if case["spkr"] != "omni" else None,
                orV_rcv=_unit(rng, case["n_rcv"]) if case["mic"] != "omni" else None,
                nb_img=[int(v) for v in case["nb"].split("x")], Tmax=case["tmax"], Tdiff=case["tdiff"],
                spkr_pattern=case["spkr"], mic_pattern=case["mic"])


def _rooms(case, seed):
    """Uneven rooms of a batch: early part to 0.4 T60 with a diffuse tail after it, or
    image sources only up to a length between t_lo and t_hi."""
    rng = np.random.default_rng(seed)
    n = case["rooms"]
    dims = np.stack([rng.uniform(3, 10, n), rng.uniform(3, 8, n), rng.uniform(2.5, 4.5, n)], axis=1)
    # lengths spread evenly over the range, in an order of the case's own: batches of one
    # case differ in their rooms, not in the sizes of their RIRs
    t = case["t_lo"] + (case["t_hi"] - case["t_lo"]) * (np.random.default_rng(n).permutation(n) + 0.5) / n
    t60 = t if case["tail"] else 1.6 * t
    beta = gpurir.beta_sabine_closed_form(dims, t60)
    rooms = []
    for i in range(n):
        tdiff = 0.4 * t[i] if case["tail"] else 0.9 * t[i]
        rooms.append(dict(room_sz=dims[i].astype(np.float32), beta=beta[i],
                          pos_src=_inside(rng, 1 + i % case["max_src"], dims[i]),
                          pos_rcv=_inside(rng, 1 + (i // 2) % case["max_rcv"], dims[i]),
                          nb_img=_counts(tdiff, dims[i]), Tmax=float(t[i]),
                          Tdiff=float(tdiff) if case["tail"] else float(t[i]),
                          spkr_pattern="omni", mic_pattern="omni", orV_src=None, orV_rcv=None))
    return rooms


def _fit(case, seed):
    """Parameters (numpy) of a fitting case, and the walls that made the measured RIRs."""
    rng = np.random.default_rng(seed)
    n, room = case["rooms"], _sizes(case["room"])
    p = dict(beta=rng.uniform(0.6, 0.95, (n, 6)).astype(np.float32),
             pos_src=np.concatenate([_inside(rng, case["n_src"], room, 0.5) for _ in range(n)]),
             pos_rcv=np.concatenate([_inside(rng, case["n_rcv"], room, 0.5) for _ in range(n)]),
             orV_rcv=_unit(rng, n * case["n_rcv"]) if case["mic"] != "omni" else None)
    return p, rng.uniform(0.6, 0.95, (n, 6)).astype(np.float32)


def _fit_rooms(case):
    room = _sizes(case["room"])
    return [dict(room_sz=room, pos_src=np.zeros((case["n_src"], 3)), pos_rcv=np.zeros((case["n_rcv"], 3)),
                 nb_img=[int(v) for v in case["nb"].split("x")], Tmax=case["tmax"], spkr_pattern="omni",
                 mic_pattern=case["mic"]) for _ in range(case["rooms"])]


def _fit_rirs(case, beta, pos_src, pos_rcv, orV_rcv):
    """Packed float64 RIRs of a fitting case in plain torch."""
    room = _sizes(case["room"])
    n_ism = _n_samples(case["tmax"], case["fs"])
    out = []
    for i in range(case["rooms"]):
        s = slice(i * case["n_src"], (i + 1) * case["n_src"])
        r = slice(i * case["n_rcv"], (i + 1) * case["n_rcv"])
        out.append(_early(room, beta[i], pos_src[s], pos_rcv[r], [int(v) for v in case["nb"].split("x")], n_ism,
                          case["fs"], "omni", case["mic"], None, orV_rcv[r] if orV_rcv is not None else None))
    return torch.cat([o.reshape(-1) for o in out])


def _walk(case, seed):
    rng = np.random.default_rng(seed)
    n, P = case["signal"], case["points"]
    sig = rng.standard_normal(n).astype(np.float32)
    decay = np.exp(-6.0 * np.arange(case["rir_len"]) / case["rir_len"]).astype(np.float32)
    rirs = rng.standard_normal((P, case["n_rcv"], case["rir_len"]), dtype=np.float32) * decay
    stamps = None
    if case["stamps"]:   # uneven steps along the path
        w = rng.uniform(0.7, 1.3, P)
        stamps = np.concatenate([[0.0], np.cumsum(w)[:-1] / w.sum()]) * n / case["fs"]
    return sig, rirs, stamps


def prepare(case, seed):
    kind, dev = case["kind"], "cuda"
    st = dict(case=case, kind=kind)
    up = lambda a: None if a is None else torch.from_numpy(a).to(dev)
    if kind == "host":
        gpurir.set_noise(case["noise"])
        st["args"] = dict(_scene(case, seed), fs=float(case["fs"]))
    elif kind == "device":
        s = _scene(case, seed)
        st["sim"] = gpurir.Simulator(mixed_precision=case["mode"] == "mp", lut=case["mode"] == "lut")
        st["sim"].set_noise(case["noise"])
        out = torch.empty((case["n_src"], case["n_rcv"], _n_samples(case["tmax"], case["fs"])), device=dev)
        st["args"] = (s["room_sz"], s["beta"], up(s["pos_src"]), up(s["pos_rcv"]), up(s["orV_src"]),
                      up(s["orV_rcv"]), gpurir.polar_patterns[case["spkr"]], gpurir.polar_patterns[case["mic"]],
                      s["nb_img"], case["tdiff"], case["tmax"], float(case["fs"]), 343.0, out)
    elif kind == "plan":
        st["plan"] = batch.BatchPlan(_rooms(case, seed), float(case["fs"]))
    elif kind == "batch":
        st["rooms"] = _rooms(case, seed)
    elif kind in ("step", "grad"):
        p, walls = _fit(case, seed)
        st["params"] = {k: up(v) for k, v in p.items()}
        with torch.no_grad():
            q = {k: None if v is None else v.double() for k, v in st["params"].items()}
            q["beta"] = up(walls).double()
            st["target"] = _fit_rirs(case, **q).float()
        for v in st["params"].values():
            if v is not None:
                v.requires_grad_(True)
        st["model"] = autograd.TorchBatch(_fit_rooms(case), float(case["fs"]))
    elif kind == "filter":
        sig, rirs, stamps = _walk(case, seed)
        st["args"] = (sig, rirs) + ((stamps, float(case["fs"])) if stamps is not None else ())
    elif kind == "traj":
        sig, rirs, stamps = _walk(case, seed)
        st["sig"], st["rirs"] = up(sig).requires_grad_(True), up(rirs).requires_grad_(True)
        st["stamps"] = dict(timestamps=stamps, fs=float(case["fs"])) if stamps is not None else {}
        g = torch.Generator(device=dev).manual_seed(seed)
        st["grad"] = torch.randn((case["signal"] + case["rir_len"] - 1, case["n_rcv"]), device=dev, generator=g,
                                 dtype=torch.float64)
    return st


def run(st):
    kind = st["kind"]
    if kind == "host":
        gpurir.seed(7)   # reproducible diffuse tails
        return gpurir.simulateRIR(**st["args"])
    if kind == "device":
        st["sim"].set_seed(7)
        return st["sim"].simulate_rir_device(*st["args"])
    if kind == "plan":
        return st["plan"].launch()
    if kind == "batch":
        gpurir.simulator().set_noise("logistic")
        gpurir.seed(7)
        return batch.simulate_batch(st["rooms"], float(st["case"]["fs"]))[0]
    if kind == "step":
        loss = st["model"].l2_step(**st["params"], target=st["target"])
        return dict(loss=loss, rirs=st["model"].last_rirs,
                    grads={k: v.grad for k, v in st["params"].items() if v is not None})
    if kind == "grad":
        rirs = st["model"](**st["params"])
        loss = ((rirs - st["target"]) ** 2).sum()
        names = [k for k, v in st["params"].items() if v is not None]
        grads = torch.autograd.grad(loss, [st["params"][k] for k in names])
        return dict(loss=loss.detach(), rirs=rirs.detach(), grads=dict(zip(names, grads)))
    if kind == "filter":
        return gpurir.simulateTrajectory(*st["args"])
    y = trajectory.simulate_trajectory_torch(st["sig"], st["rirs"], **st["stamps"])
    gs, gr = torch.autograd.grad(y, [st["sig"], st["rirs"]], st["grad"])
    return dict(y=y.detach(), grad_signal=gs, grad_rirs=gr)


# ---------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------
def _ism_work(n_img, pairs, n_ism, n_total, fs):
    """Positions are small; every output sample is written once.  Per image its delay
    and amplitude (~40 operations), per early sample one pass of the window."""
    reach = min(1.0, math.pi / 6)   # images of the box that lie within the sphere of the early part
    return 4 * pairs * n_total, pairs * (40 * reach * n_img + 2 * 0.008 * fs * n_ism)


def work(case):
    kind = case["kind"]
    if kind in ("host", "device"):
        nb = [int(v) for v in case["nb"].split("x")]
        b, f = _ism_work(nb[0] * nb[1] * nb[2], case["n_src"] * case["n_rcv"], _n_samples(case["tdiff"], case["fs"]),
                         _n_samples(case["tmax"], case["fs"]), case["fs"])
        return dict(bytes=b, flops=f)
    if kind in ("plan", "batch"):
        b = f = 0
        for r in _rooms(case, 0):
            x, y = _ism_work(int(np.prod(r["nb_img"])), len(r["pos_src"]) * len(r["pos_rcv"]),
                             _n_samples(r["Tdiff"], case["fs"]), _n_samples(r["Tmax"], case["fs"]), case["fs"])
            b, f = b + x, f + y
        return dict(bytes=b, flops=f)
    if kind in ("step", "grad"):
        nb = [int(v) for v in case["nb"].split("x")]
        n = _n_samples(case["tmax"], case["fs"])
        b, f = _ism_work(nb[0] * nb[1] * nb[2], case["rooms"] * case["n_src"] * case["n_rcv"], n, n, case["fs"])
        return dict(bytes=2 * b, flops=3 * f)   # RIRs written, target read; forward, and the adjoint twice that
    P, R, L, S = case["points"], case["n_rcv"], case["rir_len"], -(-case["signal"] // case["points"])
    n_out = case["signal"] + L - 1
    N = 1 << (S + L - 2).bit_length()
    fft = 2.5 * N * math.log2(N)
    if kind == "filter":
        return dict(bytes=4 * (case["signal"] + P * R * L) + 8 * n_out * R, flops=P * R * (2 * fft + 3 * N))
    return dict(bytes=2 * 4 * (case["signal"] + P * R * L) + 2 * 8 * n_out * R, flops=P * R * (5 * fft + 9 * N))


# ---------------------------------------------------------------------------
# What the entry points compute, in 64 bits
# ---------------------------------------------------------------------------
def _n_samples(T, fs):
    n = int(np.ceil(np.float32(T) * np.float32(fs)))
    return n + n % 2


def _gain(ct, pattern):
    if pattern == "homni":
        return (ct > 0).double()
    a = {"card": 0.5, "hypcard": 0.25, "subcard": 0.75, "bidir": 0.0}[pattern]
    return a + (1 - a) * ct


def _early(room, beta, pos_src, pos_rcv, nb, n_ism, fs, spkr, mic, orv_src, orv_rcv, c=343.0):
    """Image-source sum [n_src, n_rcv, n_ism] with the Hann-windowed sinc; float64 tensors
    beta [6], positions and orientations [n, 3]."""
    dev, f64 = beta.device, torch.float64
    Tw = int(round(float(np.float32(8e-3) * np.float32(fs))))
    H = Tw / 2.0
    k = torch.arange(math.floor(-H) + 1, math.floor(H) + 2, device=dev)
    L = [float(np.float32(v)) for v in room]
    axes = []
    for d in range(3):
        m = torch.arange(nb[d], device=dev) - nb[d] // 2
        clust, refl = torch.div(m + 1, 2, rounding_mode="floor"), m % 2
        att = torch.pow(-beta[2 * d], (clust - refl).abs().to(f64)) * torch.pow(-beta[2 * d + 1], clust.abs().to(f64))
        axes.append((2.0 * clust.to(f64) * L[d], (1 - 2 * refl).to(f64), att))
    n_img = nb[0] * nb[1] * nb[2]
    n_s, n_r = pos_src.shape[0], pos_rcv.shape[0]
    per = max(1, (1 << 24) // len(k))   # images per step over all pairs taken together
    rows_at_once = max(1, per // n_img)
    out = torch.zeros((n_s * n_r * n_ism,), dtype=f64, device=dev)
    pairs = torch.arange(n_s * n_r, device=dev)
    for p0 in range(0, n_s * n_r, rows_at_once):
        pr = pairs[p0:p0 + rows_at_once]
        s, r = torch.div(pr, n_r, rounding_mode="floor"), pr % n_r
        step = max(1, per // len(pr))
        for i0 in range(0, n_img, step):
            i = torch.arange(i0, min(i0 + step, n_img), device=dev)
            m = [torch.div(i, nb[1] * nb[2], rounding_mode="floor"),
                 torch.div(i, nb[2], rounding_mode="floor") % nb[1], i % nb[2]]
            v = [axes[d][0][m[d]][None, :] + axes[d][1][m[d]][None, :] * pos_src[s, d][:, None] -
                 pos_rcv[r, d][:, None] for d in range(3)]
            dist = torch.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
            near = dist.detach() * (fs / c) < n_ism + H
            pi, ii = torch.nonzero(near, as_tuple=True)
            dist, v = dist[pi, ii], [x[pi, ii] for x in v]
            amp = (axes[0][2][m[0]] * axes[1][2][m[1]] * axes[2][2][m[2]])[ii] / (4 * math.pi * dist)
            if spkr != "omni":
                o = orv_src / orv_src.norm(dim=1, keepdim=True)
                ct = -sum(axes[d][1][m[d]][ii] * o[s[pi], d] * v[d] for d in range(3)) / dist
                amp = amp * _gain(ct, spkr)
            if mic != "omni":
                o = orv_rcv / orv_rcv.norm(dim=1, keepdim=True)
                amp = amp * _gain(sum(o[r[pi], d] * v[d] for d in range(3)) / dist, mic)
            tau = dist * (fs / c)
            t = torch.floor(tau.detach()).long()[:, None] + k[None, :]
            x = t - tau[:, None]
            ok = (x.detach().abs() < H) & (t >= 0) & (t < n_ism)
            w = 0.5 * (1 + torch.cos(2 * math.pi / Tw * x)) * torch.sinc(x) * ok
            at = (pr[pi] * n_ism)[:, None] + t.clamp(0, n_ism - 1)
            out = out.index_add(0, at.reshape(-1), (amp[:, None] * w).reshape(-1)) if out.requires_grad or \
                amp.requires_grad else out.index_add_(0, at.reshape(-1), (amp[:, None] * w).reshape(-1))
    return out.reshape(n_s, n_r, n_ism)


def _philox_uniforms(rirs, n, seed, call, device):
    """Uniforms [len(rirs), n] of the Philox4x32-10 stream with key (seed), counter (s/4, rir, call)."""
    m32 = 0xFFFFFFFF
    blocks = (n + 3) // 4
    c = [torch.arange(blocks, device=device)[None, :].expand(len(rirs), blocks), rirs[:, None].expand(-1, blocks),
         torch.full((1, 1), call & m32, device=device), torch.full((1, 1), call >> 32, device=device)]
    k0, k1 = seed & m32, seed >> 32
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57   # products of 64 bits, their halves taken by masks
        c = [((p1 >> 32) & m32) ^ c[1] ^ k0, p1 & m32, ((p0 >> 32) & m32) ^ c[3] ^ k1, p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    w = torch.stack([x.expand(len(rirs), blocks) for x in c], dim=-1).reshape(len(rirs), -1)[:, :n]
    return ((w >> 9).double() + 0.5) / 2 ** 23


def _with_tail(early, room, beta, pos_src, pos_rcv, n_total, fs, noise, rir0=0, c=343.0, seed=7, call=0):
    """early [n_src, n_rcv, n_ism] followed by the diffuse tail."""
    n_s, n_r, n_ism = early.shape
    if n_total <= n_ism:
        return early
    dev = early.device
    L = [float(np.float32(v)) for v in room]
    b2 = 1 - beta ** 2
    Sa = (b2[0] + b2[1]) * L[1] * L[2] + (b2[2] + b2[3]) * L[0] * L[2] + (b2[4] + b2[5]) * L[0] * L[1]
    alpha = float(-13.8155 / (0.161 * L[0] * L[1] * L[2] / Sa * fs))
    tau = ((pos_src[:, None] - pos_rcv[None, :]) ** 2).sum(-1).sqrt().reshape(-1) * (fs / c)
    start = torch.ceil(torch.clamp(tau, min=float(np.float32(n_ism) - np.float32(0.01) * np.float32(fs)))).long()
    e = early.reshape(n_s * n_r, n_ism)
    t = torch.arange(n_ism, device=dev)
    count = (n_ism - start).double()
    power = (e ** 2 * (t[None, :] >= start[:, None])).sum(1) / count
    A = torch.where(count > 0, power / torch.exp(alpha * (start + count / 2 - tau)), torch.zeros_like(tau))
    n = n_total - n_ism
    u = _philox_uniforms(rir0 + torch.arange(n_s * n_r, device=dev), n + n % 4, seed, call, dev)
    if noise == "logistic":
        z = 0.551329 * torch.log(u / (1 - u + 1e-6))
    else:
        u = torch.nn.functional.pad(u, (0, -u.shape[1] % 4), value=0.5).reshape(n_s * n_r, -1, 2)
        rad = torch.sqrt(-2 * torch.log(u[..., 0]))
        z = torch.stack([rad * torch.cos(2 * math.pi * u[..., 1]), rad * torch.sin(2 * math.pi * u[..., 1])],
                        dim=-1).reshape(n_s * n_r, -1)
    s = torch.arange(n, device=dev).double()
    tail = torch.sqrt(A)[:, None] * torch.exp(0.5 * alpha * (n_ism + s[None, :] - tau[:, None])) * z[:, :n]
    return torch.cat([e, tail], dim=1).reshape(n_s, n_r, n_total)


def _room64(r, fs, noise, rir0=0):
    up = lambda a: None if a is None else torch.from_numpy(np.asarray(a, np.float32)).to("cuda").double()
    beta, ps, pr = up(r["beta"]), up(r["pos_src"]), up(r["pos_rcv"])
    n_ism, n_total = _n_samples(r["Tdiff"], fs), _n_samples(r["Tmax"], fs)
    early = _early(r["room_sz"], beta, ps, pr, r["nb_img"], n_ism, fs, r["spkr_pattern"], r["mic_pattern"],
                   up(r["orV_src"]), up(r["orV_rcv"]))
    return _with_tail(early, r["room_sz"], beta, ps, pr, n_total, fs, noise, rir0)


@torch.no_grad()
def _exact_rirs(case, seed):
    fs = case["fs"]
    if case["kind"] in ("host", "device"):
        if case["mode"] != "f32":
            return None   # the table's and the half-precision window's values are not the exact sum
        return _room64(_scene(case, seed), fs, case["noise"])
    out, rir0 = [], 0
    for r in _rooms(case, seed):
        out.append(_room64(r, fs, "logistic", rir0).reshape(-1))
        rir0 += len(r["pos_src"]) * len(r["pos_rcv"])
    return torch.cat(out)


def _exact_walk(case, seed):
    sig, rirs, stamps = _walk(case, seed)
    P, R, L, n = case["points"], case["n_rcv"], case["rir_len"], case["signal"]
    at = np.arange(P) * (n / P) if stamps is None else np.asarray(stamps) * case["fs"]
    w = np.append(at.astype(int), n)
    sig = torch.from_numpy(sig).cuda().double().requires_grad_(True)
    rirs = torch.from_numpy(rirs).cuda().double().requires_grad_(True)
    S = int(np.diff(w).max())
    N = 1 << (S + L - 2).bit_length()
    y = torch.zeros((R, n + L - 1), dtype=torch.float64, device="cuda")
    for p in range(P):
        m = int(w[p + 1] - w[p])
        conv = torch.fft.irfft(torch.fft.rfft(sig[w[p]:w[p + 1]], N)[None] * torch.fft.rfft(rirs[p], N), N)
        y = y + torch.nn.functional.pad(conv[:, :m + L - 1], (int(w[p]), n - int(w[p + 1])))
    y = y.T
    if case["kind"] == "filter":
        return y.detach()
    g = torch.Generator(device="cuda").manual_seed(seed)
    g = torch.randn((n + L - 1, R), device="cuda", generator=g, dtype=torch.float64)
    gs, gr = torch.autograd.grad(y, [sig, rirs], g)
    return dict(y=y.detach(), grad_signal=gs, grad_rirs=gr)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("filter", "traj"):
        return _exact_walk(case, seed)
    if kind not in ("step", "grad"):
        return _exact_rirs(case, seed)
    p, walls = _fit(case, seed)
    q = {k: None if v is None else torch.from_numpy(v).cuda().double() for k, v in p.items()}
    with torch.no_grad():
        target = _fit_rirs(case, **dict(q, beta=torch.from_numpy(walls).cuda().double())).float().double()
    names = [k for k, v in q.items() if v is not None]
    for k in names:
        q[k].requires_grad_(True)
    rirs = _fit_rirs(case, **q)
    loss = ((rirs - target) ** 2).sum()
    grads = torch.autograd.grad(loss, [q[k] for k in names])
    return dict(loss=loss.detach(), rirs=rirs.detach(), grads=dict(zip(names, grads)))
