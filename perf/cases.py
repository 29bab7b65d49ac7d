"""What this framework is used for, as cases that can be timed and compared.

Deblending is the main path: whole calls of ``deblend`` (host data in, host
data out) from one small gather to a 4-D vibroseis survey, ``deblend_batch``
over many gathers, and ``solve_learned`` on a planned problem.  Beside it the
network's training gradient and ``blend``, which makes the blended input.
Sizes are those of the benchmark workloads and the tests, and odd ones: real
surveys seldom divide into their windows.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import agdeblend_b200 as agd
from agdeblend_b200 import warmstart
from agdeblend_b200.nn import WarmStartNet

RATE = 250  # samples per second
LIVE, BAD, MISSING = 0, 1, 2
PAD, TARGET = 0.25, 1e-3
FLOOR = 0.05  # of the window fold, in the warm start
SWEEP = 256  # samples


def listed():
    return [
        # one small receiver gather while parameters are tried out: launches and set-up
        dict(name="gather_small", kind="gather", shots=40, nt=200, ws=16, wt=128, its=30,
             dtype="float32"),
        # the benchmark's 2-D receiver gather
        dict(name="gather", kind="gather", shots=128, nt=512, ws=32, wt=256, its=100,
             dtype="float32"),
        # a gather in double precision, of a size that no window divides
        dict(name="gather_f64", kind="gather", shots=217, nt=901, ws=64, wt=256, its=60,
             dtype="float64"),
        # a line's gathers solved together: uneven gathers, mixed windows
        dict(name="gathers", kind="batch", n=64, shots0=100, shots1=400, nt0=512, nt1=2048,
             its=100, dtype="float32"),
        # the benchmark's headline survey: two sources, 3-D, a production run
        dict(name="survey_3d", kind="survey3d", vols=2, ch=64, shots=128, nt=1024, wc=16, ws=32,
             wt=256, its=200, dtype="float32"),
        # a 3-D survey whose windows come out uneven (18, 17 for 16; 35, 34 for 32)
        dict(name="survey_3d_ragged", kind="survey3d", vols=1, ch=37, shots=101, nt=873, wc=16,
             ws=32, wt=256, its=60, dtype="float32"),
        # a small 3-D survey in double precision
        dict(name="survey_3d_f64", kind="survey3d", vols=2, ch=24, shots=64, nt=1024, wc=16,
             ws=32, wt=256, its=40, dtype="float64"),
        # 4-D vibroseis with a sweep, of a size that its windows do not divide
        dict(name="vibroseis_ragged", kind="vibroseis", sy=18, sx=27, ch=21, nt=1500, ws=16,
             wt=256, its=20, dtype="float32"),
        # the benchmark's full vibroseis survey, the largest: a quick look
        dict(name="vibroseis_full", kind="vibroseis", sy=32, sx=64, ch=32, nt=2048, ws=16,
             wt=256, its=20, dtype="float32"),
        # the learned warm start of the 3-D survey: network estimate, then 20 iterations
        dict(name="learned", kind="learned", vols=2, ch=64, shots=128, nt=1024, wc=16, ws=32,
             wt=256, its=100, begin=80),
        # loss and gradient of one training batch of the warm-start network
        dict(name="train_batch", kind="train", n=32, h=32, w=256, channels=1, base=32),
        # blending a 3-D survey's unblended traces, as before a test of the method
        dict(name="blend", kind="blend", vols=2, ch=64, shots=128, nt=1024, mode=0,
             dtype="float32"),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["gather", "gather", "batch", "survey3d", "survey3d", "survey3d",
                       "vibroseis", "learned", "train", "blend"])
    if kind == "gather":
        ws, wt = rng.choice([(16, 128), (32, 256), (64, 256)])
        return dict(kind=kind, shots=_log(rng, ws, 400), nt=_log(rng, max(200, wt), 2048), ws=ws, wt=wt,
                    its=_log(rng, 30, 100), dtype=rng.choice(["float32", "float32", "float64"]))
    if kind == "batch":
        return dict(kind=kind, n=_log(rng, 4, 64), shots0=100, shots1=rng.randrange(120, 401),
                    nt0=512, nt1=rng.randrange(600, 2049), its=_log(rng, 30, 100),
                    dtype="float32")
    if kind == "survey3d":
        wc, ws = rng.choice([(16, 16), (16, 32), (16, 32)])
        dtype = rng.choice(["float32", "float32", "float32", "float64"])
        top = (64, 128) if dtype == "float32" else (32, 96)
        return dict(kind=kind, vols=rng.randrange(1, 3), ch=_log(rng, wc, top[0]),
                    shots=_log(rng, ws, top[1]), nt=_log(rng, 500, 1100), wc=wc, ws=ws,
                    wt=rng.choice([128, 256, 256]), its=_log(rng, 20, 60), dtype=dtype)
    if kind == "vibroseis":
        return dict(kind=kind, sy=_log(rng, 16, 24), sx=_log(rng, 16, 32), ch=_log(rng, 16, 24),
                    nt=_log(rng, 1000, 2048), ws=16, wt=256, its=_log(rng, 5, 12),
                    dtype="float32")
    if kind == "learned":
        its = rng.randrange(40, 101)
        return dict(kind=kind, vols=rng.randrange(1, 3), ch=_log(rng, 16, 64),
                    shots=_log(rng, 32, 128), nt=_log(rng, 500, 1024), wc=16, ws=32, wt=256,
                    its=its, begin=its - rng.randrange(10, 31))
    if kind == "train":
        return dict(kind=kind, n=_log(rng, 4, 48), h=8 * rng.randrange(2, 7),
                    w=8 * rng.randrange(8, 41), channels=rng.choice([1, 3]), base=32)
    return dict(kind=kind, vols=rng.randrange(1, 3), ch=_log(rng, 8, 64),
                shots=_log(rng, 16, 128), nt=_log(rng, 300, 1024), mode=rng.choice([0, 1]),
                dtype=rng.choice(["float32", "float64"]))


# ------------------------------------------------------------------ inputs


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _events(gen, off, nt):
    """[traces][nt]: six linear and six hyperbolic Ricker events over the offsets `off` (m),
    with 1 % noise."""
    dev = off.device
    out = torch.zeros(off.numel(), nt, device=dev)
    k = torch.arange(-16, 17, device=dev)
    for e in range(12):
        u = torch.rand(3, generator=gen).tolist()
        amp = float(torch.randn(1, generator=gen))
        t0 = (0.1 + 0.8 * u[0]) * nt / RATE
        if e < 6:
            t = t0 + (0.8 * u[1] - 0.4) * 1e-3 * off
        else:
            t = torch.sqrt(t0 ** 2 + (off / (1500 + 2000 * u[1])) ** 2)
        s = t * RATE
        idx = torch.floor(s).long()[:, None] + k
        a = (math.pi * 20 * (idx - s[:, None]) / RATE) ** 2
        val = amp * (1 - 2 * a) * torch.exp(-a)
        ok = (idx >= 0) & (idx < nt)
        out.scatter_add_(1, idx.clamp(0, nt - 1), val * ok)
    g = torch.Generator(device=dev)
    g.manual_seed(int(torch.randint(1 << 30, (1,), generator=gen)))
    rms = out.square().mean().sqrt()
    return out + 0.01 * rms * torch.randn(out.shape, generator=g, device=dev)


def _sweep():
    t = np.arange(SWEEP) / RATE
    w = np.sin(2 * np.pi * (8 * t + 0.5 * 72 / (SWEEP / RATE) * t * t))
    m = SWEEP // 10
    ramp = 0.5 * (1 - np.cos(np.pi * np.arange(m) / m))
    w[:m] *= ramp
    w[-m:] *= ramp[::-1]
    return w


def _pseudo(sts, chs, tts, truths):
    """Each patch's blended traces: all non-missing traces summed into one record per channel,
    the spans of bad traces muted, and read back at each trace's own time."""
    dev = truths[0].device
    t0 = min(int(s.min()) for s in sts)
    nts = [x.shape[1] for x in truths]
    length = max(int(s.max()) for s in sts) - t0 + max(nts)
    nch = max(int(c.max()) for c in chs) + 1
    rec = torch.zeros(nch * length, dtype=torch.float64, device=dev)
    mute = torch.zeros(nch * length, dtype=torch.bool, device=dev)
    at = []
    for s, c, nt in zip(sts, chs, nts):
        base = torch.as_tensor(c.astype(np.int64) * length + s - t0, device=dev)
        at.append((base, torch.arange(nt, device=dev)))
    for (base, k), tt, x in zip(at, tts, truths):
        live = torch.as_tensor(tt != MISSING, device=dev)
        bad = torch.as_tensor(tt == BAD, device=dev)
        rec.index_add_(0, (base[live, None] + k).reshape(-1), x[live].reshape(-1).double())
        mute[(base[bad, None] + k).reshape(-1)] = True
    rec[mute] = 0
    out = []
    for (base, k), tt, x in zip(at, tts, truths):
        live = torch.as_tensor(tt != MISSING, device=dev)
        out.append((rec[base[:, None] + k] * live[:, None]).to(x.dtype))
    return out


def _gather(gen, shots, nt, ws, wt):
    off = (torch.arange(shots, device=_device()) - shots // 2) * 12.5
    st = np.round(np.cumsum(0.8 + 0.4 * torch.rand(shots, generator=gen).numpy()) * RATE)
    return dict(volumes=[0], window_shapes=[[ws, wt]], coords=[[0]], shapes=[[shots, nt]],
                shottimes=[st.astype(np.int64)], channels=[np.zeros(shots, np.int32)],
                trace_types=[np.zeros(shots, np.int32)], truth=[_events(gen, off, nt)])


def _survey3d(gen, c):
    ch, shots, nt, vols = c["ch"], c["shots"], c["nt"], c["vols"]
    dev = _device()
    ci, si = np.repeat(np.arange(ch), shots), np.tile(np.arange(shots), ch)
    off = torch.as_tensor((si - shots // 2) * 12.5 + (ci - ch // 2) * 25.0, device=dev).float()
    gap = 3.0 + 1.25 * nt / RATE  # two breaks in the recording
    p = dict(volumes=list(range(vols)), coords=[[0, 0]] * vols, shapes=[[ch, shots, nt]] * vols,
             window_shapes=[[c.get("wc", 16), c.get("ws", 32), c.get("wt", 256)]] * vols,
             shottimes=[], channels=[], trace_types=[], truth=[])
    for v in range(vols):
        k = np.arange(shots)
        t = 1.2 * k + 0.6 * v + 0.5 * torch.rand(shots, generator=gen).numpy()
        t = t + gap * (k > shots // 3) + gap * (k > 2 * shots // 3)
        u = torch.rand(ch * shots, generator=gen).numpy()
        tt = np.where(u < 0.04, BAD, np.where(u < 0.08, MISSING, LIVE)).astype(np.int32)
        tt[0] = LIVE
        p["shottimes"].append(np.round(t * RATE).astype(np.int64)[si])
        p["channels"].append(ci.astype(np.int32))
        p["trace_types"].append(tt)
        p["truth"].append(_events(gen, off, nt))
    return p


def _vibroseis(gen, c):
    sy, sx, ch, nt = c["sy"], c["sx"], c["ch"], c["nt"]
    iy, ix, ic = (v.reshape(-1) for v in np.meshgrid(np.arange(sy), np.arange(sx), np.arange(ch),
                                                     indexing="ij"))
    off = np.sqrt(((ix - sx / 2) * 25.0) ** 2 + ((iy - sy / 2) * 25.0) ** 2) + (ic - ch / 2) * 12.5
    x = _events(gen, torch.as_tensor(off, device=_device()).float(), nt)
    n = nt + SWEEP
    spec = torch.fft.rfft(torch.as_tensor(_sweep(), device=x.device).float(), n)
    for a in range(0, x.shape[0], 8192):
        x[a: a + 8192] = torch.fft.irfft(torch.fft.rfft(x[a: a + 8192], n) * spec, n)[:, :nt]
    st = np.round(np.cumsum(0.8 + 0.4 * torch.rand(sy * sx, generator=gen).numpy()) * RATE)
    n_tr = sy * sx * ch
    return dict(volumes=[0], window_shapes=[[c["ws"]] * 3 + [c["wt"]]], coords=[[0, 0, 0]],
                shapes=[[sy, sx, ch, nt]], shottimes=[st.astype(np.int64)[iy * sx + ix]],
                channels=[ic.astype(np.int32)], trace_types=[np.zeros(n_tr, np.int32)],
                truth=[x], wavelets=[_sweep()], wavelet_idxs=[np.zeros(n_tr, np.int32)])


def _problem(case, seed):
    """deblend's arguments of one problem, its data as tensors [traces][samples]."""
    gen = torch.Generator().manual_seed(seed)
    kind = case["kind"]
    if kind == "gather":
        p = _gather(gen, case["shots"], case["nt"], case["ws"], case["wt"])
    elif kind == "vibroseis":
        p = _vibroseis(gen, case)
    else:
        p = _survey3d(gen, case)
    dtype = torch.float64 if case.get("dtype") == "float64" else torch.float32
    truth = [x.to(dtype) for x in p.pop("truth")]
    if kind == "blend":
        p["data"] = truth
    else:
        p["data"] = _pseudo(p["shottimes"], p["channels"], p["trace_types"], truth)
    if "wavelets" in p:
        p["wavelets"] = [w.astype(case["dtype"]) for w in p["wavelets"]]
    return p


def _batch(case, seed):
    gen = torch.Generator().manual_seed(seed)
    sizes = np.random.default_rng(3000)  # the sizes are the case's, the data the seed's
    got = []
    for _ in range(case["n"]):
        shots = int(sizes.integers(case["shots0"], case["shots1"] + 1))
        nt = int(sizes.integers(case["nt0"], case["nt1"] + 1))
        ws, wt = [(16, 128), (32, 256), (64, 256)][int(sizes.integers(0, 3))]
        p = _gather(gen, shots, nt, ws, wt)
        p["data"] = _pseudo(p["shottimes"], p["channels"], p["trace_types"], p.pop("truth"))
        got.append(p)
    return got


def _to_host(p):
    p["data"] = [x.reshape(s).cpu().numpy() for x, s in zip(p["data"], p["shapes"])]
    return p


def _train_arrays(case, seed):
    """A batch as the training set has it: blended windows with unit RMS, and their targets."""
    g = torch.Generator().manual_seed(seed)
    n, h, w = case["n"], case["h"], case["w"]
    off = (torch.arange(n * h, device=_device()) % h - h // 2) * 12.5
    y = _events(g, off, w).cpu().numpy().reshape(n, h, w)
    y = y / np.sqrt(np.mean(y * y))
    rng = np.random.default_rng(seed)
    x = np.stack([y + 0.5 * np.roll(y, 1 + i, axis=0)[:, rng.permutation(h)]
                  for i in range(case["channels"])], -1)
    x = x[..., 0] if case["channels"] == 1 else x
    return np.ascontiguousarray(x, np.float32), np.ascontiguousarray(y, np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ps = [_to_host(p) for p in _batch(case, seed)]
        for p in ps:
            p.pop("shapes")
        return dict(kind=kind, problems=ps, its=case["its"])
    if kind == "train":
        x, y = _train_arrays(case, seed)
        return dict(kind=kind, x=x, y=y, net=WarmStartNet(case["base"], seed=1,
                                                          in_channels=case["channels"]))
    p = _to_host(_problem(case, seed))
    shapes = p.pop("shapes")
    if kind == "blend":
        # read back at the same shots, the traces with a bad record too (muted)
        tt = [np.where(t == BAD, LIVE, t).astype(np.int32) for t in p["trace_types"]]
        return dict(kind=kind, args=[p["shottimes"], p["channels"], p["trace_types"], p["data"]],
                    options=dict(blend_mode=case["mode"], trace_types_out=tt))
    if kind == "learned":
        data = p.pop("data")
        return dict(kind=kind, data=data, its=case["its"], begin=case["begin"],
                    net=WarmStartNet(32, seed=1),
                    problem=agd.Problem(n_dims=[3] * len(shapes), shapes=shapes, **p))
    return dict(kind=kind, args=p, its=case["its"])


def run(state):
    kind = state["kind"]
    if kind == "batch":
        return agd.deblend_batch(state["problems"], 1.0, state["its"])
    if kind == "train":
        return state["net"].loss_grad(state["x"], state["y"])
    if kind == "blend":
        return agd.blend(*state["args"], **state["options"])
    if kind == "learned":
        return warmstart.solve_learned(state["problem"], state["net"], state["data"], 1.0,
                                       state["its"], state["begin"])
    return agd.deblend(initial_factor=1.0, n_its=state["its"], print_freq=0, **state["args"])


# ------------------------------------------------------------------ work


def _windows(n, length):
    """(start, length) of the windows along one axis."""
    half = length // 2
    count = 1 if length == n else n // half - 1
    base = (n - half) // count + half
    larger = n - half - (base - half) * count
    out, start = [], 0
    for i in range(count):
        out.append((start, base + (i < larger)))
        start += out[-1][1] - half
    return out


def _padded(n):
    return int(math.ceil(n * (1 + PAD)))


def _sizes(shape, window, wl=1):
    """Complex model values, FFT operations of one transform, record samples (an upper bound:
    every trace apart) of one patch."""
    h = window[-1] // 2
    steps = -(-(shape[-1] - wl + 1) // h) + 1
    values = flops = traces = 0
    axes = [_windows(n, w) for n, w in zip(shape[:-1], window[:-1])]
    for combo in np.ndindex(*[len(a) for a in axes]):
        dims = [_padded(axes[d][i][1]) for d, i in enumerate(combo)]
        n = math.prod(dims)
        pt = _padded(window[-1])
        values += steps * n * (pt // 2 + 1)
        flops += steps * n * (pt // 2 + 1) * 5 * math.log2(n)
        cropped = math.prod(axes[d][i][1] for d, i in enumerate(combo))
        flops += steps * cropped * 2.5 * pt * math.log2(pt)
        traces += cropped
    return values, flops, traces


def work(case):
    kind = case["kind"]
    size = 8 if case.get("dtype") == "float64" else 4
    if kind == "train":
        pixels = case["n"] * case["h"] * case["w"]
        return dict(bytes=pixels * 4 * (case["channels"] + 1) + 2 * 4 * 1.16e6,
                    flops=3 * 2 * 83520 * pixels)
    if kind == "batch":
        sizes = np.random.default_rng(3000)
        patches = []
        for _ in range(case["n"]):
            shots = int(sizes.integers(case["shots0"], case["shots1"] + 1))
            nt = int(sizes.integers(case["nt0"], case["nt1"] + 1))
            w = [(16, 128), (32, 256), (64, 256)][int(sizes.integers(0, 3))]
            patches.append(([shots, nt], w, 1))
    elif kind == "gather":
        patches = [([case["shots"], case["nt"]], [case["ws"], case["wt"]], 1)]
    elif kind == "vibroseis":
        patches = [([case["sy"], case["sx"], case["ch"], case["nt"]],
                    [case["ws"]] * 3 + [case["wt"]], SWEEP)]
    else:
        patches = [([case["ch"], case["shots"], case["nt"]],
                    [case.get("wc", 16), case.get("ws", 32), case.get("wt", 256)], 1)
                   for _ in range(case["vols"])]
    data = sum(math.prod(s) for s, _, _ in patches)
    if kind == "blend":
        return dict(bytes=2 * data * size, flops=2 * data)
    got = [_sizes(*p) for p in patches]
    values, flops = sum(g[0] for g in got), sum(g[1] for g in got)
    its = case["its"] - case.get("begin", 0)
    # an iteration reads the model for the operator, reads and writes it for the update
    total = dict(bytes=2 * data * size + its * 3 * values * 2 * size, flops=2 * its * flops)
    if kind == "learned":
        total["flops"] += 2 * 83520 * data
    return total


# ------------------------------------------------------------------ 64 bits


def _taper(n, left, right):
    half = n // 2
    w = np.ones(n)
    if left:
        w[:half] = 0.5 * (1 - np.cos(np.pi * np.arange(half) / half))
    if right:
        w[n - half:] = 0.5 * (1 - np.cos(np.pi * (half + np.arange(half)) / half))
    return w


class _Exact:
    """The method in float64 on plain tensors: windows of one shape are one batch."""

    def __init__(self, p):
        dev = _device()
        self.p, self.dev = p, dev
        wav = p.get("wavelets")
        wl = len(wav[0]) if wav else 1
        self.groups, starts, self.raw = {}, [], []
        conv = []
        for s, win in zip(p["shapes"], p["window_shapes"]):
            h = win[-1] // 2
            steps = -(-(s[-1] - wl + 1) // h) + 1
            conv.append((h, steps, (steps + 1) * h + wl - 1))
        t0 = min(int(st.min()) - c[0] for st, c in zip(p["shottimes"], conv))
        self.length = max(int(st.max()) - c[0] + c[2]
                          for st, c in zip(p["shottimes"], conv)) - t0
        nch = max(int(c.max()) for c in p["channels"]) + 1
        self.n_rec = nch * self.length
        self.mute = torch.zeros(self.n_rec, dtype=torch.bool, device=dev)
        for q, (s, win) in enumerate(zip(p["shapes"], p["window_shapes"])):
            h, steps, c = conv[q]
            tt = p["trace_types"][q]
            base = p["channels"][q].astype(np.int64) * self.length + p["shottimes"][q] - h - t0
            bad = torch.as_tensor(base[tt == BAD], device=dev)
            self.mute[(bad[:, None] + torch.arange(c, device=dev)).reshape(-1)] = True
            self.raw.append((torch.as_tensor(base + h, device=dev),
                             torch.as_tensor(tt != MISSING, device=dev)))
            axes = [_windows(n, w) for n, w in zip(s[:-1], win[:-1])]
            for combo in np.ndindex(*[len(a) for a in axes]):
                lens, idx, taper = [], np.zeros(1, np.int64), np.ones(1)
                for d, i in enumerate(combo):
                    a, n = axes[d][i]
                    lens.append(n)
                    t = _taper(n, i > 0, i + 1 < len(axes[d]))
                    idx = (idx[:, None] * s[d] + a + np.arange(n)).reshape(-1)
                    taper = (taper[:, None] * t).reshape(-1)
                if not (tt[idx] == LIVE).any():
                    continue
                full = lens + [win[-1]]
                padded = [_padded(n) for n in full]
                key = (tuple(full), steps, c)
                g = self.groups.setdefault(key, dict(pad=padded, steps=steps, conv=c, h=h,
                                                     lens=full, at=[], live=[], taper=[],
                                                     trace=[], q=[]))
                g["at"].append(base[idx])
                g["live"].append(tt[idx] != MISSING)
                g["taper"].append(taper)
                g["trace"].append(idx)
                g["q"].append(q)
        self.chunks = []
        for g in self.groups.values():
            n = math.prod(g["pad"][:-1]) * (g["pad"][-1] // 2 + 1) * g["steps"]
            per = max(1, (1 << 25) // n)
            for a in range(0, len(g["at"]), per):
                c = dict(g, q=g["q"][a: a + per])
                for k in ("at", "live", "taper", "trace"):
                    c[k] = torch.as_tensor(np.stack(g[k][a: a + per]), device=dev)
                c["scale"] = c["taper"] / math.sqrt(math.prod(g["pad"]))
                c["tt"] = torch.as_tensor(_taper(g["lens"][-1], True, True), device=dev)
                self.chunks.append(c)
        self.spec = None
        if wav:
            c = conv[0][2]
            w = torch.as_tensor(np.asarray(wav[0], np.float64), device=dev)
            ang = torch.angle(torch.fft.rfft(w, c))
            self.spec = torch.polar(torch.ones_like(ang), ang)
        fold = torch.zeros(self.n_rec, dtype=torch.float64, device=dev)
        for c in self.chunks:
            self._add(c, c["taper"][..., None].expand(-1, -1, c["conv"]), fold)
        self.step = 0.5 / max(1.0, float(fold.max()))

    def _index(self, c):
        return c["at"][..., None] + torch.arange(c["conv"], device=self.dev)

    def _add(self, c, y, rec):
        y = y * c["live"][..., None]
        rec.index_add_(0, self._index(c).reshape(-1), y.reshape(-1))

    def _wave(self, y, sign):
        if self.spec is None:
            return y
        s = self.spec if sign > 0 else self.spec.conj()
        return torch.fft.irfft(torch.fft.rfft(y) * s, y.shape[-1])

    def traces(self, c, x, wave=True):
        """The window traces [W][traces][conv] of the model x [W][T][P..][F]."""
        D = len(c["lens"]) - 1
        for d in range(D):
            x = torch.fft.ifft(x, dim=2 + d, norm="forward").narrow(2 + d, 0, c["lens"][d])
        x = x.reshape(x.shape[0], c["steps"], -1, x.shape[-1]).clone()
        x[..., 0].imag.zero_()
        if c["pad"][-1] % 2 == 0:
            x[..., -1].imag.zero_()
        u = torch.fft.irfft(x, c["pad"][-1], norm="forward")[..., : c["lens"][-1]]
        u = u * c["tt"] * c["scale"][:, None, :, None]
        y = torch.zeros(u.shape[0], u.shape[2], c["conv"], dtype=torch.float64, device=self.dev)
        for t in range(c["steps"]):
            y[..., t * c["h"]: t * c["h"] + c["lens"][-1]] += u[:, t]
        return self._wave(y, 1) if wave else y

    def model(self, c, y, double=True, wave=True):
        """The adjoint of traces()."""
        y = self._wave(y, -1) if wave else y
        n, D = c["lens"][-1], len(c["lens"]) - 1
        u = torch.stack([y[..., t * c["h"]: t * c["h"] + n] for t in range(c["steps"])], 1)
        u = u * c["tt"] * c["scale"][:, None, :, None]
        x = torch.fft.rfft(u, c["pad"][-1])
        if double:
            x[..., 1: 1 + (c["pad"][-1] - 1) // 2] *= 2
        x = x.reshape(x.shape[0], c["steps"], *c["lens"][:-1], x.shape[-1])
        for d in range(D):
            x = torch.fft.fft(x, c["pad"][d], dim=2 + d)
        return x

    def forward(self, model):
        rec = torch.zeros(self.n_rec, dtype=torch.float64, device=self.dev)
        for c, x in zip(self.chunks, model):
            self._add(c, self.traces(c, x), rec)
        rec[self.mute] = 0
        return rec

    def gathered(self, c, rec):
        return rec[self._index(c)] * c["live"][..., None]

    def input(self):
        rec = torch.zeros(self.n_rec, dtype=torch.float64, device=self.dev)
        count = torch.zeros_like(rec)
        for (base, live), x in zip(self.raw, self.p["data"]):
            x = x.double()
            at = (base[live, None] + torch.arange(x.shape[1], device=self.dev)).reshape(-1)
            rec.index_add_(0, at, x[live].reshape(-1))
            count.index_add_(0, at, torch.ones_like(at, dtype=torch.float64))
        rec = rec / count.clamp(min=1)
        rec[self.mute] = 0
        return rec

    def output(self, model, wave=True):
        out = [torch.zeros(x.shape, dtype=torch.float64, device=self.dev)
               for x in self.p["data"]]
        for c, x in zip(self.chunks, model):
            y = self.traces(c, x, wave)
            for i, q in enumerate(c["q"]):
                out[q].index_add_(0, c["trace"][i],
                                  y[i, :, c["h"]: c["h"] + out[q].shape[1]])
        return out

    def start(self, its):
        """The record, the first model and the thresholds of all iterations."""
        d = self.input()
        model = [-self.step * self.model(c, self.gathered(c, d)) for c in self.chunks]
        top = max(float(x.abs().max()) for x in model)
        decay = math.exp(math.log(TARGET) / its)
        ld = math.log(decay)
        first = int((ld * (its - 1.0) + 1.0) / ld)
        lamb, lambs = top, [top]
        for it in range(1, its):
            lamb = lamb * decay if it < first else (
                (its - 1 - it) * top * decay ** first / (its - 1 - first))
            lambs.append(lamb)
        return d, model, lambs

    @staticmethod
    def shrink(x, lamb):
        a = x.abs()
        return x * ((a - lamb).clamp(min=0) / a.clamp(min=1e-300))

    def iterate(self, d, model, lambs):
        for lamb in lambs:
            r = self.forward(model) - d
            r[self.mute] = 0
            for i, c in enumerate(self.chunks):
                g = self.model(c, self.gathered(c, r))
                model[i] = self.shrink(model[i].sub_(g, alpha=self.step), lamb)
                del g
        return model

    def solve(self, its):
        d, model, lambs = self.start(its)
        model = [self.shrink(x, lambs[0]) for x in model]
        return self.output(self.iterate(d, model, lambs[1:]))

    def warm(self, values, wave=True):
        """The model whose windows, weighted by their own tapers, sum to `values`."""
        model = []
        for c in self.chunks:
            y = torch.zeros(c["at"].shape + (c["conv"],), dtype=torch.float64, device=self.dev)
            for i, q in enumerate(c["q"]):
                v = values[q]
                y[i, :, c["h"]: c["h"] + v.shape[1]] = v[c["trace"][i]]
            model.append(self.model(c, y, double=False, wave=wave))
        return model

    def solve_warm(self, its, begin, estimate):
        d, _, lambs = self.start(its)
        fold = self.output(self.warm([torch.ones_like(e) for e in estimate], False), False)
        model = self.warm([e / f.clamp(min=FLOOR) for e, f in zip(estimate, fold)])
        return self.output(self.iterate(d, model, lambs[begin:]))


def _net(params, base, channels):
    """The network on [n][channels][h][w] in float64, with its weights as leaves."""
    c = base
    plan = [(channels, c), (c, c), (c, 2 * c), (2 * c, 2 * c), (2 * c, 4 * c), (4 * c, 4 * c),
            (4 * c, 8 * c), (8 * c, 4 * c), (4 * c, 4 * c), (4 * c, 2 * c), (2 * c, 2 * c),
            (2 * c, c), (c, c), (c, 1)]
    layers, off = [], 0
    for ci, co in plan:
        w = params[off: off + 9 * ci * co].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        layers.append((w, params[off + 9 * ci * co: off + 9 * ci * co + co]))
        off += 9 * ci * co + co
    F = torch.nn.functional

    def conv(x, i):
        w, b = layers[i]
        cols = F.unfold(x, 3, padding=1)
        y = (w.reshape(w.shape[0], -1) @ cols + b[:, None]).reshape(
            x.shape[0], -1, *x.shape[2:])
        return torch.relu(y) if i + 1 < len(layers) else y

    def up(x, skip):
        return F.interpolate(x, scale_factor=2, mode="nearest") + skip

    def net(x):
        s1 = conv(conv(x, 0), 1)
        s2 = conv(conv(F.avg_pool2d(s1, 2), 2), 3)
        s3 = conv(conv(F.avg_pool2d(s2, 2), 4), 5)
        b = conv(conv(F.avg_pool2d(s3, 2), 6), 7)
        d3 = conv(conv(up(b, s3), 8), 9)
        d2 = conv(conv(up(d3, s2), 10), 11)
        return x[:, :1] + conv(conv(up(d2, s1), 12), 13)

    return net


def _params(base, channels):
    net = WarmStartNet(base, seed=1, in_channels=channels)  # the weights that prepare() gives
    p = torch.as_tensor(net.params(), device=_device()).double()
    net.close()
    return p


def _host(outs, shapes):
    return [x.reshape(tuple(s)).cpu().numpy() for x, s in zip(outs, shapes)]


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [_host(_Exact(p).solve(case["its"]), p["shapes"]) for p in _batch(case, seed)]
    if kind == "train":
        x, y = (torch.as_tensor(v, device=_device()).double() for v in _train_arrays(case, seed))
        x = x[:, None] if x.ndim == 3 else x.permute(0, 3, 1, 2)
        params = _params(case["base"], case["channels"]).requires_grad_(True)
        with torch.enable_grad():
            loss = (_net(params, case["base"], case["channels"])(x)[:, 0] - y).square().mean()
            loss.backward()
        return float(loss), params.grad.cpu().numpy()
    p = _problem(case, seed)
    if kind == "blend":
        p["window_shapes"] = [[s[0], s[1], 2] for s in p["shapes"]]
        return _host(_blend(p, case["mode"]), p["shapes"])
    if kind == "learned":
        net = _net(_params(32, 1), 32, 1)
        est = []
        for x, s in zip(p["data"], p["shapes"]):
            img = x.double().reshape(s)
            rms = img.square().mean((1, 2), keepdim=True).sqrt()
            rms[rms == 0] = 1
            pad = [0, -s[2] % 8, 0, -s[1] % 8]
            img = torch.nn.functional.pad(img / rms, pad)
            e = torch.cat([net(i[None, None])[:, 0] for i in img])
            est.append((e[:, : s[1], : s[2]] * rms).reshape(-1, s[2]))
        return _host(_Exact(p).solve_warm(case["its"], case["begin"], est), p["shapes"])
    return _host(_Exact(p).solve(case["its"]), p["shapes"])


def _blend(p, mode):
    """Sum (0) or mean (1) of the traces in the record, muted, read back."""
    dev = _device()
    t0 = min(int(s.min()) for s in p["shottimes"])
    nt = [s[-1] for s in p["shapes"]]
    length = max(int(s.max()) for s in p["shottimes"]) - t0 + max(nt)
    n = (max(int(c.max()) for c in p["channels"]) + 1) * length
    rec, count = (torch.zeros(n, dtype=torch.float64, device=dev) for _ in range(2))
    mute = torch.zeros(n, dtype=torch.bool, device=dev)
    at = []
    for s, c, tt, x in zip(p["shottimes"], p["channels"], p["trace_types"], p["data"]):
        base = torch.as_tensor(c.astype(np.int64) * length + s - t0, device=dev)
        i = base[:, None] + torch.arange(x.shape[1], device=dev)
        live = torch.as_tensor(tt != MISSING, device=dev)
        rec.index_add_(0, i[live].reshape(-1), x[live].reshape(-1).double())
        count.index_add_(0, i[live].reshape(-1), torch.ones_like(x[live]).reshape(-1).double())
        mute[i[torch.as_tensor(tt == BAD, device=dev)].reshape(-1)] = True
        at.append((i, live))
    if mode == 1:
        rec = rec / count.clamp(min=1)
    rec[mute] = 0
    return [rec[i] * live[:, None] for i, live in at]
