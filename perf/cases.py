"""
The workloads that the framework's speed is judged by, through its public
entry points: the learned surrogate (serving, whole calls, training) and the
resolution step of a fit.  They need only the libraries that build from this
repository alone (``sasmodels_b200.build.build_support``); the per-model
engines are generated from sasmodels' plugin sources, which a checkout of
this repository does not hold, so they are not among these cases.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same
ranges, ``prepare(case, seed)`` makes what a program holds before the call,
``run(state)`` is one pass, ``work(case)`` the bytes and operations a pass
cannot do without, ``exact(case, seed)`` the same results in 64 bits.
"""

import math
import os
import types

import numpy as np
import torch

from sasmodels_b200 import build as _build

# a checkout that was not built yet builds the libraries that it can
if not all(os.path.exists(os.path.join(_build.LIB, "libsasb200_%s.so" % s))
           for s in ("mlp", "resolution")):
    _build.build_support()

from sasmodels_b200.resolution import Pinhole1D, Pinhole2D, Slit1D, nllf_sets  # noqa: E402
from sasmodels_b200.surrogate import DOMAIN, MLP, Surrogate, pad128  # noqa: E402

HID, NIN = 256, 16
#: oversampling bins (radial x angular) of a 2D resolution cell per accuracy
BINS = {"low": (3, 4), "med": (5, 6), "high": (5, 12), "xhigh": (10, 20)}
#: multiply-adds of the network per row, counted once
ROW_FLOPS = 2*(NIN*HID + 3*HID*HID + HID)
WEIGHT_BYTES = 2*(NIN*HID + 3*HID*HID) + 4*5*HID
HUBER, LR, TOTAL, WARMUP, STEP0 = 0.02, 2e-3, 100000, 200, 1000


def listed():
    return [
        # one measured 1D curve smeared by its pinhole resolution, as each
        # step of a single fit does: the smallest call, all latency
        dict(name="pinhole_curve", kind="pinhole", nq=200, width=0.08),
        # one USANS-like curve smeared by a slit with length and width
        dict(name="slit_curve", kind="slit", nq=251, length=0.05, width=0.004),
        # one 2D detector image at the accuracy used for a final fit
        dict(name="image_256_high", kind="image", side=256, accuracy="high"),
        # the resolution and chi-squared of a small fit population on a short
        # data set (odd sizes)
        dict(name="fit_61x181", kind="fit", sets=61, nq=181, width=0.06),
        # the same for a whole population (the size of the fit benchmark) on a
        # finely binned curve
        dict(name="fit_4096x1000", kind="fit", sets=4096, nq=1000, width=0.05),
        # the surrogate network on one curve's points (interactive use)
        dict(name="serve_curve", kind="serve", rows=1000),
        # a batch of curves that fills neither the last tile nor the last wave
        dict(name="serve_ragged", kind="serve", rows=50021),
        # bulk serving, the size of the network's own benchmark
        dict(name="serve_bulk", kind="serve", rows=4000000),
        # parameter columns already on the GPU: features, then the network
        dict(name="points_500k", kind="points", rows=500009),
        # the user's whole call: host arrays in, I(q) and the fallback mask out
        # (network, error gate, domain check)
        dict(name="iq_100_curves", kind="iq", curves=100, nq=1000),
        # one captured training step at the training batch
        dict(name="train_8192", kind="train", batch=8192),
        # a data-parallel rank's gradients of a ragged slice
        dict(name="grad_3001", kind="grad", rows=3001),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pinhole", "slit", "image", "fit", "serve", "serve", "points", "iq",
                       "train", "grad"])
    if kind == "pinhole":
        return dict(kind=kind, nq=_log_int(rng, 30, 2000), width=round(rng.uniform(0.01, 0.15), 4))
    if kind == "slit":
        return dict(kind=kind, nq=_log_int(rng, 30, 1000), length=round(rng.uniform(0.01, 0.1), 4),
                    width=rng.choice([0.0, round(rng.uniform(0.001, 0.01), 5)]))
    if kind == "image":
        return dict(kind=kind, side=_log_int(rng, 32, 256), accuracy=rng.choice(sorted(BINS)))
    if kind == "fit":
        return dict(kind=kind, sets=_log_int(rng, 8, 4096), nq=_log_int(rng, 50, 1000),
                    width=round(rng.uniform(0.02, 0.05), 4))
    if kind == "serve":
        return dict(kind=kind, rows=_log_int(rng, 1, 4000000))
    if kind == "points":
        return dict(kind=kind, rows=_log_int(rng, 1000, 1000000))
    if kind == "iq":
        return dict(kind=kind, curves=_log_int(rng, 1, 100), nq=_log_int(rng, 50, 1000))
    if kind == "train":
        return dict(kind=kind, batch=128*_log_int(rng, 1, 128))
    return dict(kind="grad", rows=_log_int(rng, 1, 16384))


# ------------------------------------------------------------------ inputs --

def _dev():
    return torch.device("cuda", torch.cuda.current_device())


_STREAMS = {}


def _stream():
    """The one stream that this program runs its networks on."""
    return _STREAMS.setdefault(_dev(), torch.cuda.Stream(_dev()))


def _rng(case, seed):
    return np.random.default_rng([int(seed) & 0x7fffffff, len(case["kind"])])


def _gen(seed, k=0):
    g = torch.Generator(device=_dev())
    g.manual_seed(int(seed)*7 + k)
    return g


def _edges(x):
    return np.hstack([x[0] - 0.5*(x[1] - x[0]), 0.5*(x[1:] + x[:-1]),
                      x[-1] + 0.5*(x[-1] - x[-2])])


def _curve(q, radius, scale, background):
    """Sphere-like scattering curves (rows: radius, scale)."""
    x = q[None, :].abs()*radius[:, None]
    f = 3.0*(torch.sin(x) - x*torch.cos(x))/x**3
    return scale[:, None]*f*f + background


def _pinhole_grid(case):
    """Measured q, 1-sigma widths and the calculation grid that covers every
    q's window, with steps like the end intervals."""
    q = np.logspace(-3, math.log10(0.5), case["nq"])
    dq = case["width"]*q
    lo = np.arange(q[0] - (q[1] - q[0]), max(np.min(q - 2.5*dq), 0.05*q[0]), -(q[1] - q[0]))[::-1]
    step = q[-1] - q[-2]
    hi = q[-1] + step*np.arange(1, int(math.ceil(3.0*dq[-1]/step)) + 1)
    return q, dq, np.concatenate([lo, q, hi])


def _slit_grid(case):
    q = np.logspace(-3, -1, case["nq"])
    qmax = math.sqrt((q[-1] + case["width"])**2 + case["length"]**2)
    ratio = q[1]/q[0]
    n = int(math.ceil(math.log(qmax/q[-1])/math.log(ratio)))
    lo = q[0]*ratio**-np.arange(1.0, 1 + int(math.log(40.0)/math.log(ratio)))[::-1]
    return q, np.concatenate([lo, q, q[-1]*ratio**np.arange(1.0, n + 1)])


def _theories(case, seed, qc, sets):
    g = _gen(seed)
    dev = _dev()
    u = torch.rand((3, sets), dtype=torch.float64, device=dev, generator=g)
    q = torch.as_tensor(qc, device=dev)
    return _curve(q, 20.0 + 180.0*u[0], 0.5 + 100.0*u[1], 0.001 + 0.01*u[2][:, None])


def _image(case, seed):
    n = case["side"]
    x = np.linspace(-0.3, 0.3, n) + 1e-4
    qx, qy = [a.ravel() for a in np.meshgrid(x, x)]
    data = types.SimpleNamespace(qx_data=qx, qy_data=qy, q_data=np.sqrt(qx**2 + qy**2),
                                 dqx_data=0.02*np.abs(qx) + 2e-4, dqy_data=0.02*np.abs(qy) + 2e-4)
    nr, nphi = BINS[case["accuracy"]]
    g = _gen(seed)
    base = _curve(torch.as_tensor(data.q_data, device=_dev()),
                  40 + 60*torch.rand(1, dtype=torch.float64, device=_dev(), generator=g),
                  torch.full((1,), 100.0, dtype=torch.float64, device=_dev()), 0.01)
    noise = torch.rand((nr*nphi, n*n), dtype=torch.float64, device=_dev(), generator=g)
    return data, (base*(0.9 + 0.2*noise)).reshape(-1)


def _network(rng, halves):
    """A network's weights: spread as a trained one's, W as the bf16 values
    that serving packs (halves) or as fp32 master weights."""
    W = []
    for l in range(4):
        cols = NIN if l == 0 else HID
        w = rng.normal(0, 1.3/math.sqrt(15 if l == 0 else HID), (HID, cols)).astype(np.float32)
        if l == 0:
            w[:, 15] = 0
        if halves:
            w = torch.as_tensor(w).to(torch.bfloat16).float().numpy()
        W.append(w)
    return dict(W=W, b=[rng.normal(0, 0.1, HID).astype(np.float32) for _ in range(4)],
                w_out=rng.normal(0, 1/math.sqrt(HID), HID).astype(np.float32),
                b_out=np.array([0.1], np.float32))


def _rows(seed, rows, k):
    """Features as the compensated bf16 pair, zero beyond `rows`."""
    n_pad = pad128(rows)
    f = torch.rand((n_pad, NIN), device=_dev(), generator=_gen(seed, k))*2 - 1
    f[rows:] = 0
    f[:, 15] = 0
    hi = f.to(torch.bfloat16)
    return hi, (f - hi.float()).to(torch.bfloat16)


def _columns(seed, rows):
    """One float64 column per network input over its training domain."""
    u = torch.rand((7, rows), dtype=torch.float64, device=_dev(), generator=_gen(seed, 3))

    def span(k, key, logs=False):
        lo, hi = DOMAIN[key]
        if logs:
            return torch.exp(math.log(lo) + u[k]*(math.log(hi) - math.log(lo)))
        return lo + u[k]*(hi - lo)
    return dict(radius=span(0, "radius", True), length=span(1, "length", True),
                rpd=span(2, "rpd"), lpd=span(3, "lpd"), contrast=span(4, "contrast"),
                q=span(5, "q", True), flag=torch.round(u[6]))


def _host_columns(case, rng):
    """Flat host arrays of `curves` parameter sets over `nq` sorted q each."""
    nc, nq = case["curves"], case["nq"]

    def logs(key, size):
        lo, hi = DOMAIN[key]
        return np.clip(np.exp(rng.uniform(math.log(lo), math.log(hi), size)), lo, hi)
    sets = dict(radius=logs("radius", nc), length=logs("length", nc),
                rpd=rng.uniform(*DOMAIN["rpd"], nc), lpd=rng.uniform(*DOMAIN["lpd"], nc),
                contrast=rng.uniform(0.2, 5.0, nc)*rng.choice([-1.0, 1.0], nc),
                flag=rng.integers(0, 2, nc))
    cols = {k: np.repeat(v, nq) for k, v in sets.items()}
    cols["q"] = np.sort(logs("q", (nc, nq)), axis=1).ravel()
    cols["set"] = np.repeat(np.arange(nc), nq)
    return cols


def _targets(seed, n):
    return torch.randn(n, device=_dev(), generator=_gen(seed, 5))


def _moments(seed, state):
    """Adam moments of a run that has been going for a while."""
    g = _gen(seed, 6)
    shapes = [w.shape for w in state["W"]] + [b.shape for b in state["b"]] + [(HID,), (1,)]
    m = [3e-3*torch.randn(s, device=_dev(), generator=g) for s in shapes]
    v = [1e-4*(0.5 + 1.5*torch.rand(s, device=_dev(), generator=g)) for s in shapes]
    return m, v


def _indices(case, seed):
    return torch.randperm(4*case["batch"], device=_dev(), generator=_gen(seed, 7))[:case["batch"]]


# ----------------------------------------------------------------- the path --

def prepare(case, seed):
    kind, rng = case["kind"], _rng(case, seed)
    s = dict(kind=kind)
    if kind == "pinhole":
        q, dq, qc = _pinhole_grid(case)
        s.update(res=Pinhole1D(q, dq, q_calc=qc), theory=_theories(case, seed, qc, 1)[0])
        s["res"].apply(s["theory"])
    elif kind == "slit":
        q, qc = _slit_grid(case)
        s.update(res=Slit1D(q, q_length=case["length"], q_width=case["width"], q_calc=qc),
                 theory=_theories(case, seed, qc, 1)[0])
        s["res"].apply(s["theory"])
    elif kind == "image":
        data, theory = _image(case, seed)
        s.update(res=Pinhole2D(data, accuracy=case["accuracy"]), theory=theory)
        s["res"].apply(theory)
    elif kind == "fit":
        q, dq, qc = _pinhole_grid(case)
        noise = rng.normal(size=case["nq"])
        base = _curve(torch.as_tensor(q), torch.tensor([60.0], dtype=torch.float64),
                      torch.tensor([50.0], dtype=torch.float64), 0.01)[0].numpy()
        s.update(res=Pinhole1D(q, dq, q_calc=qc), theory=_theories(case, seed, qc, case["sets"]),
                 y=base*(1 + 0.05*noise), dy=0.05*base)
        s["res"].apply_sets(s["theory"][:1], torch.cuda.current_stream())
    elif kind in ("serve", "points"):
        s.update(net=MLP(device=_dev(), seed=0, stream=_stream()), n=case["rows"])
        s["net"].load_state(_network(rng, True))
        if kind == "serve":
            s["x"], s["x_lo"] = _rows(seed, case["rows"], 1)
        else:
            s["cols"] = _columns(seed, case["rows"])
    elif kind == "iq":
        S = Surrogate(device=_dev(), seed=0)
        S.net.load_state(_network(rng, True))
        S.gate = MLP(device=_dev(), seed=1, stream=S.net.stream)
        S.gate.load_state(_network(rng, True))
        S.y_mean, S.y_std, S.g_mean, S.g_std = -2.0, 1.5, -7.0, 1.0
        # a gate that trusts every point of the domain (no fallback)
        S.cal_tols, S.cal_thresh = np.array([1e-3, 1.0]), np.array([1e30, 1e30])
        s.update(S=S, cols=_host_columns(case, rng))
    else:
        net, state = MLP(device=_dev(), seed=0, stream=_stream()), _network(rng, False)
        n = case["batch"] if kind == "train" else case["rows"]
        net.huber = HUBER
        if kind == "train":
            x, x_lo = _rows(seed, 4*n, 2)
            y = _targets(seed, 4*n)
            torch.cuda.synchronize()
            net.train_step(x[:n], x_lo[:n], y[:n], n, 1e-3)   # loads every kernel
            net.stream.synchronize()
        net.load_state(state)
        if kind == "train":
            m, v = _moments(seed, state)
            for a, b in zip(net.m + net.v, m + v):
                a.copy_(b)
            net.step_count = STEP0
            torch.cuda.synchronize()
            s["graph"] = net.capture_training(x, x_lo, y, n, LR, TOTAL, STEP0, warmup=WARMUP)
            s.update(idx=_indices(case, seed), data=(x, x_lo, y))
        else:
            s["x"], s["x_lo"] = _rows(seed, n, 2)
            s["y"] = _targets(seed, pad128(n))
        s.update(net=net, n=n)
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind in ("pinhole", "slit", "image"):
        return s["res"].apply(s["theory"])
    if kind == "fit":
        stream = torch.cuda.current_stream()
        smeared = s["res"].apply_sets(s["theory"], stream)
        return smeared, nllf_sets(smeared, s["y"], s["dy"], stream)
    if kind == "iq":
        return s["S"].iq(s["cols"], tol=0.01)
    net = s["net"]
    if kind == "serve":
        out = net.serve(s["x"], s["x_lo"], s["n"])[:s["n"]]
    elif kind == "points":
        c = s["cols"]
        x, x_lo, n = net.features(c["radius"], c["length"], c["rpd"], c["lpd"], c["contrast"],
                                  c["q"], c["flag"])
        out = net.serve(x, x_lo, n)[:n]
        for t in (x, x_lo):
            t.record_stream(net.stream)
    elif kind == "train":
        out = [s["graph"].step(s["idx"])] + net.params + net.m + net.v
    else:
        out = net.reduced_gradients(s["x"], s["x_lo"], s["y"], s["n"])
    # the program goes on with the results on its own stream
    torch.cuda.current_stream().wait_stream(net.stream)
    return out


def work(case):
    kind = case["kind"]
    if kind in ("pinhole", "fit"):
        q, dq, qc = _pinhole_grid(case)
        lo, hi = np.searchsorted(qc, q - 2.5*dq), np.searchsorted(qc, q + 3*dq, side="right")
        band, sets = int(np.sum(hi - lo)), case.get("sets", 1)
        # each weight (about 40 operations) once, a multiply-add per set
        return dict(bytes=8.0*(sets*(len(qc) + len(q)) + 5*len(q) + len(qc)),
                    flops=42.0*band + 2.0*band*sets + 5.0*sets*len(q))
    if kind == "slit":
        q, qc = _slit_grid(case)
        k = 1 if case["width"] == 0 else 61
        lim = np.sqrt(q**2 + case["length"]**2)
        band = int(np.sum(np.searchsorted(qc, lim) - np.searchsorted(qc, q) + 2))*k
        return dict(bytes=8.0*(2*len(qc) + 4*len(q)), flops=20.0*band)
    if kind == "image":
        n, (nr, nphi) = case["side"]**2, BINS[case["accuracy"]]
        return dict(bytes=8.0*(n*nr*nphi + n + nr*nphi), flops=2.0*n*nr*nphi)
    if kind == "iq":
        n = case["curves"]*case["nq"]
        # q, the run index, I(q) and the mask cross to and from the GPU
        return dict(bytes=(8.0 + 4 + 8 + 1)*n + 2*WEIGHT_BYTES, flops=2.0*ROW_FLOPS*n)
    n = case.get("rows") or case.get("batch")
    if kind == "serve":
        return dict(bytes=68.0*n + WEIGHT_BYTES, flops=float(ROW_FLOPS*n))
    if kind == "points":
        return dict(bytes=60.0*n + WEIGHT_BYTES, flops=float(ROW_FLOPS*n))
    state = 4*(NIN*HID + 3*HID*HID + 5*HID + 1)
    moved = 7*state if kind == "train" else state + WEIGHT_BYTES
    return dict(bytes=68.0*n + moved, flops=3.0*ROW_FLOPS*n)


# ------------------------------------------------------------- in 64 bits --

def _pinhole_weights(q, dq, qc):
    dev = _dev()
    t = [torch.as_tensor(a, device=dev) for a in (q, dq, qc, _edges(qc))]
    cdf = torch.erf((t[3][None, :] - t[0][:, None])/(math.sqrt(2.0)*t[1])[:, None])
    w = cdf[:, 1:] - cdf[:, :-1]
    w[(t[2][None, :] < (t[0] - 2.5*t[1])[:, None]) | (t[2][None, :] > (t[0] + 3*t[1])[:, None])] = 0
    return w/w.sum(1, keepdim=True)


def _slit_exact(case, theory):
    q, qc = _slit_grid(case)
    e = _edges(qc)
    out = np.empty(len(q))
    kmax = 0 if case["width"] == 0 else 30
    for i, qi in enumerate(q):
        qk = qi + np.arange(-kmax, kmax + 1)*(case["width"]/30)
        lim = np.sqrt(qk**2 + case["length"]**2)
        c = np.clip(e[None, :], np.abs(qk)[:, None], lim[:, None])
        u = np.sqrt(np.maximum((c - np.abs(qk)[:, None])*(c + np.abs(qk)[:, None]), 0))
        out[i] = np.mean(((u[:, 1:] - u[:, :-1])/case["length"]) @ theory)
    return torch.as_tensor(out)


def _features(c):
    L = torch.log
    lr, ll, lq = L(c["radius"]), L(c["length"]), L(c["q"])

    def unit(v, lo, hi):
        return 2*(v - math.log(lo))/(math.log(hi) - math.log(lo)) - 1
    qr, qh = c["q"]*c["radius"], 0.5*c["q"]*c["length"]
    ar, al = torch.exp(-2*(c["rpd"]*qr)**2), torch.exp(-2*(c["lpd"]*qh)**2)
    f = [unit(lr, *DOMAIN["radius"]), unit(ll, *DOMAIN["length"]), 2*c["rpd"]/0.3 - 1,
         2*c["lpd"]/0.3 - 1, c["contrast"]/5, unit(lq, *DOMAIN["q"]), 2*c["flag"] - 1,
         L(qr)/4, L(qh)/4, torch.log1p(c["rpd"]*qr)/2, torch.log1p(c["lpd"]*qh)/2,
         ar*torch.cos(2*qr), ar*torch.sin(2*qr), al*torch.cos(2*qh), al*torch.sin(2*qh),
         torch.zeros_like(qr)]
    return torch.stack(f, dim=1)


def _forward64(x, p):
    h = x
    for l in range(4):
        h = torch.nn.functional.silu(h @ p[l].T + p[4 + l])
    return h @ p[8] + p[9]


def _params64(state):
    return [torch.as_tensor(a, device=_dev()).double()
            for a in state["W"] + state["b"] + [state["w_out"], state["b_out"]]]


def _served64(x_of, rows, state):
    p, step = _params64(state), 250000
    return torch.cat([_forward64(x_of(a, min(rows, a + step)), p) for a in range(0, rows, step)])


def _gradients64(x, y, n, state):
    p = [t.requires_grad_() for t in _params64(state)]
    d = (_forward64(x[:n], p) - y[:n].double()).abs()
    loss = torch.where(d <= HUBER, d*d, HUBER*(2*d - HUBER)).mean()
    return loss.detach(), [g.detach() for g in torch.autograd.grad(loss, p)], [t.detach() for t in p]


def exact(case, seed):
    kind, rng = case["kind"], _rng(case, seed)
    if kind == "pinhole":
        q, dq, qc = _pinhole_grid(case)
        return _pinhole_weights(q, dq, qc) @ _theories(case, seed, qc, 1)[0]
    if kind == "slit":
        return _slit_exact(case, _theories(case, seed, _slit_grid(case)[1], 1)[0].cpu().numpy())
    if kind == "image":
        _, theory = _image(case, seed)
        nr, nphi = BINS[case["accuracy"]]
        step = 3.0/nr
        r = step/2 + np.arange(nr)*step
        ring = np.exp(-0.5*(r - step/2)**2) - np.exp(-0.5*(r + step/2)**2)
        w = torch.as_tensor(np.tile(ring, nphi), device=_dev())
        return (w @ theory.view(nr*nphi, -1))/w.sum()
    if kind == "fit":
        q, dq, qc = _pinhole_grid(case)
        noise = rng.normal(size=case["nq"])
        base = _curve(torch.as_tensor(q), torch.tensor([60.0], dtype=torch.float64),
                      torch.tensor([50.0], dtype=torch.float64), 0.01)[0]
        y, dy = [v.to(_dev()) for v in (base*(1 + 0.05*torch.as_tensor(noise)), 0.05*base)]
        smeared = _theories(case, seed, qc, case["sets"]) @ _pinhole_weights(q, dq, qc).T
        return smeared, 0.5*(((smeared - y)/dy)**2).sum(1)
    if kind == "serve":
        x, x_lo = _rows(seed, case["rows"], 1)
        return _served64(lambda a, b: x[a:b].double() + x_lo[a:b].double(), case["rows"],
                         _network(rng, True))
    if kind == "points":
        c = _columns(seed, case["rows"])
        return _served64(lambda a, b: _features({k: v[a:b] for k, v in c.items()}), case["rows"],
                         _network(rng, True))
    if kind == "iq":
        state = _network(rng, True)
        _network(rng, True)                   # the gate's
        c = {k: torch.as_tensor(v, device=_dev()).double()
             for k, v in _host_columns(case, rng).items()}
        out = _served64(lambda a, b: _features({k: v[a:b] for k, v in c.items()}), len(c["q"]),
                        state)
        return torch.exp(1.5*out - 2.0)*c["contrast"]**2, None
    state = _network(rng, False)
    if kind == "grad":
        n = case["rows"]
        x, x_lo = _rows(seed, n, 2)
        loss, g, _ = _gradients64(x.double() + x_lo.double(), _targets(seed, pad128(n)), n, state)
        return [loss.reshape(1)] + g
    n, idx = case["batch"], _indices(case, seed)
    x, x_lo = _rows(seed, 4*n, 2)
    loss, g, p = _gradients64((x.double() + x_lo.double())[idx], _targets(seed, 4*n)[idx], n, state)
    m, v = _moments(seed, state)
    m = [0.9*a.double() + 0.1*b for a, b in zip(m, g)]
    v = [0.999*a.double() + 0.001*b*b for a, b in zip(v, g)]
    rate = LR*min(1.0, (STEP0 + 1)/WARMUP)*0.5*(1 + math.cos(math.pi*STEP0/TOTAL))
    c1, c2 = 1 - 0.9**(STEP0 + 1), 1 - 0.999**(STEP0 + 1)
    p = [a - rate*(b/c1)/(torch.sqrt(c/c2) + 1e-8) for a, b, c in zip(p, m, v)]
    return [loss] + p + m + v
