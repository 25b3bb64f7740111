"""Performance cases: what a user of this package runs, through its public
entry points, from the smallest calls to the largest.

A case is a dict of plain values; ``prepare`` makes what a user's program has
in hand before the call (contexts, networks, host arrays of events, images or
features -- the events of the optical transport are host data by nature),
``run`` is one whole call with its results read back.  Sizes follow the
package's benchmark configurations and tests.

Kinds:
  transport  EDE buffer (cm, eV, history) -> counters, PRF, PHS, per-history counts;
             the reference's column model, or an explicit lattice (grid 1, 2)
  batch      64 detector geometries in one launch (configuration 2)
  labels     the surrogate's Monte Carlo training labels (label_points)
  chain      x-ray front end -> EDEs on the device -> optical transport
  mtf, nnps  image-quality metrics of the transport's images
  train      surrogate training steps; predict: the network's forward pass;
  loop       the surrogate in the event pipeline with a 1 % Monte Carlo audit
"""
import os

import numpy as np
import torch

import hybridmantis_b200 as hb
from hybridmantis_b200 import analysis
from hybridmantis_b200 import surrogate as sgm
from hybridmantis_b200 import xray as xr

MODEL = os.path.join(sgm.__file__.rsplit(os.sep, 1)[0], "data", "surrogate_c4.fd2sg")

# Mean photons per x-ray of a stream and FP32 operations a photon's walk
# cannot do without (the reference's operations per photon, counted on
# configuration 1; a lattice photon meets about as many surfaces).
PHOTONS = {0: 1350.0, 1: 2340.0, 2: 2560.0, 4: 2340.0}
CHAIN_PHOTONS = 833.0
WALK_FLOPS = 9600.0


def listed():
    return [
        # the smallest call: a first look at a detector, or one buffer of a
        # coupled x-ray simulation -- latency and launches
        {"name": "first_look", "kind": "transport", "config": 0, "xrays": 25, "grid": 0, "refl": 0.0},
        # an ordinary run of odd size with a reflecting sensor (the option of
        # the reference's example)
        {"name": "ordinary", "kind": "transport", "config": 1, "xrays": 2311, "grid": 0, "refl": 0.25},
        # the headline workload: configuration 1, 100,000 x-rays
        {"name": "headline", "kind": "transport", "config": 1, "xrays": 100000, "grid": 0, "refl": 0.0},
        # explicit column lattice (square)
        {"name": "lattice", "kind": "transport", "config": 1, "xrays": 10001, "grid": 1, "refl": 0.0},
        # a scan over 64 detector geometries at the workload's stated size
        {"name": "geometry_scan", "kind": "batch", "xrays": 2000},
        # training labels: depositions in sampled geometries, 10,000 photons each
        {"name": "label_points", "kind": "labels", "geoms": 64, "points": 100, "photons": 10000},
        # the reference's example run: a 25 keV line, EDEs made on the GPU
        {"name": "xray_chain", "kind": "chain", "xrays": 20000},
        # MTF of a 501 x 501 point response image, every frequency
        {"name": "mtf_prf", "kind": "mtf", "nx": 501, "ny": 501, "freqs": 251},
        # NNPS of a stack of flat fields, nine regions each
        {"name": "nnps_stack", "kind": "nnps", "images": 16, "nx": 501, "ny": 501, "roi": 128, "rois": 3},
        # fine-tuning steps of the shipped network at its training batch
        {"name": "train_steps", "kind": "train", "points": 20000, "batch": 8192, "steps": 16},
        # predictions for a table of depositions (odd count)
        {"name": "predict_table", "kind": "predict", "rows": 50001},
        # the surrogate in the loop on the surrogate workload's detector
        {"name": "surrogate_loop", "kind": "loop", "xrays": 100000},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["transport"] * 4 + ["lattice", "batch", "labels", "chain", "mtf", "nnps", "train", "predict",
                                           "loop"])
    if kind == "transport":
        c = rng.choice([0, 1])
        return {"kind": "transport", "config": c, "xrays": _log(rng, 25, 100000), "grid": 0,
                "refl": rng.choice([0.0, 0.0, 0.25])}
    if kind == "lattice":
        return {"kind": "transport", "config": rng.choice([0, 1]), "xrays": _log(rng, 100, 10000),
                "grid": rng.choice([1, 2]), "refl": 0.0}
    if kind == "batch":
        return {"kind": "batch", "xrays": _log(rng, 100, 2000)}
    if kind == "labels":
        return {"kind": "labels", "geoms": rng.randint(2, 64), "points": rng.randint(20, 100),
                "photons": _log(rng, 1000, 10000)}
    if kind == "chain":
        return {"kind": "chain", "xrays": _log(rng, 500, 20000)}
    if kind == "mtf":
        n = rng.randint(101, 501)
        m = rng.choice([n, rng.randint(101, 501)])
        return {"kind": "mtf", "nx": n, "ny": m, "freqs": rng.randint(40, max(n, m) // 2 + 1)}
    if kind == "nnps":
        roi = rng.choice([32, 64, 100, 127, 128])
        return {"kind": "nnps", "images": rng.choice([1, rng.randint(2, 16)]), "nx": rng.randint(400, 501),
                "ny": rng.randint(400, 501), "roi": roi, "rois": rng.randint(1, 3)}
    if kind == "train":
        return {"kind": "train", "points": rng.randint(5000, 20000), "batch": 64 * rng.randint(8, 128),
                "steps": rng.randint(4, 16)}
    if kind == "predict":
        return {"kind": "predict", "rows": _log(rng, 100, 50000)}
    return {"kind": "loop", "xrays": _log(rng, 2000, 100000)}


# ------------------------------------------------------------------ inputs


def _cm(es):
    x, y, z = es.to_cm()
    return x, y, z, es.e_ev.astype(np.float64), es.hist


def _point_image(nx, ny, rng):
    """Poisson counts of a point response: a core and a wide halo."""
    x = np.arange(nx)[:, None] - 0.5 * (nx - 1)
    y = np.arange(ny)[None, :] - 0.5 * (ny - 1)
    r = np.hypot(x, y)
    return rng.poisson(4000.0 * np.exp(-r / 3.0) + 60.0 / (1.0 + (r / 20.0) ** 2)).astype(np.float64)


def _flat_fields(n, nx, ny, rng):
    """Flat-field counts, neighbouring pixels sharing light."""
    a = rng.poisson(300.0, (n, nx, ny)).astype(np.float64)
    return 0.5 * a + 0.25 * np.roll(a, 1, 1) + 0.25 * np.roll(a, 1, 2)


def _model():
    """The shipped network: normalisation box, routing hull (the detector's
    depositions) and public parameters (float32)."""
    with open(MODEL, "rb") as f:
        b = f.read()
    hidden, bins = np.frombuffer(b, np.int32, 2, 8)
    rmax = np.frombuffer(b, np.float64, 1, 16)[0]
    box, hull = np.frombuffer(b, np.float32, 16, 24), np.frombuffer(b, np.float32, 16, 24 + 64)
    n = hidden * 8 + hidden + 2 * (hidden * hidden + hidden) + 25 * hidden + 25
    return (int(hidden), int(bins), float(rmax), box[:8], box[8:], hull[:8], hull[8:],
            np.frombuffer(b, np.float32, int(n), 24 + 128))


def _features(n, rng):
    """Depositions in the shipped network's detector: depth, energy and
    distance over its routing hull."""
    _, _, _, _, _, lo, hi, _ = _model()
    return (lo + (hi - lo) * rng.random((n, 8), np.float32)).astype(np.float32)


def _label_table(n, rng):
    f = _features(n, rng)
    photons = np.full(n, 10000, np.int32)
    detected = rng.binomial(photons, 0.25 + 0.4 * rng.random(n)).astype(np.int32)
    edges = 400.0 * (np.arange(97) / 96.0) ** 2
    scale = 10.0 + 40.0 * rng.random(n)
    cdf = 1.0 - np.exp(-edges[None, :] / scale[:, None])
    p = np.concatenate([np.diff(cdf, axis=1), 1.0 - cdf[:, -1:]], axis=1)
    radial = rng.multinomial(detected, p / p.sum(1, keepdims=True)).astype(np.uint32)
    return f, photons, detected, radial


def prepare(case, seed):
    kind, s = case["kind"], {"kind": case["kind"], "case": case}
    rng = np.random.default_rng(seed)
    if kind == "transport":
        es = hb.synth_events(case["config"], case["xrays"], seed)
        es.params.sensor_refl = case["refl"]
        s["t"] = hb.OpticalTransport(es.params, seed=seed + 1, column_grid=case["grid"])
        s["events"] = _cm(es)
    elif kind == "batch":
        es = hb.synth_events(2, case["xrays"], seed)
        s["t"] = hb.OpticalTransport(es.params, seed=seed + 1)
        s["t"].set_geometries(es.geometries)
        s["events"], s["n_geom"] = es, len(es.geometries)
        s["prf"] = np.zeros((s["n_geom"],) + s["t"].prf_dims(0), np.uint64)
    elif kind == "labels":
        s["geoms"], s["seed"] = sgm.sample_geometries(case["geoms"], seed), seed + 1
    elif kind == "chain":
        p = hb.default_params(num_hist=case["xrays"], det_x=909.0, det_y=909.0, ub_x=909.0, ub_y=909.0, radius=5.1,
                              sensor_refl=0.25, yield_=0.055)
        s["front"] = xr.XrayFrontEnd(det_x_um=909.0, det_y_um=909.0, det_height_um=150.0, seed=seed + 1)
        e = np.array([25000.0, 25000.0])
        s["source"] = xr.Source(e, np.array([1.0, -1.0]), sides_cm=(0.003, 0.003, 0.0))
        s["t"] = hb.OpticalTransport(p, seed=seed + 2)
    elif kind == "mtf":
        s["image"] = _point_image(case["nx"], case["ny"], rng)
    elif kind == "nnps":
        s["images"] = _flat_fields(case["images"], case["nx"], case["ny"], rng)
    elif kind == "train":
        s["net"] = sgm.Surrogate(batch=case["batch"], lr=1e-4, seed=seed + 1)
        s["net"].load(MODEL)
        s["net"].set_data(*_label_table(case["points"], rng), n_val=case["points"] // 20)
    elif kind == "predict":
        s["net"] = sgm.Surrogate()
        s["net"].load(MODEL)
        s["features"] = _features(case["rows"], rng)
    elif kind == "loop":
        es = hb.synth_events(4, case["xrays"], seed)
        s["t"] = hb.OpticalTransport(es.params, seed=seed + 1)
        s["net"] = sgm.Surrogate()
        s["net"].load(MODEL)
        s["events"] = _cm(es)
    else:
        raise ValueError(kind)
    return s


# ------------------------------------------------------------------ one pass


def _counts(c):
    """Integer counters; the path-length sum is a float added in the order the
    photons end, which is not fixed."""
    return {k: v for k, v in c.items() if k != "photon_distance"}


def _transport_results(t):
    st = t.phs_stats()
    return {"counters": _counts(t.counters()), "prf": t.prf(), "phs": t.phs(), "per_history": t.detected_per_primary(),
            "mean": st["mean"], "swank": st["swank"]}


def run(s):
    kind, c = s["kind"], s["case"]
    if kind == "transport":
        t = s["t"]
        t.reset_tallies()
        t.submit_events(*s["events"])
        t.run_sync()
        return _transport_results(t)
    if kind == "batch":
        t = s["t"]
        t.reset_tallies()
        t.submit(s["events"])
        t.run_sync()
        phs, stats, counts = [], [], []
        for g in range(s["n_geom"]):
            s["prf"][g] = t.prf(g)
            phs.append(t.phs(g))
            st = t.phs_stats(g)
            stats.append((st["mean"], st["swank"]))
            counts.append(list(_counts(t.counters(g)).values()))
        return {"prf": s["prf"], "phs": np.array(phs), "stats": np.array(stats), "counters": np.array(counts),
                "per_history": t.detected_per_primary()}
    if kind == "labels":
        return sgm.label_points(s["geoms"], c["points"], c["photons"], s["seed"])
    if kind == "chain":
        t = s["t"]
        t.reset_tallies()
        s["front"].run(s["source"], c["xrays"])
        s["front"].submit(t)
        t.run_sync()
        return dict(_transport_results(t), edes=s["front"].num_edes())
    if kind == "mtf":
        return analysis.mtf(s["image"], 1.0, c["freqs"])
    if kind == "nnps":
        return analysis.nnps(s["images"], 3.0, c["roi"], rois_x=c["rois"], rois_y=c["rois"])
    if kind == "train":
        train, val = s["net"].train(c["steps"])
        return {"params": s["net"].params(), "train_loss": np.float32(train), "val_loss": np.float32(val)}
    if kind == "predict":
        return s["net"].predict(s["features"])
    t = s["t"]
    t.reset_tallies()
    t.submit_events(*s["events"])
    st = s["net"].run(t, 0.01)
    return dict(_transport_results(t), surrogate_events=st["surrogate_events"], audit_events=st["audit_events"],
                mc_events=st["mc_events"], surrogate_detected=st["surrogate_detected"],
                audit_mc_detected=st["audit_mc_detected"], audit_expected=np.float32(st["audit_sg_expected"]))


def work(case):
    kind = case["kind"]
    prf = 8.0 * 501 * 501
    if kind == "transport":
        n = case["xrays"]
        events = n if case["config"] == 0 else 2.5 * n
        return {"bytes": 36.0 * events + prf + 4.0 * n, "flops": n * PHOTONS[case["config"]] * WALK_FLOPS}
    if kind == "batch":
        n = 64 * case["xrays"]
        return {"bytes": 64 * prf + 30.0 * 2.5 * n, "flops": n * PHOTONS[2] * WALK_FLOPS}
    if kind == "labels":
        n = case["geoms"] * case["points"]
        return {"bytes": 97 * 4.0 * n, "flops": n * float(case["photons"]) * WALK_FLOPS}
    if kind == "chain":
        return {"bytes": 8.0 * 909 * 909, "flops": case["xrays"] * CHAIN_PHOTONS * WALK_FLOPS}
    if kind == "mtf":
        # row transforms at 2K - 1 column frequencies, then columns (half of
        # the frequency plane is the other half's conjugate), complex products
        v = 2.0 * case["freqs"] - 1
        px = float(case["nx"] * case["ny"])
        return {"bytes": 8.0 * px, "flops": 4.0 * px * case["freqs"] + 8.0 * case["nx"] * v * case["freqs"]}
    if kind == "nnps":
        r, n = float(case["roi"]), case["images"] * case["rois"] ** 2
        return {"bytes": 8.0 * (case["images"] * case["nx"] * case["ny"] + r * r), "flops": n * 6.0 * r ** 3}
    if kind == "train":
        mlp = 2.0 * (8 * 256 + 2 * 256 * 256 + 25 * 256)
        rows = case["steps"] * case["batch"]
        return {"bytes": 4.0 * case["points"] * (97 + 10), "flops": 3.0 * rows * mlp + rows * 97 * 8 * 40.0}
    if kind == "predict":
        mlp = 2.0 * (8 * 256 + 2 * 256 * 256 + 25 * 256)
        return {"bytes": case["rows"] * 4.0 * (8 + 25), "flops": case["rows"] * mlp}
    n = case["xrays"]
    # 1 % of the photons are walked (the audit); the rest cost the network per
    # event and about 100 operations per detected photon
    return {"bytes": 36.0 * 2.5 * n + prf, "flops": 2.5 * n * 2.8e5 + n * PHOTONS[4] * (0.01 * WALK_FLOPS + 30.0)}


# ------------------------------------------------------------------ 64 bits


def _mtf64(img, pixel, K):
    nx, ny = img.shape
    n = max(nx, ny)
    f = np.fft.fft2(img, (n, n))
    total = img.sum()
    k = np.arange(-(K - 1), K)
    mag = np.abs(f[np.ix_(k % n, k % n)]) / total
    b = np.rint(np.hypot(k[:, None], k[None, :])).astype(int).ravel()
    cnt = np.bincount(b, minlength=K)[:K]
    return {"freq": 1000.0 * np.arange(K) / (n * pixel), "mtf_x": np.abs(f[:K, 0]) / total,
            "mtf_y": np.abs(f[0, :K]) / total, "mtf_r": np.bincount(b, mag.ravel(), minlength=K)[:K] / cnt}


def _nnps64(imgs, pixel, roi, rois):
    n, nx, ny = imgs.shape
    x0, y0 = (nx - rois * roi) // 2, (ny - rois * roi) // 2
    mean = imgs.mean(0)
    acc, sig = np.zeros((roi, roi)), 0.0
    for a in range(rois):
        for b in range(rois):
            at = np.s_[x0 + a * roi:x0 + (a + 1) * roi, y0 + b * roi:y0 + (b + 1) * roi]
            sig += mean[at].sum()
            for im in imgs:
                d = im[at] - (mean[at] if n > 1 else mean[at].mean())
                acc += np.abs(np.fft.fft2(d)) ** 2
    m = sig / (rois * rois * roi * roi)
    corr = n / (n - 1) if n > 1 else 1.0
    n2 = acc * (pixel / 1000.0) ** 2 / roi ** 2 * corr / (n * rois * rois) / m ** 2
    k = np.arange(roi)
    k = np.where(k <= roi // 2, k, k - roi)
    b = np.rint(np.hypot(k[:, None], k[None, :])).astype(int).ravel()
    K = roi // 2 + 1
    cnt = np.bincount(b, minlength=K)[:K]
    return {"freq": 1000.0 * np.arange(K) / (roi * pixel),
            "nnps_r": np.bincount(b, n2.ravel(), minlength=K)[:K] / cnt, "nnps_2d": n2, "mean_signal": float(m)}


def _split(p, hidden):
    sizes = [(hidden, 8), (hidden,), (hidden, hidden), (hidden,), (hidden, hidden), (hidden,), (25, hidden), (25,)]
    out, o = [], 0
    for s in sizes:
        n = int(np.prod(s))
        out.append(p[o:o + n].reshape(s))
        o += n
    return out


def _net64(parts, feat, lo, hi):
    span = hi - lo
    inv = torch.where(span > 0, 1.0 / torch.where(span > 0, span, torch.ones_like(span)), torch.full_like(span, 0.5))
    h = 2.0 * (feat - lo) * inv - 1.0
    for i in range(0, 6, 2):
        h = torch.relu(h @ parts[i].T + parts[i + 1])
    return h @ parts[6].T + parts[7]


def _loss64(out, t, y, bins, rmax):
    """Per-row loss: detection cross-entropy plus the radial categories' under
    the mixture of Gaussian rings."""
    z = out[:, 0]
    ld = t * torch.nn.functional.softplus(-z) + (1.0 - t) * torch.nn.functional.softplus(z)
    w = torch.softmax(out[:, 1:9], 1)
    mu = 50.0 * torch.nn.functional.softplus(out[:, 9:17])
    sd = 10.0 * torch.exp(torch.clamp(out[:, 17:25], -6.0, 4.0))
    e = rmax * (torch.arange(bins + 1, dtype=out.dtype, device=out.device) / bins) ** 2
    x = (e - mu[..., None]) / sd[..., None]
    cdf, tail = torch.special.ndtr(x), torch.special.ndtr(-x)
    pdf = torch.exp(-0.5 * x * x) / np.sqrt(2.0 * np.pi)
    lower = x[..., :-1] < 0
    d = torch.where(lower, cdf[..., 1:] - cdf[..., :-1], tail[..., :-1] - tail[..., 1:])
    mass = mu[..., None] * d + sd[..., None] * (pdf[..., :-1] - pdf[..., 1:])
    last = mu * tail[..., -1] + sd * pdf[..., -1]
    S = mu * tail[..., 0] + sd * pdf[..., 0]
    q = (w[..., None] * torch.cat([mass, last[..., None]], -1) / S[..., None]).sum(1)
    return ld - (y * torch.log(q + 1e-12)).sum(1)


def _philox(r, step, key):
    """First two words of Philox-4x32-10 at counter (r, step, 0, 0x5347)."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [r.astype(np.uint64), np.full(len(r), step, np.uint64), np.zeros(len(r), np.uint64),
         np.full(len(r), 0x5347, np.uint64)]
    k0, k1 = key & 0xFFFFFFFF, key >> 32
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & m32, (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return (c[0] << np.uint64(32)) | c[1]


def _train64(case, seed):
    hidden, bins, rmax, lo, hi, _, _, p = _model()
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rng = np.random.default_rng(seed)
    f, ph, det, rad = _label_table(case["points"], rng)
    f, lo, hi = (torch.tensor(a, dtype=torch.float64, device=dev) for a in (f, lo, hi))
    t = torch.tensor(det / ph, dtype=torch.float64, device=dev)
    r = torch.tensor(rad.astype(np.float64), device=dev)
    y = r / torch.clamp(r.sum(1, keepdim=True), min=1.0)
    n_train = case["points"] - case["points"] // 20
    w = torch.tensor(p, dtype=torch.float64, device=dev)
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    losses = []
    for step in range(case["steps"]):
        rows = (_philox(np.arange(case["batch"]), step, seed + 1) % np.uint64(n_train)).astype(np.int64)
        i = torch.from_numpy(rows).to(dev)
        q = w.clone().requires_grad_(True)
        loss = _loss64(_net64(_split(q, hidden), f[i], lo, hi), t[i], y[i], bins, rmax).mean()
        loss.backward()
        losses.append(float(loss.detach()))
        m = 0.9 * m + 0.1 * q.grad
        v = 0.999 * v + 0.001 * q.grad ** 2
        k = step + 1
        w = w - 1e-4 * (m / (1 - 0.9 ** k)) / (torch.sqrt(v / (1 - 0.999 ** k)) + 1e-8)
    with torch.no_grad():
        val = _loss64(_net64(_split(w, hidden), f[n_train:], lo, hi), t[n_train:], y[n_train:], bins, rmax).mean()
    return {"params": w.cpu().numpy(), "train_loss": np.float64(np.mean(losses)), "val_loss": np.float64(float(val))}


def exact(case, seed):
    """64-bit values of the computed outputs; the Monte Carlo tallies are
    whole numbers without one."""
    kind, rng = case["kind"], np.random.default_rng(seed)
    if kind == "mtf":
        return _mtf64(_point_image(case["nx"], case["ny"], rng), 1.0, case["freqs"])
    if kind == "nnps":
        return _nnps64(_flat_fields(case["images"], case["nx"], case["ny"], rng), 3.0, case["roi"], case["rois"])
    if kind == "train":
        return _train64(case, seed)
    if kind == "predict":
        hidden, _, _, lo, hi, _, _, p = _model()
        parts = _split(torch.tensor(p, dtype=torch.float64), hidden)
        lo, hi = torch.tensor(lo, dtype=torch.float64), torch.tensor(hi, dtype=torch.float64)
        return _net64(parts, torch.tensor(_features(case["rows"], rng), dtype=torch.float64), lo, hi).numpy()
    return None
