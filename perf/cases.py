"""The measured work of the absolute-pose framework: what its users call, over the range they call it on.

Each case is one way a program uses the package, with synthetic correspondences of the shapes and value
distributions of the workloads in ``turboransac_b200.scenes`` (pinhole 640x480 camera, depth 0.5-4 m, pixel noise
on the inliers, outliers redrawn in the scene's box). Kinds of case:

* ``plain``   -- ``Context.estimate_absolute_pose``: one image at a time from host arrays, the reference's calling
                 pattern (a localisation loop that needs the pose before it goes on).
* ``resident``-- ``Batch``: frames uploaded once, re-estimated by one captured graph (offline evaluation).
* ``host``    -- ``estimate_batch``: many images from host arrays in one call, masks returned.
* ``stream``  -- ``estimate_batch_submit`` / ``collect``: two batches in flight from page-locked arrays, as a data
                 loader hands them over.
* ``device``  -- ``estimate_batch_device``: correspondences a GPU matcher left in device memory.
* ``serve``   -- ``Server``: a burst of requests, continuously batched.
* ``adjust``  -- ``Context.bundle_adjust``: pose refinement alone (a tracker with a pose prior).
* ``inliers`` -- ``Context.get_inliers``: an inlier mask for a known pose (map-point verification).

Outputs are every pose, mask and count a caller reads. Device times, scheduling details (engine steps, candidates
re-ranked) and the iteration counters of the refinement are diagnostics of one run and are left out.
"""
import math

import numpy as np
import torch

import turboransac_b200 as tbr
from turboransac_b200 import scenes

THRESHOLD_PX = 4.0
DEFAULT_PX = 12.0  # RansacOptions_cuda's own threshold

_ESTIMATES = ("plain", "resident", "host", "stream", "device", "serve")


def listed():
    """The listed cases, smallest call first."""
    return [
        # A mask for one image's correspondences at a pose known from elsewhere.
        {"name": "inliers_20000", "kind": "inliers", "n": 20000, "w": 0.4, "sigma": 1.0},
        # A tracker refining its predicted pose on the matches it kept.
        {"name": "adjust_6000", "kind": "adjust", "n": 6000, "w": 0.85, "sigma": 1.0},
        # Few matches, most of them right: the smallest calls of the serving range. Latency counts.
        {"name": "plain_301", "kind": "plain", "n": 301, "w": 0.6, "sigma": 1.0, "batch": 1000},
        # The plain workload: one ordinary image per call.
        {"name": "plain_2000", "kind": "plain", "n": 2000, "w": 0.4, "sigma": 1.0, "batch": 1000},
        # Options left at their defaults: 100000 samples per round, 12 px.
        {"name": "plain_defaults_1537", "kind": "plain", "n": 1537, "w": 0.5, "sigma": 1.0, "batch": 100000},
        # The scoring-bound workload: dense matches, a fixed number of samples, no refinement asked for.
        {"name": "forced_20000", "kind": "plain", "n": 20000, "w": 0.15, "sigma": 1.0, "batch": 1000,
         "forced": 4096},
        # A hard image: very dense matching with few right matches, tens of rounds.
        {"name": "plain_49999_hard", "kind": "plain", "n": 49999, "w": 0.08, "sigma": 1.0, "batch": 1000},
        # A small evaluation set from ordinary (pageable) arrays, masks wanted.
        {"name": "host_24_masks", "kind": "host", "frames": 24, "lo": 500, "hi": 12000, "w_lo": 0.2, "w_hi": 0.8},
        # A GPU matcher's output, a rig's worth of images at once.
        {"name": "device_64", "kind": "device", "frames": 64, "lo": 500, "hi": 30000, "w_lo": 0.1, "w_hi": 0.8},
        # The batched workload streamed through the submitted form, two halves in flight.
        {"name": "stream_256", "kind": "stream", "frames": 256, "lo": 500, "hi": 30000, "w_lo": 0.1, "w_hi": 0.8},
        # The batched workload with inputs resident: the headline of bench.py.
        {"name": "resident_256", "kind": "resident", "frames": 256, "lo": 500, "hi": 30000, "w_lo": 0.1, "w_hi": 0.8},
        # A burst of serving requests: sizes and inlier ratios of the serving workload.
        {"name": "serve_160", "kind": "serve", "frames": 160, "lo": 300, "hi": 50000, "w_lo": 0.1, "w_hi": 0.7},
    ]


def draw(rng):
    """One more case of the same ranges; no dearer than the largest listed one."""
    dearest = max(_cost(c) for c in listed())

    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    while True:
        kind = rng.choice(["plain", "plain", "plain", "host", "device", "stream", "resident", "serve", "adjust", "inliers"])
        sigma = round(rng.uniform(0.5, 2.0), 3)
        if kind == "plain":
            c = {"kind": kind, "n": log_int(300, 50000), "w": round(rng.uniform(0.1, 0.8), 3), "sigma": sigma,
                 "batch": rng.choice([1000, 1000, 1024, 100000])}
            what = rng.choice(["", "", "prosac", "forced"])
            if what == "prosac":
                c["prosac"] = True
            elif what == "forced":
                c["forced"] = log_int(1000, 8192)
        elif kind == "adjust":
            c = {"kind": kind, "n": log_int(200, 40000), "w": round(rng.uniform(0.7, 1.0), 3), "sigma": sigma}
        elif kind == "inliers":
            c = {"kind": kind, "n": log_int(1000, 100000), "w": round(rng.uniform(0.1, 0.8), 3), "sigma": sigma}
        else:
            hi = log_int(3000, 30000)
            c = {"kind": kind, "frames": log_int(4, 256), "lo": 300 if kind == "serve" else 500, "hi": hi, "w_lo": 0.1,
                 "w_hi": round(rng.uniform(0.5, 0.8), 3)}
        if _cost(c) <= dearest:
            return c


# ------------------------------------------------------------------ inputs --
def _seed(seed, i):
    return (int(seed) * 1_000_003 + i * 7919 + 17) & 0x7FFFFFFFFFFFFFFF


def _frames(case, seed):
    """The case's images, from the seed alone."""
    if "frames" not in case:
        f = scenes.make_frame(case["n"], case["w"], case["sigma"], _seed(seed, 0), threshold_px=_threshold(case))
        if case.get("prosac"):  # sorted by quality: right matches mostly first, as a matcher's ratio test has it
            rng = np.random.default_rng(_seed(seed, 1))
            order = np.argsort(rng.uniform(size=f.n) + ~f.inlier_gt, kind="stable")
            f.uv, f.xyz = np.ascontiguousarray(f.uv[order]), np.ascontiguousarray(f.xyz[order])
            f.inlier_gt = f.inlier_gt[order]
        return [f]
    rng = np.random.default_rng(_seed(seed, 1))
    m = case["frames"]
    # Sizes log-uniform and inlier ratios uniform, stratified so that another seed makes other inputs of the same weight.
    u = rng.permutation((np.arange(m) + 0.5) / m)
    v = (np.arange(m) + 0.5) / m
    n = np.exp(np.log(case["lo"]) + u * (np.log(case["hi"]) - np.log(case["lo"]))).round().astype(int)
    w = case["w_lo"] + v * (case["w_hi"] - case["w_lo"])
    sig = rng.uniform(0.5, 2.0, m)
    out = [scenes.make_frame(int(n[i]), float(w[i]), float(sig[i]), _seed(seed, 2 + i)) for i in range(m)]
    return [out[i] for i in rng.permutation(m)]


def _threshold(case):
    return DEFAULT_PX if case.get("batch") == 100000 else THRESHOLD_PX


def _options(case):
    ro = tbr.RansacOptions_cuda()
    ro.max_iterations = case.get("batch", 1000)
    ro.max_reproj_error = _threshold(case)
    ro.progressive_sampling = bool(case.get("prosac"))
    return ro


def _camera(f):
    return tbr.Camera_cuda(1, scenes.WIDTH, scenes.HEIGHT, [float(k) for k in f.K])


_kept = {}


def _context():
    """The context that a program keeps for its life."""
    if "ctx" not in _kept:
        _kept["ctx"] = tbr.Context(0, 4 << 30)
    return _kept["ctx"]


def _server():
    """The request loop that a serving program keeps for its life."""
    if "srv" not in _kept:
        _kept["srv"] = tbr.Server(_context(), budget_bytes=4 << 30, ransac_opt=_options({}))
    return _kept["srv"]


def _pinned(f):
    """The frame with page-locked arrays, as a data loader's workers leave them."""
    uv, xyz = torch.from_numpy(f.uv).pin_memory(), torch.from_numpy(f.xyz).pin_memory()
    f.uv, f.xyz = uv.numpy(), xyz.numpy()
    f.keep = (uv, xyz)
    return f


def _prior(f, seed):
    """A predicted pose: the true one turned by about a degree and moved by about 3 cm."""
    rng = np.random.default_rng(_seed(seed, 99))
    q = _quat_of(torch.from_numpy(f.R_gt)).numpy()
    d = np.concatenate([[1.0], rng.normal(0.0, 0.005, 3)])
    q = np.array([q[0] * d[0] - q[1:] @ d[1:], *(q[0] * d[1:] + d[0] * q[1:] + np.cross(q[1:], d[1:]))])
    return q / np.linalg.norm(q), f.t_gt + rng.normal(0.0, 0.02, 3)


def prepare(case, seed):
    kind = case["kind"]
    fr = _frames(case, seed)
    s = {"case": case, "kind": kind, "ctx": _context(), "opt": _options(case), "frames": fr}
    if kind == "resident":
        s["batch"] = tbr.Batch(s["ctx"], fr, s["opt"])
    elif kind == "stream":
        s["frames"] = [_pinned(f) for f in fr]
    elif kind == "device":
        s["frames"] = [tbr.DeviceFrame(f) for f in fr]
    elif kind == "serve":
        s["server"] = _server()
    elif kind in ("plain", "adjust", "inliers"):
        f = fr[0]
        s["camera"] = _camera(f)
        s["opt"].seed = f.seed
        s["bundle"] = tbr.BundleOptions_cuda()
        if kind == "adjust":  # the kept matches: those within reach of the prior
            q, t = _prior(f, seed)
            s["x"], s["X"] = f.uv, f.xyz
            s["pose"] = tbr.CameraPose_cuda(q, t)
        elif kind == "inliers":
            q, t = _prior(f, seed)
            s["x"], s["X"] = s["camera"].unproject(f.uv), f.xyz
            s["pose"] = tbr.CameraPose_cuda(q, t)
            s["sq"] = (2 * DEFAULT_PX / s["camera"].focal()) ** 2
    return s


# -------------------------------------------------------------------- runs --
_WHOLE = ("samples", "hypotheses", "ransac_inliers", "num_inliers", "best_sample", "best_solution")
_REAL = ("model_score", "lm_initial_cost", "lm_cost")


def _packed(rows):
    """Per-frame results as one array per field."""
    out = {"q": np.array([r["q"] for r in rows]), "t": np.array([r["t"] for r in rows])}
    for k in _WHOLE:
        out[k] = np.array([r[k] for r in rows], np.int64)
    for k in _REAL:
        out[k] = np.array([r[k] for r in rows], np.float64)
    return out


def run(state):
    kind, ctx, opt, fr = state["kind"], state["ctx"], state["opt"], state["frames"]
    if kind == "plain":
        case = state["case"]
        st, pose, inl = ctx.estimate_absolute_pose(
            fr[0].uv, fr[0].xyz, state["camera"], opt, state["bundle"], force_samples=case.get("forced", 0),
            skip_refine=bool(case.get("forced")), honor_options=bool(case.get("prosac")))
        d = st.details
        out = {"q": pose.q, "t": pose.t, "inliers": inl}
        out.update({k: d[k] for k in _WHOLE})
        out.update({k: d[k] for k in _REAL[: 1 if case.get("forced") else 3]})
        return out
    if kind == "resident":
        state["batch"].run()
        return _packed(state["batch"].results())
    if kind == "host":
        rows = tbr.estimate_batch(ctx, fr, opt, masks=True)
        return dict(_packed(rows), inliers=np.concatenate([r["inliers"] for r in rows]))
    if kind == "stream":
        h = len(fr) // 2
        first = tbr.estimate_batch_submit(ctx, fr[:h], opt)
        second = tbr.estimate_batch_submit(ctx, fr[h:], opt)
        return _packed(first.collect() + second.collect())
    if kind == "device":
        return _packed(tbr.estimate_batch_device(ctx, fr, opt))
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(f) for f in fr]
        srv.drain()
        got = {}
        while len(got) < len(ids):
            got.update({r["id"]: r for r in srv.poll()})
        return _packed([got[i] for i in ids])
    if kind == "adjust":
        pose, d = ctx.bundle_adjust(state["x"], state["X"], state["camera"], state["pose"], state["bundle"])
        return {"q": pose.q, "t": pose.t, "lm_initial_cost": d["lm_initial_cost"], "lm_cost": d["lm_cost"]}
    return {"inliers": ctx.get_inliers(state["pose"], state["x"], state["X"], state["sq"])}


# -------------------------------------------------------------------- work --
_FLOP_PAIR = 27  # one point against one hypothesis: projection 18, reciprocal, residual 4, square 3, sum
_FLOP_P3P = 1000
_FLOP_LM = 300   # one point in one refinement iteration
_HYP_PER_SAMPLE = 1.5
_LM_ITERATIONS = 12


def _frame_work(n, w, batch, forced=0):
    if forced:
        samples = forced
    else:
        need = 3.0 * math.log(1e-4) / math.log1p(-min(w, 0.999) ** 3)
        samples = batch * min(math.ceil((need + 1) / batch), math.ceil(100000 / batch))
    flops = samples * (_FLOP_P3P + _HYP_PER_SAMPLE * n * _FLOP_PAIR)
    if not forced:
        flops += _LM_ITERATIONS * w * n * _FLOP_LM
    return flops


def work(case):
    """Inputs read once (five doubles a point) and results written once; every sample's hypotheses against every
    point, as the estimator is defined, and the refinement's passes."""
    kind = case["kind"]
    if "frames" in case:
        m = case["frames"]
        span = math.log(case["hi"]) - math.log(case["lo"])
        ns = [math.exp(math.log(case["lo"]) + (i + 0.5) / m * span) for i in range(m)]
        points, mean = sum(ns), sum(ns) / m
        flops = sum(_frame_work(mean, case["w_lo"] + (i + 0.5) / m * (case["w_hi"] - case["w_lo"]), 1000)
                    for i in range(m))
        return {"bytes": 40 * points + 264 * m + (points if kind == "host" else 0), "flops": flops}
    n = case["n"]
    if kind == "inliers":
        return {"bytes": 41 * n, "flops": 30 * n}
    if kind == "adjust":
        return {"bytes": 40 * n, "flops": _LM_ITERATIONS * n * _FLOP_LM}
    return {"bytes": 41 * n + 264, "flops": _frame_work(n, case["w"], case["batch"], case.get("forced", 0))}


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


# ------------------------------------------------------------------- exact --
# The estimator in plain float64 tensors: counter-based samples, Lambda-Twist style P3P, truncated MSAC, the
# round-by-round stop rule, inliers, and the damped Gauss-Newton refinement on the Cauchy loss.
_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_F64 = torch.float64


def _philox(samples, seed):
    """Philox4x32-10 of counters (sample, 0, 0) under the 64-bit key: four uint32 columns."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [samples.astype(np.uint64) & m32, samples.astype(np.uint64) >> np.uint64(32),
         np.zeros(samples.size, np.uint64), np.zeros(samples.size, np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _triples(first, count, n, seed, prosac):
    s = np.arange(first, first + count)
    c = _philox(s, seed)
    sh = np.uint64(32)

    def pick(word, m):
        return ((word * np.asarray(m, np.uint64)) >> sh).astype(np.int64)

    i0, i1, i2 = pick(c[0], n), pick(c[1], n - 1), pick(c[2], n - 2)
    i1 += i1 >= i0
    lo, hi = np.minimum(i0, i1), np.maximum(i0, i1)
    i2 += i2 >= lo
    i2 += i2 >= hi
    out = np.stack([i0, i1, i2], 1)
    if prosac:
        k = np.arange(3, n + 1, dtype=np.float64)
        tk = 100000.0 * (k / n) * ((k - 1) / (n - 1)) * ((k - 2) / (n - 2))
        grow = np.concatenate([[1], 1 + np.cumsum(np.ceil(np.diff(tk)))]).astype(np.int64)
        m = 3 + np.searchsorted(grow[:-1], s + 1, side="right")
        j0, j1 = pick(c[0], m - 1), pick(c[1], m - 2)
        j1 += j1 >= j0
        out = np.where(((m >= n) & (grow[-1] < s + 1))[:, None], out, np.stack([j0, j1, m - 1], 1))
    return out


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _p3p(x, X):
    """Poses [R | t] (S, 4, 3, 4) of the bearings x and points X (S, 3, 3), and which of the four exist, in order."""
    d = lambda i, j: ((X[:, i] - X[:, j]) ** 2).sum(1)  # noqa: E731
    a01, a02, a12 = d(0, 1), d(0, 2), d(1, 2)
    swap02, swap01 = (a01 > a02) & (a01 > a12), (a01 <= a02) & (a02 > a12)
    ids = torch.arange(3, device=x.device).repeat(len(x), 1)
    ids = torch.where(swap02[:, None], ids[:, [2, 1, 0]], torch.where(swap01[:, None], ids[:, [1, 0, 2]], ids))
    at = ids[:, :, None].expand(-1, -1, 3)
    x, X = x.gather(1, at), X.gather(1, at)
    a01, a02, a12 = d(0, 1), d(0, 2), d(1, 2)
    a, b = a01 / a12, a02 / a12
    m01, m02, m12 = ((x[:, i] * x[:, j]).sum(1) for i, j in ((0, 1), (0, 2), (1, 2)))
    s12, s02, s01 = 1 - m12 * m12, m02 * m02 - 1, m01 * m01 - 1
    mm = -2 + 2 * m01 * m02 * m12
    k3 = 1 / (b * b * s12 + b * s02)
    c2 = k3 * ((a - 1) * s02 + 2 * a * b * s12 + b * b * s12 + b * mm)
    c1 = k3 * (a * a * s12 + 2 * a * b * s12 + a * mm + (b - 1) * s01)
    c0 = k3 * (a * a * s12 + a * s01)
    # One real root of the cubic.
    p = c1 - c2 * c2 / 3
    q = (2 * c2 ** 3 - 9 * c2 * c1) / 27 + c0
    disc = q * q / 4 + p ** 3 / 27
    one = disc > 0
    r = torch.sqrt(disc.clamp(min=0))
    cbrt = lambda v: torch.sign(v) * torch.abs(v).pow(1 / 3)  # noqa: E731
    root1 = cbrt(-q / 2 + r) + cbrt(-q / 2 - r) - c2 / 3
    pn = torch.where(disc < 0, p, -torch.ones_like(p))
    arg = (3 * q / (2 * pn) * torch.sqrt(-3 / pn)).clamp(-1, 1)
    root3 = 2 * torch.sqrt(-pn / 3) * torch.cos(torch.arccos(arg) / 3) - c2 / 3
    root0 = -c2 / 3 + torch.where(p != 0, 3 * q / torch.where(p != 0, p, torch.ones_like(p)), torch.zeros_like(p))
    s = torch.where(one, root1, torch.where(disc < 0, root3, root0))
    # The degenerate conic and its two lines.
    C00, C01, C02 = -a + s * (1 - b), -m02 * s, a * m12 + b * m12 * s
    C11, C12, C22 = s + 1, -m01, -a - b * s + 1
    A00, A11, A22 = C12 * C12 - C11 * C22, C02 * C02 - C00 * C22, C01 * C01 - C00 * C11
    A01, A02, A12 = C01 * C22 - C02 * C12, C02 * C11 - C01 * C12, C00 * C12 - C02 * C01
    col0 = (A00 > A11) & (A00 > A22)
    col1 = ~(A00 > A11) & (A11 > A22)
    sel = lambda u, v, w: torch.where(col0, u, torch.where(col1, v, w))  # noqa: E731
    sq = torch.sqrt(sel(A00, A11, A22))
    v0, v1, v2 = sel(A00, A01, A02) / sq, sel(A01, A11, A12) / sq, sel(A02, A12, A22) / sq
    lines = ((C00, C01 + v2, C02 - v1), (C00, C01 - v2, C02 + v1))
    # Depths of every root that passes the filters.
    dep, ok = [], []
    for p0, p1, p2 in lines:
        first = p0.abs() <= p1.abs()
        u0, u1 = torch.where(first, -p0 / p1, -p1 / p0), torch.where(first, -p2 / p1, -p2 / p0)
        ca = torch.where(first, 1 / (u1 * u1 - b), 1 / (-a * u1 * u1 + 2 * a * m12 * u1 - a + 1))
        cb = torch.where(first, 2 * (b * m12 - m02 * u1 + u0 * u1), 2 * (a * m12 * u0 - m01 - a * u0 * u1)) * ca
        cc = torch.where(first, u0 * u0 - 2 * m02 * u0 - b + 1, 1 - a * u0 * u0) * ca
        v = cb * cb - 4 * cc
        real = v >= float(np.float32(1e-6))
        y = torch.sqrt(v.clamp(min=0))
        neg = cb < 0
        r1 = torch.where(neg, 0.5 * (-cb + y), 2 * cc / (-cb + y))
        r2 = torch.where(neg, 0.5 * (-cb - y), 2 * cc / (-cb - y))
        for tau in (r1, r2):
            db = torch.sqrt(a12 / (tau * (tau - 2 * m12) + 1))  # first form: d2, d1 = tau d2, d0
            e1 = tau * db
            e0 = u0 * db + u1 * e1
            dc = torch.sqrt(a01 / (tau * (tau - 2 * m01) + 1))  # second form: d0, d1 = tau d0, d2
            g1 = tau * dc
            g2 = u0 * dc + u1 * g1
            dep.append(torch.stack([torch.where(first, e0, dc), torch.where(first, e1, g1), torch.where(first, db, g2)], 1))
            ok.append(real & ~(tau <= 0) & ~(torch.where(first, e0, g2) < 0))
    ok = torch.stack(ok, 1)
    done = one & (ok[:, 0] | ok[:, 1])
    ok = ok & ~(done[:, None] & torch.tensor([False, False, True, True], device=x.device))
    D = torch.stack(dep, 1)
    B = lambda v: v[:, None]  # noqa: E731
    live = ok.clone()
    for _ in range(5):  # Gauss-Newton polish of the depths
        l1, l2, l3 = D.unbind(2)
        e1 = l1 * l1 - 2 * l1 * l2 * B(m01) + l2 * l2 - B(a01)
        e2 = l1 * l1 - 2 * l1 * l3 * B(m02) + l3 * l3 - B(a02)
        e3 = l2 * l2 - 2 * l2 * l3 * B(m12) + l3 * l3 - B(a12)
        live = live & ~(e1.abs() + e2.abs() + e3.abs() < float(np.float32(1e-6)))
        x11, x12, x21 = l1 - l2 * B(m01), l2 - l1 * B(m01), l1 - l3 * B(m02)
        x23, x32, x33 = l3 - l1 * B(m02), l2 - l3 * B(m12), l3 - l2 * B(m12)
        j = 0.5 / (x11 * x23 * x32 + x12 * x21 * x33)
        step = torch.stack([(-x23 * x32 * e1 - x12 * x33 * e2 + x12 * x23 * e3) * j,
                            (-x21 * x33 * e1 + x11 * x33 * e2 - x11 * x23 * e3) * j,
                            (x21 * x32 * e1 - x11 * x32 * e2 - x12 * x21 * e3) * j], 2)
        D = torch.where(live[:, :, None], D + step, D)
    Y = D[:, :, :, None] * x[:, None]
    V1, V2 = Y[:, :, 0] - Y[:, :, 1], Y[:, :, 0] - Y[:, :, 2]
    W1, W2 = X[:, 0] - X[:, 1], X[:, 0] - X[:, 2]
    W = torch.stack([W1, W2, _cross(W1, W2)], 2)
    eye = torch.eye(3, dtype=_F64, device=x.device).expand_as(W)
    W = torch.linalg.inv_ex(W).inverse
    W = torch.where(torch.isfinite(W).all(2, True).all(1, True), W, eye)
    R = torch.stack([V1, V2, _cross(V1, V2)], 3) @ W[:, None]
    t = Y[:, :, 0] - (R @ X[:, None, 0, :, None])[..., 0]
    return torch.cat([R, t[..., None]], 3), ok


def _msac(P, xn, X, tau2):
    """Truncated scores and inlier counts of the poses P (H, 3, 4)."""
    Xh = torch.cat([X, torch.ones_like(X[:, :1])], 1).T
    score, count = [], []
    for Pc in P.split(max(1, 30_000_000 // X.shape[0])):
        z = Pc.reshape(-1, 4) @ Xh
        z = z.view(-1, 3, X.shape[0])
        r2 = (z[:, 0] / z[:, 2] - xn[:, 0]) ** 2 + (z[:, 1] / z[:, 2] - xn[:, 1]) ** 2
        inl = (r2 < tau2) & (z[:, 2] > 0)
        count.append(inl.sum(1))
        score.append(torch.where(inl, r2, torch.zeros_like(r2)).sum(1) + (X.shape[0] - count[-1]) * tau2)
    return torch.cat(score).cpu().numpy(), torch.cat(count).cpu().numpy()


def _quat_of(R):
    """Unit quaternion (w, x, y, z), from the largest of the four; w's branch where the trace is positive."""
    R = R.tolist()
    tr = R[0][0] + R[1][1] + R[2][2]
    if tr > 0:
        s = 0.5 / math.sqrt(tr + 1)
        q = [0.25 / s, (R[2][1] - R[1][2]) * s, (R[0][2] - R[2][0]) * s, (R[1][0] - R[0][1]) * s]
    else:
        i = 0 if R[0][0] > R[1][1] and R[0][0] > R[2][2] else (1 if R[1][1] > R[2][2] else 2)
        j, k = (i + 1) % 3, (i + 2) % 3
        s = 2 * math.sqrt(1 + R[i][i] - R[j][j] - R[k][k])
        q = [(R[k][j] - R[j][k]) / s, 0.0, 0.0, 0.0]
        q[1 + i], q[1 + j], q[1 + k] = 0.25 * s, (R[i][j] + R[j][i]) / s, (R[i][k] + R[k][i]) / s
    q = torch.tensor(q, dtype=_F64)
    return q / q.norm()


def _matrix_of(q):
    w, x, y, z = (float(v) for v in q)
    return torch.tensor([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                         [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                         [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]], dtype=_F64)


def _mask(q, t, xn, X, tau2):
    Z = X @ _matrix_of(q).to(X.device).T + t.to(X.device)
    r2 = (Z[:, 0] / Z[:, 2] - xn[:, 0]) ** 2 + (Z[:, 1] / Z[:, 2] - xn[:, 1]) ** 2
    return (r2 < tau2) & (Z[:, 2] > 0)


def _refine(q, t, u, X, cam, scale, iterations=100):
    """Levenberg-Marquardt on sum log(1 + r^2 / scale^2), rotation and translation both updated on the camera's
    right: R exp(w), t + R dt. Returns q, t, the first and the last cost."""
    inv = 1.0 / (scale * scale)
    f, c = torch.tensor(cam[:2], dtype=_F64, device=X.device), torch.tensor(cam[2:], dtype=_F64, device=X.device)

    def project(q, t):
        Rm = _matrix_of(q).to(X.device)
        Z = X @ Rm.T + t.to(X.device)
        r = f * Z[:, :2] / Z[:, 2:] + c - u
        r2, ok = (r * r).sum(1), Z[:, 2] >= 0
        return Rm, Z, r, r2, ok, float(torch.where(ok, torch.log1p(r2 * inv), torch.zeros_like(r2)).sum())

    def normal(state):
        Rm, Z, r, r2, ok, _ = state
        wgt = torch.where(ok, inv / (1 + r2 * inv), torch.zeros_like(r2))
        iz = 1 / Z[:, 2]
        zero = torch.zeros_like(iz)
        dZ = torch.stack([torch.stack([f[0] * iz, zero, -f[0] * Z[:, 0] * iz * iz], 1),
                          torch.stack([zero, f[1] * iz, -f[1] * Z[:, 1] * iz * iz], 1)], 1) @ Rm
        rot = torch.stack([X[:, 1:2] * dZ[:, :, 2] - X[:, 2:3] * dZ[:, :, 1],
                           X[:, 2:3] * dZ[:, :, 0] - X[:, 0:1] * dZ[:, :, 2],
                           X[:, 0:1] * dZ[:, :, 1] - X[:, 1:2] * dZ[:, :, 0]], 2)
        J = torch.cat([rot, dZ], 2)
        Jw = (J * wgt[:, None, None]).reshape(-1, 6)
        return (Jw.T @ J.reshape(-1, 6)).cpu(), (Jw.T @ r.reshape(-1)).cpu()

    state = project(q, t)
    cost = first = state[5]
    lam, fresh = 1e-3, True
    for _ in range(iterations):
        stop = False
        if fresh:
            A, g = normal(state)
            stop = float(g.norm()) < 1e-10
        step = -torch.linalg.solve(A + lam * torch.eye(6, dtype=_F64), g)
        if stop or float(step.norm()) < 1e-8:
            break
        th = float(step[:3].norm())
        d = torch.cat([torch.tensor([math.cos(th / 2)], dtype=_F64), step[:3] * (math.sin(th / 2) / th if th > 1e-6 else 0.5 - th * th / 48)])
        qn = torch.stack([q[0] * d[0] - q[1:] @ d[1:], *(q[0] * d[1:] + d[0] * q[1:] + _cross(q[1:], d[1:]))])
        tn = t + _matrix_of(q) @ step[3:]
        trial = project(qn, tn)
        if trial[5] < cost:
            q, t, cost, state, lam, fresh = qn, tn, trial[5], trial, max(1e-10, lam / 10), True
        else:
            lam, fresh = min(1e10, lam * 10), False
    return q, t, first, cost


def _estimate(f, case):
    """The whole estimate of one image: a dict of what its call returns."""
    n, B, forced = f.n, case.get("batch", 1000), case.get("forced", 0)
    K = f.K
    focal = 0.5 * (K[0] + K[1])
    tau2 = (_threshold(case) / focal) ** 2
    xn = torch.from_numpy((f.uv - K[2:]) / K[:2]).to(_DEV)
    X = torch.from_numpy(f.xyz).to(_DEV)
    rays = torch.cat([xn, torch.ones_like(xn[:, :1])], 1)
    rays = rays / rays.norm(dim=1, keepdim=True)
    best = {"score": math.inf, "count": 0, "sample": -1, "sol": -1, "P": None}
    drawn, hyps, ended = 0, 0, False
    need = 0
    while not ended:
        rounds = 1 if forced or not drawn else max(1, min((int(min(need, 100000)) - drawn) // B + 1, 4, 200000 // B))
        per = forced or B
        tr = torch.from_numpy(_triples(drawn, rounds * per, n, f.seed, case.get("prosac"))).to(_DEV)
        P, ok = _p3p(rays[tr], X[tr])
        at = ok.nonzero()
        score, count = _msac(P[ok], xn, X, tau2)
        sample, sol = at[:, 0].cpu().numpy(), (ok.cumsum(1) - 1)[ok].cpu().numpy()
        edge = np.searchsorted(sample, np.arange(rounds + 1) * per)
        for r in range(rounds):
            lo, hi = edge[r], edge[r + 1]
            hyps += int(hi - lo)
            if hi > lo:
                k = lo + int(np.argmin(score[lo:hi]))
                if score[k] < best["score"]:
                    best = {"score": float(score[k]), "count": int(count[k]), "sample": drawn + int(sample[k] - r * per),
                            "sol": int(sol[k]), "P": P[ok][k].cpu()}
            drawn += per
            w = best["count"] / n
            need = 3.0 * math.log(1.0 - 0.9999) / math.log(1.0 - w ** 3) if 0 < w < 1 else (math.inf if w <= 0 else 0)
            need = min(need if math.isinf(need) else math.ceil(need), 2 ** 31 - 1)
            if forced or drawn > need or drawn >= 100000:
                ended = True
                break  # samples of the group's later rounds are dropped
    q, t = _quat_of(best["P"][:, :3]), best["P"][:, 3]
    inl = _mask(q, t, xn, X, tau2)
    out = {"ransac_inliers": best["count"], "num_inliers": int(inl.sum()), "samples": drawn, "hypotheses": hyps,
           "best_sample": best["sample"], "best_solution": best["sol"], "model_score": best["score"],
           "inliers": inl.cpu().numpy().astype(np.uint8)}
    if forced:
        return dict(out, q=q.numpy(), t=t.numpy())
    u = torch.from_numpy(f.uv).to(_DEV)[inl] / focal
    q, t, c0, c1 = _refine(q, t, u, X[inl], [k / focal for k in K], 1.0 / focal)
    return dict(out, q=q.numpy(), t=t.numpy(), lm_initial_cost=c0, lm_cost=c1)


def exact(case, seed):
    kind = case["kind"]
    fr = _frames(case, seed)
    if kind in _ESTIMATES:
        rows = [_estimate(f, case) for f in fr]
        if kind == "plain":
            keys = ("q", "t", "inliers") + _WHOLE + _REAL[: 1 if case.get("forced") else 3]
            return {k: rows[0][k] for k in keys}
        out = _packed(rows)
        return dict(out, inliers=np.concatenate([r["inliers"] for r in rows])) if kind == "host" else out
    f = fr[0]
    q, t = (torch.from_numpy(v) for v in _prior(f, seed))
    X = torch.from_numpy(f.xyz).to(_DEV)
    if kind == "adjust":
        q, t, c0, c1 = _refine(q, t, torch.from_numpy(f.uv).to(_DEV), X, [float(k) for k in f.K], 1.0)
        return {"q": q.numpy(), "t": t.numpy(), "lm_initial_cost": c0, "lm_cost": c1}
    xn = torch.from_numpy((f.uv - f.K[2:]) / f.K[:2]).to(_DEV)
    return {"inliers": _mask(q, t, xn, X, (2 * DEFAULT_PX / (0.5 * (f.K[0] + f.K[1]))) ** 2).cpu().numpy().astype(np.uint8)}
