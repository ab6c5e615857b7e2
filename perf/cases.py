"""The measured cases: the calls a user of the tracer makes, over their real
ranges, through the Python binding of the C ABI (cortrace.Context,
cortrace.Stream) and the learned window's network (window.Network).

  field    calculate_field at n GSM positions (`-m field`, probes along a line)
  dump     one trajectory's accepted steps (`-m trajectory`)
  scan     rigidity scans (`-m cutoff`): one INFILE, or a batch of sites,
           through a batch call or as segments of a scan stream
  forward  the window network's inference on n site-directions
  train    training steps of the window network on minibatches of n samples

Positions, sites, directions, epochs and solar-wind conditions are drawn from
the seed over the ranges the learned window trains on.  A scan's step limit
is the program's -s.  The default of 25,000 makes one call take half a minute
(its longest trajectories run to the limit one step after another), so the
cases take the same calls with a lower limit: the cost of a step does not
depend on it.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cor-model_gb300"))

import cortrace as ct  # noqa: E402
import window  # noqa: E402

EXTERNAL = {"igrf": ct.EXTERNAL_NONE, "t96": ct.EXTERNAL_T96, "ts05": ct.EXTERNAL_TS05, "chaos": ct.EXTERNAL_NONE}
# FP64 operations of one field evaluation and of one accepted step (its
# rejected trials included) in the models' own formulation
FIELD_FLOPS = {"igrf": 2700, "t96": 12500, "ts05": 26000, "chaos": 430000}
STEP_FLOPS = {"igrf": 3800, "t96": 13800, "ts05": 27000}
NET_MACS = 19 * 256 + 3 * 256 * 256 + 2 * 256


def listed():
    return [
        # a handful of probe points along a field line or an orbit pass
        {"name": "field_probe_t96", "kind": "field", "model": "t96", "n": 21},
        # the field on a 1-degree map at several altitudes, internal field alone
        {"name": "field_map_igrf", "kind": "field", "model": "igrf", "n": 500003},
        # `-m field` on the 5-degree global grid with a storm-time external field
        {"name": "field_grid_ts05", "kind": "field", "model": "ts05", "n": 2664},
        # the crustal field of degree 185 over a regional map
        {"name": "field_map_chaos", "kind": "field", "model": "chaos", "n": 40001},
        # `-m trajectory`: one particle's path, step by step
        {"name": "dump_t96", "kind": "dump", "model": "t96", "n": 1, "steps": 1000},
        # one INFILE of `-m cutoff` with the asymptotic directions, 0.05 GV steps
        {"name": "scan_site_igrf", "kind": "scan", "model": "igrf", "sites": 1, "rigidities": 400, "steps": 2500,
         "zenith": 0.0, "records": True, "via": "batch"},
        # one INFILE on the fine 0.01 GV grid with an external field
        {"name": "scan_site_t96", "kind": "scan", "model": "t96", "sites": 1, "rigidities": 2000, "steps": 1000,
         "zenith": 0.0, "records": True, "via": "batch"},
        # the IGRF-only workload: 228 sites by 400 rigidities
        {"name": "scan_batch_igrf", "kind": "scan", "model": "igrf", "sites": 228, "rigidities": 400, "steps": 1000,
         "zenith": 0.0, "records": False, "via": "batch"},
        # a slice of the global grid at 0.01 GV, as segments of a scan stream
        {"name": "stream_batch_t96", "kind": "scan", "model": "t96", "sites": 33, "rigidities": 2000, "steps": 250,
         "zenith": 0.0, "records": False, "via": "stream"},
        # a served storm request: inclined directions, TS05
        {"name": "scan_storm_ts05", "kind": "scan", "model": "ts05", "sites": 9, "rigidities": 397, "steps": 400,
         "zenith": 30.0, "records": False, "via": "batch"},
        # rigidity windows for the sites of the 5-degree grid
        {"name": "window_forward", "kind": "forward", "n": 2664},
        # the trainer's minibatch
        {"name": "window_train", "kind": "train", "n": 512, "steps": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["field", "field", "dump", "scan", "scan", "scan", "forward", "train"])
    if kind == "field":
        model = rng.choice(["igrf", "t96", "ts05", "chaos"])
        return {"kind": kind, "model": model,
                "n": _log_int(rng, 1, {"igrf": 500000, "t96": 200000, "ts05": 60000, "chaos": 40000}[model])}
    if kind == "dump":
        return {"kind": kind, "model": rng.choice(["igrf", "t96", "ts05"]), "n": rng.randint(1, 3),
                "steps": rng.randint(100, 1000)}
    if kind == "scan":
        model = rng.choice(["igrf", "t96", "ts05"])
        n = _log_int(rng, 100, {"igrf": 90000, "t96": 60000, "ts05": 8000}[model])
        sites = min(_log_int(rng, 1, 228), max(1, n // 50))
        return {"kind": kind, "model": model, "sites": sites, "rigidities": max(20, min(2000, n // sites)),
                "steps": rng.randint(100, {"igrf": 900, "t96": 250, "ts05": 250}[model]),
                "zenith": rng.choice([0.0, 30.0]), "records": rng.random() < 0.5 and n < 10000,
                "via": rng.choice(["batch", "batch", "stream"])}
    if kind == "forward":
        return {"kind": kind, "n": _log_int(rng, 1, 8192)}
    return {"kind": kind, "n": _log_int(rng, 64, 2048), "steps": rng.randint(2, 8)}


def _conditions(rng, model):
    external = "ts05" if model == "ts05" else "t96"
    c = window.sample_conditions(rng, 1, external)[0]
    return ct.internal_setup("igrf14", c["time7"], parmod=c["parmod"] if model in ("t96", "ts05") else None)


def _models(model):
    return ct.model_set(ct.INTERNAL_SH, EXTERNAL[model], ct.CRUSTAL_CHAOS if model == "chaos" else ct.CRUSTAL_NONE)


def _positions(rng, model, n):
    """GSM positions [m]: isotropic directions, 1 to 12 R_E (where
    trajectories run), the crustal field within 1.5 R_E."""
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    hi = 1.5 if model == "chaos" else 12.0
    return u * (np.exp(rng.uniform(math.log(1.003), math.log(hi), n)) * ct.DEF_RE)[:, None]


def _jobs(rng, case):
    n, jobs = case["rigidities"], []
    dele = 0.01 if n >= 1000 else 0.05
    for _ in range(case["sites"]):
        lat = math.degrees(math.asin(rng.uniform(-1.0, 1.0)))
        lon = rng.uniform(0.0, 360.0)
        the1, fi1 = window.arrival_direction(lat, lon, case["zenith"], 45.0 * int(rng.integers(0, 8)))
        jobs.append(ct.make_job(lat, lon, rig=dele, rk=dele * n, dele=dele, the1=the1, fi1=fi1))
    return np.concatenate(jobs)


def _samples(rng, n):
    x = rng.normal(size=(n, window.N_IN)).astype(np.float32)
    t = np.stack([x[:, 0] - 0.5 * x[:, 3] * x[:, 1], np.tanh(x[:, 2] + 0.3 * x[:, 8])], 1).astype(np.float32)
    return torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind in ("forward", "train"):
        s["net"] = window.Network(0, max_batch=case["n"])
        s["params"] = window.init_params(seed)
        s["net"].set_params(s["params"])
        s["batches"] = [_samples(rng, case["n"]) for _ in range(case.get("steps", 1))]
        return s
    s["params"] = _conditions(rng, case["model"])
    s["models"] = _models(case["model"])
    s["ctx"] = ct.Context(0)
    if kind == "field":
        s["pos"] = _positions(rng, case["model"], case["n"])
    elif kind == "dump":
        s["jobs"] = np.concatenate([
            ct.make_job(rng.uniform(-40.0, 40.0), rng.uniform(0.0, 360.0), rig=r, rk=r, dele=1.0)
            for r in rng.uniform(1.0, 6.0, case["n"])])
    else:
        s["jobs"] = _jobs(rng, case)
        if case["via"] == "stream":
            k = min(4, case["sites"])
            s["segments"] = [np.ascontiguousarray(s["jobs"][i::k]) for i in range(k)]
            most = max(len(j) for j in s["segments"])
            s["ctx"].set_queue_order(2)
            s["stream"] = ct.Stream(s["ctx"], s["models"], step_limit=case["steps"], slots=4, max_jobs=most,
                                    max_trajectories=most * case["rigidities"], max_params=1, fixed_params=4,
                                    pool_params=64, want_records=int(case["records"]))
    return s


def _scan_outputs(res):
    out = {k: res.sites[k].copy() for k in ("r_lower", "r_upper", "r_cutoff", "n_forbidden", "n_traj")}
    out["status"] = res.status
    out["accepted_steps"] = res.counters["accepted_steps"]
    if res.records is not None:
        out |= {k: res.records[k].copy() for k in ("pos", "vel", "time", "length", "steps", "trials")}
    return out


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "field":
        return s["ctx"].field_batch(s["pos"], s["params"], s["models"])
    if kind == "dump":
        res, paths = s["ctx"].trace_steps(s["jobs"], s["params"], s["models"], step_limit=case["steps"],
                                          capacity=case["steps"])
        out = _scan_outputs(res)
        for i, p in enumerate(paths):
            # up to the capacity asked for, zeros beyond the path's end (as the C call leaves them)
            pad = case["steps"] - len(p)
            out |= {f"{k}{i}": np.pad(p[k], [(0, pad)] + [(0, 0)] * (p[k].ndim - 1))
                    for k in ("gsm", "pos", "v", "time", "length", "step")}
        return out
    if kind == "scan" and case["via"] == "batch":
        return _scan_outputs(s["ctx"].trace_batch(s["jobs"], s["params"], s["models"], step_limit=case["steps"],
                                                  want_records=case["records"]))
    if kind == "scan":
        st = s["stream"]
        tickets = [st.submit(j, s["params"], want_records=case["records"]) for j in s["segments"]]
        got = [_scan_outputs(st.wait(t)[0]) for t in tickets]
        st.drain()
        return got
    if kind == "forward":
        return s["net"].forward(s["batches"][0][0])
    # from the state's initial weights, so that every pass is the same work
    s["net"].set_params(s["params"])
    losses = [s["net"].train_step(x, t, lr=1e-3) for x, t in s["batches"]]
    return {"loss": np.array(losses, np.float32), "weights": s["net"].get_params()}


def work(case):
    kind = case["kind"]
    if kind == "field":
        return {"bytes": 48 * case["n"], "flops": FIELD_FLOPS[case["model"]] * case["n"]}
    if kind == "dump":
        return {"bytes": 80 * case["steps"] * case["n"], "flops": STEP_FLOPS[case["model"]] * case["steps"] * case["n"]}
    if kind == "scan":
        n = case["sites"] * case["rigidities"]
        # mean accepted steps of a trajectory under the step limit
        mean = min(0.8 * case["steps"], 1300.0 * (case["steps"] / 25000.0) ** 0.36)
        return {"bytes": 88 * case["sites"] + (89 if case["records"] else 1) * n,
                "flops": STEP_FLOPS[case["model"]] * mean * n}
    passes = 2 if kind == "forward" else 6 * case["steps"]
    weights = 4 * window.N_PARAMS * (1 if kind == "forward" else 7 * case["steps"])
    return {"bytes": weights + 84 * case["n"] * case.get("steps", 1), "flops": float(passes) * NET_MACS * case["n"]}


# ---- in 64 bits, without the library's kernels ---------------------------------
def _rot(p):
    return np.stack([p["a1"][0], p["a2"][0], p["a3"][0]])     # rows: GEO -> GSM


def _internal(p, x):
    """The Schmidt-scaled internal field at GEO positions x [R_E], with the
    model's truncation by radius."""
    g, h, rec = (np.asarray(p[k][0], np.float64) for k in ("g", "h", "rec"))
    r = np.linalg.norm(x, axis=1)
    rho = np.hypot(x[:, 0], x[:, 1])
    c, s = x[:, 2] / r, rho / r
    cf, sf = x[:, 0] / rho, x[:, 1] / rho
    top = np.minimum(13, 3 + 30 // (r.astype(np.int64) + 2)) + 1
    br, bt, bf = np.zeros(len(x)), np.zeros(len(x)), np.zeros(len(x))
    pmm, dmm = np.ones(len(x)), np.zeros(len(x))
    for m in range(14):
        cm, sm = np.cos(m * np.arctan2(sf, cf)), np.sin(m * np.arctan2(sf, cf))
        q, z, p2, d2 = pmm, dmm, np.zeros(len(x)), np.zeros(len(x))
        for n in range(m + 1, 15):
            i = n * (n - 1) // 2 + m
            on = n <= top
            a = np.where(on, r ** -(n + 1.0), 0.0)
            w = g[i] * cm + h[i] * sm
            br += n * a * w * q
            bt -= a * w * z
            bf += m * a * (h[i] * cm - g[i] * sm) * -q
            q, z, p2, d2 = c * q - rec[i] * p2, c * z - s * q - rec[i] * d2, q, z
        dmm, pmm = s * dmm + c * pmm, s * pmm
    bphi = bf / s
    he = br * s + bt * c
    return np.stack([he * cf - bphi * sf, he * sf + bphi * cf, br * c - bt * s], 1)


def _net(params, batches, train, lr=1e-3, decay=1e-4):
    """The network in 64 bits: its forward pass, or training steps (mean
    squared error, AdamW) with the losses before each update."""
    w = [torch.from_numpy(a.astype(np.float64)).cuda().requires_grad_(train) for a in window.split_params(params)]
    mom = [[torch.zeros_like(a), torch.zeros_like(a)] for a in w]
    losses = []
    for k, (x, t) in enumerate(batches, 1):
        y = x.double()
        for i in range(0, len(w), 2):
            y = y @ w[i].T + w[i + 1]
            y = torch.nn.functional.silu(y) if i < len(w) - 2 else y
        if not train:
            return y
        loss = ((y - t.double()) ** 2).mean()
        grads = torch.autograd.grad(loss, w)
        losses.append(float(loss))
        with torch.no_grad():
            for a, g, mv in zip(w, grads, mom):
                mv[0].mul_(0.9).add_(0.1 * g)
                mv[1].mul_(0.999).add_(0.001 * g * g)
                step = (mv[0] / (1 - 0.9 ** k)) / ((mv[1] / (1 - 0.999 ** k)).sqrt() + 1e-8)
                a -= lr * (step + (decay * a if a.dim() == 2 else 0.0))
    return {"loss": np.array(losses), "weights": torch.cat([a.detach().reshape(-1) for a in w]).cpu().numpy()}


def exact(case, seed):
    """The internal field and the network in 64 bits.  The external models are
    defined by their own thousand lines of fitted terms, and a trajectory by
    every rounding on its way, so those have no value here."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "field" and case["model"] == "igrf":
        p = _conditions(rng, case["model"])
        a = _rot(p)
        return _internal(p, _positions(rng, case["model"], case["n"]) / ct.DEF_RE @ a)
    if case["kind"] in ("forward", "train"):
        batches = [_samples(rng, case["n"]) for _ in range(case.get("steps", 1))]
        return _net(window.init_params(seed), batches, case["kind"] == "train")
    return None
