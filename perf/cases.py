"""Timing cases of the tracking paths, as a program that uses the package
calls them.

Each case is one pass through a public entry point at a size of this
package's own configurations, tests and benchmark:

* fit       Kalman fit of device-resident tracks (Context.fit_device), 10
            layers: barrel cylinders, or "steered" with two cylinders and
            eight disks. 64 tracks is the smallest golden sample (launch
            latency), 320,000 the benchmark's step.
* fit_host  the same fit from and to host buffers (Context.fit_host).
* align     the differentiable fit: summed chi2 and its gradient with
            respect to the alignment and material parameters of every layer,
            forward and backward through autograd (AlignedFit.chi2).
* event     one CMS-2017 event found as a drop-in call does it
            (Finder.find_event): upload, clone-engine finding, all
            candidates back.
* batch     many events in one batch (upload_batch, run_graph,
            download_best): the benchmark's batched finding, its PU200-like
            finding, and ragged sizes between.
* iteration one tracking iteration with the steps after the finding: the
            batch, filters, backward fit, output selection, backward search
            and the best candidates back.
* clean     the cleaning of an iteration's seeds before the finding
            (seed_clean.clean_seeds).

The finder's contexts live as long as the process, as they do in a program
that takes one batch after the other; the inputs of every pass are uploaded
in that pass.
"""
import math

import numpy as np

FIND = dict(max_cands=6, chi2_cut=30.0, zero_c2=True)

# Tracks of a steered fit cross the two cylinders before the first disk.
STEERED_MASK = 0b1111111100


def listed():
    return [
        # The smallest fit: a handful of tracks, launch latency.
        {"name": "fit 64", "kind": "fit", "tracks": 64, "steered": False, "material": True,
         "chi2": True},
        # The benchmark's fit step: 16 events of 20,000 tracks.
        {"name": "fit 320000", "kind": "fit", "tracks": 320000, "steered": False,
         "material": True, "chi2": False},
        # Forward tracks: barrel and endcap (disk) steps in one fit.
        {"name": "fit steered 50021", "kind": "fit", "tracks": 50021, "steered": True,
         "material": True, "chi2": True},
        # One event's tracks from a host program without device buffers of its own.
        {"name": "fit host 20011", "kind": "fit_host", "tracks": 20011, "steered": False,
         "material": True, "chi2": True},
        # The differentiable fit, one gradient step: the benchmark's size ...
        {"name": "align 50000", "kind": "align", "tracks": 50000, "material": True},
        # ... and a small ragged sample without material.
        {"name": "align 3001", "kind": "align", "tracks": 3001, "material": False},
        # One small and one ordinary event through the drop-in call.
        {"name": "event 120", "kind": "event", "tracks": 120, "noise": 0.01, "iteration": 0},
        {"name": "event 800", "kind": "event", "tracks": 800, "noise": 0.01, "iteration": 0},
        # The benchmark's batch: 64 events of about 3000 tracks.
        {"name": "batch 64x3000", "kind": "batch", "events": 64, "tracks": 3000, "noise": 0.01,
         "ramp": 20.0, "pileup": False},
        # High pileup: 600,000 hits per event, twice as many noise hits as signal.
        {"name": "batch 4x10000 pileup", "kind": "batch", "events": 4, "tracks": 10000,
         "noise": 2.16, "ramp": 1.0, "pileup": True},
        # A whole iteration, detachedQuadStep: two quality filters, backward fit and search.
        {"name": "iteration 16x1500", "kind": "iteration", "events": 16, "tracks": 1500,
         "noise": 0.05, "iteration": 5},
        # The cleaning of an iteration's seeds, a fifth of them with near-duplicates.
        {"name": "clean 32x3000", "kind": "clean", "events": 32, "tracks": 3000, "noise": 0.01},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit_host", "align", "event", "batch", "batch", "iteration",
                       "clean"])
    if kind == "fit":
        return {"kind": "fit", "tracks": _log_int(rng, 33, 320000), "steered": rng.random() < 0.4,
                "material": rng.random() < 0.7, "chi2": rng.random() < 0.5}
    if kind == "fit_host":
        return {"kind": "fit_host", "tracks": _log_int(rng, 500, 60000), "steered": False,
                "material": rng.random() < 0.7, "chi2": rng.random() < 0.5}
    if kind == "align":
        return {"kind": "align", "tracks": _log_int(rng, 300, 50000),
                "material": rng.random() < 0.7}
    if kind == "event":
        return {"kind": "event", "tracks": _log_int(rng, 100, 4000),
                "noise": round(rng.uniform(0.0, 0.5), 3), "iteration": rng.choice([0, 1, 3, 6])}
    if kind == "batch":
        events = _log_int(rng, 2, 64)
        return {"kind": "batch", "events": events,
                "tracks": _log_int(rng, 300, min(10000, 150000 // events)),
                "noise": round(rng.uniform(0.0, 0.3), 3), "ramp": 1.0, "pileup": False}
    if kind == "clean":
        return {"kind": "clean", "events": _log_int(rng, 1, 32), "tracks": _log_int(rng, 200, 3000),
                "noise": 0.01}
    return {"kind": "iteration", "events": _log_int(rng, 1, 16), "tracks": _log_int(rng, 300, 1500),
            "noise": round(rng.uniform(0.0, 0.2), 3), "iteration": rng.choice([0, 2, 5, 9])}


# ------------------------------------------------------------------ inputs
def _fit_event(case, seed):
    from mkfit_b200 import synth
    if case.get("steered"):
        return synth.gen_fit_event_steered(case["tracks"], seed=seed)
    return synth.gen_fit_event(case["tracks"], seed=seed)


def _align_event(case, seed):
    """Toy tracks on a misaligned detector: layer offsets N(0, 20 um),
    material 1 +- 0.1 of nominal."""
    from mkfit_b200 import synth
    rng = np.random.default_rng(seed)
    return synth.gen_fit_event(case["tracks"], seed=seed, align_rphi=rng.normal(0, 0.002, 10),
                               align_z=rng.normal(0, 0.002, 10),
                               mat_scale=1 + rng.uniform(-0.1, 0.1, 10))


def _align_theta(seed):
    """Parameters of a step on the way to the minimum: a few microns and a
    percent from nominal."""
    rng = np.random.default_rng([seed, 1])
    t = np.zeros((10, 3), np.float32)
    t[:, :2] = rng.normal(0, 0.0005, (10, 2))
    t[:, 2] = 1 + rng.normal(0, 0.01, 10)
    return t


def _rotated(ev, angle):
    """The event turned about the beam line by `angle`: the layers and the
    material are the same all around, the hits' bins, modules and the seeds'
    directions are not."""
    from mkfit_b200.synth import CmsEvent
    c, s = math.cos(angle), math.sin(angle)
    d = dict(ev.__dict__)
    pos, err = ev.hit_pos.astype(np.float64), ev.hit_err.astype(np.float64)
    d["hit_pos"] = np.stack([c * pos[0] - s * pos[1], s * pos[0] + c * pos[1],
                             pos[2]]).astype(np.float32)
    xx, xy, yy, zx, zy, zz = err
    d["hit_err"] = np.stack([c * c * xx - 2 * c * s * xy + s * s * yy,
                             c * s * (xx - yy) + (c * c - s * s) * xy,
                             s * s * xx + 2 * c * s * xy + c * c * yy,
                             c * zx - s * zy, s * zx + c * zy, zz]).astype(np.float32)
    par = ev.seed_par.astype(np.float64)
    phi = np.mod(par[4] + angle + math.pi, 2 * math.pi) - math.pi
    d["seed_par"] = np.stack([c * par[0] - s * par[1], s * par[0] + c * par[1], par[2], par[3],
                              phi, par[5]]).astype(np.float32)
    return CmsEvent(**d)


# Events generated for one batch; the others are these, turned.
BASE_EVENTS = 2


def _seeds_kept(ev, n):
    """The event with its first `n` seeds."""
    from mkfit_b200.synth import CmsEvent
    assert ev.n_seeds >= n
    d = dict(ev.__dict__)
    for k in ("seed_par", "seed_err"):
        d[k] = np.ascontiguousarray(d[k][:, :n])
    for k in ("seed_chg", "seed_nhits", "seed_hit_layer", "seed_hit_index", "seed_mc"):
        d[k] = np.ascontiguousarray(d[k][:n])
    return CmsEvent(**d)


def _events(case, seed):
    """The case's events. The number of seeds of each event follows from the
    case alone (about `tracks`, uneven as Poisson counts are)."""
    from mkfit_b200 import synth
    from mkfit_b200.geometry import cms2017
    rng = np.random.default_rng([seed, 2])
    n_ev, pu, n = case.get("events", 1), case.get("pileup", False), case["tracks"]
    kw = dict(noise_frac=case["noise"])
    if case.get("ramp", 1.0) != 1.0:
        kw["noise_scale"] = synth.density_ramp(cms2017().n_layers, case["ramp"])
    if pu:
        kw.update(pt_range=(0.3, 50.0), eta_max=2.5)
    base = [synth.gen_cms_event(int(1.01 * n + 3 * math.sqrt(n)) + 10,
                                seed=1000 * (seed % (1 << 40)) + i, **kw)
            for i in range(min(n_ev, 1 if pu else BASE_EVENTS))]
    sizes = np.random.default_rng([n_ev, n]).normal(n, math.sqrt(n) / 2, n_ev)
    out = []
    for i in range(n_ev):
        ev = base[i % len(base)]
        if i >= len(base):
            ev = _rotated(ev, float(rng.uniform(-math.pi, math.pi)))
        k = n if n_ev == 1 else int(min(sizes[i], n + 1.5 * math.sqrt(n)))
        out.append(_seeds_kept(ev, k))
    return out


def _clean_seeds_in(case, seed):
    """Seeds with near-duplicates, 1.2 per track, of every event."""
    from mkfit_b200 import synth
    seeds, n = [], int(1.2 * case["tracks"])
    for i, e in enumerate(_events(case, seed)):
        s = synth.with_duplicate_seeds(_seeds_kept(e, min(e.n_seeds, case["tracks"])), frac=0.25,
                                       seed=seed + i)
        assert len(s["chg"]) >= n
        seeds.append({k: v[:, :n] if k in ("par", "err") else v[:n] for k, v in s.items()})
    return seeds


_kept = {}


def _context(kind):
    """The process's context of one kind of work."""
    if kind not in _kept:
        from mkfit_b200 import Context
        _kept[kind] = Context(0)
    return _kept[kind]


def _finder(iteration):
    key = ("finder", iteration)
    if key not in _kept:
        from mkfit_b200.finder import FindConfig, Finder
        _kept[key] = Finder(_context(key + ("context",)), FindConfig(iteration=iteration, **FIND))
    return _kept[key]


def prepare(case, seed):
    import torch
    from mkfit_b200 import FitBuffers, capi
    kind = case["kind"]
    if kind in ("fit", "fit_host"):
        ev = _fit_event(case, seed)
        steered = bool(case.get("steered"))
        ctx = _context(("fit", steered))
        ctx.set_material(ev.rl_grid, ev.xi_grid)
        args = dict(pflags=capi.PF_MATERIAL if case["material"] else capi.PF_NONE,
                    endcap_mask=STEERED_MASK if steered else 0, with_chi2=case["chi2"])
        if kind == "fit":
            return dict(kind=kind, ctx=ctx, dev=FitBuffers.upload(ev),
                        out=FitBuffers.outputs(ev.n), args=args)
        pin = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()  # noqa: E731
        n, nl = ev.n, ev.hit_pos.shape[0]
        # The layout the call takes without a copy: [3 | 6][layer, track].
        hp = pin(ev.hit_pos.transpose(1, 0, 2).reshape(3, nl * n)).reshape(3, nl, n)
        he = pin(ev.hit_err.transpose(1, 0, 2).reshape(6, nl * n)).reshape(6, nl, n)
        out = dict(par=pin(np.zeros((6, n), np.float32)), err=pin(np.zeros((21, n), np.float32)),
                   chg=pin(np.zeros(n, np.int32)), chi2=pin(np.zeros(n, np.float32)))
        return dict(kind=kind, ctx=ctx, ins=(pin(ev.par), pin(ev.err), pin(ev.chg),
                                             hp.transpose(1, 0, 2), he.transpose(1, 0, 2)),
                    out=out, args=args)
    if kind == "align":
        from mkfit_b200.align import AlignedFit
        ev = _align_event(case, seed)
        fit = AlignedFit(_context(("align", case["material"])), ev, material=case["material"])
        theta = torch.from_numpy(_align_theta(seed)).cuda().requires_grad_()
        return dict(kind=kind, fit=fit, theta=theta)
    from mkfit_b200.finder import output_arrays
    if kind == "event":
        return dict(kind=kind, finder=_finder(case["iteration"]), ev=_events(case, seed)[0])
    if kind == "clean":
        seeds = _clean_seeds_in(case, seed)
        begin = np.concatenate([[0], np.cumsum([len(s["chg"]) for s in seeds])]).astype(np.int32)
        cat = lambda k, ax: np.ascontiguousarray(  # noqa: E731
            np.concatenate([s[k] for s in seeds], axis=ax))
        return dict(kind=kind, ctx=_context("clean"),
                    ins=(begin, cat("par", 1), cat("chg", 0), cat("nhits", 0),
                         cat("hit_layer", 0), cat("hit_index", 0)))
    evs = _events(case, seed)
    return dict(kind=kind, finder=_finder(case.get("iteration", 0)), evs=evs,
                iteration=case.get("iteration", 0),
                out=output_arrays(sum(e.n_seeds for e in evs), 1))


# -------------------------------------------------------------------- pass
def run(state):
    kind = state["kind"]
    if kind == "fit":
        out, args = state["out"], state["args"]
        state["ctx"].fit_device(state["dev"], out, **args)
        return out if args["with_chi2"] else {k: out[k] for k in ("par", "err", "chg")}
    if kind == "fit_host":
        out, args = state["out"], state["args"]
        state["ctx"].fit_host(*state["ins"], out=out, **args)
        return out if args["with_chi2"] else {k: out[k] for k in ("par", "err", "chg")}
    if kind == "align":
        theta = state["theta"]
        theta.grad = None
        loss = state["fit"].chi2(theta)
        loss.backward()
        return {"chi2": loss.detach(), "grad": theta.grad}
    if kind == "clean":
        from mkfit_b200.seed_clean import clean_seeds
        keep, nhits, hit_layer, hit_index = clean_seeds(state["ctx"], *state["ins"])
        return {"keep": keep, "nhits": nhits, "hit_layer": hit_layer, "hit_index": hit_index}
    fnd = state["finder"]
    if kind == "event":
        return fnd.find_event(state["ev"])
    n = fnd.upload_batch(state["evs"])
    fnd.run_graph()
    if kind == "batch":
        return fnd.download_best(n, out=state["out"])
    selected = fnd.run_iteration_selection(n, iteration=state["iteration"])
    fnd.backward_search()
    return {"selected": selected, "best": fnd.download_best(n, out=state["out"])}


# -------------------------------------------------------------------- work
# FLOPs of the algorithm per unit: a fit step (propagation to the hit with
# its covariance and material, update), its adjoint, a candidate's
# propagation to a layer with the hit selection, a (candidate, hit)
# evaluation, an update.
FIT_STEP, ADJ_FWD, ADJ_BWD = 1130, 1181, 3768
LAYER_PROP, HIT_CHI2, UPDATE = 1000, 950, 1150


def work(case):
    n, kind = case["tracks"], case["kind"]
    if kind in ("fit", "fit_host"):
        # Per track: state in and out, chi2; per layer a hit and its index.
        return {"bytes": n * (2 * 112 + 10 * 40 + (4 if case["chi2"] else 0)),
                "flops": n * 10 * FIT_STEP}
    if kind == "align":
        return {"bytes": n * (112 + 10 * 40), "flops": n * 10 * (ADJ_FWD + ADJ_BWD)}
    if kind == "clean":
        # Per seed: state, charge, hit list in; verdict and merged hit list
        # out; its window against the seeds near it in eta.
        seeds = 1.2 * n * case["events"]
        return {"bytes": seeds * (24 + 8 + 32 + 8 + 128), "flops": seeds * (100 + 0.01 * n * 20)}
    # Finding: about 19 hits per track plus the noise; a track's seed of
    # three hits is followed over about 17 layers with a few candidates.
    # Bytes: hits (48 B with module and charge) and seeds (148 B) in, the
    # candidates out (a track state, its counters and its hits).
    n_ev = case.get("events", 1)
    hits = 19.2 * n * (1 + case["noise"] * (case.get("ramp", 1.0) ** 0.5))
    slots = FIND["max_cands"] if kind == "event" else 1
    by = n_ev * (48 * hits + n * (148 + slots * (37 * 4 + 512)))
    steps = 17 * n * n_ev
    pairs = 4.0 * (1 + case["noise"]) if case.get("pileup") else 1.5 * (1 + case["noise"])
    fl = steps * 4.0 * (LAYER_PROP + pairs * HIT_CHI2 + 0.6 * UPDATE)
    if kind == "iteration":
        fl += steps * UPDATE
    return {"bytes": float(by), "flops": float(fl)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("fit", "fit_host"):
        # State and covariance 1e-6, chi2 2e-5 off; an azimuth that falls on
        # the other side of +-pi moves by 2 pi (one in 320,000 tracks: 2e-4).
        return {"rel": 1e-3, "max": 0.9}
    if kind == "align":
        return {"rel": 4e-5}
    if kind == "clean":
        return "exact"  # verdicts and hit lists: whole numbers
    # Candidates: whole numbers apart from near-ties of scores and cuts, and
    # the states of the candidates that follow.
    return {"rel": 0.01, "max": 0.9, "differ": 0.005}


# ------------------------------------------------------------- 64-bit values
def _packed(C):
    return [C[:, i, j] for i in range(6) for j in range(i + 1)]


def _unpacked(e, k):
    """[k(k+1)/2][n] packed lower triangle -> [n][k][k]."""
    import torch
    rows, p = [[None] * k for _ in range(k)], 0
    for i in range(k):
        for j in range(i + 1):
            rows[i][j] = rows[j][i] = e[p]
            p += 1
    return torch.stack([torch.stack(r, -1) for r in rows], -2)


def _sincos4(x):
    x2 = x * x
    return x - 0.16666667 * x * x2, 1 - 0.5 * x2 + 0.04166667 * x2 * x2


def _to_r(p, k, r):
    """Helix to radius r in five steps with the Jacobian: (state, J, failed)."""
    import torch
    x0, y0, z0, ipt, phi, th = p
    kinv, pt = 1 / k, 1 / ipt
    r0 = torch.sqrt(x0 * x0 + y0 * y0)
    zero = torch.zeros_like(x0)
    cp, sp = torch.cos(phi), torch.sin(phi)
    px, py = cp * pt, sp * pt
    ddx, ddy, ddi, ddp, D = -x0 / r0, -y0 / r0, zero, zero, zero
    x, y = x0, y0
    fail = torch.zeros_like(x0, dtype=torch.bool)
    for it in range(5):
        r0 = torch.sqrt(x * x + y * y)
        o = r0 * pt / (px * x + py * y)
        bad = (o > 5) | (o < 0)
        fail = fail | bad
        step = torch.where(bad, zero, (r - r0) * o)
        D = D + step
        sh, ch = _sincos4(step * ipt * kinv * 0.5)
        ca, sa = 1 - 2 * sh * sh, 2 * sh * ch
        if it < 4:
            w = torch.where((r - r0).abs() < 1e-4, 1 / r0, zero)
            ax, ay, ai = -x * ipt * kinv * w, -y * ipt * kinv * w, step * kinv
            u, v = px * ca - py * sa, py * ca + px * sa
            ddx = ddx - (x * (1 + k * ax * u) + y * k * ax * v) * w
            ddy = ddy - (x * k * ay * u + y * (1 + k * ay * v)) * w
            t = ai * ipt
            ddi = ddi - k * (x * (u * t - v + py) + y * (v * t + u - px)) * pt * w
            ddp = ddp + k * (x * (py * sa - px + px * ca) - y * (px * sa - py + py * ca)) * w
        x, y = (x + 2 * k * sh * (px * ch - py * sh), y + 2 * k * sh * (py * ch + px * sh))
        px, py = px * ca - py * sa, py * ca + px * sa
    al = D * ipt * kinv
    dax, day = ddx * ipt * kinv, ddy * ipt * kinv
    dai, dap = (ipt * ddi + D) * kinv, ddp * ipt * kinv
    sa, ca = _sincos4(al)
    u, v = cp * ca - sp * sa, sp * ca + cp * sa
    sT, cT = torch.sin(th), torch.cos(th)
    one = torch.ones_like(x0)
    g = k * cT * pt / sT
    J = [[1 + k * dax * u * pt, k * day * u * pt, zero,
          k * (cp * (ipt * dai * ca - sa) + sp * ((1 - ca) - ipt * dai * sa)) * pt * pt,
          k * (dap * u - sp * sa + cp * ca - cp) * pt, zero],
         [k * dax * v * pt, 1 + k * day * v * pt, zero,
          k * (sp * (ipt * dai * ca - sa) + cp * (ipt * dai * sa - (1 - ca))) * pt * pt,
          k * (dap * v + sp * ca + cp * sa - sp) * pt, zero],
         [g * dax, g * day, one, g * (ipt * dai - al) * pt, g * dap, -k * al * pt / (sT * sT)],
         [zero, zero, zero, one, zero, zero],
         [dax, day, zero, dai, 1 + dap, zero],
         [zero, zero, zero, zero, zero, one]]
    J = torch.stack([torch.stack(r_, -1) for r_ in J], -2)
    return [x, y, z0 + g * al, ipt, phi + al, th], J, fail


def _to_z(p, k, z):
    """Helix to plane z with the Jacobian: (state, J)."""
    import torch
    x0, y0, z0, ipt, phi, th = p
    kinv, pt = 1 / k, 1 / ipt
    cp, sp, cT, sT = torch.cos(phi), torch.sin(phi), torch.cos(th), torch.sin(th)
    tT, ic2 = sT / cT, 1 / (cT * cT)
    px, py, dz = cp * pt, sp * pt, z - z0
    al = dz * tT * ipt * kinv
    sh, ch = _sincos4(al * 0.5)
    ca, sa = 1 - 2 * sh * sh, 2 * sh * ch
    u, v = px * ca - py * sa, py * ca + px * sa
    zero, one = torch.zeros_like(x0), torch.ones_like(x0)
    J = [[one, zero, -tT * ipt * u,
          k * pt * pt * (cp * (al * ca - sa) + sp * 2 * sh * (sh - al * ch)),
          -2 * k * pt * sh * (sp * ch + cp * sh), dz * ipt * u * ic2],
         [zero, one, -tT * ipt * v,
          k * pt * pt * (sp * (al * ca - sa) - cp * 2 * sh * (sh - al * ch)),
          2 * k * pt * sh * (cp * ch - sp * sh), dz * ipt * v * ic2],
         [zero] * 6, [zero, zero, zero, one, zero, zero],
         [zero, zero, -ipt * tT * kinv, tT * dz * kinv, one, ipt * dz * kinv * ic2],
         [zero, zero, zero, zero, zero, one]]
    J = torch.stack([torch.stack(r_, -1) for r_ in J], -2)
    return [x0 + 2 * k * sh * (px * ch - py * sh), y0 + 2 * k * sh * (py * ch + px * sh),
            z + zero, ipt, phi + al, th], J


def _material(rl, xi, sign, barrel, p, C):
    """Multiple scattering and energy loss of `rl` radiation lengths."""
    import torch
    th, mpi, me = p[5], 0.140, 0.0005
    on = rl >= 1e-13
    pt = 1 / p[3]
    mom = pt / torch.sin(th)
    p2 = mom * mom
    b2 = p2 / (p2 + mpi * mpi)
    beta = torch.sqrt(b2)
    inv_cos = mom / pt if barrel else 1 / torch.cos(th).abs()
    rl = torch.where(on, rl * inv_cos, torch.ones_like(rl))
    ms = (0.0136 * (1 + 0.038 * torch.log(rl)) / (beta * mom)) ** 2 * rl
    g2 = (p2 + mpi * mpi) / (mpi * mpi)
    gamma = torch.sqrt(g2)
    wmax = 2 * me * b2 * g2 / (1 + 2 * gamma * me / mpi + me * me / (mpi * mpi))
    ion = 16.0e-9 * 10.75
    dh = math.log(28.816e-9 * math.sqrt(2.33 * 0.498) / ion) + torch.log(beta * gamma) - 0.5
    dedx = 2 * (xi * inv_cos * (0.5 * torch.log(2 * me * b2 * g2 * wmax / (ion * ion)) - b2 - dh)
                / b2)
    dp = sign * dedx / beta
    add = torch.zeros_like(C)
    add[:, 3, 3] = dp * dp / (p2 * pt * pt)
    add[:, 4, 4] = ms
    add[:, 5, 5] = ms
    ipt = mom / (torch.clamp(mom + dp, min=0.001) * pt)
    return (p[:3] + [torch.where(on, ipt, p[3])] + p[4:],
            torch.where(on[:, None, None], C + add, C))


def _squash(phi):
    import torch
    phi = torch.where(phi >= math.pi, phi - 2 * math.pi, phi)
    return torch.where(phi < -math.pi, phi + 2 * math.pi, phi)


def _exact_fit(ev, mask, material, theta=None):
    """The fit of `ev`'s tracks in 64 bits: (state, covariance, chi2 per
    track); theta [steps][3]: hit shifts in r-phi and z, material scale."""
    import torch
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev, torch.float64)  # noqa: E731
    p = list(t(ev.par))
    C = _unpacked(t(ev.err), 6)
    k = t(ev.chg) * 100 / (-0.299792458 * 3.8112)
    grid = (t(ev.rl_grid), t(ev.xi_grid))
    chi2 = torch.zeros_like(k)
    for s in range(ev.hit_pos.shape[0]):
        m, M = list(t(ev.hit_pos[s])), _unpacked(t(ev.hit_err[s]), 3)
        scale = 1.0
        if theta is not None:
            rh = torch.sqrt(m[0] * m[0] + m[1] * m[1])
            m = [m[0] - theta[s, 0] * m[1] / rh, m[1] + theta[s, 0] * m[0] / rh,
                 m[2] + theta[s, 1]]
            scale = theta[s, 2]
        r = torch.sqrt(m[0] * m[0] + m[1] * m[1])
        endcap = bool((mask >> s) & 1)
        if endcap:
            q, J = _to_z(p, k, m[2])
            fail = torch.zeros_like(k, dtype=torch.bool)
            zm, rm = m[2], torch.sqrt(q[0] * q[0] + q[1] * q[1])
            sign = torch.where(m[2].abs() > p[2].abs(), 1.0, -1.0)
        else:
            q, J, fail = _to_r(p, k, r)
            zm, rm = q[2], r
            sign = torch.where(r * r > p[0] * p[0] + p[1] * p[1], 1.0, -1.0)
        Cm = C
        if material:
            zb, rb = zm.detach().abs().float().long(), rm.detach().float().long()
            on = (zb < 300) & (rb < 120) & ~fail
            at = (zb.clamp(max=299), rb.clamp(max=119))
            rl = torch.where(on, grid[0][at], torch.zeros_like(k)) * scale
            xi = torch.where(on, grid[1][at], torch.zeros_like(k)) * scale
            q, Cm = _material(rl, xi, sign, not endcap, q, C)
        q[4] = _squash(q[4])
        Cp = J @ Cm @ J.transpose(1, 2)
        p = [torch.where(fail, a, b) for a, b in zip(p, q)]
        C = torch.where(fail[:, None, None], C, Cp)
        zero, one = torch.zeros_like(k), torch.ones_like(k)
        if endcap:
            H = [[one, zero, zero], [zero, one, zero]]
        else:
            H = [[-(m[1] + p[1]) / (2 * r), (m[0] + p[0]) / (2 * r), zero], [zero, zero, one]]
        H = torch.stack([torch.stack(h, -1) for h in H], -2)
        res = (H @ torch.stack([a - b for a, b in zip(m, p)], -1)[:, :, None])
        S = H @ (C[:, :3, :3] + M) @ H.transpose(1, 2)
        det = S[:, 0, 0] * S[:, 1, 1] - S[:, 0, 1] * S[:, 1, 0]
        Si = torch.stack([torch.stack([S[:, 1, 1], -S[:, 0, 1]], -1),
                          torch.stack([-S[:, 1, 0], S[:, 0, 0]], -1)], -2) / det[:, None, None]
        chi2 = chi2 + (res.transpose(1, 2) @ Si @ res)[:, 0, 0]
        K = C[:, :, :3] @ H.transpose(1, 2) @ Si
        p = list((torch.stack(p, -1) + (K @ res)[:, :, 0]).unbind(-1))
        p[4] = _squash(p[4])
        C = C - K @ H @ C[:, :3, :]
    return p, C, chi2


def exact(case, seed):
    import torch
    kind = case["kind"]
    if kind in ("fit", "fit_host"):
        ev = _fit_event(case, seed)
        with torch.no_grad():
            p, C, chi2 = _exact_fit(ev, STEERED_MASK if case.get("steered") else 0,
                                    case["material"])
        out = dict(par=torch.stack(p), err=torch.stack(_packed(C)), chg=None)
        if case["chi2"]:
            out["chi2"] = chi2
        return out
    if kind == "align":
        ev = _align_event(case, seed)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        theta = torch.from_numpy(_align_theta(seed)).to(dev, torch.float64).requires_grad_()
        chi2 = _exact_fit(ev, 0, case["material"], theta)[2].sum()
        chi2.backward()
        return {"chi2": chi2.detach(), "grad": theta.grad}
    # A clone-engine finding in plain 64-bit torch takes minutes.
    return None
