"""Performance cases: the work a user of the engine has it do, through its public entry points.

Kinds of case:

``host``      ``BiotSavart`` on NumPy arrays, the shed and the trailing call of one evaluation
              (``WInDS.m:150,153`` on all wake nodes, ``KuttaJoukowski.m:216,218`` on the
              lifting-line points): the MATLAB-style drop-in, every copy included.
``eval``      ``eval_device`` on torch tensors and the program's own stream, both families onto
              all wake nodes and lifting-line points: one induced-velocity evaluation of a solver
              that keeps its wake on the GPU.
``noalloc``   the same evaluation through ``winds_bs_eval_device_noalloc``, for hosts that own all
              device memory.
``step``      one time step of a ``WakeBatch`` (CUDA graph) with the lifting line at
              ``WInDS.m``'s settings (relax 0.25, tol 1e-8, maxiter 30), then the rotor loads and
              the new state, as a driver that keeps the history of the run reads them.
``kin``       ``kinematics``: positions, frames and velocities of a whole run's time series.
``train``     one training epoch of the bound-circulation network (Adam, batches of 4096).
``forward``   the network's prediction for many stations (validation sets).

The single-precision path (``f32c``) returns float64 arrays of single-precision accuracy: the
tiling the autotuner picks by timing already moves them by ~1e-7. A program that keeps them keeps
them in single precision, and so do these cases; everything else keeps its own type.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

wb = importlib.import_module("winds-master_b200")
synth = importlib.import_module("winds-master_b200.synth")
kin = importlib.import_module("winds-master_b200.kin")
mlp = importlib.import_module("winds-master_b200.mlp")
wake = importlib.import_module("winds-master_b200.wake")

CO = 1000.0  # user.co, the reach cut-off in metres (WInDS's default)
CUTOFF_D = 1e-4  # user.d of the cut-off core (WInDS's default)
RELAX, TOL, MAXITER = 0.25, 1e-8, 30  # user.relax, user.tol, user.maxiter
FEATURES, WIDTH, PAD = 11, 128, 16  # the network's inputs, hidden width and padded inputs


def listed():
    return [
        # a lifting-line call of KuttaJoukowski.m on the small wake: the smallest call there is,
        # made up to 30 times per step, all latency
        dict(name="host_lifting_line", kind="host", nst=17, steps=60, core="cutoff", at="line"),
        # the small wake's evaluation from the host (6k filaments onto 3.1k nodes)
        dict(name="host_small", kind="host", nst=17, steps=60, core="visc2", at="wake"),
        # the same wake held on the GPU
        dict(name="eval_small", kind="eval", nst=17, steps=60, core="visc2", precision="f32c"),
        # an ordinary wake of odd sizes with the reference's default core
        dict(name="eval_ragged", kind="eval", nst=29, steps=347, core="cutoff", precision="f32c"),
        # two revolutions at 1 degree, 1.55e10 interactions: the large wake
        dict(name="eval_large", kind="eval", nst=41, steps=720, core="visc2", precision="f32c"),
        # the double-precision sum, for runs that must follow the reference to the last digits
        dict(name="eval_double", kind="eval", nst=23, steps=181, core="visc2", precision="f64"),
        # no allocation, fixed scratch: a solver's per-step call
        dict(name="noalloc_medium", kind="noalloc", nst=21, steps=120, core="visc2", precision="f32c"),
        # one small rotor's step: launch latency and the lifting-line iteration
        dict(name="step_small", kind="step", rotors="17x60", core="cutoff", precision="f32c"),
        # uneven rotors stepped together
        dict(name="step_batch", kind="step", rotors="41x720,17x60,29x348,33x500,20x161,38x260,24x610,35x95",
             core="visc2", precision="f32c"),
        # the kinematics of 720 steps, once per run
        dict(name="kinematics", kind="kin", nst=41, steps=720),
        # training of the start value's network on some operating points' pairs
        dict(name="train_epoch", kind="train", rows=32768),
        # its prediction on a validation set, no multiple of any tile
        dict(name="forward_rows", kind="forward", rows=100003),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "eval", "eval", "eval", "noalloc", "step", "step", "kin", "train", "forward"])
    core = rng.choice(["visc2", "cutoff"])
    nst = rng.randint(9, 41)
    if kind == "host":
        return dict(kind=kind, nst=nst, steps=_log_int(rng, 24, 240), core=core, at=rng.choice(["wake", "line"]))
    if kind == "eval":
        double = rng.random() < 0.25
        return dict(kind=kind, nst=rng.randint(9, 29) if double else nst, steps=_log_int(rng, 24, 240 if double else 720),
                    core=core, precision="f64" if double else "f32c")
    if kind == "noalloc":
        return dict(kind=kind, nst=nst, steps=_log_int(rng, 24, 360), core=core, precision="f32c")
    if kind == "step":
        rotors, total = [], 0
        for _ in range(rng.randint(1, 8)):
            r = (rng.randint(13, 41), _log_int(rng, 40, 720))
            if total + _interactions(*r) <= 2.5e10:
                rotors.append("%dx%d" % r)
                total += _interactions(*r)
        return dict(kind=kind, rotors=",".join(rotors), core=core, precision="f32c")
    if kind == "kin":
        return dict(kind=kind, nst=nst, steps=_log_int(rng, 40, 900))
    return dict(kind=kind, rows=_log_int(rng, 2000, 33000 if kind == "train" else 110000))


# ------------------------------------------------------------------ inputs
def _core(case):
    return (wb.bs.CORE_VATISTAS, 2.0) if case["core"] == "visc2" else (wb.bs.CORE_CUTOFF, CUTOFF_D)


def _wake(case, seed):
    """A helical wake of two revolutions: (families, nodes, lifting-line points)."""
    w = synth.make_wake(synth.RotorCase(nst=case["nst"], nsteps=case["steps"], dpsi_deg=720.0 / case["steps"], seed=seed))
    fams = [synth.shed_filaments(w["dom"]) + (w["gamma_shed"], w["rc_shed"]),
            synth.trail_filaments(w["dom"]) + (w["gamma_trail"], w["rc_trail"])]
    return fams, w["dom"], w["ll"]


def _points(dom, ll):
    return np.asfortranarray(np.concatenate([synth.flat_points(dom), synth.flat_points(ll)]).reshape(-1, 3, 1, 1))


def _rotor_sizes(case):
    return [tuple(int(v) for v in r.split("x")) for r in case["rotors"].split(",")]


def _interactions(nst, steps, nb=3):
    na = steps + 1
    return (nst * na * nb) * ((nst - 1) * na * nb + nst * (na - 1) * nb)


def _step_rows(case):
    """Kinematics rows of a step case: enough for a long series of passes."""
    work = sum(2 * _interactions(*r) for r in _rotor_sizes(case))
    return int(min(8000, max(300, 6.0 / max(3e-4, work / 1.2e12))))


def _rotor(nst, steps, rows, seed):
    """One rotor turning steadily at an operating point of the seed: wake and lifting-line inputs
    of ``rows`` steps (one period of the rotor's motion, repeated)."""
    rng = np.random.default_rng(seed)
    U, tsr = rng.uniform(8.0, 14.0), rng.uniform(7.0, 9.0)
    rc = synth.RotorCase(nst=nst, nsteps=steps, dpsi_deg=720.0 / steps, U=U, omega_rpm=tsr * U / 63.0 * 30.0 / np.pi,
                         yaw_deg=rng.uniform(0.0, 30.0), shear=rng.uniform(0.0, 0.3), seed=seed, jitter=0.0)
    period = steps // 2 if steps % 2 == 0 else steps
    c = synth.make_wake_case(rc, nsteps=period, pitch_deg=4.0)
    k = synth.make_kj_case(rc, nsteps=period, pitch_deg=4.0, root_cut=0.2)
    at = np.arange(rows) % period
    c.update(nsteps=rows, quarter=c["quarter"][:, :, at], trailing=c["trailing"][:, :, at], wind=c["wind"][:, at])
    for f in ("ll", "bxn", "byn", "bzn", "vblade"):
        k[f] = k[f][:, :, at]
    k.update(azimuth=k["azimuth"][at], rpm=k["rpm"][at])
    return c, k


def _rotors(case, seed, rows):
    got = [_rotor(nst, steps, rows, 1000 * seed + i) for i, (nst, steps) in enumerate(_rotor_sizes(case))]
    return [c for c, _ in got], [k for _, k in got]


def _series(case, seed):
    rng = np.random.default_rng(seed)
    rc = synth.RotorCase(nst=case["nst"], nsteps=case["steps"], dpsi_deg=720.0 / case["steps"], seed=seed)
    return synth.rotor_series(rc, case["steps"], pitch_deg=rng.uniform(0.0, 5.0), nac_yaw_deg=rng.uniform(0.0, 20.0),
                              platform_motion=True, seed=seed)


def _network(case, seed):
    """Weights of the network's initial distribution, standardised features and a smooth target."""
    rng = np.random.default_rng(seed)
    parts = []
    for k in (PAD, WIDTH, WIDTH, WIDTH):
        w = rng.normal(0.0, 1.0 / math.sqrt(FEATURES if k == PAD else k), (WIDTH, k))
        w[:, FEATURES if k == PAD else k:] = 0.0
        parts += [w.ravel(), np.zeros(WIDTH)]
    parts += [rng.normal(0.0, 1.0 / math.sqrt(WIDTH), WIDTH), np.zeros(1)]
    theta = np.concatenate(parts).astype(np.float32)
    x = rng.normal(0.0, 1.0, (case["rows"], FEATURES)).astype(np.float32)
    t = (np.sin(x[:, 0]) + 0.3 * x[:, 5] * x[:, 8] - 0.2 * x[:, 9]).astype(np.float32)
    return theta, x, t


_STREAM = None


def _stream():
    """The program's one stream (the engine's scratch is shared by the calls of a device)."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def _device(a):
    return torch.from_numpy(np.asarray(a).ravel(order="F").copy()).cuda()


# ------------------------------------------------------------------ the program's side
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, kind=kind)
    if kind == "host":
        fams, dom, ll = _wake(case, seed)
        s.update(fams=fams, P=dom if case["at"] == "wake" else ll, d="visc2" if case["core"] == "visc2" else CUTOFF_D)
    elif kind in ("eval", "noalloc"):
        fams, dom, ll = _wake(case, seed)
        P = _points(dom, ll)
        core, d = _core(case)
        s.update(fams=[(_device(F1), _device(F2), _device(g), _device(rc), F1.shape) for F1, F2, g, rc in fams],
                 P=(_device(P), P.shape), core=core, d=d, out=torch.empty(P.size, dtype=torch.float64, device="cuda"),
                 stream=_stream())
        if kind == "eval":  # the first call, on the library's own stream, picks the size's tiling
            wb.eval_device(s["fams"], s["P"], core, d, CO, s["out"], case["precision"])
            wb.sync()
        else:
            fam = (wb.bs.Family * len(s["fams"]))()
            for f, (F1, F2, g, rc, dims) in zip(fam, s["fams"]):
                f.F1, f.F2, f.gamma, f.rc = (x.data_ptr() for x in (F1, F2, g, rc))
                f.dims[:] = list(dims)
            prm = wb.bs.Params(core, d, CO, wb.bs.PREC_F32C, 0)
            call = wb.lib().winds_bs_eval_device_noalloc
            call.argtypes = [ctypes.c_void_p, ctypes.c_int] + [ctypes.c_void_p] * 5
            s.update(call=call, args=(fam, len(s["fams"]), s["P"][0].data_ptr(), (ctypes.c_longlong * 4)(*P.shape),
                                      ctypes.byref(prm), s["out"].data_ptr(), s["stream"].cuda_stream), prm=prm)
        torch.cuda.synchronize()
    elif kind == "step":
        cases, kjs = _rotors(case, seed, _step_rows(case))
        b = wake.WakeBatch(cases, integrator="pcc", d="visc2" if case["core"] == "visc2" else CUTOFF_D, co=CO,
                           precision=case["precision"])
        b.set_kj(kjs, relax=RELAX, tol=TOL, maxiter=MAXITER)
        s.update(batch=b, n=len(cases))
    elif kind == "kin":
        s["series"] = _series(case, seed)
    else:
        theta, x, t = _network(case, seed)
        m = mlp.Mlp(FEATURES, seed=seed)
        for _ in range(2):  # the first call may convert weights to 16 bits before their upload has landed
            m.params = theta
        s.update(model=m, x=x, t=t, seed=seed)
    return s


def run(s):
    kind = s["kind"]
    if kind == "host":
        (a, La), (b, Lb) = (wb.BiotSavart(F1, F2, s["P"], g, rc, s["d"], CO, "full") for F1, F2, g, rc in s["fams"])
        return dict(uind=(a + b).astype(np.float32), lengths=[La, Lb])
    if kind == "eval":
        with torch.cuda.stream(s["stream"]):
            wb.eval_device(s["fams"], s["P"], s["core"], s["d"], CO, s["out"], s["case"]["precision"],
                           stream=s["stream"].cuda_stream)
            return s["out"].float() if s["case"]["precision"] == "f32c" else s["out"]
    if kind == "noalloc":
        with torch.cuda.stream(s["stream"]):
            if s["call"](*s["args"]) != 0:
                raise RuntimeError(wb.lib().winds_bs_last_error().decode())
            return s["out"].float()
    if kind == "step":
        b = s["batch"]
        b.step(1, graph=True)
        loads = b.loads()
        f = np.float32
        return dict(loads=[v.astype(f) for v in loads],
                    state=[{k: v.astype(f) for k, v in b.state(i).items()} for i in range(s["n"])])
    if kind == "kin":
        return kin.kinematics(s["series"])
    if kind == "train":
        loss = s["model"].train(s["x"], s["t"], epochs=1, batch=4096, lr=2e-3, seed=s["seed"])
        return dict(loss=loss, params=s["model"].params)
    return s["model"].forward(s["x"])


def work(case):
    """Bytes: every input read and every output written once. Operations: 52 per interaction with
    the Vatistas core and 44 with the cut-off core (FMA = 2; rsqrt and reciprocals not counted)."""
    kind = case["kind"]
    per = 52 if case.get("core") == "visc2" else 44
    if kind in ("host", "eval", "noalloc"):
        nst, na, nb = case["nst"], case["steps"] + 1, 3
        nf = (nst - 1) * na * nb + nst * (na - 1) * nb
        line = (nst - 1) * nb
        nt = nst * na * nb + line if kind != "host" else line if case["at"] == "line" else nst * na * nb
        return dict(bytes=8 * (8 * nf + 6 * nt), flops=per * nf * nt)
    if kind == "step":
        # the corrector's two evaluations and one of the lifting line; the iteration itself needs
        # only the filaments that follow the bound circulation
        flops = bytes_ = 0
        for nst, steps in _rotor_sizes(case):
            na, nb = steps + 1, 3
            nodes, line = nst * na * nb, (nst - 1) * nb
            nf = (nst - 1) * na * nb + nst * (na - 1) * nb
            own = nb * (2 * (nst - 1) + nst)
            flops += per * (2 * _interactions(nst, steps) + line * nf + MAXITER * line * own)
            bytes_ += 8 * (4 * 3 * nodes + 4 * nf)
        return dict(bytes=bytes_, flops=flops)
    if kind == "kin":
        n = 3 * case["steps"] * 3 * (6 * case["nst"] + 8 * (case["nst"] - 1))
        return dict(bytes=8 * n, flops=20 * n)
    macs = PAD * WIDTH + 3 * WIDTH * WIDTH + WIDTH
    return dict(bytes=4 * case["rows"] * (FEATURES + 1), flops=2 * macs * case["rows"] * (3 if kind == "train" else 1))


# ------------------------------------------------------------------ the same in 64 bits
def _t(a):
    return torch.from_numpy(np.array(a, dtype=np.float64, order="C")).to("cuda" if torch.cuda.is_available() else "cpu")


def _rows(a):
    """[n, 3, m, k] -> [n*m*k, 3], the first index fastest."""
    return a.permute(3, 2, 0, 1).reshape(-1, 3)


def _flat(a):
    return a.permute(2, 1, 0).reshape(-1)


def _induced(x1, x2, gamma, rc, p, core):
    """Velocity at p [n, 3] of the filaments x1 -> x2 with squared cores rc."""
    L = x2 - x1
    L2 = (L * L).sum(1)
    out = torch.empty_like(p)
    n = max(1, int(1.2e7) // max(1, len(x1)))
    for i in range(0, len(p), n):
        q = p[i:i + n]
        ax, ay, az = (q[:, c, None] - x1[None, :, c] for c in range(3))
        bx, by, bz = (q[:, c, None] - x2[None, :, c] for c in range(3))
        r1, r2 = torch.sqrt(ax * ax + ay * ay + az * az), torch.sqrt(bx * bx + by * by + bz * bz)
        cx, cy, cz = ay * bz - az * by, az * bx - ax * bz, ax * by - ay * bx
        rr = r1 * r2
        den = rr * (rr + ax * bx + ay * by + az * bz)
        u = gamma / (4 * math.pi) * (r1 + r2)
        if core == "visc2":
            h2 = (cx * cx + cy * cy + cz * cz) / L2
            u = u * h2 / torch.sqrt(rc * rc + h2 * h2) / den
        else:
            u = u / (den + CUTOFF_D * L2)
        u = torch.where(torch.isfinite(u) & ~((r1 > CO) & (r2 > CO)), u, torch.zeros_like(u))
        out[i:i + n] = torch.stack([(u * c).sum(1) for c in (cx, cy, cz)], 1)
    return out


def _family(F1, F2, gamma, rc):
    return _rows(F1), _rows(F2), _flat(gamma), _flat(rc)


def _like(u, shape):
    return u.reshape(shape[3], shape[2], shape[0], 3).permute(2, 3, 1, 0)


def _exact_wake(case, seed):
    fams, dom, ll = _wake(case, seed)
    P = _points(dom, ll) if case["kind"] != "host" else dom if case["at"] == "wake" else ll
    u = sum(_induced(*_family(_t(F1), _t(F2), _t(g)[:, 0], _t(rc)[:, 0]), _rows(_t(P)), case["core"]) for F1, F2, g, rc in fams)
    u = _like(u, P.shape).cpu().numpy()
    if case["kind"] != "host":
        return u.ravel(order="F")
    return dict(uind=u, lengths=[((F2 - F1) ** 2).sum(1, keepdims=True) for F1, F2, _, _ in fams])


def _book(bound, prev):
    """Trailing and shed circulation from the bound column and the trailing columns before it."""
    z = torch.zeros_like(bound[:1])
    trail = torch.cat([torch.diff(torch.cat([z, bound, z]), dim=0)[:, None], prev[:, :-1]], 1)
    c = torch.cumsum(trail[:-1], 0)
    return torch.cat([bound[:, None], torch.diff(torch.cat([c, torch.zeros_like(c[:, :1])], 1), dim=1)], 1), trail


def _lengths(dom):
    return [torch.sqrt((d * d).sum(1)) for d in (dom[1:] - dom[:-1], dom[:, :, :-1] - dom[:, :, 1:])]


def _exact_step(c, k, core):
    dom, quarter, trailing = _t(c["dom"]), _t(c["quarter"]), _t(c["trailing"])
    na, dt = c["na"], c["dt"]
    age = torch.arange(na, dtype=torch.float64, device=dom.device)[None, :, None] * dt
    grow = 4 * c["alpha"] * c["delta"] * c["nu"]

    def cores(shed, trail, new, old):
        rc = [(c["rc0"] ** 2 + grow * age) * torch.ones_like(shed), (c["rc0"] ** 2 + grow * (age[:, :-1] + 0.5 * dt)) * torch.ones_like(trail)]
        for r, a, b in zip(rc, new, old):
            a, b = torch.sqrt(a[:, 1:-1]), torch.sqrt(b[:, 1:-1])
            r[:, 1:-1] = r[:, 1:-1] / (1 + (a - b) / b)
        return rc

    def velocity(dom, shed, trail, rc, p):
        return (_induced(*_family(dom[:-1], dom[1:], shed, rc[0]), p, core)
                + _induced(*_family(dom[:, :, 1:], dom[:, :, :-1], trail, rc[1]), p, core))

    def wind(s, dom):
        f = (torch.clamp(c["hub_height"] + dom[:, 2], min=1e-3) / c["hub_height"]) ** c["shear"]
        return _t(c["wind"][:, s])[None, :, None, None] * f[:, None]

    prev, bound = torch.zeros_like(_t(c["trail_gamma"])), _t(c["bound"])
    prev[:, :-1] = _t(c["trail_gamma"])[:, 1:]
    shed, trail = _book(bound, prev)
    len0 = _lengths(dom)
    rc = cores(shed, trail, len0, len0)
    uind = _like(velocity(dom, shed, trail, rc, _rows(dom)), dom.shape)
    vel = wind(0, dom) + uind
    new = torch.empty_like(dom)
    new[:, :, 0], new[:, :, 1] = quarter[:, :, 1], trailing[:, :, 1]
    new[:, :, 2:] = dom[:, :, 1:-1] + dt * vel[:, :, 1:-1]
    shed1, trail1 = _book(bound, trail)
    u1 = _like(velocity(new, shed1, trail1, cores(shed1, trail1, _lengths(new), len0), _rows(new)), dom.shape)
    v1 = wind(1, new) + u1
    new[:, :, 2:] = dom[:, :, 1:-1] + dt / 2 * (v1[:, :, 2:] + vel[:, :, 1:-1])
    # the lifting line: the velocity is linear in the circulation of the two newest shed columns
    # and the newest trailing column, so these are summed apart from the rest at each iteration
    ll, vb = _t(k["ll"])[:, :, :1], _t(k["vblade"])[:, :, 0]
    frame = [_t(k[f])[:, :, 0] for f in ("bxn", "byn", "bzn")]
    vinf, chord = torch.sqrt((vb * vb).sum(1)), _t(k["chord"])[:, None]
    p = _rows(ll)
    own_s, own_t = shed.clone(), trail.clone()
    own_s[:, 2:], own_t[:, 1:] = 0, 0
    rest = velocity(dom, shed - own_s, trail - own_t, rc, p)
    first = torch.arange(len(bound) * bound.shape[1])
    foil, offs = np.asarray(k["foil"]), np.concatenate([[0], np.cumsum(k["foil_points"])])
    for _ in range(MAXITER):
        own = _induced(*_family(dom[:-1, :, :2], dom[1:, :, :2], shed[:, :2], rc[0][:, :2]), p, core)
        own = own + _induced(*_family(dom[:, :, 1:2], dom[:, :, :1], trail[:, :1], rc[1][:, :1]), p, core)
        u = _like(rest + own, ll.shape)[:, :, 0]
        tot = torch.stack([vb[:, a] + (frame[a] * u).sum(1) for a in range(3)], 1)
        aoa = torch.rad2deg(torch.atan2(-tot[:, 1], tot[:, 0])).cpu().numpy()
        cl, cd = np.empty_like(aoa), np.empty_like(aoa)
        for f in range(len(offs) - 1):
            a, b = offs[f], offs[f + 1]
            for to, table in ((cl, k["cl"]), (cd, k["cd"])):
                to[foil == f] = np.interp(aoa[foil == f], k["aoa"][a:b], table[a:b])
        gamma = 0.5 * vinf * chord * _t(cl)
        dg = gamma - bound
        bound = bound + RELAX * dg
        if float((dg / (gamma.abs() + 1)).abs().max()) <= TOL:
            break
        shed, trail = _book(bound, prev)
    shed, trail = _book(bound, prev)
    n = lambda a: a.cpu().numpy()  # noqa: E731
    state = dict(dom=n(new), bound=n(bound), shed=n(shed), trail=n(trail), rc_shed=n(rc[0]), rc_trail=n(rc[1]), uind=n(uind))
    return _loads(k, n(vb), cl, cd, aoa), state


def _loads(k, vb, cl, cd, aoa):
    """Rotor thrust, torque and power of one step."""
    th = np.degrees(k["twist"])[:, None]
    rot = np.radians(th - 90.0)
    v1 = -(np.cos(rot) * vb[:, 0] - np.sin(rot) * vb[:, 1])
    v2 = -(np.sin(rot) * vb[:, 0] + np.cos(rot) * vb[:, 1])
    phi = np.radians(aoa - th)
    tp = np.tan(phi)
    ratio = v2 / v1 / tp
    a = ratio * (v1 - tp * v2) / (ratio * v1 + tp * v2)
    w = (v1 * (1 - a)) ** 2 + (v2 * (1 + a / ratio)) ** 2
    q = 0.5 * k["rho"] * np.asarray(k["chord"])[:, None] * w * np.asarray(k["dr_station"])[:, None]
    torque = (q * (cl * np.sin(phi) - cd * np.cos(phi)) * np.asarray(k["r_station"])[:, None]).sum()
    return (q * (cl * np.cos(phi) + cd * np.sin(phi))).sum(), torque, math.pi / 30.0 * k["rpm"][0] * torque


def _rotation(axis, deg):
    a = np.radians(deg)
    c, s, o, z = np.cos(a), np.sin(a), np.ones_like(a), np.zeros_like(a)
    m = {"x": [[o, z, z], [z, c, -s], [z, s, c]], "y": [[c, z, s], [z, o, z], [-s, z, c]], "z": [[c, -s, z], [s, c, z], [z, z, o]]}[axis]
    return np.stack([np.stack(np.broadcast_arrays(*row), -1) for row in m], -2)


def _exact_kin(r):
    nt, nb = len(r["time"]), len(r["precone"])
    pf = r["ptfm"]
    tilt = np.radians(r["shaft_tilt"])
    hub0 = np.array([r["overhang"] * np.cos(tilt), 0.0, r["ptfm_ref"] + r["tower_ht"] + r["twr2shft"] + r["overhang"] * np.sin(tilt)])
    R = _rotation("z", r["nac_yaw"]) @ _rotation("x", pf[:, 3]) @ _rotation("y", pf[:, 4]) @ _rotation("z", pf[:, 5])
    hub = pf[:, :3] + R @ hub0
    out = dict(hub=hub)
    # rotations after the twist, blade by step: [nb, nt, 3, 3]
    A = _rotation("z", pf[:, 5]) @ _rotation("y", pf[:, 4]) @ _rotation("x", pf[:, 3]) @ _rotation("z", r["nac_yaw"]) @ _rotation("y", np.full(nt, float(r["shaft_tilt"]))) @ _rotation("x", r["azimuth"])
    B = np.stack([A @ _rotation("x", np.full(nt, 360.0 / nb * b)) @ _rotation("y", np.full(nt, float(r["precone"][b])))
                  @ _rotation("z", r["pitch"][:, b] + 90.0) for b in range(nb)])
    for name, x, at in (("lead", -0.25, "_trail"), ("quarter", 0.0, "_trail"), ("trail", 0.75, "_trail"),
                        ("bound", 0.0, ""), ("colloc", 0.25, ""), ("end", 0.75, "")):
        rad, ch, tw = (r["r_trail"], r["chord_trail"], r["twist_trail"]) if at else (r["r_nodes"], r["chord"], r["twist"])
        local = np.stack([x * ch, np.zeros_like(ch), rad], -1)
        local = (_rotation("z", tw) @ local[..., None])[..., 0]
        out[name] = np.einsum("btij,nj->nitb", B, local) + hub.T[None, :, :, None]
    for q, (o, tip) in dict(t=("quarter", "trail"), n=("bound", "end")).items():
        unit = lambda d: d / np.sqrt((d * d).sum(1, keepdims=True))  # noqa: E731
        bx, bz = unit(out[tip] - out[o]), unit(np.diff(out[o], axis=0))
        bz = np.concatenate([bz[:1], bz])
        out.update({"bx" + q: bx, "bz" + q: bz, "by" + q: np.cross(bz, bx, axis=1)})
    y, h = out["bound"], abs(np.mean(np.diff(r["time"])))
    d = np.empty_like(y)
    d[:, :, 0] = (-y[:, :, 2] + 4 * y[:, :, 1] - 3 * y[:, :, 0]) / (2 * h)
    d[:, :, 1] = (y[:, :, 2] - y[:, :, 0]) / (2 * h)
    d[:, :, 2:-2] = (-y[:, :, 4:] + 8 * y[:, :, 3:-1] - 8 * y[:, :, 1:-3] + y[:, :, :-4]) / (12 * h)
    d[:, :, -2] = (y[:, :, -1] - y[:, :, -3]) / (2 * h)
    d[:, :, -1] = (3 * y[:, :, -1] - 4 * y[:, :, -2] + y[:, :, -3]) / (2 * h)
    v = out["vbound"] = r["wind"].T[None, :, :, None] - d
    out["vblade"] = np.stack([(out[f] * v).sum(1) for f in ("bxn", "byn", "bzn")], 1)
    return out


def _exact_forward(theta, x):
    th, a = _t(theta), torch.nn.functional.pad(_t(x), (0, PAD - FEATURES))
    at = 0
    for k in (PAD, WIDTH, WIDTH, WIDTH):
        w, b = th[at:at + WIDTH * k].reshape(WIDTH, k), th[at + WIDTH * k:at + WIDTH * (k + 1)]
        a = torch.nn.functional.gelu(a @ w.T + b, approximate="tanh")
        at += WIDTH * (k + 1)
    return (a @ th[at:at + WIDTH] + th[at + WIDTH]).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("host", "eval", "noalloc"):
        return _exact_wake(case, seed)
    if kind == "step":
        cases, kjs = _rotors(case, seed, 4)
        got = [_exact_step(c, k, case["core"]) for c, k in zip(cases, kjs)]
        return dict(loads=[np.array(v) for v in zip(*(g[0] for g in got))], state=[g[1] for g in got])
    if kind == "kin":
        return _exact_kin(_series(case, seed))
    theta, x, _ = _network(case, seed)
    if kind == "forward":
        return _exact_forward(theta, x)
    return None  # the epoch's order of rows is the library's own
