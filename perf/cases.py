"""The work a user of this framework has it do, as measurable cases.

Sizes and options are those of this repository's documents, tests and
benchmark: the reference's default domain (100 x 100 x 30), the 512 x 512 x 60
hill, the 1024 x 1024 x 60 double hill, ensembles of uneven members between
64 x 64 and 256 x 192, the 256 x 256 x 40 surrogate domain, and the odd small
domains of the parity tests.  A domain's state is made here and uploaded
through the reference-layout arrays, as the Fortran driver's init does.

Kinds of case:
  loop      the time loop between two outputs: n steps (one moloch() call a
            step as the driver makes them, or one run() of the captured step),
            then t, ps and some of the updated state into arrays the program
            keeps
  coupled   a host model around the step: the whole state up from pinned
            arrays, one step, t and ps back
  ensemble  many uneven domains advanced together
  surrogate the learned acoustic cycle in the place of the sound() calls
  gradient  forward and backward of the surrogate's network on one batch
  advect    WAF advection of one field in memory the caller owns

Launch shapes: `tuned` cases apply the shapes an earlier autotune() found, as
a program that caches them does; the others construct the handle and step, as
the integration notes show.
"""
import ctypes
import math

import numpy as np
import torch

import dynamical_model_gb300 as dm

# shapes autotune() picks on GB300, cached by the caller
TUNED = {"fp32_mixed": [32, 760, 1, 8, 1], "fp64": [2, 6, 10, 4, 0]}
TUNED_ENSEMBLE = [32, 536, 1, 32, 0]
FETCH = ("u", "w", "pai", "qv")  # state read back beside t and ps


def _loop(name, jx, iy, kz, mode, steps, **kw):
    c = {"name": name, "kind": "loop", "jx": jx, "iy": iy, "kz": kz, "mode": mode, "steps": steps, "graph": False,
         "lprint": False, "tuned": False, "rotllr": 1, "filters": False, "hills": 1}
    c.update(kw)
    return c


def listed():
    return [
        # one printed step of a test-sized domain: launches and latency
        _loop("tiny_fp64", 24, 20, 12, "fp64", 1, lprint=True),
        # the driver's own defaults, its loop up to a printed step
        _loop("defaults_fp64", 100, 100, 30, "fp64", 10, lprint=True, hills=0),
        # the same domain in FP32 storage, replayed as a graph
        _loop("defaults_fp32", 100, 100, 30, "fp32_mixed", 20, graph=True, hills=0),
        # parity runs: reference evaluation order, map factors, all filters, odd sizes
        _loop("options_exact", 53, 47, 21, "fp64_exact", 2, rotllr=0, filters=True),
        # the plain FP64 step on a mid-sized hilly domain
        _loop("hill_fp64", 256, 256, 60, "fp64", 2, graph=True, tuned=True),
        # an ordinary FP32 run on a domain of no round size, one call a step
        _loop("ragged_fp32", 203, 157, 45, "fp32_mixed", 10),
        # the benchmarked domain
        _loop("hill_fp32", 512, 512, 60, "fp32_mixed", 10, graph=True, tuned=True),
        # the largest domain the repository runs
        _loop("hills_fp32", 1024, 1024, 60, "fp32_mixed", 8, graph=True, tuned=True, hills=2),
        # a host model coupled every step through pinned FP64 arrays
        {"name": "coupled_fp32", "kind": "coupled", "jx": 512, "iy": 512, "kz": 60, "mode": "fp32_mixed",
         "tuned": True, "hills": 1},
        # uneven members in one batched step
        {"name": "ensemble_fp32", "kind": "ensemble", "members": 12, "mode": "fp32_mixed", "steps": 4, "tuned": True},
        # inference of the acoustic-cycle network, every cycle committed
        {"name": "surrogate_fp32", "kind": "surrogate", "jx": 256, "iy": 256, "kz": 40, "steps": 2},
        # advection of one field by a caller with its own memory
        {"name": "advect_one", "kind": "advect", "jx": 160, "iy": 128, "kz": 64, "rotllr": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop"] * 6 + ["coupled", "ensemble", "surrogate", "gradient", "advect"])
    if kind == "advect":
        jx, iy, kz = _log(rng, 24, 256), _log(rng, 24, 256), rng.randint(12, 64)
        while jx * iy * kz > 1 << 21:
            jx, iy = jx * 3 // 4, iy * 3 // 4
        return {"kind": kind, "jx": jx, "iy": iy, "kz": kz, "rotllr": rng.randint(0, 1)}
    if kind == "gradient":
        return {"kind": kind, "kz": rng.choice([20, 30, 40, 60]), "batch": rng.choice([256, 512, 1024, 4096]),
                "layer": rng.randint(0, 3)}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(3, 16), "mode": rng.choice(["fp32_mixed", "fp32_mixed", "fp64"]),
                "steps": rng.randint(1, 4), "tuned": False}
    if kind == "surrogate":
        return {"kind": kind, "jx": _log(rng, 48, 320), "iy": _log(rng, 48, 320), "kz": rng.choice([20, 30, 40, 60]),
                "steps": rng.randint(1, 3)}
    mode = rng.choice(["fp32_mixed", "fp32_mixed", "fp64"])
    hi = 640 if mode == "fp32_mixed" else 200
    jx, iy = _log(rng, 24, hi), _log(rng, 24, hi)
    if rng.random() < 0.5:  # model domains are often multiples of 8
        jx, iy = (jx + 7) // 8 * 8, (iy + 7) // 8 * 8
    kz = rng.choice([12, 18, 30, 40, 45, 60, 64, 72])
    tuned = mode in TUNED and rng.random() < 0.5
    if kind == "coupled":
        return {"kind": kind, "jx": jx, "iy": iy, "kz": kz, "mode": mode, "tuned": tuned, "hills": 1}
    c = _loop("", jx, iy, kz, mode, rng.randint(1, 6), graph=rng.random() < 0.5, lprint=rng.random() < 0.5,
              tuned=tuned, rotllr=rng.choice([1, 1, 1, 0]), filters=rng.random() < 0.15, hills=rng.randint(0, 2))
    del c["name"]
    return c


# ---- the state of a domain, FP64, arrays (k, i, j) ---------------------------
ZTOP, ZH, DX, DT, NADV, NSOUND, ANU2 = 36000.0, 12000.0, 3000.0, 30.0, 3, 5, 0.6
G, RGAS_MOL, AMD, AMW = 9.80665, 6.02214076e23 * 1.3806490e-23, 28.96454, 18.01528
RGAS, RWAT = RGAS_MOL / AMD * 1000.0, RGAS_MOL / AMW * 1000.0
CPD, CVD, P00, LRATE, TZERO, WLHV = 3.5 * RGAS, 2.5 * RGAS, 1.0e5, 0.00649, 273.15, 2500610.0
RDRCV, CPOVR, EP1, EP2 = RGAS / CVD, CPD / RGAS, AMD / AMW - 1.0, AMW / AMD
EOMEG2 = 2.0 * 7.2921159e-5


def _gzita(r):
    return -3.0 * r ** 2 + 2.0 * r ** 3 + 1.0


def _state(jx, iy, kz, seed, hills, rotllr=1, amp=0.5, wind=6.0):
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def rand(*shape):
        return 2.0 * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) - 1.0

    def f64(x):
        return torch.as_tensor(x, dtype=torch.float64, device="cuda")

    i, j = torch.meshgrid(torch.arange(1, iy + 1, device="cuda"), torch.arange(1, jx + 1, device="cuda"), indexing="ij")
    ht = torch.zeros(iy, jx, dtype=torch.float64, device="cuda")
    for n in range(hills):
        cj, ci = jx * (n + 1) / (hills + 1), iy * (n + 1) / (hills + 1)
        r = max(3.0, min(20.0, 0.12 * min(jx, iy)))
        ht += min(500.0 * hills, 100.0 * r) * torch.exp(-((j - cj) ** 2 + (i - ci) ** 2) / (r * r))
    dz = ZTOP / kz
    zita = torch.arange(kz, -1, -1, device="cuda", dtype=torch.float64) * dz
    zitah = (torch.arange(kz - 1, -1, -1, device="cuda", dtype=torch.float64) + 0.5) * dz
    zfz = ZTOP / (math.exp(ZTOP / ZH) - 1.0)

    def fm(z):
        r = (z / ZTOP)[:, None, None]
        return 1.0 / ((-6.0 * r + 6.0 * r * r) / ZTOP * ht + (zfz * torch.exp(z / ZH) / ZH)[:, None, None])

    s = {"zita": zita, "zitah": zitah, "fmz": fm(zitah), "fmzf": fm(zita),
         "zeta": ht * (_gzita(zitah / ZTOP)[:, None, None] - 1.0) + (zfz * (torch.exp(zitah / ZH) - 1.0))[:, None, None]}
    s["hx"] = (ht - torch.roll(ht, 1, 1)) / DX
    s["hy"] = (ht - torch.roll(ht, 1, 0)) / DX
    skew = 0.0 if rotllr else 0.05
    for n in ("msfx", "msfu", "msfv"):
        s[n] = 1.0 + skew * rand(iy, jx)
    s["ulat"] = 45.0 + 3.0 * rand(1, 1) + 0.01 * i
    s["vlat"] = s["ulat"] - 0.005
    z = s["zeta"]
    s["qv"] = torch.where(z < 15000.0, 0.018 * torch.exp(-z / 4000.0), f64(1.0e-8))
    s["qv"] *= 1.0 + 0.02 * rand(kz, iy, jx)
    t = torch.where(z < 15000.0, 300.0 - LRATE * z, f64(300.0 - LRATE * 15000.0))
    # hydrostatic Exner function from the ground up
    tv = t * (1.0 + EP1 * s["qv"])
    pai = torch.empty_like(t)
    ps = 101480.0
    pai[-1] = (ps * torch.exp(-G * z[-1] / (RGAS * tv[-1])) / P00) ** (RGAS / CPD)
    for k in range(kz - 2, -1, -1):
        th = 0.5 * (tv[k + 1] / pai[k + 1] + tv[k] / (pai[k + 1] - G * (z[k] - z[k + 1]) / (CPD * tv[k] / pai[k + 1])))
        pai[k] = pai[k + 1] - G * (z[k] - z[k + 1]) / (CPD * th)
    low = min(10, kz)
    t[kz - low:] += amp * rand(low, iy, jx) * pai[kz - low:]
    s["t"], s["pai"] = t, pai
    blob = torch.exp(-((j - jx / 2) ** 2 + (i - iy / 2) ** 2) / (0.2 * min(jx, iy)) ** 2) * torch.exp(-((z - 3000.0) / 1500.0) ** 2)
    s["qc"], s["qr"] = 3.0e-4 * blob, 1.0e-4 * blob
    s["qi"], s["qs"] = torch.zeros_like(t), torch.zeros_like(t)
    s["u"] = wind * rand(1, 1, 1) + 0.1 * rand(kz, iy, jx)
    s["v"] = wind * rand(1, 1, 1) + 0.1 * rand(kz, iy, jx)
    s["w"] = torch.zeros(kz + 1, iy, jx, dtype=torch.float64, device="cuda")
    return s


def _host(name, a, jx, iy, kz):
    """Reference-layout host array (Fortran order, halo rings as periodic images) of an interior (k, i, j)."""
    if a.dim() == 1:
        return a.cpu().numpy()
    b = dm.field_bounds(name, jx, iy, kz)
    jj = (torch.arange(b[0][0], b[0][1] + 1, device=a.device) - 1) % jx
    ii = (torch.arange(b[1][0], b[1][1] + 1, device=a.device) - 1) % iy
    a = a.index_select(-1, jj).index_select(-2, ii)
    out = np.empty(tuple(reversed(a.shape)), order="F")
    torch.from_numpy(out.T).copy_(a)
    return out


STATICS = ("zita", "zitah", "msfx", "msfu", "msfv", "hx", "hy", "ulat", "vlat", "zeta", "fmz", "fmzf")
TRACERS = ("qv", "qc", "qi", "qr", "qs")


def _model(case, st, stream=None):
    jx, iy, kz = case["jx"], case["iy"], case["kz"]
    opts = {}
    if case.get("filters"):
        opts = {"mo_divfilter": 1, "do_filterpai": 1, "do_filtertheta": 1}
    m = dm.Moloch(jx, iy, kz, mode=case["mode"], stream=stream, rotllr=case.get("rotllr", 1), **opts)
    arrays = {n: _host(n, st[n], jx, iy, kz) for n in ("u", "v", "w", "pai", "t")}
    arrays["qx"] = _host("qx", torch.stack([st[n] for n in TRACERS]), jx, iy, kz)
    for n in STATICS:
        m.upload(n, _host(n, st[n], jx, iy, kz))
    for n, a in arrays.items():
        m.upload(n, a)
    m.init()
    if case.get("tuned"):
        m.set_tuning(TUNED[case["mode"]])
    return m, arrays


def _empty(name, jx, iy, kz):
    return np.zeros([u - l + 1 for l, u in dm.field_bounds(name, jx, iy, kz)], order="F")


class _Outputs:
    """The arrays a program keeps for its output, FP64 as the interface has them; FP32 runs write single precision."""

    def __init__(self, m, fields):
        self.m, self.single = m, m.params.mode == dm.FP32_MIXED
        self.a = {n: _empty(n, m.jx, m.iy, m.kz) for n in ("t", "ps") + fields}
        for n in ("t", "ps"):  # pinned once, as the integration notes do
            m.host_register(self.a[n])
        self.ptr = {n: (dm.FIELD[n], self.a[n].ctypes.data_as(ctypes.POINTER(ctypes.c_double)))
                    + tuple((ctypes.c_int * 4)(*[x[q] for x in dm.field_bounds(n, m.jx, m.iy, m.kz)]) for q in (0, 1))
                    for n in fields}
        if self.single:
            self.f = {n: torch.empty(a.T.shape, dtype=torch.float32) for n, a in self.a.items()}

    def fetch(self):
        m = self.m
        m.output_start()
        for n, (f, p, lb, ub) in self.ptr.items():
            rc = m.L.moloch_gpu_download(m.h, f, p, lb, ub)
            if rc:
                raise dm.MolochError(rc, m.L.moloch_gpu_last_error().decode())
        m.output_finish(self.a["t"], self.a["ps"])
        if not self.single:
            return {n: torch.from_numpy(a.T) for n, a in self.a.items()}
        return {n: self.f[n].copy_(torch.from_numpy(a.T)) for n, a in self.a.items()}


def _members(case, seed):
    """Uneven members, sizes from the member's number alone (64..256 x 64..192, 30, 40 or 60 levels)."""
    r = np.random.RandomState(7)
    out = []
    for n in range(case["members"]):
        jx, iy, kz = int(r.randint(64, 257)), int(r.randint(64, 193)), int(r.choice([30, 40, 60]))
        if case["mode"] == "fp64":
            jx, iy = (jx + 1) // 2, (iy + 1) // 2
        out.append({"jx": jx, "iy": iy, "kz": kz, "mode": case["mode"], "seed": int(seed) * 100 + n})
    return out


def _member_state(c):
    return _state(c["jx"], c["iy"], c["kz"], c["seed"], 0, amp=1.0, wind=10.0)


def _network(kz, seed):
    """A trained network's parameters stand-in: seeded weights and the normalisation of a typical state."""
    kin, nop = -(-45 * kz // 64) * 64, -(-5 * kz // 64) * 64
    r = np.random.RandomState(seed % (1 << 31))
    dims = [(kin, 256), (256, 256), (256, 256), (256, nop)]
    layers = [((r.standard_normal((o, i)) / math.sqrt(i)).astype(np.float32), (0.1 * r.standard_normal(o)).astype(np.float32))
              for i, o in dims]
    mean = np.array([0.0, 0.0, 0.0, 0.7, 400.0], np.float32)[:, None].repeat(kz, 1)
    std = np.array([6.0, 6.0, 0.5, 0.3, 120.0], np.float32)[:, None].repeat(kz, 1)
    ystd = np.array([1e-3, 1e-3, 1e-3, 1e-7, 1e-3], np.float32)[:, None].repeat(kz, 1)
    return layers, mean, std, np.zeros_like(mean), ystd


def _surrogate(kz, seed, **kw):
    layers, xm, xs, ym, ys = _network(kz, seed)
    sur = dm.Surrogate(kz, seed=1, **kw)
    for n, (w, b) in enumerate(layers):
        sur.set_param(n, w, b)
    sur.set_stats(xm, xs, ym, ys)
    return sur


def _batch(case, seed):
    kin, nop = -(-45 * case["kz"] // 64) * 64, -(-5 * case["kz"] // 64) * 64
    r = np.random.RandomState((seed + 17) % (1 << 31))
    x = r.standard_normal((case["batch"], kin)).astype(np.float32)
    t = r.standard_normal((case["batch"], nop)).astype(np.float32)
    x[:, 45 * case["kz"]:] = 0.0
    t[:, 5 * case["kz"]:] = 0.0
    return x, t


def _field(case, seed):
    """Inputs of the one-field advection: a field, s, winds and metric terms."""
    st = _state(case["jx"], case["iy"], case["kz"], seed, 1, case["rotllr"])
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 5)
    s = 0.4 * torch.randn(case["kz"] + 1, case["iy"], case["jx"], generator=g, device="cuda", dtype=torch.float64)
    s[0], s[-1] = 0.0, 0.0
    u, v = (x + 4.0 * torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64) for x in (st["u"], st["v"]))
    return {"pp": (st["t"] / st["pai"]).contiguous(), "s": s, "u": u, "v": v, **{n: st[n].contiguous() for n in
            ("fmz", "fmzf", "msfu", "msfv", "msfx")}}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "loop":
        st = _state(case["jx"], case["iy"], case["kz"], seed, case["hills"], case["rotllr"])
        m, _ = _model(case, st)
        return {"case": case, "m": m, "out": _Outputs(m, FETCH)}
    if kind == "coupled":
        m, arrays = _model(case, _state(case["jx"], case["iy"], case["kz"], seed, case["hills"]))
        for a in arrays.values():
            m.host_register(a)
        return {"case": case, "m": m, "in": arrays, "out": _Outputs(m, ())}
    if kind == "ensemble":
        stream = torch.cuda.Stream()
        ms = [_model(c, _member_state(c), stream.cuda_stream)[0] for c in _members(case, seed)]
        ens = dm.Ensemble(ms)
        if case["tuned"]:
            ens.set_tuning(TUNED_ENSEMBLE)
        return {"case": case, "stream": stream, "ens": ens, "out": [_Outputs(m, ("u",)) for m in ms]}
    if kind == "surrogate":
        m, _ = _model(dict(case, mode="fp32_mixed"), _state(case["jx"], case["iy"], case["kz"], seed, 1))
        sur = _surrogate(case["kz"], seed, capacity=256, batch=128)
        sur.attach(m, threshold=1e30, judge_every=0)
        return {"case": case, "m": m, "sur": sur, "out": _Outputs(m, FETCH)}
    if kind == "gradient":
        x, t = _batch(case, seed)
        return {"case": case, "sur": _surrogate(case["kz"], seed, capacity=2 * case["batch"], batch=case["batch"]), "x": x, "t": t}
    return {"case": case, "f": _field(case, seed), "L": dm.lib()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "loop":
        m, d = state["m"], None
        if case["graph"]:
            m.run(case["steps"] - case["lprint"])
            if case["lprint"]:
                d = m.moloch(case["steps"], lprint=True)
        else:
            for i in range(1, case["steps"] + 1):
                d = m.moloch(i, lprint=case["lprint"] and i == case["steps"])
        out = state["out"].fetch()
        if d is not None:
            out["diag"] = np.array([d.maxps, d.minps, d.maxu, d.minu, d.maxv, d.minv, d.mass, d.energy],
                                   np.float32 if case["mode"] == "fp32_mixed" else np.float64)
        return out
    if kind == "coupled":
        m = state["m"]
        for n, a in state["in"].items():
            m.upload(n, a)
        m.moloch(1)
        return state["out"].fetch()
    if kind == "ensemble":
        state["ens"].run(case["steps"])
        return [o.fetch() for o in state["out"]]
    if kind == "surrogate":
        state["m"].run(case["steps"])
        return state["out"].fetch()
    if kind == "gradient":
        loss, gw, gb = state["sur"].gradients(state["x"], state["t"], case["layer"])
        return {"loss": np.float32(loss), "gw": gw, "gb": gb}
    f = state["f"]
    pp = f["pp"].clone()
    rc = state["L"].moloch_gpu_wafone_noalloc(
        pp.data_ptr(), *[f[n].data_ptr() for n in ("s", "u", "v", "fmz", "fmzf", "msfu", "msfv", "msfx")],
        case["jx"], case["iy"], case["kz"], DT / NADV, DX, ZTOP / case["kz"], case["rotllr"],
        torch.cuda.current_stream().cuda_stream)
    if rc:
        raise dm.MolochError(rc, state["L"].moloch_gpu_last_error().decode())
    return pp


# ---- what a pass cannot do without ------------------------------------------
STEP_WORDS = 28     # u v w pai t and five tracers in and out, zeta fmz fmzf in, p qsat tvirt rho tetav out
WAF_FLOPS = 4 * 11  # four one-dimensional passes of one field at a point
STEP_FLOPS = NADV * (NSOUND * 110 + 10 * WAF_FLOPS + 40) + 150


def _step_work(jx, iy, kz, mode, steps, fields):
    n, e = jx * iy * kz, 4 if mode == "fp32_mixed" else 8
    return {"bytes": steps * STEP_WORDS * n * e + fields * n * 8, "flops": steps * STEP_FLOPS * n}


def work(case):
    kind = case["kind"]
    if kind == "loop":
        return _step_work(case["jx"], case["iy"], case["kz"], case["mode"], case["steps"], 1 + len(FETCH))
    if kind == "coupled":
        return _step_work(case["jx"], case["iy"], case["kz"], case["mode"], 1, 11)
    if kind == "ensemble":
        w = [_step_work(c["jx"], c["iy"], c["kz"], c["mode"], case["steps"], 2) for c in _members(case, 0)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    if kind == "gradient":
        kin, nop, b = -(-45 * case["kz"] // 64) * 64, -(-5 * case["kz"] // 64) * 64, case["batch"]
        par = kin * 256 + 2 * 256 * 256 + 256 * nop
        return {"bytes": 4 * b * (kin + nop) + 2 * par + 4 * (kin, 256, 256, nop)[case["layer"]] * 256,
                "flops": 2 * b * (par + par + par - kin * 256)}
    n = case["jx"] * case["iy"] * case["kz"]
    if kind == "surrogate":
        kz, cols = case["kz"], case["jx"] * case["iy"]
        kin, nop = -(-45 * kz // 64) * 64, -(-5 * kz // 64) * 64
        w = _step_work(case["jx"], case["iy"], kz, "fp32_mixed", case["steps"], 1 + len(FETCH))
        net = 2 * cols * (kin * 256 + 2 * 256 * 256 + 256 * nop)
        w["flops"] += case["steps"] * NADV * (net - NSOUND * 110 * n)
        return w
    return {"bytes": 8 * n * 7, "flops": (WAF_FLOPS + 30) * n}


# ---- the same in plain 64-bit torch ------------------------------------------
def _W(a):
    return torch.roll(a, 1, -1)


def _E(a):
    return torch.roll(a, -1, -1)


def _S(a):
    return torch.roll(a, 1, -2)


def _N(a):
    return torch.roll(a, -1, -2)


def _pfwsat(t, p):
    td = (t - TZERO).clamp(-75.0, 100.0)
    aw = (0.611213476e+03, 0.444007856e+02, 0.143064234e+01, 0.264461437e-01, 0.305903558e-03,
          0.196237241e-05, 0.892344772e-08, -0.373208410e-10, 0.209339997e-13)
    ci = (0.611123516e+03, 0.503109514e+02, 0.188369801e+01, 0.420547422e-01, 0.614396778e-03,
          0.602780717e-05, 0.387940929e-07, 0.149436277e-09, 0.262655803e-12)

    def horner(c):
        acc = torch.full_like(td, c[8])
        for x in c[7::-1]:
            acc = acc * td + x
        return acc

    es = torch.minimum(torch.where(td >= 0.0, horner(aw), horner(ci)), 0.15 * p)
    return EP2 * (es / (p - es))


def _lap(a):
    return 0.125 * (_W(a) + _E(a) + _S(a) + _N(a)) - 0.5 * a


def _flux(pos, za, up2, dn2, a, b):
    """WAF value between cells a (behind) and b of the positive direction: limiter from the differences up2 and dn2."""
    d = b - a
    den = torch.where(d.abs() < 1.0e-30, torch.copysign(torch.full_like(d, 1.0e-30), d), d)
    r = torch.where(pos, up2, dn2) / den
    lim = torch.clamp(torch.maximum(r, (2.0 * r).clamp(max=1.0)), 0.0, 2.0)
    sg = torch.where(pos, 1.0, -1.0)
    phi = sg + za * lim - sg * lim
    return (1.0 + phi) * a + (1.0 - phi) * b


def _advect(x, s, u, v, c, rot):
    """WAF advection of one field: twice the vertical pass, then meridional, then zonal."""
    old = x
    zu, zd = c["wu"], c["wd"]
    sk, sk1 = s[:-1], s[1:]
    pos, za, half = sk1[:-1] >= 0.0, sk1[:-1] * c["dz_a"], 0.5 * sk1[:-1]
    zero = torch.zeros_like(x[:1])
    for _ in range(2):
        d = x[1:] - x[:-1]  # level k+1 minus level k (downwards)
        up2 = -torch.cat([d[1:], zero])          # x(k+1) - x(min(k+2, kz))
        dn2 = -torch.cat([zero, d[:-1]])         # x(max(k-1, 1)) - x(k)
        f = half * _flux(pos, za, up2, dn2, x[1:], x[:-1])
        ft, fb = torch.cat([zero, f]), torch.cat([f, zero])
        x = x - ft * zu + fb * zd + (sk * zu - sk1 * zd) * x
    # flux through the southern face of a cell
    vf = v if rot else v / c["mv"]
    f = 0.5 * vf * _flux(v > 0.0, vf * c["dx_a"], _S(x) - _S(_S(x)), _N(x) - x, _S(x), x)
    p0 = f * c["ws"] - _N(f) * c["wn"] + (_N(vf) * c["wn"] - vf * c["ws"]) * old
    x = x + (p0 if rot else c["mx"] ** 2 * p0)
    uf = u if rot else u / c["mu"]
    za = u * c["mu"] * c["dx_a"] if rot else uf * c["dx_a"]
    f = 0.5 * uf * _flux(u > 0.0, za, _W(x) - _W(_W(x)), _E(x) - x, _W(x), x)
    p1 = f * c["ww"] - _E(f) * c["we"] + (_E(uf) * c["we"] - uf * c["ww"]) * old
    return x + (p1 if rot else c["mx"] ** 2 * p1)


def _metrics(st, kz, rot):
    c = {"mx": st["msfx"], "mu": st["msfu"], "mv": st["msfv"], "fmz": st["fmz"], "fmzf": st["fmzf"]}
    dta = DT / NADV
    c["dz_a"], c["dx_a"] = 0.5 * dta / (ZTOP / kz), dta / DX
    f = st["fmz"]
    c["wu"], c["wd"] = c["dz_a"] * f / st["fmzf"][:-1], c["dz_a"] * f / st["fmzf"][1:]
    my, mx = (c["mx"], c["mu"]) if rot else (1.0, 1.0)
    c["wn"] = 2.0 * c["dx_a"] * f / (f + _N(f)) * (my / _N(c["mv"]) if rot else 1.0)
    c["ws"] = 2.0 * c["dx_a"] * f / (f + _S(f)) * (my / c["mv"] if rot else 1.0)
    c["we"], c["ww"] = (2.0 * c["dx_a"] * mx * f / (f + y) for y in (_E(f), _W(f)))
    return c


class _Exact:
    def __init__(self, st, rotllr, filters):
        self.rot, self.filters = bool(rotllr), filters
        self.st = st
        self.f = {n: st[n].clone() for n in ("u", "v", "w", "pai", "t") + TRACERS}
        self.kz = kz = st["t"].shape[0]
        self.c = _metrics(st, kz, self.rot)
        dts = DT / NADV / NSOUND
        self.dts, self.dx, self.dz = dts, dts / DX, dts / (ZTOP / kz)
        k = torch.arange(kz, device="cuda", dtype=torch.float64)
        self.xknu = (0.0625 + (1.0 - 0.0625) * torch.sin(0.5 * math.pi * (1.0 - k / (kz - 1))))[:, None, None]
        self.gk = _gzita(st["zita"] / ZTOP)[:, None, None]
        self.gkh = _gzita(st["zitah"] / ZTOP)[:, None, None]
        self.coru = EOMEG2 * torch.sin(st["ulat"] * math.pi / 180.0)
        self.corv = EOMEG2 * torch.sin(st["vlat"] * math.pi / 180.0)
        fz = st["fmz"]
        self.rw, self.rs = 2.0 / (fz + _W(fz)), 2.0 / (fz + _S(fz))

    def slope(self, u, v):
        """u hx + u(j+1) hx(j+1) and the same of v."""
        return u * self.st["hx"] + _E(u * self.st["hx"]) + v * self.st["hy"] + _N(v * self.st["hy"])

    def sound(self):
        f, st, c, kz, rot = self.f, self.st, self.c, self.kz, self.rot
        u, v, w, pai, tet = f["u"], f["v"], f["w"], f["pai"], f["tetav"]
        fz, ff, hx, hy = st["fmz"], st["fmzf"], st["hx"], st["hy"]
        dts, dx, dz = self.dts, self.dx, self.dz
        qv, qc, qsat, t = f["qv"], f["qc"], f["qsat"], f["t"]
        mo1 = (1.0 + 0.86 * qv + 3.2 * qc) / (1.0 + 0.96 * qv + 4.8 * qc)
        mo2 = 0.25 * qv + 4.2 * f["qwl"] + 2.1 * f["qwi"]
        lat = dts * G * WLHV * WLHV * 0.5 * (qsat[1:] + qsat[:-1]) / (CPD * RWAT * t[:-1] ** 2)
        damp = self.xknu * (0.125 * DX / dts)
        for n in range(1, NSOUND + 1):
            s = torch.zeros_like(w)
            s[1:-1] = -0.25 * self.slope(u[1:] + u[:-1], v[1:] + v[:-1]) * self.gk[1:-1]
            ws = 0.5 * self.slope(u[-1], v[-1])
            w[-1], s[-1] = ws, -ws
            if rot:
                a, b = dx * u * self.rw, dx * v * self.rs / c["mv"]
                z = fz * c["mx"] * ((_E(a) - a) + (_N(b) - b))
            else:
                a, b = dx * u / c["mu"] * self.rw, dx * v / c["mv"] * self.rs
                z = c["mx"] ** 2 * fz * ((_E(a) - a) + (_N(b) - b))
            ud, vd = u, v  # the halo rings keep the winds from before the damping
            u = u + damp * c["mu"] * (z - _W(z))
            v = v + damp * (1.0 if rot else c["mv"]) * (z - _S(z))
            z = z + 0.0625 * 0.015625 / dts * _lap(z) + fz * dz * (s[:-1] - s[1:])
            # implicit w
            wk, tk, tm, pk, pm = w[1:-1], tet[1:], tet[:-1], pai[1:], pai[:-1]
            fi = ff[1:-1]
            ro = 0.5 * CPD * fi * (tm + tk) - CPD * wk * fi * fi * n * dz * (tm - tk)
            moist = (qv[1:] > 0.96 * qsat[1:]) & (wk > 0.1)
            ro = torch.where(moist, ro + lat * wk * (n - 1) / pm * fi, ro)
            ex = wk - ro * dz * (pm - pk) - G * dts + RDRCV * ro * dz * (pm * z[:-1] - pk * z[1:])
            zcs = dz * dz * RDRCV
            zu, zd = zcs * fz[:-1] * ro * pm, zcs * fz[1:] * ro * pk
            wn, ww = w.clone(), torch.zeros_like(w)
            for k in range(kz - 1, 0, -1):
                den = 1.0 + zd[k - 1] + zu[k - 1] - zd[k - 1] * ww[k + 1]
                wn[k] = (ex[k - 1] + zd[k - 1] * wn[k + 1]) / den
                ww[k] = zu[k - 1] / den
            for k in range(1, kz):
                wn[k] += ww[k] * wn[k - 1]
            dw = torch.zeros_like(w)
            dw[1:-1] = wn[1:-1] - w[1:-1]
            w = wn
            z = (z + dz * fz * (w[:-1] - w[1:])) * mo1
            tet = tet * (1.0 + RDRCV * z * mo2)
            if self.filters:
                z = z + ANU2 * self.xknu * _lap(z)
            pold, pai = pai, pai * (1.0 - RDRCV * z)
            # momentum; at the first row and column the neighbours are the older halo values
            pw, psn = _W(pai), _S(pai)
            pw[..., 0], psn[..., 0, :] = pold[..., -1], pold[..., -1, :]
            vw, vn = _W(v), _N(v)
            vw[..., 0], vn[..., -1, :] = vd[..., -1], vd[..., 0, :]
            vwn = _N(_W(v))
            vwn[..., -1, :], vwn[..., 0] = _W(vd)[..., 0, :], _N(vd)[..., -1]
            us, ue = _S(u), _E(u)
            us[..., 0, :], ue[..., -1] = ud[..., -1, :], ud[..., 0]
            ues = _S(_E(u))
            ues[..., 0, :], ues[..., -1] = _E(ud)[..., -1, :], _S(ud)[..., 0]
            d2 = dw[:-1] + dw[1:]
            un = u + self.coru * dts * 0.25 * (v + vw + vwn + vn) - (G * dts + 0.25 * (_W(d2) + d2)) * hx * self.gkh \
                - dx * c["mu"] * 0.5 * CPD * (_W(tet) + tet) * (pai - pw)
            zcy = dx if rot else dx * c["mv"]
            vnew = v - self.corv * dts * 0.25 * (u + us + ue + ues) - (G * dts + 0.25 * (_S(d2) + d2)) * hy * self.gkh \
                - zcy * 0.5 * CPD * (_S(tet) + tet) * (pai - psn)
            u, v = un, vnew
        s[1:-1] = (w[1:-1] + s[1:-1]) * ff[1:-1]
        s[0], s[-1] = 0.0, 0.0
        f.update(u=u, v=v, w=w, pai=pai, tetav=tet, s=s)

    def network(self, net):
        """The surrogate's cycle: features, the network, the committed increments and s."""
        f, kz = self.f, self.kz
        layers, xm, xs, ym, ys = net

        def dev(a):
            return torch.as_tensor(np.asarray(a, np.float64), device="cuda")

        ni, nj = f["u"].shape[-2:]
        flds = (f["u"], f["v"], f["w"][1:], f["pai"], f["tetav"])
        planes = [((a - dev(xm)[q][:, None, None]) / dev(xs)[q][:, None, None]) for q, a in enumerate(flds)]
        inc = torch.empty(ni, nj, 5, kz, dtype=torch.float64, device="cuda")
        for lo in range(0, ni, 32):
            rows = torch.arange(lo - 1, min(lo + 33, ni + 1), device="cuda") % ni
            x = torch.stack(planes).index_select(2, rows)  # field, k, rows with a halo, j
            n = x.shape[2] - 2
            nb = [torch.roll(x, -dj, -1)[:, :, 1 + di:1 + di + n] for di in (-1, 0, 1) for dj in (-1, 0, 1)]
            h = torch.stack(nb, -1).permute(2, 3, 0, 1, 4).reshape(n * nj, 45 * kz)
            for q, (w, b) in enumerate(layers):
                w = dev(w)
                h = h @ (w[:, :45 * kz] if q == 0 else w).T + dev(b)
                h = h * torch.sigmoid(h) if q < 3 else h
            inc[lo:lo + n] = h[:, :5 * kz].reshape(n, nj, 5, kz)
        inc = inc.permute(2, 3, 0, 1) * dev(ys)[:, :, None, None] + dev(ym)[:, :, None, None]
        fr = (NSOUND - 1) / NSOUND
        ul, vl = f["u"] + fr * inc[0], f["v"] + fr * inc[1]
        f["u"], f["v"], f["pai"], f["tetav"] = f["u"] + inc[0], f["v"] + inc[1], f["pai"] + inc[3], f["tetav"] + inc[4]
        f["w"] = f["w"].clone()
        f["w"][1:] += inc[2]
        s = torch.zeros_like(f["w"])
        s[1:-1] = (f["w"][1:-1] - 0.25 * self.slope(ul[1:] + ul[:-1], vl[1:] + vl[:-1]) * self.gk[1:-1]) * self.st["fmzf"][1:-1]
        f["s"] = s

    def advection(self):
        f, kz = self.f, self.kz
        u, v, w, s = f["u"], f["v"], f["w"], f["s"]
        ux = 0.5625 * (_E(u) + u) - 0.0625 * (_E(_E(u)) + _W(u))
        vx = 0.5625 * (_N(v) + v) - 0.0625 * (_N(_N(v)) + _S(v))
        wx = 0.5 * (w[1:] + w[:-1])
        wx[1:-1] = 0.5625 * (w[2:-1] + w[1:-2]) - 0.0625 * (w[3:] + w[:-3])
        for n in ("tetav", "pai") + TRACERS:
            f[n] = _advect(f[n], s, u, v, self.c, self.rot)
        ux, vx, wx = (_advect(x, s, u, v, self.c, self.rot) for x in (ux, vx, wx))
        f["u"] = 0.5625 * (ux + _W(ux)) - 0.0625 * (_E(ux) + _W(_W(ux)))
        f["v"] = 0.5625 * (vx + _S(vx)) - 0.0625 * (_N(vx) + _S(_S(vx)))
        w = w.clone()
        w[1:-1] = 0.5 * (wx[1:] + wx[:-1])
        w[2:-2] = 0.5625 * (wx[2:-1] + wx[1:-2]) - 0.0625 * (wx[3:] + wx[:-3])
        f["w"] = w

    def step(self, net=None):
        f, st = self.f, self.st
        load = f["qc"] + f["qi"] + f["qr"] + f["qs"]
        p = f["pai"] ** CPOVR * P00
        f["qsat"] = _pfwsat(f["t"], p)
        f["qwl"], f["qwi"] = f["qc"] + f["qr"], f["qi"] + f["qs"]
        f["tetav"] = f["t"] * (1.0 + EP1 * f["qv"] - load) / f["pai"]
        pf, tf = f["pai"], f["tetav"]
        for _ in range(NADV):
            self.network(net) if net else self.sound()
            self.advection()
        if self.filters:
            x = f["pai"] - pf
            f["pai"] = x + 0.05 * _lap(x) + pf
            x = f["tetav"] - tf
            f["tetav"] = x + 0.05 * _lap(x) + tf
        tv = f["tetav"] * f["pai"]
        f["t"] = tv / (1.0 + EP1 * f["qv"] - f["qc"] - f["qi"] - f["qr"] - f["qs"])
        p = f["pai"] ** CPOVR * P00
        f["rho"] = p / (RGAS * f["t"])
        z = st["zeta"]
        lr = 0.65 * (tv[-2] - tv[-1]) / (z[-2] - z[-1]) - 0.35 * LRATE
        f["ps"] = p[-1] * torch.exp(z[-1] * G / (RGAS * (tv[-1] - 0.5 * z[-1] * lr)))

    def outputs(self, jx, iy, kz, fields):
        return {n: torch.from_numpy(_host(n, self.f[n], jx, iy, kz).T) for n in ("t", "ps") + fields}

    def diag(self):
        f = self.f
        rdz = f["rho"] * (ZTOP / self.kz) / self.st["fmz"]
        wm = 0.5 * (f["w"][1:] + f["w"][:-1])
        en = rdz * (CVD * f["t"] + G * self.st["zeta"] + 0.5 * (f["u"] ** 2 + f["v"] ** 2 + wm ** 2))
        return np.array([float(x) for x in (f["ps"].max(), f["ps"].min(), f["u"].max(), f["u"].min(), f["v"].max(),
                                            f["v"].min(), rdz.sum(), en.sum())])


def _exact_domain(case, st, steps, fields, net=None):
    x = _Exact(st, case.get("rotllr", 1), case.get("filters", False))
    for _ in range(steps):
        x.step(net)
    return x, x.outputs(case["jx"], case["iy"], case["kz"], fields)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("loop", "coupled", "surrogate"):
        steps = case.get("steps", 1)
        if case["jx"] * case["iy"] * case["kz"] * steps > 2.0e8:  # more than the time this is worth
            return None
        st = _state(case["jx"], case["iy"], case["kz"], seed, case.get("hills", 1), case.get("rotllr", 1))
        net = _network(case["kz"], seed) if kind == "surrogate" else None
        x, out = _exact_domain(case, st, steps, () if kind == "coupled" else FETCH, net)
        if case.get("lprint"):
            out["diag"] = x.diag()
        return out
    if kind == "ensemble":
        return [_exact_domain(c, _member_state(c), case["steps"], ("u",))[1] for c in _members(case, seed)]
    if kind == "gradient":
        x, t = (torch.as_tensor(a, dtype=torch.float64, device="cuda") for a in _batch(case, seed))
        m = 5 * case["kz"]
        par = [(torch.as_tensor(w, dtype=torch.float64, device="cuda").requires_grad_(),
                torch.as_tensor(b, dtype=torch.float64, device="cuda").requires_grad_()) for w, b in _network(case["kz"], seed)[0]]
        h = x
        for q, (w, b) in enumerate(par):
            h = h @ w.T + b
            h = h * torch.sigmoid(h) if q < 3 else h
        loss = ((h[:, :m] - t[:, :m]) ** 2).sum()
        gw, gb = torch.autograd.grad(loss / (x.shape[0] * m), par[case["layer"]])
        return {"loss": np.float64(loss.item()), "gw": gw.cpu(), "gb": gb.cpu()}
    f = _field(case, seed)
    return _advect(f["pp"], f["s"], f["u"], f["v"], _metrics(f, case["kz"], bool(case["rotllr"])), bool(case["rotllr"]))
