"""Work that programs built on this framework have it do, from one small simulation to a batch.

Every case goes through the package's public entry points: one simulation that lives on the GPU
(`Engine`), many that are admitted from host memory, stepped together and read back (`Batch`), and
the call without allocation.  A mixed-precision run carries FP32 accuracy, so a program keeps its
states as FP32; an FP64 run's states stay FP64.  Workloads under the method's own time-step rule
start from smooth flow or from seeded noise; those whose rule would follow rounding noise (the
blast's uniform surroundings, the stratified atmosphere) run at a fixed step.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "smaug-all_b200", "python")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from smaug_b200 import PREC_FP64, PREC_MIXED, Batch, Engine, load_library, make_params, problems  # noqa: E402

RK_STAGES = 4


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a small vortex, stepped many times between looks: launches and latency count
        {"name": "vortex_small_mixed", "kind": "engine", "problem": "vortex", "nx": 64, "ny": 48, "nz": 0, "mixed": True, "steps": 32},
        # the classic 256^2 vortex in FP64
        {"name": "vortex_256_fp64", "kind": "engine", "problem": "vortex", "nx": 256, "ny": 256, "nz": 0, "mixed": False, "steps": 16},
        # one large vortex of uneven sides in mixed precision
        {"name": "vortex_large_mixed", "kind": "engine", "problem": "vortex", "nx": 1531, "ny": 1022, "nz": 0, "mixed": True, "steps": 12},
        # the batched ensemble: sides 128..768, admitted from pinned host memory, stepped, read back
        {"name": "ensemble_mixed", "kind": "batch", "problem": "vortex", "sims": 24, "lo": 128, "hi": 768, "mixed": True, "steps": 24},
        # the same in FP64, smaller members
        {"name": "ensemble_fp64", "kind": "batch", "problem": "vortex", "sims": 12, "lo": 96, "hi": 512, "mixed": False, "steps": 12},
        # driven slices of the stratified atmosphere as the server takes them
        {"name": "slices_mixed", "kind": "batch", "problem": "atmosphere", "sims": 10, "lo": 128, "hi": 512, "mixed": True, "steps": 24},
        # a small 3-D blast: few cells for so wide a chip
        {"name": "blast_small_mixed", "kind": "engine", "problem": "blast", "nx": 26, "ny": 26, "nz": 26, "mixed": True, "steps": 16},
        # the 3-D blast at its usual size, both precisions
        {"name": "blast_128_mixed", "kind": "engine", "problem": "blast", "nx": 128, "ny": 128, "nz": 128, "mixed": True, "steps": 8},
        {"name": "blast_85_fp64", "kind": "engine", "problem": "blast", "nx": 85, "ny": 85, "nz": 85, "mixed": False, "steps": 6},
        # the 3-D stratified atmosphere: gravity, live background, driver, closed vertical boundaries
        {"name": "atmosphere_3d_mixed", "kind": "engine", "problem": "atmosphere", "nx": 128, "ny": 66, "nz": 61, "mixed": True, "steps": 8},
        # an FP64 slice whose host program takes the state back after a few steps (files, plots)
        {"name": "slice_host_fp64", "kind": "host", "problem": "atmosphere", "nx": 256, "ny": 130, "nz": 0, "mixed": False, "steps": 16},
        # a caller that may not allocate: device buffers in, device buffers out
        {"name": "vortex_noalloc_fp64", "kind": "noalloc", "problem": "vortex", "nx": 200, "ny": 151, "nz": 0, "mixed": False, "steps": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["engine2", "engine2", "engine3", "engine3", "batch", "host", "noalloc"])
    mixed = rng.random() < 0.6
    if kind == "batch":
        lo = _log(rng, 32, 200)
        return {"kind": "batch", "problem": rng.choice(["vortex", "vortex", "atmosphere"]), "sims": rng.randint(3, 14), "lo": lo,
                "hi": min(512, 2 * lo + rng.randint(0, 150)), "mixed": mixed, "steps": rng.randint(8, 20)}
    if kind == "engine3":
        n = _log(rng, 14, 100)
        if rng.random() < 0.6:
            return {"kind": "engine", "problem": "blast", "nx": n, "ny": n, "nz": n, "mixed": mixed, "steps": rng.randint(4, 8)}
        return {"kind": "engine", "problem": "atmosphere", "nx": n + rng.randint(6, 40), "ny": max(10, n - rng.randint(0, 20)),
                "nz": max(10, n - rng.randint(0, 20)), "mixed": mixed, "steps": rng.randint(4, 8)}
    # (the time-step rule looks at the last dimension's spacing: a vortex's sides stay near each other)
    if kind == "noalloc":
        ny = _log(rng, 24, 300)
        return {"kind": "noalloc", "problem": "vortex", "nx": int(ny * rng.uniform(0.6, 1.3)), "ny": ny, "nz": 0, "mixed": False,
                "steps": rng.randint(4, 12)}
    if kind == "host":
        return {"kind": "host", "problem": "atmosphere", "nx": _log(rng, 48, 400), "ny": _log(rng, 32, 300), "nz": 0, "mixed": mixed,
                "steps": rng.randint(8, 24)}
    ny = _log(rng, 32, 1100)
    return {"kind": "engine", "problem": rng.choice(["vortex", "vortex", "atmosphere"]), "nx": int(ny * rng.uniform(0.6, 1.3)), "ny": ny,
            "nz": 0, "mixed": mixed, "steps": rng.randint(8, 24)}


# ------------------------------------------------------------------ the inputs
def _atmosphere(nz, nx, ny, rng, seed):
    """A driven stratified atmosphere with 0.1 % density noise: amplitude and period as the server draws them."""
    p = problems.atmosphere(nz, nx, ny or None, noise=1e-3, seed=seed)
    p.driver["amp"] = float(rng.uniform(50.0, 500.0))
    p.driver["period"] = float(rng.uniform(120.0, 600.0))
    return p


def _blast(n, seed):
    """The blast wave, with the seed's 1 % density noise in the whole box."""
    p = problems.blast_wave(n, seed=seed)
    noise = np.random.default_rng(seed).standard_normal((n, n, n))
    p.w[0] = np.pad(1.0 + 0.01 * noise, 2, mode="wrap")
    return p


def _problem(case, seed):
    rng = np.random.default_rng(1000 + seed)
    if case["problem"] == "vortex":
        return problems.orszag_tang(case["nx"], case["ny"], b0_scale=float(rng.uniform(0.5, 1.5)), rho_noise=0.01, seed=seed)
    if case["problem"] == "blast":
        return _blast(case["nx"], seed)
    return _atmosphere(case["nx"], case["ny"], case["nz"], rng, seed)


def _members(case, seed):
    """A batch's simulations: the sizes belong to the case, the fields to the seed."""
    sizes = np.random.default_rng(case["sims"] * 7919 + case["lo"])
    rng = np.random.default_rng(1000 + seed)
    out = []
    for i in range(case["sims"]):
        n = int(round(math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        n = case["hi"] if i == 0 else n
        if case["problem"] == "vortex":
            out.append(problems.orszag_tang(n, b0_scale=float(rng.uniform(0.5, 1.5)), rho_noise=0.01, seed=100 * seed + i))
        else:
            out.append(_atmosphere(n, max(24, n // 2 if i % 2 else n), 0, rng, 100 * seed + i))
    return out


def _dt(case, prob):
    """(dt_mode, dt0): the rule, or a fixed step well inside it."""
    if case["problem"] == "atmosphere":
        return 0, 1.0e-7 * min(prob.dx)
    if case["problem"] == "blast":
        return 0, 0.03 * prob.dx[0]
    return 1, 0.0


def _delx(prob):
    return np.ascontiguousarray(np.concatenate([a.ravel() for a in prob.delx()]))


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory()


def prepare(case, seed):
    prec = PREC_MIXED if case["mixed"] else PREC_FP64
    s = {"case": case}
    if case["kind"] == "batch":
        from smaug_b200 import footprint
        probs = _members(case, seed)
        need = sum(footprint(p, prec) + 4096 for p in probs)
        s["batch"] = Batch(2, precision=prec, arena_bytes=need, max_sims=case["sims"])
        s["sims"] = []
        for p in probs:
            mode, dt0 = _dt(case, p)
            out = torch.empty(p.w.shape, dtype=torch.float64).pin_memory()
            kept = torch.empty(p.w.shape, dtype=torch.float32) if case["mixed"] else out
            s["sims"].append({"prob": p, "w": _pinned(p.w), "delx": _pinned(_delx(p)), "out": out, "kept": kept, "dt_mode": mode, "dt0": dt0})
        return s
    p = _problem(case, seed)
    mode, dt0 = _dt(case, p)
    if case["kind"] == "noalloc":
        lib = load_library()
        lib.smaug_step_noalloc.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int,
                                           ctypes.c_void_p, ctypes.POINTER(ctypes.c_double), ctypes.c_char_p, ctypes.c_size_t]
        s.update(lib=lib, params=make_params(p, rk4=True, dt_mode=mode, dt0=dt0, precision=prec), delx=torch.from_numpy(_delx(p)).cuda(),
                 w=torch.from_numpy(np.ascontiguousarray(p.w)).cuda())
        s["out"] = torch.empty_like(s["w"])
        return s
    s["engine"] = Engine(p, rk4=True, dt_mode=mode, dt0=dt0, precision=prec)
    if case["kind"] == "host":
        s["w"] = np.ascontiguousarray(p.w)
    else:
        s["w"] = torch.from_numpy(np.ascontiguousarray(p.w)).cuda()
        s["out"] = torch.empty_like(s["w"])
    return s


# ------------------------------------------------------------------ one pass
def _run_batch(s):
    """Admit every member from pinned memory, a step queued after every fourth; step; read all back; free the slots."""
    b, steps = s["batch"], s["case"]["steps"]
    slots, queued = [], 0
    for i, m in enumerate(s["sims"]):
        slots.append(b.add(m["prob"], steps, dt_mode=m["dt_mode"], dt0=m["dt0"], w=m["w"].numpy(), delx=m["delx"].numpy()))
        if i % 4 == 3:
            b.step(1)
            queued += 1
    b.step(steps)  # a member stops by itself after its own steps
    left = b.poll_end(b.poll_begin())
    if any(left[k] != 0 for k in slots):
        raise RuntimeError("a simulation did not finish")
    for k, m in zip(slots, s["sims"]):
        b.state_async(k, m["out"].numpy())
    b.io_wait()
    for k in slots:
        b.remove(k)
    if s["case"]["mixed"]:
        for m in s["sims"]:
            m["kept"].copy_(m["out"])
    return [m["kept"] for m in s["sims"]]


def run(state):
    s, case = state, state["case"]
    if case["kind"] == "batch":
        return _run_batch(s)
    if case["kind"] == "noalloc":
        err = ctypes.create_string_buffer(256)
        rc = s["lib"].smaug_step_noalloc(ctypes.byref(s["params"]), s["delx"].data_ptr(), s["w"].data_ptr(), s["out"].data_ptr(), case["steps"],
                                         torch.cuda.current_stream().cuda_stream, None, err, 256)
        if rc != 0:
            raise RuntimeError(err.value.decode())
        return s["out"]
    e = s["engine"]
    if case["kind"] == "host":
        e.set_state(s["w"])
        e.step(case["steps"])
        w = torch.from_numpy(e.state())
        return w.float() if case["mixed"] else w
    e.set_state_device(s["w"].data_ptr(), s["w"].numel())
    e.step(case["steps"])
    e.get_state_device(s["out"].data_ptr(), s["out"].numel())
    e.sync()
    return s["out"].float() if case["mixed"] else s["out"]


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Bytes: the state in and out once, and per Runge-Kutta stage the stage's input read and its output written once, in the
    type of the stage states.  Flops: the arithmetic of the method per cell and stage, counted from its formulas."""
    if case["kind"] == "batch":
        cells = sum((p[0] + 4) * (p[1] + 4) for p in _sizes(case))
        d = 2
    else:
        d = 3 if case["nz"] else 2
        cells = (case["nx"] + 4) * (case["ny"] + 4) * (case["nz"] + 4 if d == 3 else 1)
    nw, nvar = 2 + 2 * d, 4 + 3 * d
    size = 4 if case["mixed"] else 8
    stages = RK_STAGES * case["steps"]
    # per cell and stage: the fluxes of each direction once, their divergence, the face ratios, the
    # hyperviscous terms (diagonal and cross), the update and the wave speeds
    flops = d * (10 + 8 * d) + d * 4 * nw + d * (2 * d + 1) * 16 + d * (12 + 20 * d + 24 * (d - 1) * 2) + 6 * nw + 20 + 14 * d
    return {"bytes": cells * (16 * nvar + stages * 2 * nw * size), "flops": cells * stages * flops}


def _sizes(case):
    sizes = np.random.default_rng(case["sims"] * 7919 + case["lo"])
    out = []
    for i in range(case["sims"]):
        n = int(round(math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        n = case["hi"] if i == 0 else n
        out.append((n, n) if case["problem"] == "vortex" else (n, max(24, n // 2 if i % 2 else n)))
    return out


# ------------------------------------------------------------------ the method in 64 bits, in plain torch
class _Exact:
    """The split-variable MHD step of one simulation on whole arrays, FP64: 4th-order central fluxes, background energy terms,
    gravity, hyperdiffusion, driver, four-stage Runge-Kutta, periodic or contcd4 ghosts, fixed step or the time-step rule."""

    def __init__(self, prob, dt_mode, dt0, device):
        self.p, self.D, self.n = prob, prob.ndim, prob.n
        D = self.D
        self.nw = 2 + 2 * D
        self.M, self.E, self.B = 1, 1 + D, 2 + D
        t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=device)  # noqa: E731
        w = t(prob.w)
        self.w, self.eb, self.rb, self.bb = w[:self.nw].clone(), w[self.nw], w[self.nw + 1], w[self.nw + 2:]
        self.bg = w[self.nw:].clone()
        full = [t(a) for a in prob.delx()]
        self.last = full[-1]
        self.dx = []
        inner = [slice(2, 3)] * D
        for d in range(D):
            s = list(inner)
            s[self.ax(d, D)] = slice(None)
            self.dx.append(full[d][tuple(s)])
        N = self.last.numel()
        ndimp = 1 << (N - 1).bit_length()
        self.K = (ndimp + 511) // 512 * 64
        self.minsq = [float((a.reshape(-1)[:self.K] ** 2).min()) for a in full]
        self.inner = tuple([slice(2, -2)] * D)
        self.mask = torch.zeros(self.last.shape, dtype=torch.float64, device=device)
        self.mask[self.inner] = 1.0
        # cells whose gradients count as zero near a closed end (2: the outer two inner cells, 1: the outer one)
        self.z4, self.z1 = [], []
        for d in range(D):
            for width, to in ((2, self.z4), (1, self.z1)):
                m = torch.ones(self.n[d], dtype=torch.float64, device=device)
                if prob.btype[d] != 0:
                    m[2:2 + width] = 0.0
                    m[self.n[d] - 2 - width:self.n[d] - 2] = 0.0
                to.append(m.reshape([-1 if k == self.ax(d, D) else 1 for k in range(D)]))
        self.mode, self.dt, self.t = dt_mode, (dt0 if dt_mode == 0 or dt0 > 0 else 1e-8), 0.0
        self.drv = None
        if prob.driver:
            f = torch.ones([1] * D, dtype=torch.float64, device=device)
            for d in range(D):
                x = prob.xmin[d] + np.arange(self.n[d]) * prob.dx[d]
                wd = prob.driver["width"][d]
                g = np.exp(-((x - prob.driver["center"][d]) ** 2) / (wd * wd)) if wd > 0 else np.ones(self.n[d])
                f = f * t(g).reshape([-1 if k == self.ax(d, D) else 1 for k in range(D)])
            self.drv = f * prob.driver["amp"]
        self.steps, self.maxnu, self.dtdiff = 0, 0.0, 0.0
        self.ghosts(self.w)
        self.speeds = self.reduce(self.w)

    @staticmethod
    def ax(d, D):
        return D - 1 - d

    def sh(self, a, d, o):
        """a at the cell o further along d."""
        return torch.roll(a, -o, dims=a.dim() - 1 - d)

    def ghosts(self, w):
        for d in range(self.D):
            v = w.movedim(w.dim() - 1 - d, 0)
            n = self.n[d]
            src = (n - 4, n - 3, 2, 3) if self.p.btype[d] == 0 else (4, 3, n - 4, n - 5)
            for g, k in zip((0, 1, n - 2, n - 1), src):
                v[g] = v[k].clone()

    def reduce(self, w):
        gam, D = self.p.gamma, self.D
        rt = w[0] + self.rb
        m, b = w[1:1 + D], w[self.B:]
        m2, b2, bb2, bbb = (m * m).sum(0), (b * b).sum(0), (self.bb * self.bb).sum(0), (b * self.bb).sum(0)
        pk = (gam - 1) * (w[self.E] - 0.5 * m2 / rt - 0.5 * b2 - bbb)
        cs2 = gam * (pk + (gam - 1) * (self.eb - 0.5 * bb2)) / rt
        cf = (b2 + bb2 + 2 * bbb) / rt + cs2
        out = []
        for d in range(D):
            bd = self.bb[d] + b[d]
            c = torch.sqrt(0.5 * (cf + torch.sqrt(cf * cf - 4 * cs2 * bd * bd / rt))) + (m[d] / rt).abs()
            out.append(float(c.max()))
        cour = (c / self.last).reshape(-1)
        return out, float(cour.max()), float(cour[self.K:].max())

    def ratio(self, q, d):
        """max|d3 q| / max|d1 q| of the face between each cell and the next along d."""
        v = q.movedim(q.dim() - 1 - d, 0)
        n = v.shape[0]
        e = torch.cat([v[5:6], v, torch.zeros_like(v[:1])])  # the padded copy: q(5) on the left, 0 on the right
        t1 = (e[1:] - e[:-1])                                 # t1[k]: cells k-1 and k
        t3 = (3 * t1[1:-1] - (e[3:] - e[:-3])).abs()          # t3[k]: around t1[k+1]
        t1 = t1.abs()
        m1 = torch.stack([t1[o:o + n - 3] for o in range(5)]).amax(0)      # faces of the cells 1..n-3
        m3 = torch.stack([t3[o:o + n - 3] for o in range(3)]).amax(0)
        out = torch.zeros_like(v)
        out[1:n - 2] = torch.where(m1 > 0, m3 / torch.where(m1 > 0, m1, torch.ones_like(m1)), torch.zeros_like(m1))
        return out.movedim(0, q.dim() - 1 - d)

    def source(self, w, cmax):
        p, D, gam, sh = self.p, self.D, self.p.gamma, self.sh
        M, E, B = self.M, self.E, self.B
        rt = w[0] + self.rb
        m, b, e = w[1:1 + D], w[B:], w[E]
        v = m / rt
        m2, b2, bbb = (m * m).sum(0), (b * b).sum(0), (b * self.bb).sum(0)
        pt = (gam - 1) * (e - 0.5 * m2 / rt) - (gam - 2) * (bbb + 0.5 * b2)
        dL = torch.zeros_like(w)
        numax = 0.0
        bv, bbv = (b * v).sum(0), (self.bb * v).sum(0)
        ptb = (gam - 1) * self.eb - 0.5 * (gam - 2) * (self.bb * self.bb).sum(0)
        live = bool((self.bb != 0).any()) or bool((self.eb != 0).any())

        def grad4(a, d):
            return (8 * (sh(a, d, 1) - sh(a, d, -1)) - (sh(a, d, 2) - sh(a, d, -2))) / (12 * self.dx[d]) * self.z4[d]

        for d in range(D):
            F = torch.zeros_like(w)
            F[0] = m[d]
            for k in range(D):
                F[M + k] = v[d] * m[k] - b[k] * (b[d] + self.bb[d]) - self.bb[k] * b[d]
                if k != d:
                    F[B + k] = v[d] * (b[k] + self.bb[k]) - (b[d] + self.bb[d]) * v[k]
            F[M + d] += pt
            F[E] = v[d] * (e + self.eb + pt) - (b[d] + self.bb[d]) * bv - b[d] * bbv
            dL -= grad4(F, d)
            if live:
                for k in range(D):
                    gv = grad4(v[k], d)
                    if k == d:
                        dL[E] -= ptb * gv
                    dL[E] += self.bb[d] * self.bb[k] * gv
        for k in range(D):
            if p.g[k] != 0.0:
                dL[M + k] += p.g[k] * w[0]
                dL[E] += w[0] * p.g[k] * v[k]
        if not p.hyperdif:
            return dL, numax
        qe = e - 0.5 * (b2 + m2 / rt)

        def nus(q, d, f):
            r = self.ratio(q, d)
            k = self.dx[d] * (cmax[d] * float(p.chyp[f])) * self.mask
            return k * r, k * sh(r, d, -1)

        def up(a, d):
            return (sh(a, d, 1) - a) / self.dx[d] * self.z1[d]

        def down(a, d):
            return (a - sh(a, d, -1)) / self.dx[d] * self.z1[d]

        def mid(a, d):
            return (sh(a, d, 1) - sh(a, d, -1)) / (2 * self.dx[d]) * self.z1[d]

        for d in range(D):
            for q, f in ((w[0], 0), (qe, E)):
                nr, nl = nus(q, d, f)
                numax = max(numax, float(torch.maximum(nr, nl).max()))
                dL[f] += (nr * up(q, d) - nl * down(q, d)) / self.dx[d]
            for f in range(D):
                nr, nl = nus(v[f], d, M + f)
                numax = max(numax, float(torch.maximum(nr, nl).max()))
                tp, tm = nr * up(v[f], d), nl * down(v[f], d)
                fac = (1.0 if f == d else 0.5) * 0.5 / self.dx[d]
                dL[M + f] += ((rt + sh(rt, d, 1)) * tp - (rt + sh(rt, d, -1)) * tm) * fac
                dL[E] += ((m[f] + sh(m[f], d, 1)) * tp - (m[f] + sh(m[f], d, -1)) * tm) * fac
                if f != d:
                    c = mid(v[f], d) * (nr + nl) / 4
                    dL[M + d] += mid(rt * c, f)
                    dL[E] += mid(m[d] * c, f)
            for f in range(D):
                if f == d:
                    continue
                nr, nl = nus(b[f], d, B + f)
                numax = max(numax, float(torch.maximum(nr, nl).max()))
                c = mid(b[f], d) * (nr + nl) / 2
                dL[B + d] -= mid(c, f)
                dL[E] -= mid(c * b[d], f)
                tp, tm = nr * up(b[f], d), nl * down(b[f], d)
                dL[B + f] += (tp - tm) / self.dx[d]
                dL[E] += (0.5 * (b[f] + sh(b[f], d, 1)) * tp - 0.5 * (b[f] + sh(b[f], d, -1)) * tm) / self.dx[d]
        return dL, numax

    def stage(self, win, h, cmax, frac):
        dL, nu = self.source(win, cmax)
        out = self.w.clone()
        out[(slice(None),) + self.inner] += h * dL[(slice(None),) + self.inner]
        if self.drv is not None:
            per = self.p.driver["period"]
            td = math.sin(2 * math.pi * (self.t + frac * self.dt) / per) if per > 0 else 1.0
            k = self.M + self.p.driver.get("dir", 0)
            add = h * self.drv * td * (out[0] + self.rb)
            out[k][self.inner] += add[self.inner]
        return out, nu

    def step(self):
        p, D = self.p, self.D
        cmax, cour, courk = self.speeds
        self.steps += 1
        if self.mode == 1:
            if p.courant / cour > 1e-8:
                self.dt = p.courant / cour
            if self.steps > 1:
                dtd = 1e-10
                for d in range(D):
                    dtd = 0.25 / max(dtd, courk, self.maxnu / self.minsq[d])
                self.dtdiff = dtd
            if self.dtdiff > 1e-8 and self.dt > self.dtdiff:
                self.dt = self.dtdiff
        dt, nus = self.dt, []
        w1, nu = self.stage(self.w, dt / 2, cmax, 0.0)
        self.ghosts(w1)
        nus.append(nu)
        w2, nu = self.stage(w1, dt / 2, self.reduce(w1)[0], 0.5)
        self.ghosts(w2)
        nus.append(nu)
        w3, nu = self.stage(w2, dt, self.reduce(w2)[0], 0.5)
        self.ghosts(w3)
        nus.append(nu)
        acc = (w1 + 2 * w2 + w3 - 4 * self.w) / 3
        w4, nu = self.stage(w3, dt / 6, self.reduce(w3)[0], 1.0)
        nus.append(nu)
        w4 += acc
        self.ghosts(w4)
        self.w, self.speeds = w4, self.reduce(w4)
        self.maxnu = max([self.maxnu] + nus)
        self.t += dt


def _exact_state(prob, dt_mode, dt0, steps, device):
    x = _Exact(prob, dt_mode, dt0, device)
    for _ in range(steps):
        x.step()
    return torch.cat([x.w, x.bg])


def exact(case, seed):
    """run()'s answer in 64 bits by the method on whole arrays, without this framework's kernels."""
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "batch":
        return [_exact_state(p, *_dt(case, p), case["steps"], device) for p in _members(case, seed)]
    p = _problem(case, seed)
    return _exact_state(p, *_dt(case, p), case["steps"], device)
