"""The work this solver is timed on: whole solves through the public entry points.

A pass takes new initial fields from host memory through ``set_fields``, a fixed number of
Lawson-Runge-Kutta steps and ``result`` (a served mix: ``submit`` to ``wait``), as a program
that scans pulses over a fibre does. The solver, batch or server is made once, in ``prepare``,
and kept. A case is

    kind      solver (one solve), snapshots (one solve read back n_save times along the
              fibre), batch (``members`` solves advanced together), served (``members``
              requests of mixed shapes through one Server)
    modes, nt, members, steps, order (4, 6, 8: RK4, 7 and 11 stages)
    fp64      every operation in FP64, else FP32 bulk
    raman     damped (one damped sinusoid), measured (two of them: no closed recurrence),
              off
    coupling  two_mode (the 2-mode example's four values), grin (sparse, even total azimuthal
              order, about ``terms`` entries), dense (all M^4 entries)

FP32-bulk solves hand their fields on in single precision, the precision in which their
transforms and nonlinearity run; FP64 solves in double.
"""
import itertools
import math

import numpy as np
import torch

import mm_propagation_b200 as mmp
from mm_propagation_b200 import workloads as W

GAMMA = 1.4e-13     # 1/(W m)
F_R = 0.18
FWHM, WINDOW = 0.2, 20.0  # ps
DZ = 2e-4           # m per step
PHASE_PER_STEP = 5.6e-3   # rad of nonlinear phase: where RK4 with this step converges
STAGES = {4: 4, 6: 7, 8: 11}


def _case(name, kind, modes, nt, members, steps, order, fp64=False, raman="damped", coupling="grin", terms=0,
          n_save=0):
    c = dict(kind=kind, modes=modes, nt=nt, members=members, steps=steps, order=order, fp64=fp64, raman=raman,
             coupling=coupling, terms=terms, n_save=n_save)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest request of a served stream: single-mode pulse propagation, latency of one solve
        _case("one_mode_solver", "solver", 1, 2048, 1, 61, 4, terms=1),
        # the reference's plain method: its 2-mode example in FP64, fields saved along the fibre
        _case("two_mode_fp64_snapshots", "snapshots", 2, 4096, 1, 122, 4, fp64=True, coupling="two_mode", n_save=4),
        # a parameter scan of that example in FP32 bulk
        _case("two_mode_batch", "batch", 2, 4096, 128, 200, 4, coupling="two_mode"),
        # one 6-mode GRIN solve at a time, RK order 6: interactive use
        _case("six_mode_solver", "solver", 6, 16384, 1, 60, 6, terms=60),
        # the 6-mode GRIN ensemble (noise or launch-condition statistics), RK4
        _case("six_mode_batch", "batch", 6, 16384, 32, 50, 4, terms=60),
        # a converged FP64 reference solve, the 11-stage tableau
        _case("six_mode_fp64", "solver", 6, 8192, 1, 40, 8, fp64=True, terms=60),
        # an odd, small batch with a tabulated (measured) Raman response: the convolution by FFT
        _case("three_mode_measured_raman", "batch", 3, 8192, 9, 60, 4, raman="measured", terms=15),
        # Kerr-only propagation of a few long windows, 11 stages
        _case("ten_mode_kerr", "batch", 10, 32768, 3, 30, 8, raman="off", terms=167),
        # dense coupling (a fibre without symmetry), RK4
        _case("fifteen_mode_dense", "batch", 15, 8192, 16, 20, 4, coupling="dense"),
        # the largest: the 28-mode power sweep, RK order 6
        _case("twenty_eight_mode_sweep", "batch", 28, 65536, 8, 12, 6, terms=2000),
        # mixed requests through the serving loop
        _case("served_mix", "served", 10, 16384, 16, 320, 6, terms=167),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solver", "solver", "snapshots", "batch", "batch", "batch", "batch", "served"])
    modes = min(28, max(1, _log_int(rng, 1, 28)))
    nt = 2 ** rng.randint(10, 16)
    order = rng.choice([4, 4, 6, 8])
    fp64 = rng.random() < 0.25
    raman = rng.choice(["damped", "damped", "damped", "measured", "off"])
    coupling = "dense" if 2 <= modes <= 15 and rng.random() < 0.2 else "grin"
    if modes == 2 and rng.random() < 0.5:
        coupling = "two_mode"
    terms = max(1, round(60 * (modes / 6) ** 2)) if coupling == "grin" else 0
    members = 1 if kind in ("solver", "snapshots") else _log_int(rng, 2, 64)
    if kind == "served":
        modes, nt, members = min(modes, 10), min(nt, 16384), min(members, 24)
        coupling, raman = "grin", "damped"
        terms = max(1, round(60 * (modes / 6) ** 2))
    # as many steps as keep a pass below the largest listed case, at most a few hundred
    cap = 4e8 / (8 if fp64 else 1) / (4 if coupling == "dense" else 1)
    per_step = modes * nt * STAGES[order] * (2 if raman == "measured" else 1) * max(1.0, modes / 6)
    while members > 1 and per_step * members * 4 > cap:
        members = max(1, members // 2)
    most = int(min(200, max(4, cap / (per_step * members))))
    steps = _log_int(rng, min(20, most), most)
    if kind == "served":
        members, steps = max(2, members), 4 * steps
    return _case(None, kind, modes, nt, members, steps, order, fp64, raman, coupling, terms,
                 n_save=rng.randint(2, 5) if kind == "snapshots" else 0)


# ---- inputs ---------------------------------------------------------------------------------

def _azimuthal(M):
    out, group = [], 0
    while len(out) < M:
        for ell in range(group, -1, -2):
            out += [ell] if ell == 0 else [ell, ell]
        group += 1
    return out[:M]


def _coupling(case, M, rng):
    """[(p, k, l, m, Q)] in insertion order, Q in 1/m^2, symmetric in (p, k, l, m)."""
    if case["coupling"] == "two_mode":
        sr = 6.4341e12
        by_ones = [sr, sr / 3, sr / 2, -sr / 3, 0.8 * sr]
        return [(p, k, l, m, by_ones[p + k + l + m]) for p in range(2) for k in range(2) for l in range(2) for m in range(2)]
    entries = [(0, 0, c % M, c // M, 0.0) for c in range(M * M)]  # every pair, in order
    if case["coupling"] == "dense":
        g = rng.standard_normal((M,) * 4) * 1e12
        q = sum(np.transpose(g, s) for s in itertools.permutations(range(4))) / 24
        q[(np.arange(M),) * 4] += 6e12
        return entries + [(p, k, l, m, q[p, k, l, m]) for p, k, l, m in itertools.product(range(M), repeat=4)]
    az = _azimuthal(M)
    sets = [(p,) * 4 for p in range(M)]
    count = M
    cands = [s for s in itertools.combinations_with_replacement(range(M), 4)
             if sum(az[i] for i in s) % 2 == 0 and s[0] != s[3]]
    for i in rng.permutation(len(cands)):
        if count >= case["terms"]:
            break
        sets.append(cands[i])
        count += len(set(itertools.permutations(cands[i])))
    grown = []
    for s in sets:
        v = 5e12 * math.exp(0.35 * rng.standard_normal())
        grown += [(*t, v) for t in set(itertools.permutations(s))]
    return entries + sorted(grown)


def _response(case, nt):
    if case["raman"] == "off":
        return None
    t = np.arange(nt) * (WINDOW / nt)
    h = np.exp(-t / 0.032) * np.sin(t / 0.0122)
    if case["raman"] == "measured":
        h = h + 0.3 * np.exp(-t / 0.1) * np.sin(t / 0.05)
    return h / (h.sum() * (WINDOW / nt))


def _pulses(M, nt, peak_w, rng):
    t0 = FWHM / (2 * math.sqrt(math.log(2)))
    t = -WINDOW / 2 + np.arange(nt) * (WINDOW / nt)
    frac, phase, at = rng.dirichlet(np.ones(M)), rng.uniform(0, 2 * math.pi, M), rng.uniform(-1, 1, M)
    return np.stack([np.sqrt(peak_w * frac[p]) * np.exp(-((t - at[p]) ** 2) / (2 * t0 * t0) + 1j * phase[p])
                     for p in range(M)])


def _solves(case, seed):
    """The solves of a pass: dicts of the shape, the fibre and the pulse, from the seed alone.
    Members of a batch share the fibre; each has a pulse and a power of its own."""
    rng = np.random.default_rng([seed, 7])
    out = []
    fibre = None
    for i in range(case["members"]):
        M, nt, order, steps = case["modes"], case["nt"], case["order"], case["steps"]
        sub = case
        if case["kind"] == "served":  # shapes cycle through the stream's ranges up to the case's
            M = [m for m in (1, 3, 6, 10) if m <= max(M, 1)][i % sum(m <= max(M, 1) for m in (1, 3, 6, 10))]
            nt = max(1024, nt >> (i // 2) % 4)
            order = (4, order)[(i // 3) % 2]
            steps = steps * (2 + i % 5) // 4
            sub = dict(case, terms=max(1, round(60 * (M / 6) ** 2)))
        if fibre is None or case["kind"] == "served":
            beta = np.zeros((M, 3))
            beta[:, 1] = rng.uniform(-2e-3, 2e-3, M)
            beta[:, 2] = rng.uniform(0.015, 0.025, M)
            fibre = dict(beta=beta, q=_coupling(sub, M, rng), h=_response(case, nt))
        qsum = np.zeros(M)
        np.add.at(qsum, [e[0] for e in fibre["q"]], [abs(e[4]) for e in fibre["q"]])
        watt = PHASE_PER_STEP * M / (GAMMA * qsum.max() * DZ)  # the peak power of that phase a step
        spread = 500.0 ** (-i / max(1, case["members"])) if M >= 20 else rng.uniform(0.3, 1.0)
        pulse = _pulses(M, nt, 1.0, rng)
        pulse *= math.sqrt(watt * spread / float((np.abs(pulse) ** 2).sum(axis=0).max()))
        out.append(dict(fibre, M=M, nt=nt, order=order, steps=steps, phi=pulse))
    return out


def _problem(s, case):
    q = np.zeros(len(s["q"]), dtype=W.NZ_DTYPE)
    for f, v in zip(("p", "k", "l", "m", "value"), zip(*s["q"])):
        q[f] = v
    return W.Problem(n_modes=s["M"], nt=s["nt"], dispersion=s["beta"], coupling=q, initial_fields=s["phi"],
                     time_window=WINDOW, pulse_width=FWHM / (2 * math.sqrt(math.log(2))),
                     fiber_length=DZ * s["steps"], n_steps=s["steps"], method_order=s["order"],
                     nonlinearity_const=GAMMA, raman_proportion=F_R if s["h"] is not None else 0.0,
                     raman_response=s["h"], raman=s["h"] is not None,
                     flags=mmp.MMP_F_FP64 if case["fp64"] else 0)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.complex128, pin_memory=torch.cuda.is_available())
    t.numpy()[...] = a
    return t


def _hand_on(state, t):
    return t.clone() if state["case"]["fp64"] else t.to(torch.complex64)


# ---- the interface --------------------------------------------------------------------------

def prepare(case, seed):
    solves = _solves(case, seed)
    probs = [_problem(s, case) for s in solves]
    state = dict(case=case, steps=case["steps"], n_save=case["n_save"])
    if case["kind"] == "served":
        state.update(handle=mmp.Server(), probs=probs, params=[p.to_params() for p in probs])
        return state
    phi = np.stack([s["phi"] for s in solves])
    state.update(phi=_pinned(phi), out=_pinned(np.zeros_like(phi)))
    state["handle"] = mmp.Batch(probs) if case["kind"] == "batch" else mmp.Solver(probs[0])
    return state


def run(state):
    h, kind = state["handle"], state["case"]["kind"]
    if kind == "served":
        ids = [h.submit(p, params) for p, params in zip(state["probs"], state["params"])]
        return [_hand_on(state, torch.from_numpy(h.wait(i)[0])) for i in ids]
    if kind == "batch":
        for i, phi in enumerate(state["phi"]):
            h.set_fields(i, phi.numpy())
        h.propagate(state["steps"])
        for i, out in enumerate(state["out"]):
            h.result(i, out.numpy())
        return _hand_on(state, state["out"])
    h.set_fields(state["phi"][0].numpy())
    if kind == "snapshots":
        fields, z, _ = h.snapshots(state["n_save"])
        return {"fields": _hand_on(state, torch.from_numpy(fields)), "z": z}
    h.propagate(state["steps"])
    h.result(state["out"][0].numpy())
    return _hand_on(state, state["out"][0])


def _counts(s):
    """Terms merged over a pair field and its conjugate, pair fields read, (p, k) products."""
    terms = {(e[0], e[1], min(e[2], e[3]), max(e[2], e[3])) for e in s["q"] if e[4] != 0}
    return len(terms), len({t[2:] for t in terms}), len({t[:2] for t in terms})


def work(case):
    """Fields in and out once; per stage and mode a transform each way, the phase and the stage
    sum, the pair fields, their Raman convolution (a recurrence, or two transforms), the sums of
    pair fields over the terms and their products with the modes."""
    moved = ops = 0.0
    seen = {}
    for s in _solves(case, 0):
        M, nt = s["M"], s["nt"]
        if id(s["q"]) not in seen:
            seen[id(s["q"])] = _counts(s)
        terms, pairs, products = seen[id(s["q"])]
        fft = 5.0 * nt * math.log2(nt)
        raman = 0.0 if s["h"] is None else 24.0 * nt if case["raman"] == "damped" else 2 * fft + 6.0 * nt
        stage = M * (2 * fft + 40.0 * nt) + pairs * (6.0 * nt + raman) + (4.0 * terms + 8.0 * products) * nt
        ops += s["steps"] * STAGES[s["order"]] * stage + 2 * M * fft
        moved += 16.0 * M * nt * (1 + max(1, case["n_save"]))
    return {"bytes": moved, "flops": ops}


# ---- the same solves in 64 bits, from the equations --------------------------------------------

def _tableau(order):
    s = math.sqrt(21.0)
    if order == 4:
        return [[], [1 / 2], [0, 1 / 2], [0, 0, 1]], [1 / 6, 1 / 3, 1 / 3, 1 / 6], [0, 1 / 2, 1 / 2, 1]
    if order == 6:
        return ([[], [1], [3 / 8, 1 / 8], [8 / 27, 2 / 27, 8 / 27],
                 [(-21 - 9 * s) / 392, -8 * (7 + s) / 392, 48 * (7 + s) / 392, -3 * (21 + s) / 392],
                 [-5 * (231 - 51 * s) / 1960, -40 * (7 - s) / 1960, 320 * s / 1960, 3 * (21 - 121 * s) / 1960,
                  392 * (6 - s) / 1960],
                 [15 * (22 - 7 * s) / 180, 120 / 180, -40 * (5 + 7 * s) / 180, 63 * (2 + 3 * s) / 180,
                  -14 * (49 - 9 * s) / 180, 70 * (7 + s) / 180]],
                [9 / 180, 0, 64 / 180, 0, 49 / 180, 49 / 180, 9 / 180],
                [0, 1, 1 / 2, 2 / 3, (7 + s) / 14, (7 - s) / 14, 1])
    return ([[], [1 / 2], [1 / 4, 1 / 4], [1 / 7, (-7 + 3 * s) / 98, (21 - 5 * s) / 49],
             [(11 - s) / 84, 0, (18 - 4 * s) / 63, (21 + s) / 252],
             [(5 - s) / 48, 0, (9 - s) / 36, (-231 - 14 * s) / 360, (63 + 7 * s) / 80],
             [(10 + s) / 42, 0, (-432 - 92 * s) / 315, (633 + 145 * s) / 90, (-504 - 115 * s) / 70, (63 + 13 * s) / 35],
             [1 / 14, 0, 0, 0, (14 + 3 * s) / 126, (13 + 3 * s) / 63, 1 / 9],
             [1 / 32, 0, 0, 0, (91 + 21 * s) / 576, 11 / 72, (-385 + 75 * s) / 1152, (63 - 13 * s) / 128],
             [1 / 14, 0, 0, 0, 1 / 9, (-733 + 147 * s) / 2205, (515 - 111 * s) / 504, (-51 + 11 * s) / 56,
              (132 - 28 * s) / 245],
             [0, 0, 0, 0, (-42 - 7 * s) / 18, (-18 - 28 * s) / 45, (-273 + 53 * s) / 72, (301 - 53 * s) / 72,
              (28 + 28 * s) / 45, (49 + 7 * s) / 18]],
            [1 / 20, 0, 0, 0, 0, 0, 0, 49 / 180, 16 / 45, 49 / 180, 1 / 20],
            [0, 1 / 2, 1 / 2, (7 - s) / 14, (7 - s) / 14, 1 / 2, (7 + s) / 14, (7 + s) / 14, 1 / 2, (7 - s) / 14, 1])


def _solve64(s, marks):
    """The fields after each number of steps in `marks`."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    M, nt = s["M"], s["nt"]
    t0 = FWHM / (2 * math.sqrt(math.log(2)))
    ld = t0 * t0 / np.abs(s["beta"][:, 2]).max()
    max_q = max(abs(e[4]) for e in s["q"])
    cf = math.sqrt(GAMMA * ld) * math.sqrt(max_q)
    t_final = WINDOW / t0
    j = np.arange(nt)
    w = 2 * math.pi / t_final * np.where(j <= nt // 2, j, j - nt)
    b = s["beta"] * (ld / t0 ** np.arange(3))
    L = torch.tensor(b[:, :1] - b[:, 1:2] * w - b[:, 2:] / 2 * w * w, device=dev)
    dz = DZ / ld
    # a term reads the pair whose position in the order of first use is that of its own pair
    order = {}
    for p in range(M):
        for e in s["q"]:
            if e[0] == p:
                order.setdefault(e[2] + e[3] * M, len(order))
    used = sorted({order[e[2] + e[3] * M] for e in s["q"] if e[4] != 0})
    at = {v: i for i, v in enumerate(used)}
    pl = torch.tensor([v % M for v in used], device=dev)
    pm = torch.tensor([v // M for v in used], device=dev)
    Q = torch.zeros(M, M, len(used), dtype=torch.float64)
    for p, k, l, m, v in s["q"]:
        if v != 0:
            Q[p, k, at[order[l + m * M]]] += v / max_q
    Q = Q.reshape(M * M, -1).to(dev)
    fr, H = 0.0, None
    if s["h"] is not None:
        fr = F_R
        H = torch.fft.fft(torch.tensor(s["h"], device=dev)) * (t_final / nt * t0 * fr)
    a, bb, c = _tableau(s["order"])
    psi = torch.fft.fft(torch.tensor(s["phi"], device=dev) * cf)
    done, fields = 0, []
    for n in range(max(marks) + 1):
        if n in marks:
            fields.append((torch.fft.ifft(psi * torch.polar(torch.ones_like(L), L * (n * dz))) / cf).cpu())
        if n == max(marks):
            break
        N = []
        for i in range(len(bb)):
            x = psi.clone()
            for jj, v in enumerate(a[i]):
                if v:
                    x += (v * dz) * N[jj]
            E = torch.polar(torch.ones_like(L), L * ((n + c[i]) * dz))
            U = torch.fft.ifft(x * E)
            V = U[pl] * U[pm].conj()
            if H is not None:
                V = (1 - fr) * V + torch.fft.ifft(torch.fft.fft(V) * H)
            T = torch.view_as_complex((Q @ torch.view_as_real(V).reshape(len(used), -1)).reshape(M, M, nt, 2))
            N.append(1j * E.conj() * torch.fft.fft((T * U).sum(1)))
        for i, v in enumerate(bb):
            if v:
                psi = psi + (v * dz) * N[i]
    return fields


def exact(case, seed):
    solves = _solves(case, seed)
    cost = 0.0
    for s in solves:
        rows = len({(e[2], e[3]) for e in s["q"]})
        cost += s["steps"] * STAGES[s["order"]] * (1.2e-3 + s["nt"] * (s["M"] ** 2 * rows * 4 / 1.5e13 + rows * 160 / 2e12))
    if cost > 18.0:
        return None
    if case["kind"] == "snapshots":
        s, n = solves[0], case["n_save"]
        marks = [(i + 1) * (s["steps"] // n) for i in range(n - 1)] + [s["steps"]]
        return {"fields": torch.stack(_solve64(s, marks)), "z": None}
    out = [_solve64(s, [s["steps"]])[0] for s in solves]
    if case["kind"] == "batch":
        return torch.stack(out)
    return out if case["kind"] == "served" else out[0]
