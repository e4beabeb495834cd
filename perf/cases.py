"""The work that users have this framework do, as measurable cases.

Every case is one call (or one short loop body) of a user's program through
the public entry points: a propagator advanced by a number of steps, the
density-matrix frame loop, the surrogate's inference, one evaluation of its
training gradients.  ``listed()`` gives fixed cases over the real range
(smallest grids to the headline batch, powers of two and ragged sizes, FP32 and
FP64, uniform and uneven batches); ``draw(rng)`` gives more of the same ranges.
``exact`` restates each case in 64 bits with plain torch.

Observable sums of FP32 runs are returned in FP32, the precision they carry.
"""
from __future__ import annotations

import math

import numpy as np
import torch

DEV = "cuda"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one drop-in object on the 256^2 harmonic configuration in the default
        # precision, a few steps per call with the Ehrenfest lists and the
        # returned host state: the interactive use of the reference's classes,
        # where latency and launches count
        dict(name="single_f64_256", kind="single", P=256, X=256, precision="float64", steps=10),
        # the same class on an even grid that is not a power of two (the
        # reference takes any even size)
        dict(name="single_f64_98x202", kind="single", P=98, X=202, precision="float64", steps=10),
        # a batch of ragged grids, enough work to fill the GPU
        dict(name="batch_f32_600x1000", kind="batch", P=600, X=1000, precision="float32", batch=8, steps=10),
        # the headline workload: 64 double-well packets at 1024^2, FP32
        dict(name="batch_f32_1024x64", kind="batch", P=1024, X=1024, precision="float32", batch=64, steps=20),
        # the 256^2 configuration in FP64 as an ensemble that streams from HBM
        dict(name="batch_f64_256x512", kind="batch", P=256, X=256, precision="float64", batch=512, steps=20),
        # von Neumann propagation of a 1024^2 density matrix, complex64
        dict(name="rho_c64_1024", kind="rho", N=1024, precision="float32", steps=20, wigner=False),
        # the density-matrix frame loop in the default precision: a few steps,
        # then the Wigner function of the state
        dict(name="rho_c128_512_frame", kind="rho", N=512, precision="float64", steps=10, wigner=True),
        # imaginary-time steps of 16 Morse wells with their own real tables
        dict(name="bloch_f32_512x16", kind="bloch", G=512, n=16, steps=50),
        # independent instances of many grid shapes replayed as one graph
        dict(name="uneven_f32_48", kind="uneven", n=48, mix=11, steps=20),
        # laser-driven atom with dephasing: per-step separable factors, three
        # passes per step, host-built field integrals
        dict(name="strong_f32_1024x2048", kind="strong", P=1024, X=2048, precision="float32", steps=64),
        # surrogate: thermal states of 16 wells on the full grid (inference)
        dict(name="fno_predict_512x16", kind="fno_predict", G=512, n=16),
        # surrogate: gradients of one training batch (forward and backward)
        dict(name="fno_train_256x16", kind="fno_train", G=256, n=16),
    ]


_POW2 = (128, 256, 512, 1024, 2048)
_MAX_POINT_STEPS = 64 * 1024 * 1024 * 20  # the headline case


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _even(rng, lo, hi):
    return 2 * int(round(_log(rng, lo, hi) / 2))


def draw(rng):
    kind = rng.choice(["single", "single", "batch", "batch", "batch", "mask", "rho", "rho", "bloch", "uneven",
                       "strong", "fno_train", "fno_predict"])
    prec = rng.choice(["float32", "float64"])
    if kind == "single":
        if rng.random() < 0.5:
            P, X = rng.choice(_POW2[:4]), rng.choice(_POW2[:4])
        else:
            P, X = _even(rng, 60, 1000), _even(rng, 60, 1000)
        return dict(kind=kind, P=P, X=X, precision=prec, steps=rng.randint(5, 40))
    if kind == "batch":
        if rng.random() < 0.65:
            P, X = rng.choice(_POW2), rng.choice(_POW2)
        else:
            P, X = _even(rng, 100, 1200), _even(rng, 100, 1200)
        most = (64 << 20) // (P * X) // (4 if prec == "float64" else 1)
        B = max(1, min(512, int(round(_log(rng, 1, max(1, most))))))
        if not (_is_pow2(P) and _is_pow2(X)):
            B = min(B, max(1, (16 << 20) // (P * X)))
        return dict(kind=kind, P=P, X=X, precision=prec, batch=B, steps=rng.randint(5, 20))
    if kind == "mask":
        return dict(kind=kind, P=rng.choice(_POW2), X=rng.choice(_POW2), precision=prec, steps=rng.randint(5, 30))
    if kind == "rho":
        N = rng.choice(_POW2[:4])
        return dict(kind=kind, N=N, precision=prec, steps=rng.randint(5, 30), wigner=rng.random() < 0.5)
    if kind == "bloch":
        G = rng.choice((128, 256, 512))
        return dict(kind=kind, G=G, n=int(round(_log(rng, 1, 64 * (256 / G)))) if G < 512 else rng.randint(1, 24),
                    steps=rng.randint(10, 60))
    if kind == "uneven":
        return dict(kind=kind, n=rng.randint(6, 48), mix=rng.randint(0, 10 ** 6), steps=rng.randint(5, 20))
    if kind == "strong":
        return dict(kind=kind, P=rng.choice((256, 512, 1024)), X=rng.choice((512, 1024, 2048)), precision=prec,
                    steps=rng.randint(16, 80))
    if kind == "fno_train":
        return dict(kind=kind, G=rng.choice((128, 192, 256)), n=rng.randint(2, 16))
    return dict(kind=kind, G=rng.choice((256, 384, 512)), n=rng.randint(1, 16))


def _is_pow2(n):
    return n & (n - 1) == 0


# ---------------------------------------------------------------------------
# physics shared by prepare() and exact()
# ---------------------------------------------------------------------------
_AMP = 10.0


def _dw(x):
    return 0.05 * x ** 4 - x ** 2


def _ddw(x):
    return 0.2 * x ** 3 - 2.0 * x


def _harm(x):
    return 0.5 * x * x


def _ident(x):
    return 1.0 * x


def _kin(p):
    return 0.5 * p * p


def _box(case):
    """(X amplitude, P amplitude, dt, V, V') of a single / batch / mask case:
    the harmonic box for one small object and its ensemble, else the double well."""
    if case["kind"] == "single" or (case["P"] == 256 and case["X"] == 256):
        return 8.0, 7.0, 0.01, _harm, _ident
    return _AMP, _AMP, 0.005, _dw, _ddw


def _grid(P, X, XA, PA):
    dX, dP = 2.0 * XA / X, 2.0 * PA / P
    x = np.linspace(-XA, XA - dX, X)[None, :]
    p = np.linspace(-PA, PA - dP, P)[:, None]
    th = np.fft.fftfreq(P, dP / (2 * np.pi))[: P // 2 + 1][:, None]
    la = np.fft.fftfreq(X, dX / (2 * np.pi))[: X // 2 + 1][None, :]
    return x, p, th, la, dX, dP


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a)).to(DEV).to(dtype)


def _packets(case, seed, n, P, X, XA, PA):
    """n displaced Gaussian packets (n, P, X), FP64 on the GPU; width 0.5 in x."""
    rng = np.random.default_rng(seed)
    x0, p0 = _t(rng.uniform(-2, 2, n)), _t(rng.uniform(-1, 1, n))
    x, p, _, _, dX, dP = _grid(P, X, XA, PA)
    gx = torch.exp(-((_t(x[0])[None, :] - x0[:, None]) ** 2) / 0.5)
    gp = torch.exp(-0.5 * (_t(p[:, 0])[None, :] - p0[:, None]) ** 2)
    W = gp[:, :, None] * gx[:, None, :]
    return W / (W.sum(dim=(1, 2), keepdim=True) * dX * dP)


def _real(case):
    return torch.float64 if case.get("precision") == "float64" else torch.float32


def _sums(case, obs):
    """Observable sums in the precision of the run."""
    obs = obs if isinstance(obs, torch.Tensor) else np.asarray(obs)
    if case.get("precision") == "float64":
        return obs
    return obs.to(torch.float32) if isinstance(obs, torch.Tensor) else obs.astype(np.float32)


_LISTS = ("X_average", "P_average", "X_average_RHS", "P_average_RHS", "hamiltonian_average")


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    return {"case": case, **_PREPARE[case["kind"]](case, seed)}


def run(state):
    return _RUN[state["case"]["kind"]](state)


def _prep_single(case, seed):
    import fastwigner_b200 as fw

    XA, PA, dt, V, dV = _box(case)
    q = fw.WignerMoyalFTTW1D(t=0.0, dt=dt, X_gridDIM=case["X"], X_amplitude=XA, P_gridDIM=case["P"], P_amplitude=PA,
                             V=lambda _, x: V(x), K=lambda _, p: _kin(p), diff_V=lambda _, x: dV(x),
                             diff_K=lambda _, p: _ident(p), precision=case["precision"])
    q.set_wignerfunction(_packets(case, seed, 1, case["P"], case["X"], XA, PA)[0])
    return {"q": q}


def _clear(q):
    for k in _LISTS:
        getattr(q, k).clear()


def _run_single(s):
    q, case = s["q"], s["case"]
    _clear(q)
    W = q.propagate(case["steps"])
    if case["precision"] == "float32":
        W = W.astype(np.float32)
    return {"W": W, **{k: _sums(case, getattr(q, k)) for k in _LISTS}}


def _prep_batch(case, seed):
    from fastwigner_b200.batch import WignerMoyalBatch

    XA, PA, dt, V, dV = _box(case)
    q = WignerMoyalBatch(batch=case["batch"], X_gridDIM=case["X"], X_amplitude=XA, P_gridDIM=case["P"],
                         P_amplitude=PA, dt=dt, V=V, K=_kin, diff_V=dV, diff_K=_ident, precision=case["precision"])
    q.set_wignerfunctions(_packets(case, seed, case["batch"], case["P"], case["X"], XA, PA))
    return {"q": q}


def _run_batch(s):
    q, case = s["q"], s["case"]
    obs = q.propagate(case["steps"])
    return {"W": q.W, "obs": _sums(case, obs)}


def _prep_mask(case, seed):
    import fastwigner_b200 as fw

    XA, PA, dt, V, dV = _AMP, _AMP, 0.005, _dw, _ddw
    q = fw.WignerMoyalCUDA1D(t=0.0, dt=dt, X_gridDIM=case["X"], X_amplitude=XA, P_gridDIM=case["P"], P_amplitude=PA,
                             K="0.5 * P * P", V="0.05 * X * X * X * X - X * X", diff_K="P",
                             diff_V="0.2 * X * X * X - 2.0 * X", precision=case["precision"],
                             abs_boundary_x_p="pow(abs(sin(0.5 * M_PI * (X + X_amplitude) / X_amplitude)), dt * 0.5)")
    q.set_wignerfunction(_packets(case, seed, 1, case["P"], case["X"], XA, PA)[0])
    return {"q": q}


def _run_mask(s):
    q, case = s["q"], s["case"]
    _clear(q)
    W = q.propagate(case["steps"])
    return {"W": W.tensor, **{k: _sums(case, getattr(q, k)) for k in _LISTS}}


def _psi(x, seed):
    rng = np.random.default_rng(seed)
    x0, p0 = rng.uniform(-2, 2), rng.uniform(-1, 1)
    return np.exp(-((x - x0) ** 2) / (2 * 0.5 ** 2) + 1j * p0 * x)


def _prep_rho(case, seed):
    import fastwigner_b200 as fw

    q = fw.RhoVNeumannCUDA1D(X_gridDIM=case["N"], X_amplitude=_AMP, dt=0.005, t=0.0, K="0.5 * P * P",
                             V="0.05 * X * X * X * X - X * X", diff_K="P", diff_V="0.2 * X * X * X - 2.0 * X",
                             precision=case["precision"])
    psi = _t(_psi(q.X.reshape(-1), seed), torch.complex128)
    q.set_rho(psi[:, None] * psi.conj()[None, :])
    return {"q": q}


def _run_rho(s):
    q, case = s["q"], s["case"]
    _clear(q)
    r = q.propagate(case["steps"])
    out = {"rho": r.tensor, **{k: _sums(case, getattr(q, k)) for k in _LISTS}}
    if case["wigner"]:
        out["wigner"] = q.get_wignerfunction().tensor
    return out


def _wells(n, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(2, 10, n), rng.uniform(0.5, 1.5, n)


def _prep_bloch(case, seed):
    from fastwigner_b200.fno import BlochBatch, MorseBlochSetup

    setup = MorseBlochSetup(grid=case["G"])
    Ds, As = _wells(case["n"], seed)
    q = BlochBatch(setup, Ds, As).set_uniform()
    return {"q": q}


def _run_bloch(s):
    return s["q"].run(s["case"]["steps"]).W


def _mix(case):
    """Grid shapes and wells of an uneven batch (the program's fixed mix of systems)."""
    rng = np.random.default_rng(case["mix"])
    sizes = (128, 256, 512, 1024)
    return [dict(P=int(rng.choice(sizes)), X=int(rng.choice(sizes)), a=rng.uniform(0.02, 0.1),
                 b=rng.uniform(0.5, 2.0)) for _ in range(case["n"])]


def _prep_uneven(case, seed):
    from fastwigner_b200.batch import WignerMoyalUnevenBatch

    mix = _mix(case)
    specs = [dict(P_gridDIM=m["P"], X_gridDIM=m["X"], X_amplitude=_AMP, P_amplitude=_AMP,
                  V=(lambda x, m=m: m["a"] * x ** 4 - m["b"] * x ** 2), K=_kin) for m in mix]
    # the mode the autotuner picks for such mixes, fixed so that no timing decides
    q = WignerMoyalUnevenBatch(specs, dt=0.005, variant=0)
    q.set_variant(q.GROUPED)
    q.set_wignerfunctions([_packets(case, seed + 1000 * i, 1, m["P"], m["X"], _AMP, _AMP)[0].float()
                           for i, m in enumerate(mix)])
    obs = torch.empty((case["steps"], case["n"], 2), dtype=torch.float64, device=DEV)
    return {"q": q, "obs": obs}


def _run_uneven(s):
    q = s["q"]
    obs = q.propagate(s["case"]["steps"], obs=s["obs"])
    return {"W": list(q.W), "obs": obs.to(torch.float32)}


_OMEGA = 0.057
_T_LASER = 8 * 2 * math.pi / _OMEGA


def _laser(seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(0.01, 0.1), rng.uniform(1e-4, 1e-2)


def _field(E0, t):
    return E0 * np.sin(np.pi * t / _T_LASER) ** 2 * np.sin(_OMEGA * t)


_SF = dict(XA=200.0, PA=5.0, dt=0.05, t0=0.25 * _T_LASER, kT=0.1, dbeta=0.05)


def _sf_start(case, seed):
    x, p, _, _, dX, dP = _grid(case["P"], case["X"], _SF["XA"], _SF["PA"])
    rng = np.random.default_rng(seed + 7)
    x0, p0 = rng.uniform(-5, 5), rng.uniform(-0.5, 0.5)
    W = torch.exp(-0.25 * (_t(x) - x0) ** 2) * torch.exp(-4.0 * (_t(p) - p0) ** 2)
    return W / (W.sum() * dX * dP)


def _prep_strong(case, seed):
    from fastwigner_b200 import StrongFieldWigner

    E0, gamma = _laser(seed)
    q = StrongFieldWigner(X_gridDIM=case["X"], X_amplitude=_SF["XA"], P_gridDIM=case["P"], P_amplitude=_SF["PA"],
                          dt=_SF["dt"], t=_SF["t0"], V=lambda _, x: -1.0 / np.sqrt(x * x + 1.0),
                          diff_V=lambda _, x: x / (x * x + 1.0) ** 1.5, gauge="velocity",
                          E=lambda _, t: _field(E0, t), gamma=gamma, kT=_SF["kT"], dbeta=_SF["dbeta"],
                          precision=case["precision"])
    q.set_wignerfunction(_sf_start(case, seed))
    return {"q": q}


def _run_strong(s):
    q, case = s["q"], s["case"]
    _clear(q)
    q.propagate(case["steps"])
    return {"W": q.wigner_device, **{k: _sums(case, getattr(q, k)) for k in _LISTS}}


_FNO = dict(NP=3, C=32, m=16, layers=4, proj=128)


def _fno_params(seed):
    """Network parameters with the initialiser's distributions (FP32 values)."""
    rng = np.random.default_rng(seed)
    C, K = _FNO["C"], 2 * _FNO["m"] * _FNO["m"]

    def lin(o, i):
        b = 1.0 / math.sqrt(i)
        return rng.uniform(-b, b, (o, i)), rng.uniform(-b, b, (o,))

    p = {}
    p["W0"], p["b0"] = lin(C, _FNO["NP"] + 2)
    for l in range(_FNO["layers"]):
        p[f"R{l}"] = rng.uniform(0, 1.0 / (C * C), (C, C, 2, K))
        p[f"W{l + 1}"], p[f"b{l + 1}"] = lin(C, C)
    p["Q1"], p["c1"] = lin(_FNO["proj"], C)
    p["Q2"], p["c2"] = lin(1, _FNO["proj"])
    return {k: v.astype(np.float32) for k, v in p.items()}


def _fno_net(seed):
    from fastwigner_b200.fno import FNO2d

    net = FNO2d(n_params=_FNO["NP"], width=_FNO["C"], modes=(_FNO["m"], _FNO["m"]), layers=_FNO["layers"],
                proj=_FNO["proj"], seed=0)
    net.load_state_dict({**_fno_params(seed), "__in_scale__": np.ones(_FNO["NP"]),
                         "__in_shift__": np.zeros(_FNO["NP"])})
    return net


def _fno_inputs(case, seed):
    """Normalised (D, a, beta) rows and the grid coordinates over the box."""
    rng = np.random.default_rng(seed + 1)
    n, G = case["n"], case["G"]
    beta = np.exp(rng.uniform(math.log(2.0), math.log(20.0), n))
    raw = np.stack([rng.uniform(2, 10, n), rng.uniform(0.5, 1.5, n), beta], axis=1)
    xs = ((-8.0 + 16.0 / G * np.arange(G)) / 8.0).astype(np.float32)
    return raw, xs


def _norm(raw):
    return np.stack([raw[:, 0] / 10.0, raw[:, 1], np.log(raw[:, 2]) / np.log(20.0)], axis=1)


def _fno_target(raw, G):
    """Anharmonic-looking corrections: differences of two Gaussians per sample."""
    x = _t(-8.0 + 16.0 / G * np.arange(G))
    w = _t(raw[:, 1] * np.sqrt(2.0 * raw[:, 0]))[:, None, None]
    r = 0.5 * x[None, :, None] ** 2
    a = torch.exp(-2.0 / w * (r + 0.5 * (w * (x[None, None, :] + 2.0)) ** 2))
    b = torch.exp(-2.0 / w * (r + 0.5 * (w * (x[None, None, :] + 1.8)) ** 2))
    return (b - a).float()


def _prep_fno_train(case, seed):
    raw, xs = _fno_inputs(case, seed)
    return {"net": _fno_net(seed), "X": _norm(raw), "xs": xs, "T": _fno_target(raw, case["G"])}


def _run_fno_train(s):
    net = s["net"]
    loss, dY = net.loss_and_grad(s["X"], s["xs"], s["xs"], s["T"])
    grads = net.backward(dY)
    return {"loss": loss, "dY": dY, "grads": dict(grads)}


def _prep_fno_predict(case, seed):
    from fastwigner_b200.fno import BlochSurrogate, MorseBlochSetup

    raw, _ = _fno_inputs(case, seed)
    sur = BlochSurrogate(MorseBlochSetup(grid=case["G"]), _fno_net(seed))
    return {"sur": sur, "D": raw[:, 0], "a": raw[:, 1], "beta": float(raw[0, 2])}


def _run_fno_predict(s):
    return s["sur"].predict(s["D"], s["a"], s["beta"])


_PREPARE = dict(single=_prep_single, batch=_prep_batch, mask=_prep_mask, rho=_prep_rho, bloch=_prep_bloch,
                uneven=_prep_uneven, strong=_prep_strong, fno_train=_prep_fno_train, fno_predict=_prep_fno_predict)
_RUN = dict(single=_run_single, batch=_run_batch, mask=_run_mask, rho=_run_rho, bloch=_run_bloch,
            uneven=_run_uneven, strong=_run_strong, fno_train=_run_fno_train, fno_predict=_run_fno_predict)


# ---------------------------------------------------------------------------
# work of one pass: state read and written once, tables and inputs read once
# ---------------------------------------------------------------------------
def _phase_work(P, X, B, tables, steps, real, passes=2, extra_reals=0, tab_complex=True):
    pts = P * X * B
    tab = ((P // 2 + 1) * X + P * (X // 2 + 1)) * tables * real * (2 if tab_complex else 1)
    by = pts * real * (2 + extra_reals) + tab
    lg = math.log2(P) * (passes - 1) + math.log2(X)
    return by, steps * pts * (5.0 * lg + 10.0 * passes)  # real-data transforms there and back, factor products


def work(case):
    k = case["kind"]
    r = 8 if case.get("precision") == "float64" else 4
    if k in ("single", "batch", "mask"):
        by, fl = _phase_work(case["P"], case["X"], case.get("batch", 1), 1, case["steps"], r, extra_reals=k == "mask")
        return {"bytes": by, "flops": fl}
    if k == "bloch":
        by, fl = _phase_work(case["G"], case["G"], case["n"], case["n"], case["steps"], 4, tab_complex=False)
        return {"bytes": by, "flops": fl}
    if k == "uneven":
        parts = [_phase_work(m["P"], m["X"], 1, 1, case["steps"], 4) for m in _mix(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if k == "strong":
        by, fl = _phase_work(case["P"], case["X"], 1, 1, case["steps"], r, passes=3, extra_reals=1)
        return {"bytes": by + case["steps"] * (case["X"] // 2 + 1) * 2 * r, "flops": fl}
    if k == "rho":
        N = case["N"]
        step = N * N * (20.0 * math.log2(N) + 26.0)
        fl = case["steps"] * step
        by = 4 * r * N * N
        if case["wigner"]:
            fl += N * N * 35.0 * math.log2(N)
            by += 2 * r * N * N
        return {"bytes": by, "flops": fl}
    G, n, C, m = case["G"], case["n"], _FNO["C"], _FNO["m"]
    pix = G * G * n
    layer = pix * (2.0 * C * C + 2 * 2.0 * C * 2 * m) + n * C * 4 * 2.0 * (2 * 2 * m) * 2 * G * m / 2
    fwd = _FNO["layers"] * layer + pix * 2.0 * (C * (_FNO["NP"] + 2) + _FNO["proj"] * (C + 1))
    params = sum(v.size for v in _fno_params(0).values()) * 4
    if k == "fno_predict":
        return {"bytes": pix * 4 + params, "flops": fwd}
    return {"bytes": pix * 4 * 2 + 2 * params, "flops": 3 * fwd}


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------
def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)


def _half(W, tab, dim, n):
    F = torch.fft.rfft(W, dim=dim)
    F *= tab
    return torch.fft.irfft(F, n=n, dim=dim)


def _tabs(P, X, XA, PA, dt, V):
    x, p, th, la, dX, dP = _grid(P, X, XA, PA)
    x, p, th, la = _t(x), _t(p), _t(th), _t(la)
    ev = torch.exp(-0.5j * dt * (V(x - 0.5 * th) - V(x + 0.5 * th)))
    ek = torch.exp(-1j * dt * (_kin(p + 0.5 * la) - _kin(p - 0.5 * la)))
    return ev, ek, dX * dP


def _weights(P, X, XA, PA, V, dV):
    x, p, *_ = _grid(P, X, XA, PA)
    x, p = _t(x[0]), _t(p[:, 0])
    return torch.stack([x, dV(x), V(x)]), torch.stack([p, p, _kin(p)])


def _steps(W, ev, ek, dxdp, steps, wx=None, wp=None, mask=None):
    """Normalised V/2 K V/2 steps; per step and instance [sum W, sum W^2, x sums, p sums]."""
    n = W.shape[0]
    P, X = W.shape[-2:]
    obs = []
    for _ in range(steps):
        W = _half(_half(_half(W, ev, 1, P), ek, 2, X), ev, 1, P)
        if mask is not None:
            W = W * mask
        s = W.sum(dim=(1, 2))
        rec = [s, (W * W).sum(dim=(1, 2))]
        if wx is not None:
            rec += list((W.sum(dim=1) @ wx.T).T) + list((W.sum(dim=2) @ wp.T).T)
        obs.append(torch.stack(rec, dim=1))
        W = W / (s * dxdp).view(n, 1, 1)
    return W, torch.stack(obs)


def _averages(o):
    S = o[:, 0]
    return {"X_average": (o[:, 2] / S).cpu().numpy(), "P_average": (o[:, 5] / S).cpu().numpy(),
            "X_average_RHS": (o[:, 6] / S).cpu().numpy(), "P_average_RHS": (-o[:, 3] / S).cpu().numpy(),
            "hamiltonian_average": ((o[:, 7] + o[:, 4]) / S).cpu().numpy()}


def _exact_phase(case, seed):
    k = case["kind"]
    P, X = case["P"], case["X"]
    XA, PA, dt, V, dV = (_AMP, _AMP, 0.005, _dw, _ddw) if k == "mask" else _box(case)
    ev, ek, dxdp = _tabs(P, X, XA, PA, dt, V)
    wx, wp = _weights(P, X, XA, PA, V, dV)
    B = case.get("batch", 1)
    W0 = _packets(case, seed, B, P, X, XA, PA).to(_real(case)).double()
    mask = None
    if k == "mask":
        x, _, _, _, dX, _ = _grid(P, X, XA, PA)
        mask = torch.abs(torch.sin(0.5 * math.pi * (_t(x) + XA) / XA)) ** (0.5 * dt)
    Ws, obs = [], []
    per = max(1, (32 << 20) // (P * X))
    for b in range(0, B, per):
        W, o = _steps(W0[b:b + per], ev, ek, dxdp, case["steps"], wx, wp, mask)
        Ws.append(W)
        obs.append(o)
    W, obs = torch.cat(Ws), torch.cat(obs, dim=1)
    if k == "batch":
        return {"W": W, "obs": obs}
    return {"W": W[0].cpu().numpy() if k == "single" else W[0], **_averages(obs[:, 0])}


def _exact_rho(case, seed):
    N, dt = case["N"], 0.005
    dX = 2.0 * _AMP / N
    x = dX * (np.arange(N) - 0.5 * N)
    freq = np.fft.fftfreq(N, dX / (2 * np.pi))
    dP = freq[1] - freq[0]
    pk = dP * ((np.arange(N) + N // 2) % N - 0.5 * N)
    psi = _t(_psi(np.linspace(-_AMP, _AMP - dX, N), seed), torch.complex128)
    rho = psi[:, None] * psi.conj()[None, :]
    rho = rho / (torch.diagonal(rho).sum() * dX)
    xt, pt = _t(x), _t(pk)
    uV, uK = torch.exp(-0.5j * dt * _dw(xt)), torch.exp(-1j * dt * _kin(pt))
    eV, eK = uV[None, :] * uV.conj()[:, None], uK[None, :] * uK.conj()[:, None]
    rows = []
    for _ in range(case["steps"]):
        rho = eV * torch.fft.ifft2(torch.fft.fft2(rho * eV) * eK)
        tr = torch.diagonal(rho).sum()
        d = torch.diagonal(rho) / tr
        m = [torch.diagonal(torch.fft.ifft(torch.fft.fft(rho, dim=1) * g, dim=1)).sum() / tr for g in (pt, _kin(pt))]
        rows.append(torch.stack([(d * xt).sum(), m[0], m[0], -(d * _ddw(xt)).sum(), m[1] + (d * _dw(xt)).sum()]).real)
        rho = rho / (tr * dX)
    rows = torch.stack(rows).cpu().numpy()
    out = {"rho": rho, **{k: rows[:, i] for i, k in enumerate(_LISTS)}}
    if case["wigner"]:
        a, b = math.tan(math.pi / 8.0), -math.sin(math.pi / 4.0)
        px = torch.exp(-1j * a * pt[None, :] * xt[:, None])
        py = torch.exp(-1j * b * xt[None, :] * pt[:, None])
        w = torch.fft.ifft(torch.fft.fft(rho, dim=1) * px, dim=1)
        w = torch.fft.ifft(torch.fft.fft(w, dim=0) * py, dim=0)
        w = torch.fft.ifft(torch.fft.fft(w, dim=1) * px, dim=1)
        sg = _t(1.0 - 2.0 * (np.arange(N) % 2))[:, None]
        w = sg * torch.fft.ifft(sg * w, dim=0)
        out["wigner"] = w / (w.sum() * 0.5 * dX * dP)
    return out


def _exact_bloch(case, seed):
    G, n, db = case["G"], case["n"], 1e-3
    x, p, th, la, dX, dP = _grid(G, G, 8.0, 8.0)
    x, p, th, la = _t(x), _t(p), _t(th), _t(la)
    Ds, As = _wells(n, seed)
    out = []
    for D, a in zip(Ds, As):
        V = lambda u: D * (1.0 - torch.exp(-a * (u + 2.0))) ** 2  # noqa: E731, B023
        vs = V(x - 0.5 * th) + V(x + 0.5 * th)
        ks = _kin(p + 0.5 * la) + _kin(p - 0.5 * la)
        W = torch.full((1, G, G), 1.0 / (dX * dP * G * G), dtype=torch.float64, device=DEV)
        out.append(_steps(W, torch.exp(-0.25 * db * (vs - vs.min())), torch.exp(-0.5 * db * (ks - ks.min())),
                          dX * dP, case["steps"])[0])
    return torch.cat(out)


def _exact_uneven(case, seed):
    Ws, obs = [], []
    for i, m in enumerate(_mix(case)):
        V = lambda u, m=m: m["a"] * u ** 4 - m["b"] * u ** 2  # noqa: E731
        ev, ek, dxdp = _tabs(m["P"], m["X"], _AMP, _AMP, 0.005, V)
        W0 = _packets(case, seed + 1000 * i, 1, m["P"], m["X"], _AMP, _AMP)
        W, o = _steps(W0, ev, ek, dxdp, case["steps"])
        Ws.append(W[0])
        obs.append(o[:, 0])
    return {"W": Ws, "obs": torch.stack(obs, dim=1)}


def _exact_strong(case, seed):
    E0, gamma = _laser(seed)
    P, X, dt = case["P"], case["X"], _SF["dt"]
    x, p, th, la, dX, dP = _grid(P, X, _SF["XA"], _SF["PA"])
    x, p, th, la = _t(x), _t(p), _t(th), _t(la)
    dxdp = dX * dP
    V = lambda u: -1.0 / torch.sqrt(u * u + 1.0)  # noqa: E731
    dV = lambda u: u / (u * u + 1.0) ** 1.5  # noqa: E731
    t0 = _SF["t0"]
    gx, gw = np.polynomial.legendre.leggauss(200)

    def A(t):  # -int_0^t E, one 200-point rule over at most a few optical cycles per piece
        edges = np.linspace(0.0, t, 9)
        h = 0.5 * np.diff(edges)
        mid = 0.5 * (edges[1:] + edges[:-1])
        return -float((h[:, None] * gw * _field(E0, mid[:, None] + h[:, None] * gx)).sum())

    A0 = A(t0)
    n = round(1.0 / (_SF["kT"] * _SF["dbeta"]))
    db = 1.0 / (_SF["kT"] * n)
    vs = V(x - 0.5 * th) + V(x + 0.5 * th)
    ks = _kin(p + A0 + 0.5 * la) + _kin(p + A0 - 0.5 * la)
    bv, bk = torch.exp(-0.5 * db * (vs - vs.min())), torch.exp(-db * (ks - ks.min()))
    W = torch.full((1, P, X), 1.0 / (dxdp * P * X), dtype=torch.float64, device=DEV)
    gibbs = _steps(W, bv, bk, dxdp, n)[0][0]
    c = math.exp(-0.5 * gamma * dt)
    s0 = gibbs * (1 - c)
    ev = torch.exp(-0.5j * dt * (V(x - 0.5 * th) - V(x + 0.5 * th)))
    W = _sf_start(case, seed)
    rows = []
    gx_mean, gp_mean = (gibbs * x).sum() / gibbs.sum(), (gibbs * p).sum() / gibbs.sum()
    for k in range(case["steps"]):
        a = A(t0 + dt * (k + 1))
        ek = torch.exp(-1j * dt * la * (p + a))
        W = c * W + s0
        W = _half(_half(_half(W, ev, 0, P), ek, 1, X), ev, 0, P)
        W = c * W + s0
        S = W.sum()
        av = lambda f: (W * f).sum() / S  # noqa: E731, B023
        xm, pm = av(x), av(p)
        rows.append(torch.stack([xm, pm, pm + a + gamma * (gx_mean - xm), -av(dV(x)) + gamma * (gp_mean - pm),
                                 av(0.5 * (p + a) ** 2) + av(V(x))]))
        W = W / (S * dxdp)
    rows = torch.stack(rows).cpu().numpy()
    return {"W": W, **{k: rows[:, i] for i, k in enumerate(_LISTS)}}


def _fno_forward(par, X, xs, G):
    """The surrogate network in plain FP64 torch (differentiable in `par`)."""
    m, C, n = _FNO["m"], _FNO["C"], X.shape[0]
    kp = np.concatenate([np.arange(m), np.arange(G - m, G)])
    f = torch.cat([X[:, :, None, None].expand(n, _FNO["NP"], G, G), xs[None, None, None, :].expand(n, 1, G, G),
                   xs[None, None, :, None].expand(n, 1, G, G)], dim=1)
    ch = lambda w, b, v: torch.einsum("oi,bixy->boxy", w, v) + b[None, :, None, None]  # noqa: E731
    v = ch(par["W0"], par["b0"], f)
    for l in range(_FNO["layers"]):
        F = torch.fft.rfft2(v, norm="forward")[:, :, kp, :m].reshape(n, C, 2 * m * m)
        O = torch.einsum("bik,iok->bok", F, torch.complex(par[f"R{l}"][:, :, 0], par[f"R{l}"][:, :, 1]))
        O = O.reshape(n, C, 2 * m, m)
        full = torch.zeros((n, C, G, G // 2 + 1), dtype=O.dtype, device=DEV)
        full[:, :, kp, :m] = O
        y = torch.fft.irfft(torch.fft.ifft(full, dim=2, norm="forward"), n=G, dim=3, norm="forward")
        v = y + ch(par[f"W{l + 1}"], par[f"b{l + 1}"], v)
        if l < _FNO["layers"] - 1:
            v = torch.nn.functional.gelu(v)
    out = []
    for b in range(n):  # the 128-channel hidden layer one sample at a time
        a = torch.nn.functional.gelu(ch(par["Q1"], par["c1"], v[b:b + 1]))
        out.append(ch(par["Q2"], par["c2"], a)[:, 0])
    return torch.cat(out)


def _exact_fno_train(case, seed):
    raw, xs = _fno_inputs(case, seed)
    G = case["G"]
    par = {k: _t(v).requires_grad_() for k, v in _fno_params(seed).items()}
    T = _fno_target(raw, G).double()
    Y = _fno_forward(par, _t(_norm(raw).astype(np.float32)), _t(xs), G)
    Yd = Y.detach().requires_grad_()
    loss = (((Yd - T) ** 2).sum(dim=(1, 2)) / (T ** 2).sum(dim=(1, 2))).mean()
    loss.backward()
    Y.backward(Yd.grad)
    return {"loss": float(loss), "dY": Yd.grad, "grads": {k: v.grad for k, v in par.items()}}


def _exact_fno_predict(case, seed):
    raw, _ = _fno_inputs(case, seed)
    n, G = case["n"], case["G"]
    raw[:, 2] = raw[0, 2]
    x = -8.0 + 16.0 / G * np.arange(G)
    par = {k: _t(v) for k, v in _fno_params(seed).items()}
    xs = _t((np.linspace(-8.0, 8.0 - 16.0 / G, G) / 8.0).astype(np.float32))
    res = []
    for b in range(n):
        Y = _fno_forward(par, _t(_norm(raw[b:b + 1]).astype(np.float32)), xs, G)[0]
        w = raw[b, 1] * math.sqrt(2.0 * raw[b, 0])
        H = 0.5 * _t(x)[:, None] ** 2 + 0.5 * (w * (_t(x)[None, :] + 2.0)) ** 2
        base = torch.exp(-2.0 / w * math.tanh(0.5 * raw[b, 2] * w) * (H - H.min()))
        base = base / base.sum()
        o = base + base.max() * Y
        res.append(o / (o.sum() * (16.0 / G) ** 2))
    return torch.stack(res)


_EXACT = dict(single=_exact_phase, batch=_exact_phase, mask=_exact_phase, rho=_exact_rho, bloch=_exact_bloch,
              uneven=_exact_uneven, strong=_exact_strong, fno_train=_exact_fno_train, fno_predict=_exact_fno_predict)
