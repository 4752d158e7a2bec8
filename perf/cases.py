"""Performance cases of the framework: what its users have it do, through its
public entry points, from the smallest calls to the benchmark's grid.

listed() names the fixed cases and draw(rng) gives one more of the same
ranges; prepare(case, seed) makes what a user's program holds before the call,
run(state) makes one pass, work(case) says what a pass cannot do without, and
exact(case, seed) gives a pass's outputs in plain torch in 64 bits.

Kinds of cases:
  flow   `steps` steps of DeviceFlowfield.run, then the state is downloaded (a
         program's run between two outputs).  Set-ups: "rsbi", a Mach 2 shock
         in air and an H2-O2 bubble; "znd", the 1D detonation initiation;
         "odw", the oblique detonation over a wedge, from a developed state.
  host   the reference's convention: the state lives in host arrays and the
         member calls (decode, ghost fill, dt, advection, chemistry) work on it.
  infer  the learned chemistry's network over device arrays.
  train  optimiser steps of that network from given weights.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from eu3d_b200 import gpu
from eu3d_b200 import surrogate as S
from eu3d_b200.cases import odw_case, setup_odw
from eu3d_b200.readers import load_h2_ja919, make_grid, stoichiometric_h2_air

ATM = 101325.0
R_GAS = 8.31434
RU_CAL = 1.987
BC = {"rsbi": gpu.BC_RSBI, "znd": gpu.BC_TRANSMISSIVE, "odw": gpu.BC_ODM}
REACT = {"imex": gpu.REACT_IMEX, "none": gpu.REACT_NONE, "surrogate": gpu.REACT_SURROGATE,
         "adaptive": gpu.REACT_ADAPTIVE}
ADV = {"ee": gpu.ADV_EE, "rk2": gpu.ADV_SSPRK2, "rk3": gpu.ADV_SSPRK3}
STAGES = {"ee": 1, "rk2": 2, "rk3": 3}
DIFF = {"muscl1": gpu.DIFF_MUSCL1, "muscl2": gpu.DIFF_MUSCL2, "weno": gpu.DIFF_WENO}


def _flow(name, setup, ni, nj, nk, bits, react, adv, diff, cfl, steps):
    return dict(name=name, kind="flow", setup=setup, ni=ni, nj=nj, nk=nk, bits=bits, react=react, adv=adv, diff=diff,
                cfl=cfl, steps=steps)


def listed():
    return [
        # the 1D ZND detonation at its full size, FP64 throughout: the smallest
        # run a user makes, bound by launches
        _flow("znd_1d_fp64", "znd", 4000, 2, 2, 64, "imex", "rk2", "muscl2", 0.3, 20),
        # the reference's shipped grid and scheme: 2D shock-bubble, explicit Euler,
        # one-step IMEX, FP64 (the constructor's default)
        _flow("rsbi_2d_fp64_ee", "rsbi", 241, 81, 2, 64, "imex", "ee", "muscl2", 0.3, 20),
        # the 2D oblique detonation of the benchmark's odw2d configuration
        _flow("odw_2d_fp32_imex", "odw", 1024, 512, 2, 32, "imex", "rk2", "muscl2", 0.5, 20),
        # the accuracy reference of the learned chemistry, and the runs its
        # training snapshots come from: all-FP64 flow with the adaptive integrator
        _flow("odw_2d_fp64_adaptive", "odw", 512, 256, 2, 64, "adaptive", "rk2", "muscl2", 0.5, 10),
        # the 3D shock-bubble in the default precision at an intermediate size
        _flow("rsbi_3d_fp64", "rsbi", 160, 160, 160, 64, "imex", "rk2", "muscl2", 0.5, 8),
        # the 3D shock-bubble at its benchmark size, FP32 flux
        _flow("rsbi_3d_fp32", "rsbi", 256, 256, 256, 32, "imex", "rk2", "muscl2", 0.5, 10),
        # ragged extents with the other reconstruction and time scheme
        _flow("rsbi_3d_fp32_weno_rk3", "rsbi", 150, 131, 97, 32, "imex", "rk3", "weno", 0.5, 10),
        # the benchmark's flagship: 3D oblique detonation with the learned chemistry,
        # half the benchmark's span so that several states fit the card
        _flow("odw_3d_fp32_surrogate", "odw", 512, 256, 128, 32, "surrogate", "rk2", "muscl2", 0.5, 40),
        # a ported program that keeps the reference's host arrays: every step
        # uploads, calls the members and downloads (hot reacting mixture)
        dict(name="host_step_fp64_imex", kind="host", ni=121, nj=81, nk=61, bits=64, react="imex", dt=0.0),
        # the same with the reference's adaptive trapezoid (Euler::Trapezoid type 1), warm gas
        dict(name="host_step_fp64_trapezoid", kind="host", ni=241, nj=81, nk=2, bits=64, react="trapezoid", dt=5e-9),
        # the learned chemistry's network alone, at the benchmark's state count and ragged
        dict(name="network_infer", kind="infer", n=4194304 - 37),
        # fitting the network: the recipe's batch size
        dict(name="network_train", kind="train", samples=131072, batch=8192, steps=200),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("rsbi", "rsbi", "rsbi", "odw", "odw", "znd", "host", "host", "infer", "train"))
    if kind == "rsbi":
        bits = rng.choice((32, 64))
        cells = math.exp(rng.uniform(math.log(2e4), math.log(8e6 if bits == 32 else 3e6)))
        nk = rng.choice((2, _logint(rng, 9, 160)))
        ni = max(17, min(600, int(math.sqrt(cells / nk) * rng.uniform(0.8, 2.0))))
        nj = max(9, min(600, int(cells / nk / ni)))
        adv = rng.choice(("ee", "rk2", "rk2", "rk3"))
        return dict(kind="flow", setup="rsbi", ni=ni, nj=nj, nk=nk, bits=bits,
                    react=rng.choice(("imex", "imex", "none")), adv=adv,
                    diff=rng.choice(("muscl1", "muscl2", "muscl2", "weno")), cfl=0.3 if adv == "ee" else 0.5,
                    steps=rng.randint(4, 10))
    if kind == "odw":
        react = rng.choice(("surrogate", "surrogate", "imex", "adaptive"))
        nj = _logint(rng, 96, 256 if react == "adaptive" else 320)
        nk = 2 if react == "adaptive" else rng.choice((2, _logint(rng, 5, 64)))
        return dict(kind="flow", setup="odw", ni=2 * nj + rng.randint(0, 9), nj=nj, nk=nk,
                    bits=32 if react == "surrogate" else rng.choice((32, 64)), react=react, adv="rk2", diff="muscl2",
                    cfl=0.5, steps=rng.randint(4, 10))
    if kind == "znd":
        return dict(kind="flow", setup="znd", ni=_logint(rng, 500, 8000), nj=2, nk=2, bits=rng.choice((32, 64)),
                    react=rng.choice(("imex", "adaptive")), adv="rk2", diff="muscl2", cfl=0.3, steps=rng.randint(5, 20))
    if kind == "host":
        react = rng.choice(("imex", "trapezoid"))
        return dict(kind="host", ni=_logint(rng, 16, 200), nj=_logint(rng, 9, 100), nk=rng.choice((2, _logint(rng, 3, 40))),
                    bits=rng.choice((32, 64)), react=react, dt=5e-9 if react == "trapezoid" else 0.0)
    if kind == "infer":
        return dict(kind="infer", n=_logint(rng, 200, 4_000_000))
    return dict(kind="train", samples=_logint(rng, 10_000, 131_072), batch=256 * rng.randint(1, 32),
                steps=rng.randint(20, 200))


# ------------------------------------------------------------------ inputs
_MECH = None


def _mech():
    global _MECH
    if _MECH is None:
        _MECH = load_h2_ja919()
    return _MECH


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=_device())


def _pick(cond, a, b):
    return torch.where(cond, _t(a), _t(b))


def _thermo(T):
    """Per-species Cp/R, H/R, S/R lists at T (NASA-9, two ranges split at 1000 K)."""
    m = _mech()
    hi = T >= 1000.0
    lnT, i1 = torch.log(T), 1.0 / T
    cp, h, s = [], [], []
    for k in range(m.NS):
        a = [_pick(hi, m.c1[q][k], m.c0[q][k]) for q in range(9)]
        cp.append(a[0] * i1 * i1 + a[1] * i1 + a[2] + T * (a[3] + T * (a[4] + T * (a[5] + T * a[6]))))
        h.append(-a[0] * i1 + a[1] * lnT + a[7] + T * (a[2] + T * (a[3] / 2 + T * (a[4] / 3 + T * (a[5] / 4 + T * a[6] / 5)))))
        s.append(-a[0] * i1 * i1 / 2 - a[1] * i1 + a[2] * lnT + a[8] + T * (a[3] + T * (a[4] / 2 + T * (a[5] / 3 + T * a[6] / 4))))
    return cp, h, s


def _conserved(P, T, U, V, W, Y):
    """(..., 13) conserved variables of a primitive state; Y (..., 9)."""
    m = _mech()
    ri = [R_GAS / float(w) for w in m.mw]
    _, h, _ = _thermo(T)
    rg = sum(Y[..., k] * ri[k] for k in range(9)) * 1e3
    e = sum(Y[..., k] * (ri[k] * h[k] - ri[k] * T) for k in range(9)) * 1e3
    D = P / (rg * T)
    mom = torch.stack((D * U, D * V, D * W, D * e + 0.5 * D * (U * U + V * V + W * W)), dim=-1)
    return torch.cat((D[..., None] * Y, mom), dim=-1)


def _grid(case):
    if case.get("setup") == "znd":
        dx = 0.1 / (case["ni"] - 1)
        return make_grid(case["ni"], 0.0, 0.1, 2, 0.0, dx, 2, 0.0, dx, 2, fixed_ghosts=True)
    dx = (0.1 if case["kind"] == "flow" else 0.01) / (case["ni"] - 1)
    return make_grid(case["ni"], 0.0, dx * (case["ni"] - 1), case["nj"], 0.0, dx * max(case["nj"] - 1, 1), case["nk"],
                     0.0, dx * max(case["nk"] - 1, 1), 2, fixed_ghosts=True)


def _axes(g):
    return (_t(g.xnode)[:, None, None], _t(g.ynode)[None, :, None], _t(g.znode)[None, None, :])


def _mixture(moles):
    m = _mech()
    y = np.zeros(m.NS)
    for k, v in moles.items():
        y[m.species.index(k)] = v * m.mw[m.species.index(k)]
    return y / y.sum()


def _initial(case, seed):
    """The start of a "rsbi" or "znd" run, or the mixture of a "host" step, on
    every cell (ghosts included): grid, CS (NI, NJ, NK, 13) and T."""
    rng = np.random.default_rng(seed)
    g = _grid(case)
    x, y, z = _axes(g)
    shape = (g.ni + 4, g.nj + 4, g.nk + 4)
    if case["kind"] == "host":
        gen = torch.Generator(device=_device()).manual_seed(int(seed) & 0x7FFFFFFF)

        def noise(k=1):
            return torch.randn(shape + (() if k == 1 else (k,)), generator=gen, device=_device(), dtype=torch.float64)

        ph = rng.uniform(0, 2 * np.pi, 8)
        ax, ay, az = (2 * math.pi * torch.linspace(0, 1, n, dtype=torch.float64, device=_device()) for n in shape)
        ax, ay, az = ax[:, None, None], ay[None, :, None], az[None, None, :]
        sm = 0.5 + 0.25 * (torch.sin(ax + ph[0]) * torch.cos(ay + ph[1]) + torch.sin(az + ph[2]) * torch.cos(ax + ph[3]))
        # (the reference's trapezoid does not bear a hotter gas or more radicals)
        lo, span, rad = (1100.0, 1500.0, 1e-3) if case["react"] == "imex" else (450.0, 530.0, 1e-3)
        T = lo + span * torch.clamp(sm + 0.02 * noise(), 0, 1)
        P = ATM * (1.0 + 0.3 * torch.sin(ay + ph[4]) * torch.sin(az + ph[5]) + 0.02 * noise().clamp(-3, 3))
        U = 300.0 * torch.sin(ax + ph[6]) + 30.0 * noise()
        V = 200.0 * torch.cos(ay + ph[7]) + 20.0 * noise()
        W = 100.0 * torch.sin(az + ph[0]) + 10.0 * noise()
        m = _mech()
        X = torch.zeros(shape + (9,), dtype=torch.float64, device=_device())
        sp = m.species.index
        X[..., sp("H2")] = 2.0 * (1 + 0.3 * torch.sin(ax + ay))
        X[..., sp("O2")] = 1.0 + 0.2 * torch.cos(ay + az)
        X[..., sp("N2")] = 3.76
        r = torch.rand(shape + (6,), generator=gen, device=_device(), dtype=torch.float64)
        for n, k in enumerate(("H", "O", "OH", "HO2", "H2O2")):
            X[..., sp(k)] = rad * (0.2 + 0.8 * r[..., n])
        X[..., sp("H2O")] = 0.3 * r[..., 5]
        Y = X * _t(m.mw)
        Y = Y / Y.sum(-1, keepdim=True)
        return g, _conserved(P, T, U, V, W, Y), T
    zero = torch.zeros(shape, dtype=torch.float64, device=_device())
    if case["setup"] == "znd":
        drv = (x < 0.005).expand(shape)
        wave = 1.0 + 0.01 * torch.sin(2 * math.pi * x / 0.1 * rng.integers(3, 9) + rng.uniform(0, 6.28)).expand(shape)
        P = _pick(drv, 30 * ATM, ATM)
        T = torch.where(drv, 3000.0 + 0 * wave, 300.0 * wave)
        Y = torch.where(drv[..., None], _t(_mixture({"H2O": 2.0, "N2": 3.76})), _t(stoichiometric_h2_air(_mech())))
        return g, _conserved(P, T, zero, zero, zero, Y), T
    # shock-bubble: Mach 2 shock from x = 0.1 Lx towards a wavy H2-O2 bubble;
    # the gas ahead carries 1 % smooth seeded temperature waves
    L = [float(a[-3] - a[2]) for a in (g.xnode, g.ynode, g.znode)]
    dx = float(g.xnode[3] - g.xnode[2])
    flat = case["nk"] < 8
    cx, cy, cz = x - 0.45 * L[0], y - 0.5 * L[1], (0 * z if flat else z - 0.5 * L[2])
    R0 = 0.25 * min(L[:2] if flat else L)
    r = torch.sqrt(cx * cx + cy * cy + cz * cz)
    th, phi = torch.atan2(cy + 0 * cx, cx + 0 * cy), torch.atan2(cz + 0 * cx, torch.sqrt(cx * cx + cy * cy) + 1e-30)
    wob = sum(float(rng.uniform(-1, 1)) * torch.cos(n * th + float(rng.uniform(0, 6.28))) * torch.cos((n % 3) * phi)
              for n in range(2, 7)) / 5
    chi = 0.5 * (1.0 - torch.tanh((r - R0 * (1 + 0.05 * wob)) / (2.0 * dx)))
    Y = chi[..., None] * _t(_mixture({"H2": 2.0, "O2": 1.0})) + (1 - chi[..., None]) * _t(_mixture({"O2": 1.0, "N2": 3.76}))
    ph = rng.uniform(0, 6.28, 3)
    wave = 1.0 + 0.01 * (torch.sin(6.28 * 4 * x / L[0] + ph[0]) * torch.cos(6.28 * 3 * y / L[1] + ph[1])
                         * (1.0 if flat else torch.cos(6.28 * 2 * z / L[2] + ph[2])))
    m2 = 4.0
    P1 = ATM * (1 + 2 * 1.4 / 2.4 * (m2 - 1))
    T1 = 300.0 * (2 + 0.4 * m2) / (2.4 * m2) * P1 / ATM
    U1 = 2.0 * (1 - (2 + 0.4 * m2) / (2.4 * m2)) * math.sqrt(1.4 * 287 * 300.0)
    post = (x < 0.1 * L[0]).expand(shape)
    T = torch.where(post, T1, 300.0 * wave.expand(shape))
    return g, _conserved(_pick(post, P1, ATM), T, _pick(post, U1, 0.0), zero, zero, Y), T


def _pinned(shape):
    t = torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return t, t.numpy()


def _host(t):
    p, a = _pinned(tuple(t.shape))
    p.copy_(t)
    return a


def _prepare_flow(case, seed):
    m = _mech()
    out = {}
    if case["setup"] == "odw":
        # a developed oblique detonation: the 2D case run from the free stream
        # with the learned chemistry, extruded along z
        model = S.SurrogateModel.load(S.DEFAULT_MODEL)
        c2 = odw_case(m, case["ni"], case["nj"], 2, seed=int(seed) & 0x7FFFFFFF)
        d2 = gpu.DeviceFlowfield(m, c2.grid, gpu.QUIRKS_FIXED, flux_bits=32)
        setup_odw(d2, c2)
        s2 = model.attach(d2, 0, gate=S.GATE)
        d2.run(1500, react=gpu.REACT_SURROGATE, timeadv=gpu.ADV_SSPRK2, bc_kind=gpu.BC_ODM, cfl=0.5, final_time=1.0)
        cs2, T2 = d2.download("CS")[:, :, 2], d2.download("T")[:, :, 2]
        d2.set_surrogate(None)
        s2.close()
        d2.close()
        c3 = odw_case(m, case["ni"], case["nj"], case["nk"], seed=int(seed) & 0x7FFFFFFF)
        dev = gpu.DeviceFlowfield(m, c3.grid, gpu.QUIRKS_FIXED, flux_bits=case["bits"])
        setup_odw(dev, c3)
        dev.set_elements(S.atoms_matrix(m))
        if case["react"] == "surrogate":
            out["sur"] = model.attach(dev, 4099, gate=S.GATE)
        nk = case["nk"] + 4
        cs = _t(cs2)[:, :, None].expand(-1, -1, nk, -1)
        T = _t(T2)[:, :, None].expand(-1, -1, nk)
    else:
        g, cs, T = _initial(case, seed)
        dev = gpu.DeviceFlowfield(m, g, gpu.QUIRKS_FIXED, flux_bits=case["bits"])
        dev.set_elements(S.atoms_matrix(m))
    a = _host(cs)
    dev.upload("CS", a)
    b = _host(T)
    dev.upload("T", b)
    dev.update_after_cs()
    dev.synchronize()
    # the download goes to the pinned arrays the state came from
    out.update(dev=dev, CS=a, T=b, steps=case["steps"],
               kw=dict(react=REACT[case["react"]], timeadv=ADV[case["adv"]], diff=DIFF[case["diff"]],
                       bc_kind=BC[case["setup"]], cfl=case["cfl"], final_time=1.0))
    return out


def _network_inputs(n, seed):
    gen = torch.Generator(device=_device()).manual_seed(int(seed) & 0x7FFFFFFF)
    X = torch.zeros((n, 16), dtype=torch.float32, device=_device())
    X[:, :12] = torch.randn((n, 12), generator=gen, device=_device())
    for col, src in ((12, 0), (13, 1), (14, 11)):
        X[:, col] = (X[:, src] - X[:, src].bfloat16().float()) * 256.0
    return X


def _small_handle():
    return gpu.DeviceFlowfield(_mech(), make_grid(8, 0.0, 1.0, 4, 0.0, 1.0, 2, 0.0, 1.0, 2, fixed_ghosts=True),
                               gpu.QUIRKS_FIXED, flux_bits=32)


def prepare(case, seed):
    m = _mech()
    st = dict(kind=case["kind"], case=case)
    if case["kind"] == "flow":
        st.update(_prepare_flow(case, seed))
    elif case["kind"] == "host":
        g, cs, T = _initial(case, seed)
        dev = gpu.DeviceFlowfield(m, g, gpu.QUIRKS_FIXED, flux_bits=case["bits"])
        st.update(dev=dev, CS=_host(cs), T=_host(T), CS1=_pinned(tuple(cs.shape))[1], T1=_pinned(tuple(T.shape))[1],
                  P1=_pinned(tuple(T.shape))[1])
    elif case["kind"] == "infer":
        dev = _small_handle()
        X = _network_inputs(case["n"], seed)
        st.update(dev=dev, sur=S.SurrogateModel.load(S.DEFAULT_MODEL).attach(dev), X=X,
                  out=torch.zeros((case["n"], 16), dtype=torch.float32, device=X.device), n=case["n"])
    else:
        dev = _small_handle()
        sur = gpu.DeviceSurrogate(dev, case["samples"], S.atoms_matrix(m))
        rec = S.Recipe()
        env = (rec.T_range[0], rec.T_range[1], np.log(rec.p_atm_range[0]), np.log(rec.p_atm_range[1]),
               np.log(rec.dt_range[0]), np.log(rec.dt_range[1]))
        sur.add_random(case["samples"], env, S.species_index(m), int(seed) & 0x7FFFFFFF)
        sur.label(gpu.REACT_ADAPTIVE, rec.label_cap)
        X, Lb = sur.dataset(0, min(case["samples"], 32768))
        sur.set_norm(S.make_norm(m, X, Lb, rec.Ta, rec.Tr, env, delta=rec.delta, lin_quantile=rec.lin_quantile,
                                 lin_T=rec.lin_T))
        st.update(dev=dev, sur=sur, p0=S.init_params(int(seed) & 0x7FFFFFFF), batch=case["batch"], steps=case["steps"])
    return st


def run(state):
    kind = state["kind"]
    dev = state["dev"]
    if kind == "flow":
        dev.run(state["steps"], **state["kw"])
        return {"CS": dev.download("CS", state["CS"]), "T": dev.download("T", state["T"])}
    if kind == "host":
        case = state["case"]
        dev.upload("CS", state["CS"])
        dev.upload("T", state["T"])
        dev.update_after_cs()
        dev.boundary(gpu.BC_RSBI)
        if case["react"] == "imex":
            dev.set_time(0.0)
            dt = dev.cfl(0.3, 1.0)
            dev.advection()
            dev.imex()
        else:
            dev.dt = dt = case["dt"]
            dev.advection()
            dev.trapezoid(1)
        return {"CS": dev.download("CS", state["CS1"]), "T": dev.download("T", state["T1"]),
                "P": dev.download("P", state["P1"]), "dt": dt}
    if kind == "infer":
        state["sur"].infer_device(state["X"].data_ptr(), state["n"], state["out"].data_ptr(),
                                  torch.cuda.current_stream().cuda_stream)
        return state["out"]
    sur = state["sur"]
    sur.set_params(state["p0"])
    losses = sur.train(state["steps"], state["batch"], 2e-3, 2e-5, 20, 1234)
    return {"losses": losses, "params": sur.get_params()}


# FP64 work of the reference's chemistry per cell: one IMEX step, one adaptive
# substep (about two a cell here), and the flux sweeps and decode of a stage
FLOP_IMEX, FLOP_SUBSTEP, FLOP_STAGE, FLOP_NET = 8277, 7923, 1800, 71168


def work(case):
    if case["kind"] == "infer":
        return {"bytes": case["n"] * 128.0, "flops": case["n"] * float(FLOP_NET)}
    if case["kind"] == "train":
        n = float(case["steps"] * case["batch"])
        return {"bytes": n * 96.0 + case["steps"] * 37264 * 24.0, "flops": 3.0 * n * FLOP_NET}
    cells = float(case["ni"]) * case["nj"] * case["nk"]
    if case["kind"] == "host":
        chem = FLOP_IMEX if case["react"] == "imex" else 2 * FLOP_SUBSTEP
        return {"bytes": cells * (14 + 15) * 8.0, "flops": cells * (chem + 2 * FLOP_STAGE)}
    st = STAGES[case["adv"]]
    # CS and T read and written once a stage; the wedge's solid cells (38 % of
    # the oblique detonation's grid) take no part
    share = 0.62 if case["setup"] == "odw" else 1.0
    chem = {"imex": FLOP_IMEX, "none": 0, "adaptive": 2 * FLOP_SUBSTEP, "surrogate": 0.2 * FLOP_NET}[case["react"]]
    return {"bytes": share * cells * case["steps"] * 224.0 * st,
            "flops": share * cells * case["steps"] * (st * FLOP_STAGE + chem)}


# ------------------------------------------------- the same in 64-bit torch
def _mix(Y, T):
    """Cp (J/kg/K), R (J/kg/K) of mass fractions Y[9] at T."""
    cp, _, _ = _thermo(T)
    ri = [R_GAS / float(w) for w in _mech().mw]
    return sum(Y[k] * ri[k] * cp[k] for k in range(9)) * 1e3, sum(Y[k] * ri[k] for k in range(9)) * 1e3


def _decode(cs, T):
    """Primitives (D U V W P H G Y0..8), T of conserved cs (13, ...)."""
    m = _mech()
    ri = [R_GAS / float(w) for w in m.mw]
    D = cs[:9].sum(0)
    Y = cs[:9] / D
    U, V, W = cs[9] / D, cs[10] / D, cs[11] / D
    E = cs[12] / D - 0.5 * (U * U + V * V + W * W)
    A = [[sum(Y[k] * (ri[k] * float(c[q][k])) for k in range(9)) for q in range(8)] for c in (m.c0, m.c1)]
    R = sum(Y[k] * ri[k] for k in range(9))
    done = torch.zeros_like(T, dtype=torch.bool)
    for _ in range(10):
        hi = T >= 1000.0
        a = [torch.where(hi, A[1][q], A[0][q]) for q in range(8)]
        h = -a[0] / T + a[1] * torch.log(T) + a[7] + T * (a[2] + T * (a[3] / 2 + T * (a[4] / 3 + T * (a[5] / 4 + T * a[6] / 5))))
        cp = a[0] / (T * T) + a[1] / T + a[2] + T * (a[3] + T * (a[4] + T * (a[5] + T * a[6])))
        dT = (h - E * 1e-3 - R * T) / (cp - R)
        T = torch.where(done, T, T - dT)
        done = done | (dT.abs() < 1e-6)
        if bool(done.all()):
            break
    hi = T >= 1000.0
    a = [torch.where(hi, A[1][q], A[0][q]) for q in range(7)]
    cp = (a[0] / (T * T) + a[1] / T + a[2] + T * (a[3] + T * (a[4] + T * (a[5] + T * a[6])))) * 1e3
    Rg = R * 1e3
    P = T * D * Rg
    return torch.cat((torch.stack((D, U, V, W, P, P / D + E, cp / (cp - Rg))), Y)), T, E


def _ghosts(q, T, kind):
    """RSBI (mirrors; the lower y wall recomputes its thermodynamics) or
    transmissive ends (copies, zero gradient in x)."""
    ri = [R_GAS / float(w) for w in _mech().mw]
    for ax in (1, 2, 3):
        n = q.shape[ax] - 4
        pairs = [(0, 3), (1, 2), (n + 2, n + 1), (n + 3, n)]
        if kind == "znd" and ax == 1:
            pairs = [(0, 2), (1, 2), (n + 2, n + 1), (n + 3, n + 1)]
        for d, s in pairs:
            q.select(ax, d).copy_(q.select(ax, s))
            T.select(ax - 1, d).copy_(T.select(ax - 1, s))
            if kind == "rsbi" and ax == 2 and d < 2:
                v, t = q.select(2, d), T.select(1, d)
                ok = t > 0
                tt = torch.where(ok, t, 300.0)
                cp, R = _mix(v[7:], tt)
                _, h, _ = _thermo(tt)
                v[0] = torch.where(ok, v[4] / (tt * torch.where(ok, R, 1.0)), v[0])
                v[5] = torch.where(ok, sum(v[7 + k] * ri[k] * h[k] for k in range(9)) * 1e3, v[5])
                v[6] = torch.where(ok, cp / (cp - R), v[6])


def _face(a, b, c, diff):
    """State of cell b at the face towards c."""
    if diff == "muscl1":
        return b
    A0, A1 = b - a, c - b
    if diff == "weno":
        q0, q1 = (1e-6 + A0 * A0) ** 2, (1e-6 + A1 * A1) ** 2
        w0 = q1 / (q1 + 2 * q0)
        return b + 0.5 * (A1 + w0 * (A0 - A1))
    r = A1 / (A0 + 1e-12)
    lim = torch.where(r > 0, torch.where(r >= 1, A0, A0 * r), 0.0)
    return b + 0.5 * lim


def _fluxes(q, ax, diff):
    """AUSM fluxes (13, ...) of the n + 1 faces along axis ax of the interior."""
    n = q.shape[ax] - 4
    idx = [slice(None)] * 4
    for o in (1, 2, 3):
        if o != ax:
            idx[o] = slice(2, q.shape[o] - 2)
    v = q[tuple(idx)]
    c = [v.narrow(ax, k, n + 1) for k in range(4)]

    def L(f):
        return _face(c[0][f], c[1][f], c[2][f], diff)

    def Rt(f):
        if diff == "muscl2":
            A1, A2 = c[2][f] - c[1][f], c[3][f] - c[2][f]
            r = A1 / (A2 + 1e-12)
            return c[2][f] - 0.5 * torch.where(r > 0, torch.where(r >= 1, A2, A2 * r), 0.0)
        return _face(c[3][f], c[2][f], c[1][f], diff)

    un = ax
    DL, DR, PL, PR, NL, NR = L(0), Rt(0), L(4), Rt(4), L(un), Rt(un)
    CI = 0.5 * (torch.sqrt(L(6) * PL / DL) + torch.sqrt(Rt(6) * PR / DR))
    ML, MR = NL / CI, NR / CI

    def split(M, s):
        m2 = (M * M - 1) ** 2
        sub = M.abs() < 1
        b = torch.where(sub, s * 0.25 * (M + s) ** 2 + s * 0.125 * m2, 0.5 * (M + s * M.abs()))
        g = torch.where(sub, 0.25 * (M + s) ** 2 * (2 - s * M) + s * 3.0 / 16.0 * M * m2, (0.5 * (M + s * M.abs())) / torch.where(sub, 1.0, M))
        return b, g

    b1, g1 = split(ML, 1.0)
    b2, g2 = split(MR, -1.0)
    VI = (b1 + b2) * CI
    left = VI >= 0

    def up(f):
        return torch.where(left, L(f), Rt(f))

    Ds = torch.where(left, DL, DR)
    vel = [torch.where(left, NL, NR) if f == un else up(f) for f in (1, 2, 3)]
    VD = VI * Ds
    out = torch.empty((13,) + tuple(VD.shape), dtype=VD.dtype, device=VD.device)
    for s in range(9):
        out[s] = VD * up(7 + s)
    for f in range(3):
        out[9 + f] = VD * vel[f]
    out[9 + un - 1] += g1 * PL + g2 * PR
    out[12] = VI * (Ds * up(5) + 0.5 * Ds * (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2))
    return out


def _residual(q, g, dt, diff):
    r = None
    for ax, node in ((1, g.xnode), (2, g.ynode), (3, g.znode)):
        n = q.shape[ax] - 4
        F = _fluxes(q, ax, diff)
        shape = [1, 1, 1, 1]
        shape[ax] = n
        h = (_t(node)[2:-2] - _t(node)[1:-3]).reshape(shape)
        d = -(dt / h) * (F.narrow(ax, 1, n) - F.narrow(ax, 0, n))
        r = d if r is None else r + d
        del F
    return r


def _rates(T, Mc):
    """Per reaction: (KF, KB, product of reactants, of products, third body)."""
    m = _mech()
    _, h, s = _thermo(T)
    G = [R_GAS * (h[k] - s[k] * T) for k in range(9)]
    for r in range(m.NR):
        kf = float(m.af[r]) * T ** float(m.bf[r]) * torch.exp(-float(m.eaf[r]) / (RU_CAL * T))
        nu = m.stoi_b[:, r] - m.stoi_f[:, r]
        dg = sum(float(nu[k]) * G[k] for k in range(9) if nu[k])
        x = float(nu.sum())
        kc = torch.exp(-dg / (R_GAS * T)) * (ATM * 1e-6 / (R_GAS * T)) ** x
        rf, rb = 1.0, 1.0
        for k in range(9):
            for _ in range(int(m.stoi_f[k, r])):
                rf = rf * Mc[k]
            for _ in range(int(m.stoi_b[k, r])):
                rb = rb * Mc[k]
        tb = sum(float(m.react_tb[k, r]) * Mc[k] for k in range(9) if m.react_tb[k, r])
        tb = torch.where(tb == 0, 1.0, tb) if torch.is_tensor(tb) else 1.0
        yield r, nu, kf, kf / kc, rf, rb, tb


def _imex(cs, T, res, dt):
    """One Diagonalized + Update_IMEX step of cs (13, n) at T with residual res."""
    m = _mech()
    mw = [float(w) for w in m.mw]
    ri = [R_GAS / w for w in mw]
    D = cs[:9].sum(0)
    U, V, W = cs[9] / D, cs[10] / D, cs[11] / D
    cp, h, _ = _thermo(T)
    Cp = sum(cs[k] / D * ri[k] * cp[k] for k in range(9)) * 1e3
    CV = Cp - sum(cs[k] / D * ri[k] for k in range(9)) * 1e3
    ke = 0.5 * (U * U + V * V + W * W)
    PT = [(ke - ri[k] * h[k] * 1e3 + ri[k] * 1e3 * T) / (CV * D) for k in range(9)]
    Mc = [cs[k] / mw[k] * 1e-3 for k in range(9)]
    Di = [cs[k] * 1e-3 for k in range(9)]
    Wi, MD = [torch.zeros_like(T) for _ in range(9)], [torch.zeros_like(T) for _ in range(9)]
    for r, nu, kf, kb, rf, rb, tb in _rates(T, Mc):
        rr = kf * rf - kb * rb
        w2 = rr * (float(m.bf[r]) / T + float(m.eaf[r]) / (RU_CAL * T * T))
        for k in range(9):
            if not nu[k]:
                continue
            w1 = 0.0
            if m.stoi_f[k, r]:
                w1 = w1 + kf * float(m.stoi_f[k, r]) * rf / Di[k]
            if m.stoi_b[k, r]:
                w1 = w1 - kb * float(m.stoi_b[k, r]) * rb / Di[k]
            w1 = torch.where(Di[k] == 0, 0.0, w1) if torch.is_tensor(w1) else w1
            Wi[k] += float(nu[k]) * tb * rr
            MD[k] += float(nu[k]) * ((w1 + w2 * PT[k]) * tb + rr * float(m.react_tb[k, r]) / mw[k])
    new = cs + res
    for k in range(9):
        new[k] = cs[k] + (res[k] + mw[k] * Wi[k] * 1e3 * dt) / (1.0 - dt * mw[k] * MD[k])
    return new


def _trapezoid(cs, T, dt):
    """TrapezoidPrediction and its substeps for cs (13, n) after the flux update."""
    m = _mech()
    mw = [float(w) for w in m.mw]

    def terms(c, T):
        Mc = [c[k] / mw[k] * 1e-3 for k in range(9)]
        Wi, P, Q = ([torch.zeros_like(T) for _ in range(9)] for _ in range(3))
        for r, nu, kf, kb, rf, rb, tb in _rates(T, Mc):
            for k in range(9):
                f, b = float(m.stoi_f[k, r]), float(m.stoi_b[k, r])
                Wi[k] += (b - f) * tb * (kf * rf - kb * rb)
                if f or b:
                    Q[k] += b * kf * rf + f * kb * rb * tb
                    P[k] += b * kb * rb + f * kf * rf * tb
        return Mc, Wi, P, Q

    q, T, E = _decode(cs, T)
    _, Wi, _, _ = terms(cs, T)
    lim = torch.full_like(T, dt)
    for k in range(9):
        w = mw[k] * Wi[k]
        t = (cs[k] * 1e-3 / w).abs()
        lim = torch.where((q[7 + k] >= 1e-6) & (w != 0) & (t < lim), t, lim)
    n = torch.ceil(dt / lim).clamp(min=1)
    h = dt / n
    for step in range(int(n.max())):
        go = torch.nonzero(n > step)[:, 0]
        c, hh, t = cs[:, go].clone(), h[go], T[go]
        Mc, _, P, Q = terms(c, t)
        for k in range(9):
            p = torch.where(Mc[k] == 0, 0.0, P[k] / Mc[k])
            c[k] = ((1 - hh / 2 * p) * c[k] * 1e-3 + hh * mw[k] * Q[k]) / (1 + hh / 2 * p) * 1e3
        D, vel = c[:9].sum(0), q[1:4, go]
        c[9:12] = vel * D
        c[12] = D * E[go] + 0.5 * D * (vel ** 2).sum(0)
        q1, T1, E1 = _decode(c, t)
        cs[:, go], q[:, go], T[go], E[go] = c, q1, T1, E1
    return cs


def _chunks(n, size=1 << 21):
    return [slice(i, min(n, i + size)) for i in range(0, n, size)]


def _decode_all(cs, T, q):
    """Decodes the interior of the ghosted q, T from interior cs (13, i, j, k)."""
    inner = (slice(2, -2),) * 3
    f, t = cs.reshape(13, -1), T[inner].reshape(-1)
    qn, tn = torch.empty((16, f.shape[1]), dtype=f.dtype, device=f.device), torch.empty_like(t)
    for s in _chunks(f.shape[1]):
        qn[:, s], tn[s], _ = _decode(f[:, s], t[s])
    q[(slice(None),) + inner] = qn.reshape((16,) + tuple(cs.shape[1:]))
    T[inner] = tn.reshape(cs.shape[1:])


def exact(case, seed):
    m = _mech()
    if case["kind"] == "train":
        return None  # hundreds of dependent optimiser steps on batches that the device draws
    if case["kind"] == "infer":
        p = _t(S.SurrogateModel.load(S.DEFAULT_MODEL).params)
        h = _network_inputs(case["n"], seed)
        outs = []
        for s in _chunks(case["n"], 1 << 19):
            x, o = h[s].double(), 0
            for k, (i, j) in enumerate(((16, 128), (128, 128), (128, 128), (128, 16))):
                x = x @ p[o:o + i * j].reshape(i, j) + p[o + i * j:o + i * j + j]
                o += i * j + j
                if k < 3:
                    x = 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))
            outs.append(x)
        return torch.cat(outs)
    if case["kind"] == "flow" and (case["setup"] == "odw" or case["react"] == "adaptive"):
        # the start of these runs is the program's own developed state, and their
        # chemistry picks substeps or a network's answer per cell by thresholds
        return None
    g, cs0, T = _initial(case, seed)
    host = case["kind"] == "host"
    bc = "rsbi" if host else case["setup"]
    CS = cs0.permute(3, 0, 1, 2)
    inner = (slice(None),) + (slice(2, -2),) * 3
    cs = CS[inner].clone()
    q = torch.zeros((16,) + tuple(T.shape), dtype=torch.float64, device=T.device)
    T = T.clone()
    _decode_all(cs, T, q)
    adv, diff = ("ee", "muscl2") if host else (case["adv"], case["diff"])
    cfl = 0.3 if host else case["cfl"]
    P1, dt = None, case.get("dt", 0.0)
    for _ in range(1 if host else case["steps"]):
        if not host or case["react"] == "imex":
            v = q[inner]
            C = torch.sqrt(v[6] * v[4] / v[0])
            dt = cfl * min(float((float(n[1] - n[0]) / (v[1 + k].abs() + C)).min())
                           for k, n in enumerate((g.xnode, g.ynode, g.znode)))
        _ghosts(q, T, bc)
        res = _residual(q, g, dt, diff)
        if adv == "rk2":
            c1 = cs + res
            _decode_all(c1, T, q)
            _ghosts(q, T, bc)
            cs = 0.5 * cs + 0.5 * (c1 + _residual(q, g, dt, diff))
        elif adv == "rk3":
            c1 = cs + res
            _decode_all(c1, T, q)
            _ghosts(q, T, bc)
            c1 = 0.75 * cs + 0.25 * (c1 + _residual(q, g, dt, diff))
            _decode_all(c1, T, q)
            _ghosts(q, T, bc)
            cs = cs / 3.0 + 2.0 / 3.0 * (c1 + _residual(q, g, dt, diff))
        if adv != "ee":
            _decode_all(cs, T, q)
            res = torch.zeros_like(cs)
        f, rf, Tf = cs.reshape(13, -1), res.reshape(13, -1), T[inner[1:]].reshape(-1)
        new = torch.empty_like(f)
        for s in _chunks(f.shape[1]):
            if case["react"] == "imex":
                new[:, s] = _imex(f[:, s], Tf[s], rf[:, s], dt)
            elif case["react"] == "none":
                new[:, s] = f[:, s] + rf[:, s]
            else:
                new[:, s] = _trapezoid(f[:, s] + rf[:, s], Tf[s], dt)
        cs = new.reshape(cs.shape)
        _decode_all(cs, T, q)
    full = CS.clone()
    full[inner] = cs
    out = {"CS": full.permute(1, 2, 3, 0).contiguous(), "T": T}
    if host:
        out.update(P=q[4], dt=dt)
    return out
