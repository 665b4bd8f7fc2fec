"""The performance cases of the framework: the calls its users make, through
the public entry points (pmhd.Solver, pmhd.Ensemble, pmhd.Euler2D and the C ABI
of the learned correction's layers), over the sizes, precisions and options
they are used with.

A case is a dict of plain values.  `kind` selects the path:

  mhd       a pmhd.Solver segment: upload a state, advance a number of steps,
            read the state back (what a run between two snapshots does)
  ensemble  a pmhd.Ensemble segment: advance every member, read all states
  euler     a pmhd.Euler2D segment: advance, read the primitives
  layer     one layer of the correction network on the tensor cores: forward,
            backward, or both (a training step of that layer)

exact() states the same schemes in plain torch, in binary64.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "precision-study_b200"))
import pmhd  # noqa: E402

GAMMA, CFL, ALPHA, TOL = 5.0 / 3.0, 0.25, 0.18, 1.0e-4


def listed():
    return [
        # Small periodic grid in binary64: the coarse grid of the learned
        # correction and of convergence studies; bound by step latency.
        {"name": "ot_64_fp64", "kind": "mhd", "problem": "ot", "nx": 64, "ny": 64, "precision": "fp64",
         "order": "muscl", "solver": "hlld", "steps": 64},
        # The reference's own protocol grid (192^2) in binary32.
        {"name": "ot_192_fp32", "kind": "mhd", "problem": "ot", "nx": 192, "ny": 192, "precision": "fp32",
         "order": "muscl", "solver": "hlld", "steps": 64},
        # Shear layer between reflecting walls on an odd, ragged grid.
        {"name": "kh_walls_509x331_fp64", "kind": "mhd", "problem": "kh", "nx": 509, "ny": 331, "precision": "fp64",
         "order": "muscl", "solver": "hlld", "steps": 32},
        # The mixed-precision policy at a medium grid.
        {"name": "ot_1024_mixed", "kind": "mhd", "problem": "ot", "nx": 1024, "ny": 1024, "precision": "mixed",
         "order": "muscl", "solver": "hlld", "steps": 32},
        # A large production grid in binary64.
        {"name": "ot_2048_fp64", "kind": "mhd", "problem": "ot", "nx": 2048, "ny": 2048, "precision": "fp64",
         "order": "muscl", "solver": "hlld", "steps": 24},
        # The one-stage MUSCL-Hancock scheme in binary64.
        {"name": "hancock_512_fp64", "kind": "mhd", "problem": "ot", "nx": 512, "ny": 512, "precision": "fp64",
         "order": "hancock", "solver": "hlld", "steps": 64},
        # A parameter sweep of small uneven grids in shared launches.
        {"name": "ensemble_16_mixed", "kind": "ensemble", "members": 16, "n_min": 64, "n_max": 256,
         "precision": "mixed", "steps": 100},
        # The Haas-Sturtevant shock-bubble program's grid.
        {"name": "bubble_500x197_fp64", "kind": "euler", "config": 100, "nx": 500, "ny": 197, "precision": "fp64",
         "solver": "hllc", "steps": 256},
        # A Liska-Wendroff Riemann problem in binary32.
        {"name": "lw3_1024_fp32", "kind": "euler", "config": 3, "nx": 1024, "ny": 1024, "precision": "fp32",
         "solver": "hllc", "steps": 64},
        # The correction network's hidden layer over a training batch at
        # 512^2: forward, and its two backward passes.
        {"name": "layer_forward_8x512", "kind": "layer", "part": "forward", "batch": 8, "h": 512, "w": 512,
         "c_out": 32},
        {"name": "layer_backward_8x512", "kind": "layer", "part": "backward", "batch": 8, "h": 512, "w": 512,
         "c_out": 32},
        # The same layer's training step at the 64^2 grids the correction
        # is trained on.
        {"name": "layer_train_8x64", "kind": "layer", "part": "both", "batch": 8, "h": 64, "w": 64, "c_out": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["mhd", "ensemble", "euler", "layer"], [6, 1, 3, 4])[0]
    if kind == "mhd":
        nx, ny = _log_int(rng, 48, 2048), _log_int(rng, 48, 2048)
        return {"kind": kind, "problem": rng.choice(["ot", "ot", "kh", "pulse"]), "nx": nx, "ny": ny,
                "precision": rng.choice(["fp64", "fp64", "fp32", "mixed"]),
                "order": rng.choice(["muscl", "muscl", "hancock"]),
                "solver": rng.choice(["hlld", "hlld", "hlld", "hll"]),
                "steps": max(8, min(64, 60_000_000 // (nx * ny)))}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(6, 20), "n_min": rng.randint(48, 96),
                "n_max": rng.randint(128, 256), "precision": rng.choice(["mixed", "fp64"]),
                "steps": rng.randint(24, 64)}
    if kind == "euler":
        config = rng.choice([100, 3, 6, 12])
        nx, ny = (_log_int(rng, 128, 1024), _log_int(rng, 64, 512)) if config == 100 else [_log_int(rng, 100, 1500)] * 2
        return {"kind": kind, "config": config, "nx": nx, "ny": ny, "precision": rng.choice(["fp64", "fp32"]),
                "solver": rng.choice(["hllc", "hllc", "hll"]), "steps": max(32, min(256, 80_000_000 // (nx * ny)))}
    # Layers: the grids the correction runs on (multiples of 64) and odd ones.
    size = rng.choice([(64, 64), (128, 128), (256, 256), (512, 512), None, None])
    h, w = size if size else (_log_int(rng, 24, 512), _log_int(rng, 24, 512))
    return {"kind": kind, "part": rng.choice(["forward", "backward", "both"]), "batch": rng.randint(1, 8), "h": h,
            "w": w, "c_out": rng.choice([32, 32, 16])}


# ---- inputs -------------------------------------------------------------------


def _domain(case):
    """(x_min, x_max, y_min, y_max), boundary kinds of an mhd case."""
    if case["problem"] == "kh":
        return (0.0, 1.0, -1.0, 1.0), (0, 0, 1, 1)
    if case["problem"] == "pulse":
        return (0.0, 1.0, 0.0, 1.0), (2, 2, 2, 2)
    return (0.0, 1.0, 0.0, 1.0), (0, 0, 0, 0)


def _conserved(P):
    rho, vx, vy, vz, p, bx, by, bz, psi = P
    e = p / (GAMMA - 1.0) + 0.5 * rho * (vx * vx + vy * vy + vz * vz) + 0.5 * (bx * bx + by * by + bz * bz)
    return np.stack([rho, rho * vx, rho * vy, rho * vz, e, bx, by, bz, psi], axis=-1)


def _initial(case, seed):
    """Initial conserved state [ny][nx][9] of an mhd case, in its storage type."""
    rng = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    (x0, x1, y0, y1), _ = _domain(case)
    x = (x0 + (np.arange(nx) + 0.5) * (x1 - x0) / nx)[None, :]
    y = (y0 + (np.arange(ny) + 0.5) * (y1 - y0) / ny)[:, None]
    one, tau = np.ones((ny, nx)), 2.0 * np.pi
    if case["problem"] == "ot":  # Orszag-Tang, its field scaled, its phases shifted
        b0, a, b = rng.uniform(0.7, 1.3), rng.uniform(), rng.uniform()
        f = b0 / math.sqrt(4.0 * np.pi)
        P = [25.0 / (36.0 * np.pi) * one, -np.sin(tau * (y + b)) * one, np.sin(tau * (x + a)) * one,
             0.2 * np.sin(tau * (x + y)) * one, 5.0 / (12.0 * np.pi) * one, -f * np.sin(tau * (y + b)) * one,
             f * np.sin(2.0 * tau * (x + a)) * one, 0.1 * np.cos(tau * (x - y)) * one, 0.0 * one]
    elif case["problem"] == "kh":  # a perturbed shear layer between walls
        width, amp, ph = rng.uniform(0.04, 0.08), rng.uniform(0.005, 0.02), rng.uniform()
        P = [one, 0.5 * np.tanh(y / width) * one, amp * np.sin(tau * (x + ph)) * np.exp(-y * y / 0.01), 0.0 * one, one,
             0.1 * one, 0.0 * one, 0.0 * one, 0.0 * one]
    else:  # a pressure pulse in an oblique field, open sides
        cx, cy, th = rng.uniform(0.4, 0.6), rng.uniform(0.4, 0.6), rng.uniform(0.2, 1.2)
        g = np.exp(-((x - cx) ** 2 + (y - cy) ** 2) / 0.01)
        P = [1.0 + 0.5 * g, 0.1 * one, -0.05 * one, 0.0 * one, 0.5 + 2.0 * g, 0.5 * math.cos(th) * one,
             0.5 * math.sin(th) * one, 0.1 * one, 0.0 * one]
    return np.ascontiguousarray(_conserved(P).astype(np.float32 if case["precision"] == "fp32" else np.float64))


def _members(case, seed):
    """(n, field factor) of every member of an ensemble case; the sizes are
    the case's, the fields the seed's."""
    rng = np.random.default_rng(seed)
    count, lo, hi = case["members"], case["n_min"], case["n_max"]
    sizes = [int(round(lo * (hi / lo) ** ((k % 5) / 4.0))) for k in range(count)]
    return [(n, float(b)) for n, b in zip(sizes, rng.uniform(0.5, 1.5, count))]


def _euler_offset(case, seed):
    """Steps the run has already taken when the timed segment starts."""
    return 2 * (np.random.default_rng(seed).integers(4, 44) if case["kind"] == "euler" else 0)


def _layer_inputs(case, seed):
    """bf16 operands of a layer on the GPU: x [B][H][W][32] its input, wt its
    weights [c_out][9][32], bias, dz the gradient of its output, zprev the
    pre-activation x came from."""
    B, H, W, co = case["batch"], case["h"], case["w"], case["c_out"]
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    zprev = torch.randn((B, H, W, 32), generator=g, device="cuda").to(torch.bfloat16)
    x = torch.nn.functional.gelu(zprev.float(), approximate="tanh").to(torch.bfloat16)
    wt = (0.08 * torch.randn((co, 9, 32), generator=g, device="cuda")).to(torch.bfloat16)
    bias = 0.1 * torch.randn((co,), generator=g, device="cuda")
    dz = (1e-2 * torch.randn((B, H, W, co), generator=g, device="cuda")).to(torch.bfloat16)
    return {"x": x, "wt": wt, "bias": bias, "dz": dz, "zprev": zprev}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mhd":
        dom, bc = _domain(case)
        U0 = torch.from_numpy(_initial(case, seed)).pin_memory()
        out = torch.empty_like(U0).pin_memory()
        s = pmhd.Solver(nx=case["nx"], ny=case["ny"], precision=case["precision"], order=case["order"],
                        solver=case["solver"], cfl=CFL, alpha=ALPHA, domain=dom, bc=bc)
        return {"case": case, "solver": s, "U0": U0.numpy(), "out": out.numpy()}
    if kind == "ensemble":
        ms = [pmhd.member(n, n, pmhd.PROBLEM_ORSZAG_TANG, (b0,), t_end=1e9) for n, b0 in _members(case, seed)]
        return {"case": case, "ensemble": pmhd.Ensemble(ms, precision=case["precision"], cfl=CFL, alpha=ALPHA)}
    if kind == "euler":
        config = "shock_bubble" if case["config"] == 100 else case["config"]
        e = pmhd.Euler2D(case["nx"], case["ny"], config=config, solver=case["solver"], precision=case["precision"])
        e.advance(1e9, int(_euler_offset(case, seed)))
        return {"case": case, "euler": e}
    s = _layer_inputs(case, seed)
    s["case"] = case
    s["wt_t"] = s["wt"].permute(2, 1, 0).contiguous()  # [32][9][c_out], the backward pass's weights
    return s


# ---- one pass -------------------------------------------------------------------


def _fp(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_float))


def _ok(rc):
    if rc != pmhd.OK:
        raise RuntimeError(pmhd.strerror(rc))


def _layer_forward(s):
    """z and gelu(z) of a hidden layer (c_out 32), the fp32 output of the last
    one (c_out 16)."""
    x, L = s["x"], pmhd.load()
    B, H, W, _ = x.shape
    if s["case"]["c_out"] == 16:
        o = torch.empty((B, H, W, 16), dtype=torch.float32, device=x.device)
        _ok(L.pmhd_conv3x3(pmhd.CONV_LINEAR, x.data_ptr(), B, H, W, 32, s["wt"].data_ptr(), _fp(s["bias"]), 16, None,
                           o.data_ptr(), None, None))
        return {"out": o}
    z, a = torch.empty_like(x), torch.empty_like(x)
    _ok(L.pmhd_conv3x3(pmhd.CONV_GELU, x.data_ptr(), B, H, W, 32, s["wt"].data_ptr(), _fp(s["bias"]), 32, None,
                       z.data_ptr(), a.data_ptr(), None))
    return {"z": z, "a": a}


def _layer_backward(s):
    """Gradients of the layer's weights and bias, and of the previous layer's
    pre-activation."""
    x, dz, L = s["x"], s["dz"], pmhd.load()
    B, H, W, _ = x.shape
    co = s["case"]["c_out"]
    dw = torch.zeros((co, 9, 32), dtype=torch.float32, device=x.device)
    db = torch.zeros((co,), dtype=torch.float32, device=x.device)
    dzp = torch.empty_like(x)
    _ok(L.pmhd_conv3x3_wgrad(x.data_ptr(), dz.data_ptr(), B, H, W, 32, co, _fp(dw), _fp(db), None))
    _ok(L.pmhd_conv3x3(pmhd.CONV_DGELU, dz.data_ptr(), B, H, W, co, s["wt_t"].data_ptr(), None, 32,
                       s["zprev"].data_ptr(), dzp.data_ptr(), None, None))
    return {"dw": dw, "db": db, "dzprev": dzp}


def run(state):
    case = state["case"]
    if case["kind"] == "mhd":
        s = state["solver"]
        s.set_state(state["U0"])
        st = s.advance(max_steps=case["steps"])
        return {"U": s.get_state(out=state["out"]), "t": st.t}
    if case["kind"] == "ensemble":
        e = state["ensemble"]
        e.advance(max_steps=case["steps"])
        return [e.get_state(k) for k in range(len(e))]
    if case["kind"] == "euler":
        e = state["euler"]
        e.advance(1e9, case["steps"])
        return {"W": e.prims(), "t": e.t}
    out = {}
    if case["part"] in ("forward", "both"):
        out.update(_layer_forward(state))
    if case["part"] in ("backward", "both"):
        out.update(_layer_backward(state))
    return out


def work(case):
    """Bytes and operations of one pass.  A time step reads and writes the
    state once; operations are those of the scheme's reconstruction, Riemann
    solutions and update, counted once per cell (about 900 a stage for the
    MHD scheme, 500 a step for the Euler one)."""
    kind = case["kind"]
    if kind in ("mhd", "ensemble"):
        word = 4 if case["precision"] == "fp32" else 8
        cells = case["nx"] * case["ny"] if kind == "mhd" else sum(n * n for n, _ in _members(case, 0))
        per = 1200 if case.get("order") == "hancock" else 1800
        return {"bytes": cells * 9 * word * 2 * case["steps"], "flops": cells * per * case["steps"]}
    if kind == "euler":
        cells, word = case["nx"] * case["ny"], 4 if case["precision"] == "fp32" else 8
        return {"bytes": cells * 4 * word * 2 * case["steps"], "flops": cells * 500 * case["steps"]}
    pixels, co = case["batch"] * case["h"] * case["w"], case["c_out"]
    gemm = 2 * 9 * 32 * co * pixels
    fwd = {"bytes": pixels * (64 + (128 if co == 32 else 64)), "flops": gemm}
    bwd = {"bytes": pixels * (64 + 64 + 64 + 2 * co), "flops": 2 * gemm}
    parts = {"forward": [fwd], "backward": [bwd], "both": [fwd, bwd]}[case["part"]]
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


# ---- the same in plain binary64 -----------------------------------------------------


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _sides(A, axis, lo, hi, flip):
    """A [9][ny][nx] with two ghost layers on both sides of axis (2 = x, 1 = y)."""
    n = A.shape[axis]

    def take(idx, mirror):
        g = A.index_select(axis, torch.tensor(idx, device=A.device))
        if mirror:
            g = g.clone()
            for k in flip:
                g[k] = -g[k]
        return g

    left = {0: ([n - 2, n - 1], False), 1: ([1, 0], True), 2: ([0, 0], False)}[lo]
    right = {0: ([0, 1], False), 1: ([n - 1, n - 2], True), 2: ([n - 1, n - 1], False)}[hi]
    return torch.cat([take(*left), A, take(*right)], dim=axis)


def _mhd_prim(U):
    rho = U[0].clamp(min=1e-12)
    v = U[1:4] / rho
    p = (GAMMA - 1.0) * (U[4] - 0.5 * rho * (v * v).sum(0) - 0.5 * (U[5:8] * U[5:8]).sum(0))
    return torch.cat([rho[None], v, p[None], U[5:9]])


def _mhd_cons(P):
    e = P[4] / (GAMMA - 1.0) + 0.5 * P[0] * (P[1:4] * P[1:4]).sum(0) + 0.5 * (P[5:8] * P[5:8]).sum(0)
    return torch.cat([P[0:1], P[0] * P[1:4], e[None], P[5:9]])


def _usable(P):
    return (P[0] > 1e-12) & (P[4] > 1e-12) & torch.isfinite(P).all(0)


def _fast_speed(P, n):
    rho, p = P[0].clamp(min=1e-12), P[4].clamp(min=1e-12)
    a2, b2 = GAMMA * p / rho, (P[5:8] * P[5:8]).sum(0) / rho
    disc = ((a2 + b2) ** 2 - 4.0 * a2 * P[5 + n] ** 2 / rho).clamp(min=0.0)
    return torch.sqrt((0.5 * (a2 + b2 + torch.sqrt(disc))).clamp(min=0.0))


def _max_speed(U):
    P = _mhd_prim(U)
    return float(torch.maximum(P[1].abs() + _fast_speed(P, 0), P[2].abs() + _fast_speed(P, 1)).max())


def _mhd_flux(W, e):
    pt = W[4] + 0.5 * (W[5:8] * W[5:8]).sum(0)
    m = W[0] * W[1]
    vb = (W[1:4] * W[5:8]).sum(0)
    return torch.stack([m, m * W[1] + pt - W[5] * W[5], m * W[2] - W[5] * W[6], m * W[3] - W[5] * W[7],
                        (e + pt) * W[1] - W[5] * vb, torch.zeros_like(m), W[1] * W[6] - W[5] * W[2],
                        W[1] * W[7] - W[5] * W[3]])


def _positive(U):
    W = _mhd_prim(torch.cat([U, torch.zeros_like(U[:1])]))
    return (U[0] > 1e-12) & (W[4] > 1e-12)


def _star(U, W, s, sm, pts, bn):
    """One side's star state of HLLD (Miyoshi & Kusano 2005), and whether it is usable."""
    rho, vn, e = W[0], W[1], U[4]
    smv, sms = s - vn, s - sm
    ok = ~(sms.abs() <= TOL * torch.maximum(s.abs(), sm.abs()))
    rs = rho * smv / sms
    ok &= rs > 1e-12
    den = rho * smv * sms - bn * bn
    ok &= ~(den.abs() <= TOL * ((rho * smv * sms).abs() + bn * bn))
    pt = W[4].clamp(min=1e-12) + 0.5 * (bn * bn + W[6] ** 2 + W[7] ** 2)
    vt = [W[2 + k] - bn * W[6 + k] * (sm - vn) / den for k in (0, 1)]
    bt = [W[6 + k] * (rho * smv * smv - bn * bn) / den for k in (0, 1)]
    vb = vn * bn + W[2] * W[6] + W[3] * W[7]
    vbs = sm * bn + vt[0] * bt[0] + vt[1] * bt[1]
    es = (smv * e - pt * vn + pts * sm + bn * (vb - vbs)) / sms
    Us = torch.stack([rs, rs * sm, rs * vt[0], rs * vt[1], es, bn, bt[0], bt[1]])
    return Us, vt, bt, vbs, ok & _positive(Us)


def _riemann(UL, UR, ch, hlld):
    """GLM + HLLD (or HLL) flux along the first direction of 9-slot states."""
    bn = 0.5 * (UL[5] + UR[5]) - 0.5 * (UR[8] - UL[8]) / ch
    ps = 0.5 * (UL[8] + UR[8]) - 0.5 * ch * (UR[5] - UL[5])
    UL, UR = UL.clone(), UR.clone()
    UL[5], UR[5] = bn, bn
    WL, WR = _mhd_prim(UL), _mhd_prim(UR)
    UL, UR = UL[:8], UR[:8]
    FL, FR = _mhd_flux(WL, UL[4]), _mhd_flux(WR, UR[4])
    cL, cR = _fast_speed(WL, 0), _fast_speed(WR, 0)
    sL, sR = torch.minimum(WL[1] - cL, WR[1] - cR), torch.maximum(WL[1] + cL, WR[1] + cR)
    F = (sR * FL - sL * FR + sL * sR * (UR - UL)) / (sR - sL)
    if hlld:
        ptL = WL[4].clamp(min=1e-12) + 0.5 * (bn * bn + WL[6] ** 2 + WL[7] ** 2)
        ptR = WR[4].clamp(min=1e-12) + 0.5 * (bn * bn + WR[6] ** 2 + WR[7] ** 2)
        dL, dR = WL[0] * (sL - WL[1]), WR[0] * (sR - WR[1])
        b2 = torch.maximum(ptL - WL[4].clamp(min=1e-12), ptR - WR[4].clamp(min=1e-12)) * 2.0
        ok = ~((dR - dL).abs() <= TOL * (dR.abs() + dL.abs())) & ~(bn.abs() <= TOL * torch.sqrt(b2))
        sm = (dR * WR[1] - dL * WL[1] + ptL - ptR) / (dR - dL)
        pts = 0.5 * (ptL + dL * (sm - WL[1]) + ptR + dR * (sm - WR[1]))
        Ls, vL, bL, vbL, okL = _star(UL, WL, sL, sm, pts, bn)
        Rs, vR, bR, vbR, okR = _star(UR, WR, sR, sm, pts, bn)
        ok &= okL & okR
        qL, qR = torch.sqrt(Ls[0].clamp(min=1e-12)), torch.sqrt(Rs[0].clamp(min=1e-12))
        sgn = torch.where(bn < 0, -1.0, 1.0)
        vD = [(qL * vL[k] + qR * vR[k] + sgn * (bR[k] - bL[k])) / (qL + qR) for k in (0, 1)]
        bD = [(qL * bR[k] + qR * bL[k] + sgn * qL * qR * (vR[k] - vL[k])) / (qL + qR) for k in (0, 1)]
        vbD = sm * bn + vD[0] * bD[0] + vD[1] * bD[1]
        LD = torch.stack([Ls[0], Ls[1], Ls[0] * vD[0], Ls[0] * vD[1], Ls[4] - sgn * qL * (vbL - vbD), bn, bD[0], bD[1]])
        RD = torch.stack([Rs[0], Rs[1], Rs[0] * vD[0], Rs[0] * vD[1], Rs[4] + sgn * qR * (vbR - vbD), bn, bD[0], bD[1]])
        ok &= _positive(LD) & _positive(RD)
        sLs, sRs = sm - bn.abs() / qL, sm + bn.abs() / qR
        GL = FL + sL * (Ls - UL)
        GL = torch.where(sLs >= 0, GL, GL + sLs * (LD - Ls))
        GR = FR + sR * (Rs - UR)
        GR = torch.where(sRs >= 0, GR + sRs * (RD - Rs), GR)
        F = torch.where(ok, torch.where(sm >= 0, GL, GR), F)
    F = torch.where(sL >= 0, FL, torch.where(sR <= 0, FR, F))
    F[5] = ps
    return torch.cat([F, (ch * ch * bn)[None]])


def _minmod(a, b):
    return torch.where(a * b <= 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _faces(P):
    """Limited faces of cells 1 .. n-2 along the last axis, from primitives."""
    c = P[..., 1:-1]
    s = 0.5 * _minmod(c - P[..., :-2], P[..., 2:] - c)
    l, r = c - s, c + s
    ok = _usable(l) & _usable(r)
    return torch.where(ok, l, c), torch.where(ok, r, c)


_SWAP = [0, 2, 1, 3, 4, 6, 5, 7, 8]


def _turn(A):
    """Exchanges x and y of a [9][..][..] field."""
    return A[_SWAP].transpose(1, 2)


def _mhd_rhs(U, ch, dx, dy, bc, hlld):
    G = _mhd_prim(_sides(_sides(U, 2, bc[0], bc[1], (1, 5)), 1, bc[2], bc[3], (2, 6)))

    def part(P, d):  # P [9][rows][n + 4]: flux difference over its interior cells
        l, r = _faces(P)
        F = _riemann(_mhd_cons(r[..., :-1]), _mhd_cons(l[..., 1:]), ch, hlld)
        return (F[..., 1:] - F[..., :-1]) / d

    rhs = -part(G[:, 2:-2, :], dx) - _turn(part(_turn(G[:, :, 2:-2]), dy))
    rhs[8] -= ch / ALPHA * U[8]
    return rhs


def _phys(U, ch):
    F = _mhd_flux(_mhd_prim(U), U[4])
    F[5] = U[8]
    return torch.cat([F, (ch * ch * U[5])[None]])


def _hancock_rhs(U, ch, dx, dy, dt, bc, hlld):
    G = _mhd_prim(_sides(_sides(U, 2, bc[0], bc[1], (1, 5)), 1, bc[2], bc[3], (2, 6)))
    xl, xr = [_mhd_cons(f) for f in _faces(G[:, 1:-1, :])]
    yl, yr = [_mhd_cons(_turn(f)) for f in _faces(_turn(G[:, :, 1:-1]))]
    corr = 0.5 * dt / dx * (_phys(xr, ch) - _phys(xl, ch))
    corr = corr + 0.5 * dt / dy * (_turn(_phys(_turn(yr), ch)) - _turn(_phys(_turn(yl), ch)))

    def evolve(f):
        h = f - corr
        h[8] -= 0.5 * dt * ch / ALPHA * f[8]
        return torch.where((h[0] > 1e-12) & _usable(_mhd_prim(h)), h, f)

    xl, xr, yl, yr = evolve(xl), evolve(xr), evolve(yl), evolve(yr)
    Fx = _riemann(xr[:, 1:-1, :-1], xl[:, 1:-1, 1:], ch, hlld)
    Fy = _riemann(_turn(yr[:, :-1, 1:-1]), _turn(yl[:, 1:, 1:-1]), ch, hlld)
    rhs = -(Fx[..., 1:] - Fx[..., :-1]) / dx - _turn((Fy[..., 1:] - Fy[..., :-1]) / dy)
    rhs[8] -= ch / ALPHA * U[8]
    return rhs


def _mhd_exact(U, dom, bc, order, hlld, steps):
    """`steps` steps from U [ny][nx][9] binary64; returns (state, time)."""
    U = torch.from_numpy(U).to(_dev()).permute(2, 0, 1).contiguous()
    dx, dy = (dom[1] - dom[0]) / U.shape[2], (dom[3] - dom[2]) / U.shape[1]
    t = 0.0
    for _ in range(steps):
        ch = max(_max_speed(U), 1e-12)
        dt = CFL / (ch / dx + ch / dy)
        if order == "hancock":
            U = U + dt * _hancock_rhs(U, ch, dx, dy, dt, bc, hlld)
        else:
            V = U + dt * _mhd_rhs(U, ch, dx, dy, bc, hlld)
            U = 0.5 * U + 0.5 * (V + dt * _mhd_rhs(V, ch, dx, dy, bc, hlld))
        t += dt
    return U.permute(1, 2, 0).contiguous(), t


def _ot(n, b0):
    x = ((np.arange(n) + 0.5) / n)[None, :]
    y = ((np.arange(n) + 0.5) / n)[:, None]
    one, tau, f = np.ones((n, n)), 2.0 * np.pi, b0 / math.sqrt(4.0 * np.pi)
    z = 0.0 * one
    return _conserved([25.0 / (36.0 * np.pi) * one, -np.sin(tau * y) * one, np.sin(tau * x) * one, z,
                       5.0 / (12.0 * np.pi) * one, -f * np.sin(tau * y) * one, f * np.sin(2.0 * tau * x) * one, z, z])


_LW = {3: [(0.5197, -0.6259, -0.3109, 0.4), (1.0, 0.1, -0.3109, 1.0), (0.8, 0.1, 0.4276, 0.4),
           (0.5197, -0.6259, 0.4276, 0.4)],
       6: [(1.0, 0.75, -0.5, 1.0), (2.0, 0.75, 0.5, 1.0), (1.0, -0.75, 0.5, 1.0), (3.0, -0.75, -0.5, 1.0)],
       12: [(0.5313, 0.0, 0.0, 0.4), (1.0, 0.7276, 0.0, 1.0), (0.8, 0.0, 0.0, 1.0), (1.0, 0.0, 0.7276, 1.0)]}


def _euler_initial(case):
    """Initial primitives [4][ny][nx] and cell sizes; positions in the run's type."""
    T = np.float32 if case["precision"] == "fp32" else np.float64
    nx, ny = case["nx"], case["ny"]
    bubble = case["config"] == 100
    dx = T(0.225 if bubble else 1.0) / T(nx)
    dy = T(0.089 if bubble else 1.0) / T(ny)
    if bubble:
        x = ((np.arange(nx) + 0.5) * float(dx)).astype(T)[None, :]
        y = ((np.arange(ny) + 0.5) * float(dy)).astype(T)[:, None]
        M, g, rho1, p1 = 1.22, 1.4, 1.29, 101325.0
        rho2 = rho1 * ((g + 1) * M * M) / ((g - 1) * M * M + 2)
        p2 = p1 * (2 * g * M * M - (g - 1)) / (g + 1)
        u2 = math.sqrt(g * p1 / rho1) * M * (1 - rho1 / rho2)
        ex, ey = (x.astype(np.float64) - 0.035).astype(T), (y.astype(np.float64) - 0.089 / 2.0).astype(T)
        inside = ex * ex + ey * ey < T(0.025 * 0.025)
        post = (x.astype(np.float64) < 0.005) & ~inside
        W = np.zeros((4, ny, nx))
        W[0], W[3] = rho1, p1
        W[0][inside] = 0.214
        W[:, post] = np.array([rho2, u2, 0.0, p2])[:, None]
        return W, float(dx), float(dy)
    x = (np.arange(nx).astype(T) + T(0.5)) * dx
    y = (np.arange(ny).astype(T) + T(0.5)) * dy
    right, top = (x >= T(0.5))[None, :], (y >= T(0.5))[:, None]
    q = np.array(_LW[case["config"]])
    W = np.empty((4, ny, nx))
    for k in range(4):
        W[k] = np.where(top, np.where(right, q[0, k], q[1, k]), np.where(right, q[3, k], q[2, k]))
    return W, float(dx), float(dy)


def _euler_cons(W):
    return torch.stack([W[0], W[0] * W[1], W[0] * W[2], W[3] / 0.4 + 0.5 * W[0] * (W[1] ** 2 + W[2] ** 2)])


def _euler_prim(U):
    return torch.stack([U[0], U[1] / U[0], U[2] / U[0], 0.4 * (U[3] - 0.5 * (U[1] ** 2 + U[2] ** 2) / U[0])])


def _euler_flux(W, E):
    m = W[0] * W[1]
    return torch.stack([m, m * W[1] + W[3], m * W[2], (E + W[3]) * W[1]])


def _euler_sweep(U, ratio, hll):
    """One MUSCL-Hancock sweep along x of U [4][rows][n], transmissive ends."""
    G = torch.cat([U[..., :1], U[..., :1], U, U[..., -1:], U[..., -1:]], dim=-1)
    W = _euler_prim(G)
    c = W[..., 1:-1]
    s = 0.5 * _minmod(c - W[..., :-2], W[..., 2:] - c)
    ul, ur = _euler_cons(c - s), _euler_cons(c + s)
    d = 0.5 * ratio * (_euler_flux(c + s, ur[3]) - _euler_flux(c - s, ul[3]))
    L, R = _euler_prim(ur - d)[..., :-1], _euler_prim(ul - d)[..., 1:]
    UL, UR = _euler_cons(L), _euler_cons(R)
    FL, FR = _euler_flux(L, UL[3]), _euler_flux(R, UR[3])
    cL, cR = torch.sqrt(1.4 * L[3] / L[0]), torch.sqrt(1.4 * R[3] / R[0])
    SL, SR = torch.minimum(L[1] - cL, R[1] - cR), torch.maximum(L[1] + cL, R[1] + cR)
    if hll:
        F = torch.where(SR > 0, (SR * FL - SL * FR + SL * SR * (UR - UL)) / (SR - SL), FR)
    else:
        aL, aR = L[0] * (SL - L[1]), R[0] * (SR - R[1])
        Ss = (R[3] - L[3] + aL * L[1] - aR * R[1]) / (aL - aR)

        def star(V, S, a, E):
            k = a / (S - Ss)
            return torch.stack([k, k * Ss, k * V[2], k * (E / V[0] + (Ss - V[1]) * (Ss + V[3] / a))])

        F = torch.where(Ss > 0, FL + SL * (star(L, SL, aL, UL[3]) - UL),
                        torch.where(SR > 0, FR + SR * (star(R, SR, aR, UR[3]) - UR), FR))
    F = torch.where(SL > 0, FL, F)
    return U - ratio * (F[..., 1:] - F[..., :-1])


def _euler_exact(case, steps):
    W, dx, dy = _euler_initial(case)
    U, t, hll = _euler_cons(torch.from_numpy(W).to(_dev())), 0.0, case["solver"] == "hll"
    turn = lambda A: A[[0, 2, 1, 3]].transpose(1, 2)  # noqa: E731
    for n in range(steps):
        W = _euler_prim(U)
        c = torch.sqrt(1.4 * W[3] / W[0])
        dt = 0.8 * min(dx / float((W[1].abs() + c).max()), dy / float((W[2].abs() + c).max()))
        for axis in ((0, 1) if n % 2 == 0 else (1, 0)):
            U = _euler_sweep(U, dt / dx, hll) if axis == 0 else turn(_euler_sweep(turn(U), dt / dy, hll))
        t += dt
    return {"W": _euler_prim(U).permute(1, 2, 0).contiguous(), "t": t}


def _layer_exact(case, seed):
    s = {k: v.double() for k, v in _layer_inputs(case, seed).items()}
    x, wt, dz, zp = s["x"], s["wt"], s["dz"], s["zprev"]
    taps = [(t // 3 - 1, t % 3 - 1) for t in range(9)]

    def gelu(z):
        return z * torch.sigmoid(2.0 * math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3))

    out = {}
    if case["part"] in ("forward", "both"):
        z = s["bias"] + sum(torch.roll(x, (-dy, -dx), (1, 2)) @ wt[:, t].T for t, (dy, dx) in enumerate(taps))
        out.update({"out": z} if case["c_out"] == 16 else {"z": z, "a": gelu(z)})
    if case["part"] in ("backward", "both"):
        flat = dz.reshape(-1, dz.shape[3])
        out["dw"] = torch.stack([flat.T @ torch.roll(x, (-dy, -dx), (1, 2)).reshape(-1, 32) for dy, dx in taps], dim=1)
        out["db"] = flat.sum(0)
        da = sum(torch.roll(dz, (dy, dx), (1, 2)) @ wt[:, t] for t, (dy, dx) in enumerate(taps))
        a = 2.0 * math.sqrt(2.0 / math.pi)
        g = torch.sigmoid(a * (zp + 0.044715 * zp ** 3))
        out["dzprev"] = da * (g + zp * g * (1.0 - g) * a * (1.0 + 3.0 * 0.044715 * zp * zp))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "mhd":
        dom, bc = _domain(case)
        U, t = _mhd_exact(_initial(case, seed).astype(np.float64), dom, bc, case["order"], case["solver"] == "hlld",
                          case["steps"])
        return {"U": U, "t": t}
    if kind == "ensemble":
        return [_mhd_exact(_ot(n, b0), (0.0, 1.0, 0.0, 1.0), (0, 0, 0, 0), "muscl", True, case["steps"])[0]
                for n, b0 in _members(case, seed)]
    if kind == "euler":
        return _euler_exact(case, int(_euler_offset(case, seed)) + case["steps"])
    return _layer_exact(case, seed)
