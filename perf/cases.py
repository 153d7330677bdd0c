"""Performance cases of the framework: whole calls through its public entry
points, as the programs that use it make them.

Kinds of call
  run      an initial state in, `steps` RK2 steps, the final state out: the
           stretch between two snapshots of a simulation
  loop     the same through the reference driver's loop: one step, a crash
           check and a read of dt at a time
  batch    an ensemble of uneven periodic runs stepped together
  adjoint  a recorded forward run and its reverse: the gradients of a
           final-state misfit in the initial state and the resistivity

`exact` restates the step in plain torch at 64 bits (the stage-1-EMF step,
the CT-Contact step, both wall kinds used here, and the gradient through
automatic differentiation).
"""
import math

import torch

from resistivemhd_gpu_b200 import Batch, Solver, setups

GAMMA, CFL, EPS = 5.0 / 3.0, 0.4, 1e-20
G = 3   # ghost layers per side
FLOPS_PER_CELL_STEP = 3419   # operations of one RK2 step per cell (adds, multiplies, divisions, roots)
SIZES_BATCH = (128, 192, 256, 384, 512)


def listed():
    return [
        # a driver on a test-sized current sheet: every launch and wait counts
        {"name": "loop_harris_96x48", "kind": "loop", "flow": "harris", "n": 96, "m": 48, "steps": 20,
         "precision": "fp64_exact"},
        # a driver on the smallest ensemble grid
        {"name": "loop_ot_128_fast", "kind": "loop", "flow": "ot", "n": 128, "m": 128, "steps": 40,
         "precision": "fp64_fast"},
        # the Orszag-Tang vortex of the examples, drop-in arithmetic
        {"name": "run_ot_256", "kind": "run", "flow": "ot", "n": 256, "m": 256, "steps": 100,
         "precision": "fp64_exact"},
        # a ragged shear layer: neither side a multiple of any tile
        {"name": "run_kh_601x347_fast", "kind": "run", "flow": "kh", "n": 601, "m": 347, "steps": 50,
         "precision": "fp64_fast"},
        # the benchmark's Harris sheet, drop-in arithmetic, tuned as the benchmark tunes it
        {"name": "run_harris_2048x1024", "kind": "run", "flow": "harris", "n": 2048, "m": 1024, "steps": 40,
         "precision": "fp64_exact", "autotune": True},
        # the same sheet with fused multiply-add
        {"name": "run_harris_2048x1024_fast", "kind": "run", "flow": "harris", "n": 2048, "m": 1024, "steps": 12,
         "precision": "fp64_fast", "autotune": True},
        # the same sheet with single-precision fluxes
        {"name": "run_harris_2048x1024_bulk", "kind": "run", "flow": "harris", "n": 2048, "m": 1024, "steps": 12,
         "precision": "fp32_bulk", "autotune": True},
        # the plasmoid-unstable thin sheet, the largest grid of the configurations
        {"name": "run_plasmoid_8192x4096_bulk", "kind": "run", "flow": "plasmoid", "n": 8192, "m": 4096, "steps": 12,
         "precision": "fp32_bulk", "autotune": True},
        # the constrained-transport option of the multi-GPU library
        {"name": "run_contact_1024x512", "kind": "run", "flow": "harris", "n": 1024, "m": 512, "steps": 20,
         "precision": "fp64_exact", "ct": "contact"},
        # an ensemble of small uneven grids, tuned as the benchmark tunes it
        {"name": "batch_24_bulk", "kind": "batch", "runs": 24, "steps": 20, "precision": "fp32_bulk",
         "autotune": True},
        # the inverse problem: square-root checkpoints, drop-in forward
        {"name": "adjoint_ot_512", "kind": "adjoint", "flow": "ot", "n": 512, "m": 512, "steps": 36,
         "interval": 0, "precision": "fp64_exact"},
        # a small, ragged grid with symmetric walls and the whole trajectory kept
        {"name": "adjoint_smooth_150x90_tape", "kind": "adjoint", "flow": "smooth", "n": 150, "m": 90, "steps": 36,
         "interval": -1, "precision": "fp64_exact"},
    ]


def draw(rng):
    """A case of the same ranges: sizes over their logarithm, odd ones too."""
    kind = rng.choice(("loop", "run", "run", "run", "contact", "batch", "adjoint"))
    precision = rng.choice(("fp64_exact", "fp64_fast", "fp32_bulk"))
    if kind == "batch":
        return {"kind": "batch", "runs": rng.randint(4, 32), "steps": rng.randint(8, 24), "precision": precision,
                "autotune": rng.random() < 0.5}
    lo, hi = {"loop": (32, 256), "run": (48, 4096), "contact": (64, 2048), "adjoint": (48, 640)}[kind]
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    m = max(lo, min(hi, int(round(n * math.exp(rng.uniform(-0.9, 0.5))))))
    flow = rng.choice(("ot", "kh", "harris"))
    case = {"kind": kind, "flow": flow, "n": n, "m": m, "precision": precision}
    if kind == "adjoint":
        case.update(flow=rng.choice(("ot", "smooth")), steps=rng.randint(9, 36), interval=rng.choice((0, -1)),
                    precision="fp64_exact")
        return case
    budget = 20_000_000 if precision == "fp32_bulk" else 60_000_000
    steps = budget // (n * m)
    top = {"loop": 40, "run": 100, "contact": 20}[kind]
    case["steps"] = max(4, min(top if precision != "fp32_bulk" else 12, steps))
    if kind == "contact":
        case.update(kind="run", ct="contact", precision="fp64_exact")
    return case


# ---- initial states (interior n x m cells and 3 ghost layers per side) ----

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _noise(g, nx, ny):
    return 2.0 * torch.rand((nx, ny), generator=g, dtype=torch.float64, device="cuda") - 1.0


def _centres(n, lo, d):
    return lo + (torch.arange(n, dtype=torch.float64, device="cuda") - G + 0.5) * d


def _curl(az, dx, dy):
    """Face B of corner values az (nx+1, ny+1): discretely divergence free."""
    return (az[1:, 1:] - az[1:, :-1]) / dy, -(az[1:, 1:] - az[:-1, 1:]) / dx


def _cell_centred(bx, by):
    return 0.5 * (bx + torch.cat([bx[:1], bx[:-1]], 0)), 0.5 * (by + torch.cat([by[:, :1], by[:, :-1]], 1))


def _pack(rho, u, v, w, bx, by, bz, p):
    bxc, byc = _cell_centred(bx, by)
    e = p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v + w * w) + 0.5 * (bxc * bxc + byc * byc + bz * bz)
    return torch.stack([rho, rho * u, rho * v, rho * w, bx, by, bz, e], -1).contiguous()


def _problem(flow, n, m, g, rough=0.0, smooth_eta=False):
    """(AoS state on the GPU, dx, dy, scalar eta, eta table or None, wall
    kind).  `rough`: relative noise of the density and pressure."""
    nx, ny = n + 2 * G, m + 2 * G
    one = torch.ones((nx, ny), dtype=torch.float64, device="cuda")
    rn = 1.0 + rough * _noise(g, nx, ny), 1.0 + rough * _noise(g, nx, ny)
    table = None
    if flow == "ot":
        dx, dy, eta, walls = 2 * math.pi / n, 2 * math.pi / m, 1e-3, "periodic"
        x, y = _centres(nx, 0.0, dx)[:, None] * one, _centres(ny, 0.0, dy)[None, :] * one
        u, v = -torch.sin(y) + 1e-6 * _noise(g, nx, ny), torch.sin(x) + 1e-6 * _noise(g, nx, ny)
        state = _pack(GAMMA * GAMMA * rn[0], u, v, 0 * one, -torch.sin(y), torch.sin(2 * x), 0 * one, GAMMA * rn[1])
        if smooth_eta:
            a, b = (2 * math.pi * torch.rand(2, generator=g, dtype=torch.float64, device="cuda")).tolist()
            table = 1e-3 * torch.exp(0.5 * (torch.cos(2 * x + a) + torch.cos(3 * y + b)))
    elif flow == "kh":
        dx, dy, eta, walls, wid = 1.0 / n, 1.0 / m, 1e-3, "periodic", 0.05
        x, y = _centres(nx, 0.0, dx)[:, None] * one, torch.remainder(_centres(ny, 0.0, dy), 1.0)[None, :] * one
        u = 0.5 * (torch.tanh((y - 0.25) / wid) - torch.tanh((y - 0.75) / wid) - 1.0)
        env = torch.exp(-((y - 0.25) ** 2) / (2 * wid * wid)) + torch.exp(-((y - 0.75) ** 2) / (2 * wid * wid))
        v = 1e-2 * (torch.sin(2 * math.pi * x) + _noise(g, nx, ny)) * env
        state = _pack(rn[0], u, v, 0 * one, 0.1 * one, 0 * one, 0 * one, rn[1])
    elif flow == "smooth":
        # every field varies in both directions, between mirror walls
        dx, dy, eta, walls, tau = 1.0 / n, 1.3 / m, 2e-3, "symmetric", 2 * math.pi
        x, y = _centres(nx, 0.0, dx)[:, None] * one, _centres(ny, 0.0, dy)[None, :] * one / 1.3
        xc = (torch.arange(nx + 1, dtype=torch.float64, device="cuda") - G)[:, None] / n
        yc = (torch.arange(ny + 1, dtype=torch.float64, device="cuda") - G)[None, :] / m
        az = 0.15 * torch.cos(tau * xc) * torch.cos(tau * yc) + 0.1 * torch.sin(tau * (xc + 2 * yc))
        bx, by = _curl(az + 1e-3 * _noise(g, nx + 1, ny + 1), dx, dy)
        state = _pack(1.0 + 0.3 * torch.sin(tau * x) * torch.cos(tau * y) + 0.01 * _noise(g, nx, ny),
                      0.4 * torch.sin(tau * y) + 0.05 * _noise(g, nx, ny),
                      -0.3 * torch.sin(tau * x) + 0.05 * _noise(g, nx, ny),
                      0.2 * torch.cos(tau * x) * torch.sin(tau * y) + 0.05 * _noise(g, nx, ny), bx, by,
                      0.3 * torch.cos(tau * (x - y)) + 0.05 * _noise(g, nx, ny),
                      0.8 + 0.2 * torch.cos(tau * (x + y)) + 0.01 * _noise(g, nx, ny))
        table = eta * (1.0 + 0.5 * torch.sin(tau * x) ** 2 * torch.cos(tau * y) ** 2)
    else:
        wid, beta, amp, eta0, bump = (0.1, 0.1, 1e-4, 1e-5, 0.0) if flow == "plasmoid" else (0.5, 0.2, 1e-3, 1e-3, 1e-2)
        lx, ly, walls = 128.0, 64.0, "symmetric"
        dx, dy, eta = lx / n, ly / m, eta0 + bump
        x, y = _centres(nx, -lx / 2, dx)[:, None], _centres(ny, -ly / 2, dy)[None, :]
        xc = -lx / 2 + (torch.arange(nx + 1, dtype=torch.float64, device="cuda") - G)[:, None] * dx
        yc = -ly / 2 + (torch.arange(ny + 1, dtype=torch.float64, device="cuda") - G)[None, :] * dy
        az = wid * torch.log(torch.cosh(yc / wid)) + 0.03 * torch.cos(2 * math.pi * xc / lx) * torch.cos(math.pi * yc / ly)
        bx, by = _curl(az, dx, dy)
        sech2 = 1.0 / torch.cosh(y / wid) ** 2
        state = _pack((sech2 + beta) * rn[0], amp * _noise(g, nx, ny), amp * _noise(g, nx, ny), 0 * one, bx, by,
                      0 * one, 0.5 * (beta + sech2) * rn[1])
        if bump:
            table = eta0 + bump * torch.exp(-(x * x + y * y))
    if table is not None:
        eta = float(table.max())
    return state, dx, dy, eta, table, walls


def _case_problem(case, seed):
    adj = case["kind"] == "adjoint"
    return _problem(case["flow"], case["n"], case["m"], _gen(seed), rough=1e-3 if adj else 0.0, smooth_eta=adj)


def _batch_problems(case, seed):
    g = _gen(seed)
    sizes = torch.randint(len(SIZES_BATCH), (case["runs"],), generator=_gen(case["runs"]), device="cuda").tolist()
    etas = torch.exp(math.log(1e-4) + math.log(1e2) * torch.rand(case["runs"], generator=g, device="cuda",
                                                                 dtype=torch.float64)).tolist()
    out = []
    for r in range(case["runs"]):
        n = SIZES_BATCH[sizes[r]]
        state, dx, dy, _, _, walls = _problem("ot" if r % 2 == 0 else "kh", n, n, g)
        out.append((state, dx, dy, etas[r], None, walls))
    return out


def _seed_field(nx, ny, seed):
    """dJ/dU_N of a misfit of the interior's density and field."""
    s = torch.zeros((nx, ny, 8), dtype=torch.float64, device="cuda")
    g = _gen(seed + 7919)
    for f in (0, 4, 5, 6):
        s[G:-G, G:-G, f] = _noise(g, nx - 2 * G, ny - 2 * G)
    return s


# ---- the calls ----

def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def prepare(case, seed):
    if case["kind"] == "batch":
        probs = _batch_problems(case, seed)
        batch = Batch([setups.Setup("run", p[0].cpu().numpy(), p[1], p[2], GAMMA, CFL, EPS, p[3], None, p[5])
                       for p in probs], precision=case["precision"])
        if case.get("autotune"):
            batch.autotune(4)
        return {"case": case, "batch": batch, "initial": [p[0] for p in probs],
                "out": [_pinned(*p[0].shape) for p in probs]}
    state, dx, dy, eta, table, walls = _case_problem(case, seed)
    nx, ny = state.shape[:2]
    s = Solver(nx, ny, dx, dy, gamma=GAMMA, cfl=CFL, eps=EPS, eta=eta, bc=walls, precision=case["precision"],
               ct=case.get("ct", "stage1"))
    if table is not None:
        s.set_eta_table(table.cpu().numpy())
    torch.cuda.synchronize()
    st = {"case": case, "solver": s, "initial": state}
    if case["kind"] == "adjoint":
        st["seed"] = _seed_field(nx, ny, seed).cpu().numpy()
    else:
        st["out"] = _pinned(nx, ny, 8)
    if case.get("autotune"):
        s.set_state_device(state.data_ptr())
        s.autotune(4)
    return st


def run(st):
    case = st["case"]
    if case["kind"] == "batch":
        b = st["batch"]
        for r in range(len(b)):
            b[r].set_state_device(st["initial"][r].data_ptr())
        b.run(case["steps"])
        return [b[r].get_state(st["out"][r]) for r in range(len(b))]
    s = st["solver"]
    s.set_state_device(st["initial"].data_ptr())
    if case["kind"] == "adjoint":
        s.adjoint_forward(case["steps"], case["interval"])
        grad_state, grad_eta = s.adjoint_backward(st["seed"])
        return {"dts": s.adjoint_dts(), "grad_state": grad_state, "grad_eta": grad_eta}
    if case["kind"] == "loop":
        t = 0.0
        for _ in range(case["steps"]):
            s.step()
            if s.check_crashed():
                break
            t += s.dt
        return {"state": s.get_state(st["out"]), "time": t}
    s.run(case["steps"])
    return {"state": s.get_state(st["out"]), "dt": s.dt}


def work(case):
    """A step reads and writes the state (and reads the resistivity table);
    the reverse of a step costs at least the step's own operations twice."""
    if case["kind"] == "batch":
        sizes = torch.randint(len(SIZES_BATCH), (case["runs"],), generator=_gen(case["runs"]), device="cuda").tolist()
        cells, table = sum(SIZES_BATCH[k] ** 2 for k in sizes), 0
    else:
        cells = case["n"] * case["m"]
        table = 8 if case["flow"] == "harris" or case["kind"] == "adjoint" else 0
    k = 3 if case["kind"] == "adjoint" else 1
    return {"bytes": float(cells) * case["steps"] * (128 + table) * k,
            "flops": float(cells) * case["steps"] * FLOPS_PER_CELL_STEP * k}


# ---- the step in plain torch at 64 bits; a state is a list of 8 (nx, ny) fields ----

def _sqrt(x):
    """sqrt with derivative 0 at 0, NaN below."""
    pos = x > 0
    return torch.where(pos, torch.sqrt(torch.where(pos, x, torch.ones_like(x))),
                       torch.where(x == 0, torch.zeros_like(x), torch.full_like(x, math.nan)))


def _minmod(x, y):
    ax, sy = x.abs(), torch.where(x < 0, -y, y)
    pick = torch.where(sy < ax, sy, ax)
    m = torch.where(pick < EPS, torch.full_like(pick, EPS), pick)
    return torch.where(x > 0, m, torch.where(x < 0, -m, torch.zeros_like(m)))


def _hlld(L, R):
    """Flux of (rho, u, v, w, bn, b1, b2, p) states: mass, three momenta,
    induction of b1 and b2, energy."""
    g1 = GAMMA - 1.0
    bX = L[4]

    def outer(q):
        rho, u, v, w, _, b1, b2, p = q
        bb = bX * bX + b1 * b1 + b2 * b2
        e = p / g1 + 0.5 * rho * (u * u + v * v + w * w) + 0.5 * bb
        cs, ca, va = _sqrt(GAMMA * p / rho), _sqrt(bb / rho), _sqrt(bX * bX / rho)
        s = cs * cs + ca * ca
        return e, p + 0.5 * bb, _sqrt(0.5 * (s + _sqrt(s * s - 4.0 * cs * cs * va * va)))

    rL, uL, vL, wL, _, yL, zL, _ = L
    rR, uR, vR, wR, _, yR, zR, _ = R
    (eL, ptL, cfL), (eR, ptR, cfR) = outer(L), outer(R)
    cf = torch.where(cfL < cfR, cfR, cfL)
    SL = torch.where(uR < uL, uR, uL) - cf
    SR = torch.where(uL < uR, uR, uL) + cf
    SL = torch.where(0.0 < SL, torch.zeros_like(SL), SL)
    SR = torch.where(SR < 0.0, torch.zeros_like(SR), SR)
    den = (SR - uR) * rR - (SL - uL) * rL + EPS
    SM = ((SR - uR) * rR * uR - (SL - uL) * rL * uL - ptR + ptL) / den
    pt1 = ((SR - uR) * rR * ptL - (SL - uL) * rL * ptR + rL * rR * (SR - uR) * (SL - uL) * (uR - uL)) / den

    def star(S, r, u, v, w, y, z, e, pt):
        d = r * (S - u) * (S - SM) - bX * bX + EPS
        n = r * (S - u) * (S - u) - bX * bX
        r1 = r * (S - u) / (S - SM + EPS)
        v1, w1 = v - bX * y * (SM - u) / d, w - bX * z * (SM - u) / d
        y1, z1 = y * n / d, z * n / d
        vb1 = SM * bX + v1 * y1 + w1 * z1
        e1 = ((S - u) * e - pt * u + pt1 * SM + bX * ((u * bX + v * y + w * z) - vb1)) / (S - SM + EPS)
        return r1, v1, w1, y1, z1, e1, vb1

    r1L, v1L, w1L, y1L, z1L, e1L, vbL = star(SL, rL, uL, vL, wL, yL, zL, eL, ptL)
    r1R, v1R, w1R, y1R, z1R, e1R, vbR = star(SR, rR, uR, vR, wR, yR, zR, eR, ptR)
    S1L, S1R = SM - _sqrt(bX * bX / r1L), SM + _sqrt(bX * bX / r1R)
    qL, qR, sg = _sqrt(r1L), _sqrt(r1R), torch.sign(bX)
    qLR, dq = _sqrt(r1L * r1R), qL + qR + EPS
    v2 = (qL * v1L + qR * v1R + (y1R - y1L) * sg) / dq
    w2 = (qL * w1L + qR * w1R + (z1R - z1L) * sg) / dq
    y2 = (qL * y1R + qR * y1L + qLR * (v1R - v1L) * sg) / dq
    z2 = (qL * z1R + qR * z1L + qLR * (w1R - w1L) * sg) / dq
    vb2 = SM * bX + v2 * y2 + w2 * z2
    e2L, e2R = e1L - qL * (vbL - vb2) * sg, e1R + qR * (vbR - vb2) * sg
    oL, oR = SL > 0.0, SR <= 0.0
    mL, iL = (SL <= 0.0) & (0.0 < S1L), (S1L <= 0.0) & (0.0 < SM)
    mR, iR = (S1R <= 0.0) & (0.0 < SR), (SM <= 0.0) & (0.0 < S1R)
    nan = torch.full_like(SM, math.nan)

    def pick(a, b, c, d, e, f):
        return torch.where(oL, a, torch.where(oR, d, torch.where(mL, b, torch.where(iL, c, torch.where(
            mR, e, torch.where(iR, f, nan))))))

    r = pick(rL, r1L, r1L, rR, r1R, r1R)
    u = pick(uL, SM, SM, uR, SM, SM)
    v = pick(vL, v1L, v2, vR, v1R, v2)
    w = pick(wL, w1L, w2, wR, w1R, w2)
    y = pick(yL, y1L, y2, yR, y1R, y2)
    z = pick(zL, z1L, z2, zR, z1R, z2)
    e = pick(eL, e1L, e2L, eR, e1R, e2R)
    pt = pick(ptL, pt1, pt1, ptR, pt1, pt1)
    return (r * u, r * u * u + pt - bX * bX, r * u * v - bX * y, r * u * w - bX * z, u * y - v * bX, u * z - w * bX,
            (e + pt) * u - bX * (bX * u + y * v + z * w))


def _fluxes(U, dx, dy, eta):
    """x fluxes at i = 2 .. nx-4, j = 2 .. ny-3 and y fluxes at i = 2 ..
    nx-3, j = 2 .. ny-4, as dicts by field index, resistive terms included."""
    rho, mx, my, mz, bx, by, bz, e = U
    nx, ny = rho.shape
    bxc, byc = torch.cat([bx[:1], 0.5 * (bx[1:] + bx[:-1])], 0), torch.cat([by[:, :1], 0.5 * (by[:, 1:] + by[:, :-1])], 1)
    u, v, w = mx / rho, my / rho, mz / rho

    def pressure(a, b, c, p, q, r):
        return (GAMMA - 1.0) * (e - 0.5 * (rho * (a * a + b * b + c * c)) - 0.5 * (p * p + q * q + r * r))

    def states(q, bn, at):
        L, R = [], []
        for a in q:
            qm, q0, qp, qpp = (at(a, d) for d in (-1, 0, 1, 2))
            L.append(q0 + 0.5 * _minmod(q0 - qm, qp - q0))
            R.append(qp - 0.5 * _minmod(qp - q0, qpp - qp))
        b = 0.5 * (at(bn, 0) + at(bn, 1))
        return L[:4] + [b] + L[4:], R[:4] + [b] + R[4:]

    def at_x(a, d):
        return a[2 + d:nx - 3 + d, 2:ny - 2]

    def at_y(a, d):
        return a[2:nx - 2, 2 + d:ny - 3 + d]

    # the current at i = 1 .. nx-2, j = 1 .. ny-2, and eta J in place on the full grid
    def full(a):
        return torch.nn.functional.pad(a, (1, 1, 1, 1))

    et = eta[1:-1, 1:-1] if torch.is_tensor(eta) else eta
    ex = full(et * ((bz[1:-1, 2:] - bz[1:-1, :-2]) / (2.0 * dy)))
    ey = full(et * (-(bz[2:, 1:-1] - bz[:-2, 1:-1]) / (2.0 * dx)))
    ez = full(et * ((byc[2:, 1:-1] - byc[:-2, 1:-1]) / (2.0 * dx) - (bxc[1:-1, 2:] - bxc[1:-1, :-2]) / (2.0 * dy)))

    def mean(at, a, b=None):
        a0, a1 = at(a, 0), at(a, 1)
        return 0.5 * (a0 + a1) if b is None else 0.5 * (a0 * at(b, 0) + a1 * at(b, 1))

    f = _hlld(*states((rho, u, v, w, byc, bz, pressure(u, v, w, bxc, byc, bz)), bxc, at_x))
    F = {0: f[0], 1: f[1], 2: f[2], 3: f[3], 5: f[4] - mean(at_x, ez), 6: f[5] + mean(at_x, ey),
         7: f[6] + (mean(at_x, ey, bz) - mean(at_x, ez, byc))}
    f = _hlld(*states((rho, v, w, u, bz, bxc, pressure(v, w, u, byc, bz, bxc)), byc, at_y))
    Gf = {0: f[0], 1: f[3], 2: f[1], 3: f[2], 4: f[5] + mean(at_y, ez), 6: f[4] - mean(at_y, ex),
          7: f[6] + (mean(at_y, ez, bxc) - mean(at_y, ex, bz))}
    return F, Gf, bxc, byc


def _fill(I, row2, walls, dx, dy):
    """Full fields from interior ones; row2: face bY of the lower wall, which
    the mirror x walls read."""
    if walls == "periodic":
        out = [torch.cat([a[-3:], a, a[:3]], 0) for a in I]
        return [torch.cat([a[:, -3:], a, a[:, :3]], 1) for a in out]
    out = [torch.cat([a[:3].flip(0), a, a[-3:].flip(0)], 0) for a in I]
    bx, by = I[4], torch.cat([row2[:, None], I[5]], 1)
    D = (by[:, 1:] - by[:, :-1]) / dy * dx
    l2 = bx[0] + D[0]
    l1 = l2 + D[0]
    h1 = bx[-1] - D[-1]
    h2 = h1 - D[-2]
    out[4] = torch.cat([torch.stack([l1 + D[1], l1, l2]), bx, torch.stack([h1, h2, h2 - D[-3]])], 0)
    bx, by = out[4], out[5]
    E = torch.cat([torch.zeros_like(bx[:1]), (bx[1:] - bx[:-1]) / dx * dy], 0)
    l2 = by[:, 0] + E[:, 0]
    l1 = l2 + E[:, 0]
    h1 = by[:, -1] - E[:, -1]
    h2 = h1 - E[:, -2]
    lo, hi = torch.stack([l1 + E[:, 1], l1, l2], 1), torch.stack([h1, h2, h2 - E[:, -3]], 1)
    out = [torch.cat([a[:, :3].flip(1), a, a[:, -3:].flip(1)], 1) for a in out]
    out[5] = torch.cat([lo, by, hi], 1)
    return out


def _inner(a):
    return a[G:-G, G:-G]


def _dt(U, dx, dy, eta):
    rho, mx, my, mz, bx, by, bz, e = U
    u, v, w = mx / rho, my / rho, mz / rho
    bb = bx * bx + by * by + bz * bz
    p = (GAMMA - 1.0) * (e - 0.5 * rho * (u * u + v * v + w * w) - 0.5 * bb)
    c = torch.sqrt(torch.sqrt(GAMMA * p / rho) ** 2 + torch.sqrt(bb / rho) ** 2)
    a = (u.abs() + c) / dx + (v.abs() + c) / dy
    first = bool(torch.isnan(a[0, 0]))
    lim = min(dx * dx / eta, dy * dy / eta) if eta > 0 else math.inf
    return (lim if first else min(1.0 / (float(torch.nan_to_num(a, nan=0.0).max()) + EPS), lim)) * CFL


def _less_div(u, F, Gf, f, dt, dx, dy):
    """u - dt div of field f over the interior."""
    if f in F:
        u = u - dt / dx * (F[f][1:, 1:-1] - F[f][:-1, 1:-1])
    if f in Gf:
        u = u - dt / dy * (Gf[f][1:-1, 1:] - Gf[f][1:-1, :-1])
    return u


def _step(U, dt, dx, dy, eta, walls):
    F, Gf, _, _ = _fluxes(U, dx, dy, eta)
    ez = 0.25 * (Gf[4][:-1] + Gf[4][1:] - F[5][:, :-1] - F[5][:, 1:])   # corners i = 2 .. nx-4, j = 2 .. ny-4
    W = [_less_div(_inner(U[f]), F, Gf, f, dt, dx, dy) if f not in (4, 5) else None for f in range(8)]
    W[4] = _inner(U[4]) - dt / dy * (ez[1:, 1:] - ez[1:, :-1])
    W[5] = _inner(U[5]) + dt / dx * (ez[1:, 1:] - ez[:-1, 1:])
    row2 = U[5][G:-G, 2] + dt / dx * (ez[1:, 0] - ez[:-1, 0])
    S = _fill(W, row2, walls, dx, dy)
    F, Gf, _, _ = _fluxes(S, dx, dy, eta)
    V = [0.5 * _less_div(_inner(U[f]) + W[f], F, Gf, f, dt, dx, dy) if f not in (4, 5) else W[f] for f in range(8)]
    return _fill(V, row2, walls, dx, dy)


def _reference_emf(U, bx, by, dx, dy, eta):
    """u bY - v bX - eta jZ at i = 2 .. nx-3, j = 2 .. ny-3 from face B."""
    def s(a, di=0, dj=0):
        return a[2 + di:a.shape[0] - 2 + di, 2 + dj:a.shape[1] - 2 + dj]
    jz = 0.25 * ((s(by, 1) - s(by)) / dx - (s(bx, 0, 1) - s(bx)) / dy
                 + (s(by, 1, -1) - s(by, 0, -1)) / dx - (s(bx) - s(bx, 0, -1)) / dy
                 + (s(by, 0, -1) - s(by, -1, -1)) / dx - (s(bx, -1) - s(bx, -1, -1)) / dy
                 + (s(by) - s(by, -1)) / dx - (s(bx, -1, 1) - s(bx, -1)) / dy)
    et = s(eta) if torch.is_tensor(eta) else eta
    return s(U[1]) / s(U[0]) * (0.5 * (s(by) + s(by, 0, -1))) - s(U[2]) / s(U[0]) * (0.5 * (s(bx) + s(bx, -1))) - et * jz


def _contact_emf(F, Gf, ref):
    """Corner EMFs i = 2 .. nx-4, j = 2 .. ny-4 of one stage."""
    f5, f5n, g4, g4e = F[5][:, :-1], F[5][:, 1:], Gf[4][:-1], Gf[4][1:]
    sf, sfn, sg, sge = (torch.sign(a) for a in (F[0][:, :-1], F[0][:, 1:], Gf[0][:-1], Gf[0][1:]))
    c, ce, cn, cne = ref[:-1, :-1], ref[1:, :-1], ref[:-1, 1:], ref[1:, 1:]
    s = (1 + sf) * (g4 + c) + (1 - sf) * (g4e + ce)
    n = (1 + sfn) * (-cn - g4) + (1 - sfn) * (-cne - g4e)
    w = -(1 + sg) * (f5 - c) - (1 - sg) * (f5n - cn)
    e = -(1 + sge) * (ce - f5) - (1 - sge) * (cne - f5n)
    return 0.25 * (-f5 - f5n + g4 + g4e) + 0.125 * (s - n + w - e)


def _contact_step(U, dt, dx, dy, eta, walls):
    def smooth(bxc, byc):
        return (torch.cat([0.5 * (bxc[:-1] + bxc[1:]), bxc[-1:]], 0),
                torch.cat([0.5 * (byc[:, :-1] + byc[:, 1:]), byc[:, -1:]], 1))

    def wall(by, F):   # by of row 2 less its x flux difference
        return by[G:-G, 2] - dt / dx * (F[5][1:, 0] - F[5][:-1, 0])

    F1, G1, bxc, byc = _fluxes(U, dx, dy, eta)
    sx, sy = smooth(bxc, byc)
    old = _contact_emf(F1, G1, _reference_emf(U, sx, sy, dx, dy, eta))
    base = list(U)
    base[4], base[5] = sx, sy
    W = [_less_div(_inner(base[f]), F1, G1, f, dt, dx, dy) for f in range(8)]
    S = _fill(W, wall(sy, F1), walls, dx, dy)
    F2, G2, bxc, byc = _fluxes(S, dx, dy, eta)
    tx, ty = smooth(bxc, byc)
    bar = list(S)
    bar[4], bar[5] = tx, ty
    C = [0.5 * _less_div(_inner(base[f]) + _inner(bar[f]), F2, G2, f, dt, dx, dy) for f in range(8)]
    row2 = 0.5 * (sy[G:-G, 2] + wall(ty, F2))
    full = _fill(C, row2, walls, dx, dy)
    now = _contact_emf(F2, G2, _reference_emf(full, full[4], full[5], dx, dy, eta))
    ez = 0.5 * (old + now)
    C[4] = _inner(U[4]) - dt / dy * (ez[1:, 1:] - ez[1:, :-1])
    C[5] = _inner(U[5]) + dt / dx * (ez[1:, 1:] - ez[:-1, 1:])
    return _fill(C, U[5][G:-G, 2] + dt / dx * (ez[1:, 0] - ez[:-1, 0]), walls, dx, dy)


def _start(fields, walls, dx, dy):
    return _fill([_inner(a) for a in fields], fields[5][G:-G, 2], walls, dx, dy)


def _evolve(problem, steps, ct="stage1"):
    """(final AoS state, dts)"""
    state, dx, dy, eta, table, walls = problem
    U = _start([state[..., f].contiguous() for f in range(8)], walls, dx, dy)
    advance = _contact_step if ct == "contact" else _step
    dts = []
    for _ in range(steps):
        dts.append(_dt(U, dx, dy, eta))
        U = advance(U, dts[-1], dx, dy, eta if table is None else table, walls)
    return torch.stack(U, -1), dts


def _gradient(problem, seed_field, steps):
    state, dx, dy, eta, table, walls = problem
    leaf = [state[..., f].clone().requires_grad_(True) for f in range(8)]
    first = _start(leaf, walls, dx, dy)
    U, kept, dts = [a.detach() for a in first], [], []
    for _ in range(steps):
        kept.append(U)
        dts.append(_dt(U, dx, dy, eta))
        U = _step(U, dts[-1], dx, dy, table, walls)
    bar = [seed_field[..., f].contiguous() for f in range(8)]
    eta_bar = torch.zeros_like(table)
    for U, dt in zip(reversed(kept), reversed(dts)):
        x = [a.clone().requires_grad_(True) for a in U]
        t = table.clone().requires_grad_(True)
        grads = torch.autograd.grad(_step(x, dt, dx, dy, t, walls), x + [t], bar, allow_unused=True)
        bar = [torch.zeros_like(a) if d is None else d for a, d in zip(x, grads)]
        eta_bar = eta_bar + grads[8]
    grads = torch.autograd.grad(first, leaf, bar, allow_unused=True)
    out = torch.stack([torch.zeros_like(a) if d is None else d for a, d in zip(leaf, grads)], -1)
    return out, eta_bar, dts


def exact(case, seed):
    if case["kind"] == "batch":
        return [_evolve(p, case["steps"])[0] for p in _batch_problems(case, seed)]
    problem = _case_problem(case, seed)
    if case["kind"] == "adjoint":
        nx, ny = problem[0].shape[:2]
        grad_state, grad_eta, dts = _gradient(problem, _seed_field(nx, ny, seed), case["steps"])
        return {"dts": torch.tensor(dts, dtype=torch.float64), "grad_state": grad_state, "grad_eta": grad_eta}
    state, dts = _evolve(problem, case["steps"], case.get("ct", "stage1"))
    return {"state": state, "time": sum(dts)} if case["kind"] == "loop" else {"state": state, "dt": dts[-1]}
