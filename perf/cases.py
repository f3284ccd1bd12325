"""Performance cases of the framework: evaluations of the phi^4 objective through its Python entry
points (rcmps_b200.objective, rcmps_b200.optimizer).

States are i.i.d. complex Gaussian R and K (times `scale`), or their Z2-symmetric block form, with
the stationary density of each state in hand, as an optimizer or a sweep holds them. Settings are
the optimizer's defaults (half window 30, 512 Gauss nodes per half, tolerances 1e-13/1e-12, 512
kinetic nodes) unless a case says otherwise.

A case is one of these calls:
  objective    one state through objective(): the call that every L-BFGS trial makes;
  refined      the same at the validation run's refined controls;
  ode          the same with every term by ODEs (mode "ode");
  batch        fg_phi4_batch() over n states of one D, half of them Z2-symmetric with `kind` mixed;
  uneven       fg_phi4_batch() over n states of D from 8 to `d` with a tolerance pair per state;
  stationary   stationary_state(): the density that every trial solves before its objective;
  lbfgs        optimizer.optimize() for a number of iterations.
"""
import math
import os
import sys
from types import SimpleNamespace

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.getcwd(), "rcmpscore.jl_b200"))

from rcmps_b200 import objective as api  # noqa: E402
from rcmps_b200 import optimizer  # noqa: E402

DEFAULTS = dict(half_window=30.0, n_quad=512, nodes=512)
REFINED = dict(half_window=40.0, n_quad=1024, nodes=1024)


def listed():
    return [
        # the smallest bond dimension that is optimized in earnest: latency of a single trial
        dict(name="trial_d8", call="objective", d=8, kind="random", g=2.0, scale=0.2),
        # a trial of a Z2-symmetric run on its packed route, in the small range
        dict(name="trial_d16_z2", call="objective", d=16, kind="z2", g=2.0, scale=0.2),
        # ordinary trials, no symmetry
        dict(name="trial_d32", call="objective", d=32, kind="random", g=2.0, scale=0.2),
        dict(name="trial_d64", call="objective", d=64, kind="random", g=2.0, scale=0.2),
        # the largest bond dimension, on the packed route (where published runs used it)
        dict(name="trial_d128_z2", call="objective", d=128, kind="z2", g=2.0, scale=0.2),
        # validation of an optimized state at refined controls; D no multiple of a tile
        dict(name="validate_d25", call="refined", d=25, kind="random", g=1.3, scale=0.2),
        # the all-ODE route that the Julia package takes by default
        dict(name="ode_d16", call="ode", d=16, kind="random", g=2.0, scale=0.2),
        # sweeps: the benchmark's 32 states at D = 64, half of them Z2-symmetric
        dict(name="sweep_32x64", call="batch", d=64, n=32, kind="mixed", g=2.0, scale=0.2),
        # 64 states at D = 32
        dict(name="sweep_64x32", call="batch", d=32, n=64, kind="random", g=2.0, scale=0.2),
        # a qualification run: uneven sizes and tolerances in one call
        dict(name="uneven_16", call="uneven", d=100, n=16, kind="random", g=2.0, scale=0.2),
        # the density solve in front of each trial
        dict(name="density_d64", call="stationary", d=64, kind="random", g=2.0, scale=0.2),
        # two iterations of the optimizer: density, objective, direction, line search
        dict(name="optimize_d16", call="lbfgs", d=16, iterations=2, kind="random", g=2.0, scale=0.2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["objective", "objective", "objective", "batch", "batch", "uneven", "refined", "ode",
                       "stationary", "lbfgs"])
    case = dict(call=call, kind="random", g=round(rng.uniform(0.5, 3.0), 3), scale=round(rng.uniform(0.12, 0.22), 3))
    if call == "objective":
        case["kind"] = rng.choice(["random", "z2"])
        case["d"] = _log_int(rng, 4, 128 if case["kind"] == "z2" else 80)
    elif call == "batch":
        case["d"] = _log_int(rng, 6, 64)
        case["n"] = _log_int(rng, 2, max(2, min(64, 32 * 64 ** 3 // case["d"] ** 3)))
        case["kind"] = rng.choice(["random", "mixed"])
    elif call == "uneven":
        case["d"] = rng.randint(40, 90)
        case["n"] = rng.randint(4, 16)
    elif call == "refined":
        case["d"] = _log_int(rng, 4, 40)
    elif call == "ode":
        case["d"] = _log_int(rng, 4, 32)
    elif call == "stationary":
        case["kind"] = rng.choice(["random", "z2"])
        case["d"] = _log_int(rng, 4, 128)
    else:
        case["d"] = _log_int(rng, 4, 24)
        case["iterations"] = rng.randint(1, 2)
    if case["kind"] in ("z2", "mixed"):
        case["d"] += case["d"] % 2
    return case


# ----------------------------------------------------------------------------- inputs
def _state(rng, d, z2, scale):
    def block(n):
        return (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * (scale / math.sqrt(2.0))
    if not z2:
        r, a = block(d), block(d)
        return r, (a + a.conj().T) / 2
    n = d // 2
    zero = np.zeros((n, n), complex)
    k1, k2 = block(n), block(n)
    r = np.block([[zero, block(n)], [block(n), zero]])
    return r, np.block([[(k1 + k1.conj().T) / 2, zero], [zero, (k2 + k2.conj().T) / 2]])


def _left_canonical(r, k):
    return -1j * k - r.conj().T @ r / 2


def _density(r, k, z2):
    """The stationary density, L(rho) = 0: rho <- rho - a N^-1 L(rho) with the no-jump part
    N(X) = Q X + X Q^dag inverted in the eigenbasis of Q. a = 1 is the jump chain, whose period of
    two on a Z2-symmetric state a = 1/2 damps."""
    q = _left_canonical(r, k)
    lam, v = np.linalg.eig(q)
    q, r, lam, v, vi = (torch.from_numpy(x).cuda() for x in (q, r, lam, v, np.linalg.inv(v)))
    a = (0.5 if z2 else 1.0) / (lam[:, None] + lam.conj()[None, :])
    rh, vh, vih = _herm(r), _herm(v), _herm(vi)
    rho = torch.eye(len(q), dtype=q.dtype, device=q.device) / len(q)
    for i in range(200):
        res = q @ rho
        step = v @ (a * (vi @ (res + _herm(res) + r @ rho @ rh) @ vih)) @ vh
        rho = rho - step
        rho = rho + _herm(rho)
        rho = rho / torch.trace(rho).real
        if i % 8 == 7 and float(torch.linalg.norm(step) / torch.linalg.norm(rho)) <= 1e-14:
            break
    rho = rho.cpu().numpy()
    rho = (rho + rho.conj().T) / 2
    if z2:
        n = len(rho) // 2
        rho[:n, n:] = 0
        rho[n:, :n] = 0
    return rho


def prepare(case, seed):
    rng = np.random.default_rng([seed, 77])
    call, d, n = case["call"], case["d"], case.get("n", 1)
    dims = [d] * n
    if call == "uneven":   # D from 8 to the largest, spread over the logarithm
        dims = [int(round(8 * (d / 8) ** (1 - 0.6180339887 * i % 1.0))) for i in range(n)]
    s = SimpleNamespace(call=call, case=case, R=[], K=[], rho=[], Q=[], z2=[])
    for i, di in enumerate(dims):
        z2 = case["kind"] == "z2" or (case["kind"] == "mixed" and i >= n // 2)
        r, k = _state(rng, di, z2, case["scale"])
        s.R.append(r)
        s.K.append(k)
        s.z2.append(z2)
        s.Q.append(_left_canonical(r, k))
        s.rho.append(None if call in ("stationary",) else _density(r, k, z2))
    s.g = [case["g"]] if n == 1 else [float(x) for x in rng.uniform(0.5, 3.0, n)]
    s.args = SimpleNamespace(packed_z2=all(s.z2))
    if call == "refined":
        s.args = SimpleNamespace(window=40.0, quadrature=1024, atol=1e-14, rtol=1e-13, nodes=1024)
    elif call == "ode":
        s.args = SimpleNamespace(mode="ode")
    s.settings = api.settings_from_args(None, symmetry=api.SYMMETRY_AUTO)
    s.tolerances = None
    if call == "uneven":
        s.tolerances = [(float(rng.choice([1e-10, 1e-12])), float(rng.choice([1e-10, 1e-12]))) for _ in dims]
    if call == "lbfgs":
        s.callable = lambda r, k, rho: api.objective(r, k, rho, s.g[0], s.args)
        s.energy, s.gradient, _ = s.callable(s.R[0], s.K[0], s.rho[0])
        s.controls = optimizer.OptimizationControls(max_iterations=case["iterations"])
    return s


def run(s):
    if s.call in ("objective", "refined", "ode"):
        energy, gradient, _ = api.objective(s.R[0], s.K[0], s.rho[0], s.g[0], s.args)
        return energy, gradient
    if s.call in ("batch", "uneven"):
        energies, gradients, _ = api.fg_phi4_batch(s.R, s.K, s.rho, s.g, s.settings, tolerances=s.tolerances)
        return energies, np.concatenate([x.ravel() for x in gradients])
    if s.call == "stationary":
        return api.stationary_state(s.Q[0], s.R[0])[0]
    for event in optimizer.optimize(s.R[0], s.K[0], s.rho[0], s.energy, s.gradient, s.callable, s.controls):
        pass
    end = event["state"]
    return end["energy"], end["gradient"], end["R"], end["K"]


# ----------------------------------------------------------------------------- work
def _evaluation_flops(d, z2, nodes, channels):
    """Real flops of one evaluation. Trajectory: 4 complex D^3 products per channel in each of about
    2000 D^(1/4) right-hand sides; pullback: 9 products per Gauss node; kinetic: 4 products per node
    for each of two operators. A Z2-symmetric state needs a quarter of the dense products."""
    products = 4 * channels * 2000 * d ** 0.25 + 9 * 2 * nodes + 8 * nodes
    return 8 * d ** 3 * products * (0.25 if z2 else 1.0)


def work(case):
    d, n, call = case["d"], case.get("n", 1), case["call"]
    nodes = REFINED["nodes"] if call == "refined" else DEFAULTS["nodes"]
    if call == "stationary":   # a few tens of applications of L, 6 products each
        return dict(bytes=3 * 16 * d * d, flops=40 * 6 * 8 * d ** 3)
    one = _evaluation_flops(d, case["kind"] == "z2", nodes, 26 if call == "ode" else 7)
    if call == "batch":
        half = _evaluation_flops(d, True, nodes, 7)
        flops = n * one if case["kind"] == "random" else (n // 2) * one + (n - n // 2) * half
    elif call == "uneven":     # D^3 averaged over a logarithmic spread from 8 to d
        flops = one * (1 + (n - 1) / (3 * math.log(d / 8)))
    elif call == "lbfgs":
        flops = one * (case["iterations"] + 1)
    else:
        flops = one
    return dict(bytes=4 * 16 * d * d * n, flops=flops)


# ----------------------------------------------------------------------------- 64-bit values
def _source(t):
    """2 |t| J(t^2) = 2 sqrt(a) K_{1/4}(a^2) / (2^(9/4) sqrt(pi) Gamma(5/4)), a = |t|, with
    K_nu(x) = int_0^inf exp(-x cosh u) cosh(nu u) du by the trapezoidal rule."""
    a = np.abs(np.asarray(t, dtype=float))
    x = np.maximum(a * a, 1e-300)
    u = np.arange(0.0, 60.0, 0.04)
    out = np.empty_like(a)
    norm = 2.0 ** 2.25 * math.sqrt(math.pi) * math.gamma(1.25)
    for i in range(0, len(a), 512):
        xs = x[i:i + 512, None]
        with np.errstate(over="ignore", under="ignore"):
            f = np.exp(-xs * np.cosh(u)) * np.cosh(0.25 * u)
        out[i:i + 512] = 0.04 * (f.sum(axis=1) - 0.5 * f[:, 0])
    return np.where(a > 0, 2.0 * np.sqrt(a) * out / norm, 1.0 / math.sqrt(math.pi))


def _herm(x):
    return x.conj().transpose(-1, -2).resolve_conj()


def _superoperator(q, r):
    """Row-major matrix of L(X) = Q X + X Q^dag + R X R^dag."""
    q, r = q.resolve_conj().contiguous(), r.resolve_conj().contiguous()
    eye = torch.eye(len(q), dtype=q.dtype, device=q.device)
    return torch.kron(q, eye) + torch.kron(eye, q.conj().resolve_conj()) + torch.kron(r, r.conj().resolve_conj())


def _exact_quartic(q, r, rho, half_window, n_quad):
    """Value, covector and environment of the quartic term: the seven linear channel equations from
    one Gauss node to the next by extrapolated midpoint steps of order 16."""
    d, dev = len(q), q.device
    x, w = np.polynomial.legendre.leggauss(n_quad)
    half = math.sqrt(half_window) / 2
    points = np.concatenate([-((x + 1) * half)[::-1], (x + 1) * half])
    weights = np.concatenate([(w * half)[::-1], w * half])
    Q = torch.stack([q] * 3 + [_herm(q)] * 4)
    R = torch.stack([r] * 3 + [_herm(r)] * 4)
    QR, Qh, Rh = torch.cat([Q, R], dim=1), _herm(Q), _herm(R)
    fixed = torch.zeros((7, d, d), dtype=q.dtype, device=dev)
    fixed[0] = r @ rho + rho @ _herm(r)
    fixed[6] = 4 * (r + _herm(r))
    src = torch.tensor([0, 0, 1, 4, 5, 6, 6], device=dev)
    coef = torch.tensor([0.0, 2, 3, 1, 2, 3, 0], device=dev, dtype=torch.float64).view(7, 1, 1)
    trace = (r.conj() + r.transpose(0, 1)) * 4

    def rhs(jac, s, y):
        qp = QR @ y
        p = qp[:, d:]
        m = torch.baddbmm(qp[:, :d] + y @ Qh, p, Rh)
        ins = p[src]
        return torch.add(m * jac, torch.addcmul(fixed, ins + _herm(ins), coef), alpha=s)

    norm = float(2 * torch.linalg.matrix_norm(q, 2) + torch.linalg.matrix_norm(r, 2) ** 2)
    stops = np.unique(np.concatenate([points, [0.0, math.sqrt(half_window)]]))
    steps, t = [], -math.sqrt(half_window)
    for stop in stops:
        m = max(1, math.ceil((stop - t) * 2 * max(abs(t), abs(stop)) * norm / 1.2))
        steps += [(t + (stop - t) * i / m, (stop - t) / m, i == m - 1) for i in range(m)]
        t = stop
    seq = [2, 4, 6, 8, 10, 12, 14, 16]
    offsets = np.concatenate([np.arange(n + 1) / n for n in seq])
    times = np.array([a for a, _, _ in steps])[:, None] + np.array([h for _, h, _ in steps])[:, None] * offsets
    sources = _source(times.ravel()).reshape(times.shape)
    y = torch.zeros((7, d, d), dtype=q.dtype, device=dev)
    value = torch.zeros((), dtype=torch.float64, device=dev)
    kept = []
    for row, (_, h, last) in enumerate(steps):
        s, jac, at, table = sources[row], 2 * np.abs(times[row]), 0, []
        for n in seq:
            sub = h / n
            y0, y1 = y, y + sub * rhs(jac[at], s[at], y)
            v0 = torch.zeros_like(value)
            v1 = v0 + sub * s[at] * (trace * y0[2]).sum().real
            for i in range(1, n):
                y0, y1 = y1, y0 + (2 * sub) * rhs(jac[at + i], s[at + i], y1)
                v0, v1 = v1, v0 + (2 * sub * s[at + i]) * (trace * y0[2]).sum().real
            end = (y1 + y0 + sub * rhs(jac[at + n], s[at + n], y1)) / 2
            vend = (v1 + v0 + sub * s[at + n] * (trace * y1[2]).sum().real) / 2
            at += n + 1
            new = [(end, vend)]
            for j, (py, pv) in enumerate(table):
                k = (n / seq[len(table) - 1 - j]) ** 2 - 1
                new.append((new[j][0] + (new[j][0] - py) / k, new[j][1] + (new[j][1] - pv) / k))
            table = new
        y, value = table[-1][0], value + table[-1][1]
        if last:
            kept.append(y)
    at = {float(v): i for i, v in enumerate(stops)}
    samples = torch.stack([kept[at[float(p)]] for p in points])
    n = len(points)
    eye = torch.eye(d, dtype=q.dtype, device=dev)
    back = samples.flip(0)
    f = [rho.expand(n, d, d), samples[:, 0], samples[:, 1], samples[:, 2]]
    b = [back[:, 3], back[:, 4], back[:, 5], back[:, 6], eye.expand(n, d, d)]
    wi = torch.tensor(weights * 2 * np.abs(points), device=dev).view(n, 1, 1)
    ji = torch.tensor(weights * _source(points), device=dev).view(n, 1, 1)
    rh = _herm(r)
    m = sum((wi * (f[k] @ (rh @ b[k] - b[k] @ rh)) + ji * (k + 1) * (f[k] @ b[k + 1])).sum(0) for k in range(4))
    nn = sum((wi * ((b[k] @ r - r @ b[k]) @ f[k]) + ji * (k + 1) * (b[k + 1] @ f[k])).sum(0) for k in range(4))
    env = kept[-1][3]
    return value, (m + _herm(nn)) / 2, (env + _herm(env)) / 2


def _exact_kinetic(q, r, rho, nodes):
    """Value, covector and environment of both kinetic terms by dense solves at every node."""
    d, dev = len(q), q.device
    x, w = np.polynomial.legendre.leggauss(nodes)
    shifts, weights = np.cos(0.25 * math.pi * (x + 1)), 0.5 * w
    rh, qh = _herm(r), _herm(q)
    lq, la = _superoperator(q, r), _superoperator(qh, rh)
    eye = torch.eye(d * d, dtype=q.dtype, device=dev)
    ops = [r, q @ r - r @ q]
    fwd = torch.stack([(rho @ _herm(o)).reshape(-1) for o in ops], dim=1)
    adj = torch.stack([_herm(o).reshape(-1) for o in ops], dim=1)
    value = torch.zeros((), dtype=torch.float64, device=dev)
    acc = [[torch.zeros((d, d), dtype=q.dtype, device=dev) for _ in range(5)] for _ in ops]
    for c, wt in zip(shifts, weights):
        xs = torch.linalg.solve(eye - c * lq, fwd)
        as_ = torch.linalg.solve(eye - c * la, adj)
        for o, op in enumerate(ops):
            X, a = xs[:, o].reshape(d, d), _herm(as_[:, o].reshape(d, d))
            value = value + wt * (op * X.transpose(0, 1)).sum().real
            t = acc[o]
            t[0] += wt * c * (X @ (rh @ a - a @ rh))
            t[1] += wt * c * ((a @ r - r @ a) @ X)
            t[2] += wt * X
            t[3] += wt * (a @ rho)
            t[4] += wt * (_herm(op) @ a)
    cov, env = 0, 0
    for o, (m, nn, u, v, e) in enumerate(acc):
        if o == 0:
            m, nn = m + u, nn + v
        else:
            m = m + u @ q - q @ u - r @ u @ rh + u @ r @ rh
            nn = nn + qh @ v - v @ qh - r @ v @ rh + r @ rh @ v
        cov = cov + (m + _herm(nn)) / 2
        env = env + (e + _herm(e)) / 2
    return value, cov, env


def exact(case, seed):
    d, call = case["d"], case["call"]
    if call not in ("objective", "refined", "stationary") or d > (64 if call == "stationary" else 16):
        return None
    s = prepare(case, seed)
    q, r = (torch.from_numpy(x).cuda() for x in (s.Q[0], s.R[0]))
    eye = torch.eye(d, dtype=q.dtype, device=q.device)
    flat = eye.reshape(-1)
    if call == "stationary":
        a = -_superoperator(q, r) + torch.outer(flat, flat) / d
        rho = torch.linalg.solve(a, flat / d).reshape(d, d)
        rho = rho / torch.trace(rho)
        return (rho + _herm(rho)) / 2
    c = REFINED if call == "refined" else DEFAULTS
    rho = torch.from_numpy(s.rho[0]).cuda()
    v4, m4, e4 = _exact_quartic(q, r, rho, c["half_window"], c["n_quad"])
    vk, mk, ek = _exact_kinetic(q, r, rho, c["nodes"])
    g = s.g[0]
    cov, env = g * m4 + mk, g * e4 + ek
    b = env - torch.trace(rho @ env) * eye
    a = -_superoperator(_herm(q), _herm(r)) + torch.outer(flat, rho.transpose(0, 1).reshape(-1))
    h = torch.linalg.solve(a, b.reshape(-1)).reshape(d, d)
    rh = _herm(r)
    cov = cov + rho @ rh @ h - rho @ h @ rh
    grad = _herm(torch.linalg.solve(rho + 1e-3 * eye, cov))
    return float(g * v4 + vk), grad
