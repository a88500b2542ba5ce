"""The work that is timed: scoring, model correlations, chains and the proposal network's
training step, each through the package's public calls.

``listed()`` gives the cases, ``draw(rng)`` one more of the same ranges, ``prepare`` makes
what a program has in hand before the call, ``run`` is one pass, ``work`` the bytes and
operations that a pass cannot do without and ``exact`` the outputs in 64 bits.

Inputs: a seeded molecule (C / N / O / S atoms in a ball) expanded to the SH coefficients
of its intensity on K shells; a target histogram, the molecule's own model c3 scaled to a
number of triplets and Poisson-sampled; proposals, each one annealing move away from the
molecule (a random plane rotation per even order, applied to every shell).
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "threephotons.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import tp3  # noqa: E402
from tp3 import learned  # noqa: E402
from tp3.chains import Chains  # noqa: E402

_MODES = {"auto": tp3.TP3_MODE_AUTO, "tf32": tp3.TP3_MODE_TC_TF32X3}
_LARGEST_FLOPS = 2.1e11  # about the work of the largest listed case


def listed():
    return [
        # one structure of the small configuration scored on its own, as an interactive
        # user or a sequential annealer does: launches and latency
        {"name": "energy_one_L8", "kind": "energy", "L": 8, "K": 8, "N": 16, "LMAX": 9, "n": 1, "mode": "auto"},
        # one structure at production size through the same call
        {"name": "energy_one_L18", "kind": "energy", "L": 18, "K": 26, "N": 32, "LMAX": 25, "n": 1, "mode": "auto"},
        # the 50 proposals of the initial temperature, host arrays in and energies out
        {"name": "energy_host_L12", "kind": "host", "L": 12, "K": 17, "N": 22, "LMAX": 13, "n": 50, "mode": "auto"},
        # the production batch, device resident
        {"name": "energy_batch_L18", "kind": "device", "L": 18, "K": 26, "N": 32, "LMAX": 25, "n": 64, "mode": "auto"},
        # a small ragged-sized batch of a mid-size basis: too few proposals to fill waves evenly
        {"name": "energy_batch_L14", "kind": "device", "L": 14, "K": 21, "N": 24, "LMAX": 16, "n": 7, "mode": "auto"},
        # the largest expansion
        {"name": "energy_batch_L24", "kind": "device", "L": 24, "K": 30, "N": 32, "LMAX": 25, "n": 32, "mode": "auto"},
        # the more exact split mode
        {"name": "energy_tf32_L18", "kind": "device", "L": 18, "K": 26, "N": 32, "LMAX": 25, "n": 32, "mode": "tf32"},
        # chains of mixed orders and shells, each against its own histogram, in one launch
        {"name": "ragged_L18", "kind": "ragged", "L": 18, "K": 26, "N": 32, "LMAX": 25, "n": 48, "hists": 6,
         "mode": "auto"},
        # a curved Ewald sphere (lambda != 0), as the reference's own GPU test runs
        {"name": "lambda_L18", "kind": "device", "L": 18, "K": 26, "N": 32, "LMAX": 25, "n": 12, "mode": "auto",
         "lambda": 2.5},
        # model correlations on the full grid, for making or inspecting histograms
        {"name": "c3_L18", "kind": "c3", "L": 18, "K": 26, "N": 32, "LMAX": 25, "n": 4, "mode": "auto"},
        # annealing chains with speculative candidates at a mid size: graph replays, then the
        # state a driver logs and checkpoints
        {"name": "chains_L12", "kind": "chains", "L": 12, "K": 16, "N": 16, "LMAX": 13, "n": 16, "ncand": 16,
         "launches": 8, "mode": "auto"},
        # one training step of the proposal network: loss and gradient of 128 logged candidates
        {"name": "mlp_grad_L18", "kind": "mlp", "L": 18, "K": 26, "n": 128, "hidden": 512},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["energy", "host", "device", "device", "device", "tf32", "ragged", "lambda", "c3", "chains", "mlp"])
    if kind == "mlp":
        n = rng.choice([32, 64, 128])  # training rows (candidates x shells) are a multiple of 128
        return {"kind": "mlp", "L": rng.choice([8, 12, 16, 18]), "K": rng.randint(2, 26 * n // 128) * 128 // n, "n": n,
                "hidden": rng.choice([128, 256, 384, 512])}
    c = {"kind": {"tf32": "device", "lambda": "device"}.get(kind, kind),
         "L": rng.choice([6, 8, 10, 12, 14, 16, 18, 20, 22, 24]), "K": rng.randint(5, 30),
         "N": 2 * rng.randint(6, 16), "mode": "tf32" if kind == "tf32" else "auto"}
    if kind in ("lambda", "chains", "ragged"):
        c["L"] = min(c["L"], 18)
        c["K"] = max(8, min(c["K"], 26))
    if kind == "ragged":
        c["L"] = max(c["L"], 12)
    c["LMAX"] = c["L"] + rng.randint(1, 4)
    if kind == "energy":
        c["n"] = 1
        return c
    if kind == "lambda":
        c["lambda"] = rng.choice([1.0, 2.5])
    if kind == "chains":
        c.update(ncand=rng.choice([4, 8, 16]), launches=rng.randint(2, 10))
    top = {"host": 96, "device": 96, "tf32": 64, "ragged": 64, "lambda": 16, "c3": 6, "chains": 24}[kind]
    c["n"] = _logint(rng, 2, top)
    while c["n"] > 2 and work(c)["flops"] > _LARGEST_FLOPS:
        c["n"] = c["n"] * 2 // 3
    if kind == "ragged":
        c["hists"] = rng.randint(2, min(8, c["n"]))
    while kind == "chains" and c["launches"] > 1 and work(c)["flops"] > _LARGEST_FLOPS:
        c["launches"] //= 2
    return c


# ---- the mathematics in 64 bits (numpy and torch) ---------------------------------------

def _sean(l, m, LMAX):
    """Index of (l, m) in a shell's LMAX^2 coefficients: m >= 0 column by column, then m < 0."""
    b = LMAX - 1
    if m >= 0:
        return m * (b + 1) - (m * (m - 1)) // 2 + (l - m)
    return (b * (b + 3)) // 2 + 1 + ((b + m) * (b + m + 1)) // 2 + (l - abs(m))


def _legendre(lmax, x):
    """Orthonormal associated Legendre values P[l, m] (0 <= m <= l <= lmax) at x, Condon-Shortley."""
    x = np.asarray(x, dtype=np.float64)
    P = np.zeros((lmax + 1, lmax + 1) + x.shape)
    s = np.sqrt(np.maximum(0.0, 1.0 - x * x))
    P[0, 0] = math.sqrt(1.0 / (4.0 * math.pi))
    for m in range(1, lmax + 1):
        P[m, m] = -math.sqrt((2 * m + 1) / (2.0 * m)) * s * P[m - 1, m - 1]
    for m in range(lmax):
        P[m + 1, m] = math.sqrt(2 * m + 3.0) * x * P[m, m]
        for l in range(m + 2, lmax + 1):
            a = math.sqrt((4.0 * l * l - 1.0) / (l * l - m * m))
            b = math.sqrt(((l - 1.0) ** 2 - m * m) / (4.0 * (l - 1.0) ** 2 - 1.0))
            P[l, m] = a * (x * P[l - 1, m] - b * P[l - 2, m])
    return P


def _signed(P, l):
    """Rows m = -l..l of order l."""
    return np.stack([P[l, abs(m)] * ((-1.0) ** abs(m) if m < 0 else 1.0) for m in range(-l, l + 1)])


def _w000(l1, l2, l3):
    J = l1 + l2 + l3
    g = J // 2
    f = math.factorial
    top = f(g) ** 2 * f(J - 2 * l1) * f(J - 2 * l2) * f(J - 2 * l3)
    low = f(J + 1) * (f(g - l1) * f(g - l2) * f(g - l3)) ** 2
    return (-1) ** g * math.sqrt(top / low)


@functools.lru_cache(maxsize=None)
def _w3j(L):
    """{(l1, l2, l3): w[m1, m3]}, the 3j symbols (l1 l2 l3; m1 -m1-m3 m3) of even orders up to L,
    from Gaunt integrals by quadrature divided by the (0 0 0) symbol."""
    x, wx = np.polynomial.legendre.leggauss(3 * L // 2 + 2)
    P = _legendre(L, x)
    S = {l: _signed(P, l) for l in range(0, L + 1, 2)}
    out = {}
    for l1 in range(0, L + 1, 2):
        for l2 in range(0, L + 1, 2):
            for l3 in range(abs(l1 - l2), min(l1 + l2, L) + 1, 2):
                m1, m3 = np.arange(-l1, l1 + 1)[:, None], np.arange(-l3, l3 + 1)[None, :]
                m2 = -m1 - m3
                ok = np.abs(m2) <= l2
                G = np.einsum("ax,abx,bx,x->ab", S[l1], S[l2][np.where(ok, m2 + l2, 0)], S[l3], wx, optimize=True)
                s = math.sqrt((2 * l1 + 1) * (2 * l2 + 1) * (2 * l3 + 1) / (4 * math.pi)) * _w000(l1, l2, l3)
                out[l1, l2, l3] = np.where(ok, 2 * math.pi * G / s, 0.0)
    return out


@functools.lru_cache(maxsize=None)
def _triples(K):
    return np.array([(a, b, c) for a in range(K) for b in range(a + 1) for c in range(b + 1)], dtype=np.int64)


def _angles(N):
    """alpha and beta of grid row g = a + N b."""
    a = (np.arange(N) + 0.5) * math.pi / N
    b = (np.arange(2 * N) + 0.5) * math.pi / N
    return np.tile(a, 2 * N), np.repeat(b, N)


def _c3(coeff, LMAX, L, K, N, lam=0.0, dq=0.0):
    """Model c3 of real-function coefficients [n, K, LMAX^2] (complex128, GPU): [n, klength, 2 N^2]."""
    dev, n = coeff.device, coeff.shape[0]
    W = _w3j(L)
    tri = torch.from_numpy(_triples(K)).to(dev)
    ki = (tri[:, 0] * K + tri[:, 1]) * K + tri[:, 2]
    al, be = (torch.from_numpy(v).to(dev) for v in _angles(N))
    c = {l: coeff[:, :, [_sean(l, m, LMAX) for m in range(-l, l + 1)]] for l in range(0, L + 1, 2)}
    theta = np.arccos(np.arange(1, K + 1) * lam * dq / (4 * math.pi))
    P = _legendre(L, np.cos(theta) if lam else np.zeros(K))
    Y = {l: torch.from_numpy(np.ascontiguousarray(_signed(P, l).T)).to(dev) for l in range(0, L + 1, 2)}  # [K, m]
    pairs, pid = [], {}
    for m2 in range(0, L + 1):
        for m3 in range(-L, L + 1):
            if m2 > 0 or m3 >= 0:
                pid[m2, m3] = len(pairs)
                pairs.append((m2, m3))
    H = torch.zeros((n, tri.shape[0], len(pairs)), dtype=torch.float64, device=dev) if lam else None
    T, Hw = [], []
    for (l1, l2, l3), w in W.items():
        wt = torch.from_numpy(w).to(dev)                                   # [m1, m3]
        m1, m3 = torch.arange(-l1, l1 + 1, device=dev), torch.arange(-l3, l3 + 1, device=dev)
        m2 = -m1[:, None] - m3[None, :]
        ok = m2.abs() <= l2
        c2 = c[l2][:, :, torch.where(ok, m2 + l2, 0)]                      # [n, K, m1, m3]
        A = (c[l1][:, None] * wt.T[None, :, None, :])                      # [n, m3, K, m1]
        D = A @ c2.permute(0, 3, 2, 1)                                     # [n, m3, k1, k2]
        D = D.reshape(n, 2 * l3 + 1, K * K).transpose(1, 2) @ c[l3].transpose(1, 2)
        t = D.real.reshape(n, K * K * K)[:, ki]                            # [n, klength]
        e = torch.nonzero(wt.abs() > 1e-13)
        e2, e3 = m2[e[:, 0], e[:, 1]], m3[e[:, 1]]
        neg = (e2 < 0) | ((e2 == 0) & (e3 < 0))
        q = torch.tensor([pid[k] for k in zip(torch.where(neg, -e2, e2).tolist(), torch.where(neg, -e3, e3).tolist())],
                         device=dev)
        if lam:
            f = (wt[e[:, 0], e[:, 1]][None] * Y[l1][tri[:, 0]][:, e[:, 0]] * Y[l2][tri[:, 1]][:, e2 + l2]
                 * Y[l3][tri[:, 2]][:, e[:, 1]])                           # [klength, entries]
            g = torch.zeros((tri.shape[0], len(pairs)), dtype=torch.float64, device=dev).index_add_(1, q, f)
            H += t[:, :, None] * g[None]
        else:
            f = wt[e[:, 0], e[:, 1]] * Y[l1][0][e[:, 0]] * Y[l2][0][e2 + l2] * Y[l3][0][e[:, 1]]
            Hw.append(torch.zeros(len(pairs), dtype=torch.float64, device=dev).index_add_(0, q, f))
            T.append(t)
    if not lam:
        H = torch.stack(T, dim=2) @ torch.stack(Hw)
    pq = torch.tensor(pairs, dtype=torch.float64, device=dev)
    return H @ torch.cos(pq[:, :1] * al[None] + pq[:, 1:] * be[None])


def _factors(K):
    t = _triples(K)
    same = (t[:, 0] == t[:, 1]).astype(int) + (t[:, 1] == t[:, 2])
    return np.where(same == 2, 1.0, np.where(same == 1, 3.0, 6.0))


def _energy(c3, q, K):
    """Bayes energies of c3 [n, klength, G] against histogram slabs q [klength, G] (FP64)."""
    p = torch.clamp(c3, min=1e-30)
    s = -((q / q.abs().sum(1, keepdim=True))[None] * torch.log(p / p.sum(2, keepdim=True))).sum(2)
    return s @ torch.from_numpy(_factors(K)).to(c3.device)


# ---- inputs -----------------------------------------------------------------------------

def _molecule(g, LMAX, K, dev):
    """Intensity coefficients [K, LMAX^2] of a seeded molecule of 200 to 400 atoms, shells at
    q_k = k pi / 38."""
    atoms = int(torch.randint(200, 401, (1,), generator=g))
    v = torch.randn((atoms, 3), generator=g, dtype=torch.float64)
    pos = 13.0 * torch.rand((atoms, 1), generator=g, dtype=torch.float64) ** (1 / 3) * v / v.norm(dim=1, keepdim=True)
    kind = torch.multinomial(torch.tensor([0.60, 0.20, 0.18, 0.02]), atoms, replacement=True, generator=g)
    R = torch.tensor([0.7, 0.65, 0.6, 1.0], dtype=torch.float64)[kind].to(dev)
    B = torch.tensor([6.0, 7.0, 8.0, 16.0], dtype=torch.float64)[kind].to(dev)
    nt, nphi = 2 * LMAX, 4 * LMAX
    x, wx = np.polynomial.legendre.leggauss(nt)
    phi = (np.arange(nphi) + 0.5) * (2 * math.pi / nphi)
    st = np.sqrt(1 - x * x)
    dirs = np.stack([np.outer(st, np.cos(phi)), np.outer(st, np.sin(phi)), np.outer(x, np.ones(nphi))], -1).reshape(-1, 3)
    proj = torch.from_numpy(dirs).to(dev) @ pos.to(dev).T                   # [points, atoms]
    P = _legendre(LMAX - 1, x)
    out = torch.zeros((K, LMAX * LMAX), dtype=torch.complex128, device=dev)
    E = torch.from_numpy(np.exp(-1j * np.outer(phi, np.arange(LMAX)))).to(dev) * (2 * math.pi / nphi)
    Pw = torch.from_numpy(P * wx).to(dev)                                   # [l, m, theta]
    for k in range(1, K + 1):
        q = k * math.pi / 38.0
        f = B * torch.exp(-0.5 * R * R * q * q)
        I = (torch.cos(q * proj) @ f) ** 2 + (torch.sin(q * proj) @ f) ** 2
        Im = I.reshape(nt, nphi).to(torch.complex128) @ E                   # [theta, m]
        cl = torch.einsum("lmt,tm->lm", Pw.to(torch.complex128), Im)
        for l in range(LMAX):
            m = torch.arange(l + 1, device=dev)
            out[k - 1, [_sean(l, int(i), LMAX) for i in range(l + 1)]] = cl[l, : l + 1]
            out[k - 1, [_sean(l, -int(i), LMAX) for i in range(l + 1)]] = (
                torch.conj(cl[l, : l + 1]) * (1 - 2 * (m % 2)).to(torch.float64))
    for l in range(LMAX):
        out[:, _sean(l, 0, LMAX)] = out[:, _sean(l, 0, LMAX)].real.to(torch.complex128)
    return out


def _proposals(base, n, L, LMAX, g):
    """n annealing moves of base [K, LMAX^2]: per even order a rotation by N(0, sigma_l) in a
    random plane of its 2l+1 real coefficients, sigma_l = (pi / 4)(l - 1), on every shell."""
    dev = base.device
    out = base[None].repeat(n, 1, 1)
    for l in range(2, L + 1, 2):
        ip = [_sean(l, m, LMAX) for m in range(0, l + 1)]
        im = [_sean(l, -m, LMAX) for m in range(1, l + 1)]
        c = base[:, ip]
        x = torch.cat([c[:, :1].real, math.sqrt(2) * c[:, 1:].real, math.sqrt(2) * c[:, 1:].imag], dim=1)
        p, q = (torch.randn((n, 2 * l + 1), generator=g, dtype=torch.float64) for _ in range(2))
        beta = (torch.randn((n, 1), generator=g, dtype=torch.float64) * (math.pi / 4) * (l - 1)).to(dev)
        p = p / p.norm(dim=1, keepdim=True)
        q = q - (p * q).sum(1, keepdim=True) * p
        p, q = p.to(dev), (q / q.norm(dim=1, keepdim=True)).to(dev)
        xp, xq = p @ x.T, q @ x.T                                           # [n, K]
        cm, s = torch.cos(beta) - 1, torch.sin(beta)
        y = x[None] + (cm * xp - s * xq)[:, :, None] * p[:, None] + (cm * xq + s * xp)[:, :, None] * q[:, None]
        z = torch.complex(y[..., 1 : l + 1], y[..., l + 1 :]) / math.sqrt(2)
        out[:, :, ip[0]] = y[..., 0].to(torch.complex128)
        out[:, :, ip[1:]] = z
        sg = torch.tensor([(-1.0) ** m for m in range(1, l + 1)], dtype=torch.float64, device=dev)
        out[:, :, im] = torch.conj(z) * sg
    return out


_DQ = math.pi / 38.0  # shell spacing of the lambda != 0 cases


def _shape(case):
    return (case["L"], case["K"], case["N"], case["LMAX"], float(case.get("lambda", 0.0)), case.get("hists", 1))


@functools.lru_cache(maxsize=None)
def _problem(L, K, N, LMAX, lam, nh):
    """What a program is given once: per histogram the molecule [K, LMAX^2] (GPU), its (L, K)
    and its measured counts [klength, G]."""
    g = torch.Generator().manual_seed(17)
    out = []
    for h in range(nh):
        Lh, Kh = L, K
        if h > 0:
            Kh = int(torch.randint(max(4, K * 3 // 5), K + 1, (1,), generator=g))
            Lh = L - 2 * int(torch.randint(0, 4, (1,), generator=g))
        base = _molecule(g, LMAX, K, torch.device("cuda"))
        c3 = torch.clamp(_c3(base[None, :Kh], LMAX, Lh, Kh, N, lam, _DQ)[0], min=0.0)
        rate = (c3 * ((1e9 if K >= 16 else 1e8) / c3.sum())).cpu().numpy()
        q = np.random.default_rng([h, 5]).poisson(rate).astype(np.float64)
        out.append((base, Lh, Kh, torch.from_numpy(np.maximum(q, 1e-30))))
    return out


def _inputs(case, seed):
    """The case's n proposals [n, K, LMAX^2] (GPU) and the histogram index of each."""
    g = torch.Generator().manual_seed(1_000_003 * int(seed) + 17)
    prob = _problem(*_shape(case))
    per = [case["n"] // len(prob) + (h < case["n"] % len(prob)) for h in range(len(prob))]
    c = [_proposals(base, m, case["L"], case["LMAX"], g) for (base, _, _, _), m in zip(prob, per)]
    return torch.cat(c), [h for h, m in enumerate(per) for _ in range(m)]


def _five_d(q, K, N):
    """Histogram slabs [klength, G] as the N x 2N x K x K x K array of the API."""
    t = _triples(K)
    full = np.zeros((K, K, K, 2 * N * N))
    full[t[:, 0], t[:, 1], t[:, 2]] = q.numpy()
    return full.reshape(K, K, K, 2 * N, N).transpose(4, 3, 2, 1, 0)


@functools.lru_cache(maxsize=None)
def _basis(L, K, N, LMAX, lam, nh):
    """The basis with its histogram, or histograms: a program keeps it for all that it scores."""
    b = tp3.calculate_basis(L, LMAX, N, K, lam, _DQ if lam else 0.0)
    prob = _problem(L, K, N, LMAX, lam, nh)
    hist = [_five_d(q, Kh, N) for _, _, Kh, q in prob]
    if nh > 1:
        b.set_histograms(hist, [Kh for _, _, Kh, _ in prob])
    else:
        b.set_histogram(hist[0])
    return b, hist[0]


@functools.lru_cache(maxsize=None)
def _small_basis():
    return tp3.calculate_basis(8, 9, 16, 8)


def _mlp_inputs(case, seed):
    """Feature rows (BF16), logged steps, weights and targets of n candidates of K shells, and
    the network's parameters ((out, in) weights and biases layer by layer, one vector)."""
    dev = torch.device("cuda")
    g = torch.Generator().manual_seed(7_000_003 * int(seed) + 3)
    n_in, H = learned.n_in_for(case["L"]), case["hidden"]
    rows, nc = case["n"] * case["K"], (case["L"] + 1) ** 2
    x = torch.zeros((rows, learned.n_in_pad(n_in)))
    v = torch.randn((rows, nc), generator=g)
    x[:, :nc] = 8.0 * v / v.norm(dim=1, keepdim=True)
    x[:, nc:n_in] = torch.randn((rows, n_in - nc), generator=g)
    steps = torch.randn((rows, 3), generator=g)
    w = torch.rand(rows, generator=g)
    t = torch.randn((case["n"], 2), generator=g)
    t[:, 1] = 1.0 / case["n"]
    par = []
    for a, b, scale in ((n_in, H, 1.0), (H, H, 1.0), (H, H, 1.0), (H, 6, 0.05)):
        par.append(((2 * torch.rand(b * a, generator=g) - 1) * scale * math.sqrt(6.0 / a)))
        par.append((2 * torch.rand(b, generator=g) - 1) * 0.1)
    return x.to(torch.bfloat16).to(dev), steps.to(dev), w.to(dev), t.to(dev), torch.cat(par)


def _mlp_exact(case, seed):
    """Loss and gradient in 64 bits: three ReLU layers, drift u = o[0:3] and log-scale
    s = -3 + 4 tanh(o[3:6]); regression of the targets on the steps through u plus the
    weighted Gaussian NLL of the steps under s."""
    x, v, w, t, par = _mlp_inputs(case, seed)
    n_in, H = learned.n_in_for(case["L"]), case["hidden"]
    p = par.to(x.device).double().requires_grad_(True)
    a, at = x[:, :n_in].double(), 0
    for i, (fi, fo) in enumerate(((n_in, H), (H, H), (H, H), (H, 6))):
        a = a @ p[at : at + fi * fo].reshape(fo, fi).T + p[at + fi * fo : at + fi * fo + fo]
        a = torch.relu(a) if i < 3 else a
        at += fi * fo + fo
    u, s, v, w, t = a[:, :3], -3.0 + 4.0 * torch.tanh(a[:, 3:]), v.double(), w.double(), t.double()
    nll = (w[:, None] * (s + 0.5 * v * v * torch.exp(-2 * s) + 0.5 * math.log(2 * math.pi))).sum()
    r = t[:, 0] - (u * v).reshape(case["n"], -1).sum(1)
    loss = nll + (0.5 * t[:, 1] * r * r).sum()
    loss.backward()
    return [float(loss.detach()), p.grad]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        x, v, w, t, par = _mlp_inputs(case, seed)
        net = learned.ProposalMLP(_small_basis(), learned.n_in_for(case["L"]), hidden=case["hidden"], max_rows=x.shape[0])
        net.set_params(par.numpy())
        torch.cuda.synchronize()
        return {"case": case, "net": net, "x": x, "v": v, "w": w, "t": t}
    b, hist = _basis(*_shape(case))
    b.set_mode(_MODES[case["mode"]])
    c, which = _inputs(case, seed)
    s = {"case": case, "basis": b}
    if kind == "energy":
        s["volume"] = tp3.SphericalHarmonicsVolume(c[0].cpu().numpy(), case["LMAX"], case["K"], 38.0)
        s["hist"] = hist
    elif kind == "host":
        s["host"] = c.cpu().numpy()
    elif kind == "chains":
        # a hot start, as annealing begins: most moves are accepted
        s["chains"] = Chains(b, c.cpu().numpy(), 50.0, math.pi / 4, 1.02, 0.9999, 11 + int(seed), ncand=case["ncand"])
    else:
        s["c"] = torch.view_as_real(c).contiguous()
        s["E"] = torch.empty(case["n"], dtype=torch.float64, device="cuda")
    if kind == "c3":
        s["c3"] = torch.empty((case["n"], b.klength, 2 * b.N ** 2), dtype=torch.float32, device="cuda")
    if kind == "ragged":
        prob = _problem(*_shape(case))
        s["lkh"] = torch.tensor([(prob[h][1], prob[h][2], h) for h in which], dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return s


def run(state):
    case, b = state["case"], state.get("basis")
    kind, n = case["kind"], case["n"]
    if kind == "energy":
        return tp3.energy(state["volume"], b, state["hist"])
    if kind == "host":
        return b.energy_batch(state["host"])
    if kind == "device":
        b.energy_batch_device(n, state["c"].data_ptr(), state["E"].data_ptr())
        return state["E"]
    if kind == "ragged":
        b.energy_batch_ragged_device(n, state["c"].data_ptr(), state["lkh"].data_ptr(), state["E"].data_ptr())
        return state["E"]
    if kind == "c3":
        b.c3_batch_device(n, state["c"].data_ptr(), state["c3"].data_ptr())
        return state["c3"]
    if kind == "chains":
        state["chains"].run(case["launches"])
        return {**state["chains"].state(), "coeff": state["chains"].coeff()}
    rows = state["x"].shape[0]
    loss, grad = state["net"].loss_grad(rows, state["x"].data_ptr(), state["v"].data_ptr(), state["w"].data_ptr(),
                                        state["t"].data_ptr(), case["K"])
    return [loss, grad]


def exact(case, seed):
    if case["kind"] == "chains":
        return None  # decisions along a trajectory
    if case["kind"] == "mlp":
        return _mlp_exact(case, seed)
    c, which = _inputs(case, seed)
    L, N, LMAX, lam = case["L"], case["N"], case["LMAX"], float(case.get("lambda", 0.0))
    if case["kind"] == "c3":
        return _c3(c, LMAX, L, case["K"], N)
    E = torch.empty(len(which), dtype=torch.float64, device=c.device)
    for h, (_, Lh, Kh, q) in enumerate(_problem(*_shape(case))):
        q = q.to(c.device)
        for i in torch.tensor([p for p, hp in enumerate(which) if hp == h]).split(4):
            E[i] = _energy(_c3(c[i][:, :Kh], LMAX, Lh, Kh, N, lam, _DQ), q, Kh)
    return float(E[0]) if case["kind"] == "energy" else E


@functools.lru_cache(maxsize=None)
def _counts(L):
    """(shell products, their order sums, third-shell products) per shell pair / triple, l-triples
    and Fourier pairs, of a real function's orders 0, 2, .., L."""
    prod = sums = third = nlt = 0
    for l1 in range(0, L + 1, 2):
        for l2 in range(0, L + 1, 2):
            lo, hi = abs(l1 - l2), min(l1 + l2, L)
            for m3 in range(0, hi + 1):
                m1 = max(0, min(l1, l2 - m3) - max(-l1, -l2 - m3) + 1)
                prod += m1
                sums += m1 * len([l for l in range(lo, hi + 1, 2) if l >= m3])
            for l3 in range(lo, hi + 1, 2):
                third += l3 + 1
                nlt += 1
    return prod, sums, third, nlt


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "mlp":
        rows, H, a = n * case["K"], case["hidden"], learned.n_in_pad(learned.n_in_for(case["L"]))
        params = a * H + 2 * H * H + 6 * H + 3 * H + 6
        return {"bytes": rows * (2 * a + 16) + params * 6, "flops": 6.0 * rows * (a * H + 2 * H * H + 6 * H) - 2.0 * rows * a * H}
    L, K, N = case["L"], case["K"], case["N"]
    prod, sums, third, nlt = _counts(L)
    klen, npair, G = K * (K + 1) * (K + 2) // 6, K * (K + 1) // 2, 2 * N * N
    coef = K * (L + 1) * (L + 2) // 2 * 16
    couple = npair * (8.0 * prod + 4.0 * sums) + klen * 4.0 * third
    if case.get("lambda"):
        pairs = L * (L + 1) + L + 1
        entries = sum(w.size for w in _w3j(L).values()) if L <= 18 else 0
        angular = klen * (2.0 * entries + 2.0 * pairs * G)
    else:
        angular = klen * 2.0 * nlt * G / 4
    if kind == "chains":
        n = n * case["ncand"] * case["launches"]  # proposals
    bayes = 0.0 if kind == "c3" else 4.0 * klen * G / 4
    byts = n * coef + (n * klen * G * 4.0 if kind == "c3" else klen * G + 8 * n)
    return {"bytes": byts, "flops": n * (couple + angular + bayes)}
