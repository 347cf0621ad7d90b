"""Sums of many chunks are rounded after each addition as a loop of double additions
rounds, but formed 32 terms at a time in integers (loop.cu, sum_in_order): its steps,
restated, against the loop, and a large subhalo's energy on the GPU."""
import struct

import numpy as np
import pytest

HIDDEN = 1 << 52


def _bits(d):
    return struct.unpack("<q", struct.pack("<d", d))[0]


def _double(b):
    return struct.unpack("<d", struct.pack("<Q", b & (1 << 64) - 1))[0]


def sum_in_order(x):
    t, fast = 0.0, 0
    for g in range(0, len(x), 32):
        v = list(x[g:g + 32]) + [0.0] * (32 - len(x[g:g + 32]))
        tb = _bits(t)
        te = tb >> 52 & 0x7FF
        s = tb & HIDDEN - 1 | HIDDEN
        s = -s if tb < 0 else s
        ok = 64 < te < 2046
        q, up, tie = [], [], []
        for a in v:
            b = _bits(a)
            e = b >> 52 & 0x7FF
            m = b & HIDDEN - 1 | (HIDDEN if e else 0)
            m = -m if b < 0 else m
            d = te - max(e, 1)
            ok = ok and d >= 0
            sh = min(max(d, 0), 62)
            frac2 = (m & (1 << sh) - 1) << 1
            q.append(m >> sh)
            tie.append(frac2 == 1 << sh)
            up.append(int(frac2 > 1 << sh))
        odd = [not tie[i] and (q[i] + up[i]) & 1 for i in range(32)]
        for i in range(32):
            if tie[i]:
                prev = [j for j in range(i) if tie[j]]
                first = prev[-1] + 1 if prev else 0
                parity = sum(odd[first:i]) + (0 if prev else s & 1)
                up[i] = (parity + (q[i] & 1)) & 1
        pre = np.cumsum([q[i] + up[i] for i in range(32)], dtype=object)
        for i in range(32):
            at = s + pre[i] - up[i]
            ok = ok and (at if at >= 0 else -at - 1) >> 52 == 1
        if ok:
            s += pre[31]
            t = _double((te << 52) + (abs(s) - HIDDEN) | (1 << 63 if s < 0 else 0))
            fast += 1
        else:
            for a in x[g:g + 32]:
                t = t + a
    return t, fast


def _terms(kind, n, rng):
    if kind == "masses":
        return [1024 * float(np.float32(1e-4))] * n
    if kind == "positive":
        return [float(a) for a in rng.uniform(0.5, 2, n)]
    if kind == "signed":
        return [float(a) for a in rng.normal(0, 1, n)]
    if kind == "wide":
        return [float(a) for a in rng.normal(0, 1, n) * 10.0 ** rng.uniform(-25, 3, n)]
    if kind == "ties":  # halves and odd multiples of the sum's last place
        return [2.0 ** 52] + [float(a) / 2 for a in rng.integers(-9, 10, n - 1)]
    if kind == "borders":  # about the powers of two
        return [2.0 ** 20] + [float(a) * 2.0 ** -33 for a in rng.integers(-3, 4, n - 1)]
    x = [float(a) for a in rng.normal(5, 1, n)]
    x[n // 2] = {"inf": float("inf"), "nan": float("nan"), "zero": -0.0, "tiny": 5e-324}[kind]
    return x


@pytest.mark.parametrize("kind", ["masses", "positive", "signed", "wide", "ties", "borders", "inf",
                                  "nan", "zero", "tiny"])
def test_equals_the_loop(kind):
    rng = np.random.default_rng(20261205)
    fast = 0
    for n in (1, 31, 32, 33, 64, 200, 1999):
        for _ in range(4):
            x = _terms(kind, n, rng)
            t = 0.0
            for a in x:
                t = t + a
            s, f = sum_in_order(x)
            assert struct.pack("<d", s) == struct.pack("<d", t) or (t != t and s != s)
            fast += f
    assert fast > 0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [64_512, 64_513, 65_537, 200_001])
def test_energy_of_a_large_subhalo(n):
    """E_tot = sum m (E_i - phi_i / 2), about the line of 64 chunks; each E_i is
    rounded to float, so the sums agree to 2^-23 of their terms' sizes."""
    torch = pytest.importorskip("torch")
    from hbtplus_gb300 import synthetic as S
    from hbtplus_gb300.adjoint import energy_gradient
    from hbtplus_gb300.unbind import Unbinder
    sub = S.single_subhalo(n=n, seed=n, contaminant_frac=0.0)
    p = S.default_params()
    with Unbinder(p) as ub:
        E, pot = ub.binding_energies(sub["pos"], sub["vel"], sub["mass"], sub["ref_pos"],
                                     sub["ref_vel"])
        t = {k: torch.as_tensor(sub[k]).cuda() for k in ("pos", "vel", "mass")}
        E_tot = energy_gradient(ub, t["pos"], t["vel"], t["mass"], [0, n], sub["ref_pos"],
                                sub["ref_vel"], with_grad=False)[0].item()
    m = sub["mass"].astype(np.float64)
    want = np.sum(m * (E - pot / 2))
    bound = 2.0 ** -23 * np.sum(m * (np.abs(E) + np.abs(pot)))
    assert abs(E_tot - want) <= bound
