"""IP-Sat maps against a plain restatement, at the sizes where the kernels'
staging and scans end: nucleon counts around the four that are evaluated side
by side and the 256 that are staged at a time, rows around a warp and a block
(2048 rows are two blocks of rows), round and elliptic nucleons.

The restatement evaluates the same formulas cell by cell in numpy doubles:
every value is a chain of some 40 correctly rounded operations and a few
library functions of at most 2 ulp, so 1e-12 of the maximum for the thickness
(up to 300 terms) and 1e-11 relative for g^2 mu^2 (a contracting fixed point)."""
import math

import numpy as np
import pytest

import ipglasma_b200 as ipg

pytestmark = pytest.mark.gpu

HB = 0.1973269718
NY, NT, DY = 44, 200, 0.25
BG, RATIO, ROOTS, XF, G = 4.0, 0.8, 5020.0, 0.5, 2.0


def table():
    T = 1e-4 * (9.44 / 1e-4) ** (np.arange(NT) / (NT - 1))
    y = DY * np.arange(NY)
    return T, 2.2 * T[:, None] ** 0.92 * np.exp(0.28 * y[None, :])


def thickness(xyz, shift, phi, norm, N, L, xi):
    x = -L / 2 + L / N * np.arange(N)
    T = np.zeros((N, N))
    for (px, py, _), f, gn in zip(xyz, phi, norm):
        dx, dy = (px + shift) - x[:, None], py - x[None, :]
        b2 = dx * dx + dy * dy + xi * (dx * math.cos(f) + dy * math.sin(f)) ** 2
        T += math.sqrt(1 + xi) * np.exp(-b2 / HB ** 2 / (2 * BG)) / (2 * math.pi * BG) * gn
    return T


def qs2(T, y, tab):
    Ts, Q = tab
    k = min(max(int(math.floor(y / DY + 1e-7)), 0), NY - 2)
    fy = (y - k * DY) / DY
    if T < Ts[0]:
        return 0.0
    i = int(np.searchsorted(Ts, T, side="right")) - 1
    f = (T - Ts[i]) / (Ts[i + 1] - Ts[i])
    down, up = (f * Q[i + 1, j] + (1 - f) * Q[i, j] for j in (k, k + 1))
    return fy * up + (1 - fy) * down


def fixed_point(T, y, a, tab):
    g2, dev = 0.0, 1.0
    while abs(dev) > 0.001:
        assert y >= 0
        q = math.sqrt(qs2(T, y, tab))
        if q == 0:
            return 0.0, y
        g2 = q * q / RATIO / RATIO * a * a / HB / HB / G / G
        new = math.log(0.01 / (q * XF / ROOTS))
        dev, y = y - new, new
    return g2, y


@pytest.mark.parametrize("N,L,nA,nB,xi,rmax", [
    (8, 3.0, 1, 1, 0.0, 3.0), (32, 6.0, 4, 5, 0.0, 2.0), (64, 8.0, 3, 7, 0.4, 1.0),
    (128, 10.0, 257, 256, 0.0, 0.6), (1024, 12.0, 2, 1, 0.0, 0.25),
    (2048, 12.0, 1, 2, 0.3, 0.3)])
def test_maps_match_a_plain_restatement(N, L, nA, nB, xi, rmax):
    rng = np.random.default_rng(N + nA)
    A, B = rng.normal(0, 0.12 * L, (nA, 3)), rng.normal(0, 0.12 * L, (nB, 3))
    if nA + nB < 4:  # a few nucleons: on top of one another, near the last rows
        A[:], B[:] = [0.42 * L, 0.1, 0], [0.42 * L, 0.15, 0]
    phi = [rng.uniform(0, 6.28, n) for n in (nA, nB)]
    norm = [rng.uniform(0.7, 1.3, n) for n in (nA, nB)]
    tab, b = table(), 0.1
    with ipg.Event(ipg.Config(size=N, L=L, Ny=1, maxtime=0.1)) as ev:
        ev.set_nuclei_ipsat(A, B, b, tab, BG=BG, QsmuRatio=RATIO, proton_anisotropy=xi,
                            roots=ROOTS, x_factor=XF, rmax=rmax, phiA=phi[0], phiB=phi[1],
                            normA=norm[0], normB=norm[1])
        th, g2 = ev.thickness(), ev.g2mu()
    T = [thickness(p, s * b / 2, f, w, N, L, xi).ravel()
         for p, s, f, w in ((A, -1, phi[0], norm[0]), (B, 1, phi[1], norm[1]))]
    for k in range(2):
        assert np.abs(th[k] - T[k]).max() <= 1e-12 * T[k].max()
    with np.errstate(divide="ignore"):
        d = [np.sqrt(np.maximum(-2 * BG * np.log(2 * math.pi * BG * t), 0)) * HB for t in th]
    inside = np.flatnonzero((d[0] < rmax) & (d[1] < rmax))
    assert inside.size and (np.abs(d[0] - rmax) > 1e-9).all() and (np.abs(d[1] - rmax) > 1e-9).all()
    want, y = np.zeros((2, N * N)), 0.0
    for p in inside:  # A starts from the rapidity that B ended on at the cell before
        want[0, p], _ = fixed_point(th[0, p], y, L / N, tab)
        want[1, p], y = fixed_point(th[1, p], 0.0, L / N, tab)
    for k in range(2):
        assert np.array_equal(g2[k] > 0, want[k] > 0)
        m = want[k] > 0
        assert np.max(np.abs(g2[k][m] / want[k][m] - 1)) < 1e-11
