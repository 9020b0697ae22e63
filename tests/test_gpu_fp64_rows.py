"""Double-precision Legendre passes against sums in extended precision (numpy longdouble)."""

import math

import numpy as np
import pytest
import torch

from gmaster_b200 import _lib, sht

pytestmark = pytest.mark.gpu

LD = np.longdouble
PI = LD(np.pi) + LD(1.2246467991473532e-16)


def _rows(nside, lmax, m, s):
    """(F, G) = half the sum and difference of the rows s' = -s, +s (s = 0: the rows and zero),
    degrees max(m, s)..lmax by northern rings."""
    i = np.arange(1, 2 * nside + 1).astype(LD)
    n = LD(nside)
    xm1 = np.where(i < n, -i * i / (3 * n * n), (n - 2 * i) / (3 * n))
    x, half = 1 + xm1, (np.sqrt(1 + xm1 / 2), np.sqrt(-xm1 / 2))   # cos, sin of theta / 2
    l0, out = max(m, s), []
    for sp in (0,) if s == 0 else (-s, s):
        if m >= s:
            c, p = math.comb(2 * m, m + sp), (m + sp, m - sp)
            sign = -1 if (m - sp) & 1 else 1
        else:
            c, p = math.comb(2 * s, s + m), (s + m, s - m) if sp > 0 else (s - m, s + m)
            sign = 1 if sp > 0 else (-1) ** (m + s)
        v = np.zeros((lmax + 1 - l0, x.size), LD)
        v[0] = sign * np.sqrt(LD(2 * l0 + 1) / (4 * PI) * LD(c)) * half[0] ** p[0] * half[1] ** p[1]
        last = None
        for l in range(l0 + 1, lmax + 1):
            ll, mm = LD(l), LD(m)
            a = np.sqrt((2 * ll + 1) * (2 * ll - 1) / ((ll - mm) * (ll + mm) * (ll - s) * (ll + s))) * ll
            c0 = mm * sp / ((ll - 1) * ll) if s else LD(0)
            v[l - l0] = a * (x - c0) * v[l - 1 - l0] - (a / last * v[l - 2 - l0] if last else 0)
            last = a
        out.append(v)
    if s == 0:
        return out[0], np.zeros_like(out[0])
    return (out[0] + out[1]) / 2, (out[0] - out[1]) / 2


@pytest.mark.parametrize("nside,lmax,spin", [(64, 191, 0), (64, 191, 2), (32, 70, 0), (32, 70, 2)])
def test_fp64_passes_against_extended_precision(cuda, nside, lmax, spin):
    """Relative error of both passes below 1.5e-14: the seeds are powers of two of logarithms up
    to about 100 in size, rounded to 2^-53 of themselves (two terms), the steps unamplified."""
    r = np.random.default_rng(nside)
    plan = sht.get_plan(nside, lmax)
    nc, L = (1 if spin == 0 else 2), lmax + 1
    rhs = r.normal(size=(L, 2 * nside, nc, 4))
    alm = r.normal(size=(nc, plan.nelem)) + 1j * r.normal(size=(nc, plan.nelem))
    want_alm = np.zeros(alm.shape, np.clongdouble)
    want_syn = np.zeros(rhs.shape, LD)
    for m in range(L):
        l0 = max(m, spin)
        if l0 > lmax:
            continue
        F, G = _rows(nside, lmax, m, spin)
        ell = np.arange(l0, L)
        odd = (((ell + m) & 1) == 1)[:, None]
        g = rhs[m].astype(LD)
        h = [[g[:, c, 2 * p] + 1j * g[:, c, 2 * p + 1] for p in (0, 1)] for c in range(nc)]
        same = [np.where(odd, hc[1], hc[0]) for hc in h]
        other = [np.where(odd, hc[0], hc[1]) for hc in h]
        at = m * (2 * lmax + 1 - m) // 2 + ell
        a = [alm[c, at].astype(np.clongdouble)[:, None] for c in range(nc)]
        if spin == 0:
            want_alm[0, at] = (F * same[0]).sum(1)
            terms = [(F * a[0], 0 * F)]
        else:
            want_alm[0, at] = -(F * same[0] + 1j * G * other[1]).sum(1)
            want_alm[1, at] = -(F * same[1] - 1j * G * other[0]).sum(1)
            terms = [(-F * a[0], -1j * G * a[1]), (-F * a[1], 1j * G * a[0])]
        sign = np.where(odd, -1, 1)
        for c, (f, d) in enumerate(terms):
            north, south = (f + d).sum(0), (sign * (f - d)).sum(0)
            want_syn[m, :, c] = np.stack([north.real, north.imag, south.real, south.imag], -1)

    def rel(got, want):
        return float(np.sqrt((np.abs(got - want) ** 2).sum() / (np.abs(want) ** 2).sum()))

    got = torch.zeros((nc, plan.nelem), dtype=torch.complex128, device="cuda")
    sht.legendre_analysis(plan, spin, torch.from_numpy(rhs).cuda(), got, 1.0, _lib.FP64)
    assert rel(got.cpu().numpy(), want_alm) < 1.5e-14
    syn = sht.legendre_synthesis(plan, spin, torch.from_numpy(alm).cuda(), nc, _lib.FP64)
    assert rel(syn.cpu().numpy(), want_syn) < 1.5e-14
