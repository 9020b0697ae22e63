"""Ring fold of the one-field passes (k_fold_lanes): the residual against its definition in
double precision, and the two-step ring synthesis against the one-step kernel, at rings
shorter and longer than the band limit, with lanes and components that fill a CTA in part.

Bound: sums of at most L / 4 aliases in the working precision (1e-13 double, 3e-6 single), and
for the inverse transforms FFTs of at most 1024 points beside them."""

import pytest
import torch

from gmaster_b200 import _lib, sht

pytestmark = pytest.mark.gpu

CASES = [(1, 1, 1), (1, 7, 3), (2, 5, 2), (4, 12, 1), (16, 48, 5), (32, 20, 2), (128, 384, 1), (256, 701, 9)]


def _operands(nside, L, ncomp, prec):
    plan = sht.get_plan(nside, L - 1)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(nside + L)
    syn = torch.randn((L, plan.nlanes, ncomp, 4), generator=gen, dtype=torch.float64, device="cuda")
    return plan, syn.to(sht._real_dtype(prec)), 1e-13 if prec == _lib.FP64 else 3e-6


@pytest.mark.parametrize("prec", [_lib.FP64, _lib.MIXED])
@pytest.mark.parametrize("nside,L,ncomp", CASES)
def test_fold_residual_matches_definition(cuda, nside, L, ncomp, prec):
    plan, syn, tol = _operands(nside, L, ncomp, prec)
    rhs = torch.flip(syn, (0,)).contiguous()
    got = sht.fold_residual(plan, syn, rhs, prec).to(torch.float64)
    c = torch.view_as_complex(syn.to(torch.float64).unflatten(3, (2, 2)).contiguous())   # (L, lane, comp, N/S)
    sh = sht.shifted_flags(nside)
    want = torch.empty_like(got)
    for j in range(plan.nlanes):
        n = 4 * min(j + 1, nside)
        m = torch.arange(L, device="cuda")
        s = (1 - 2 * ((m // n) % 2)).to(torch.float64) if sh[j] else torch.ones(L, device="cuda", dtype=torch.float64)
        neg = (1 - 2 * (((m + n - 1) // n) % 2)).to(torch.float64) if sh[j] else s * 0 + 1   # order -m = r - t n
        P = torch.zeros((n,) + c[:, j].shape[1:], dtype=torch.complex128, device="cuda")
        P.index_add_(0, m % n, c[:, j] * s[:, None, None])
        P.index_add_(0, (-m[1:]) % n, c[1:, j].conj() * neg[1:, None, None])
        g = P[m % n] * s[:, None, None] * (4 * torch.pi / plan.npix * n)
        if j == plan.nlanes - 1:
            g[..., 1] = 0
        want[:, j] = torch.view_as_real(torch.stack([g[..., 0] + g[..., 1], g[..., 0] - g[..., 1]], 2)).flatten(2)
    want -= rhs.to(torch.float64)
    assert float((got - want).abs().max() / want.abs().max()) < tol


@pytest.mark.parametrize("prec", [_lib.FP64, _lib.MIXED])
@pytest.mark.parametrize("nside,L,ncomp", CASES)
def test_two_step_synthesis_matches_one_step(cuda, monkeypatch, nside, L, ncomp, prec):
    plan, syn, tol = _operands(nside, L, ncomp, prec)
    want = torch.empty((ncomp, plan.npix), dtype=torch.float64, device="cuda")
    _lib.call("gm_ring_synthesis", prec, nside, L, ncomp, _lib.ptr(syn), _lib.ptr(plan.tw), _lib.ptr(plan.shifted),
              _lib.ptr(want), _lib.stream_handle(plan.device))
    for limit in (1 << 30, 2 * int(_lib.load().gm_ring_fold_bytes(prec, nside))):   # at once, two at a time
        monkeypatch.setattr(sht, "RING_FOLD_BYTES", limit)
        got = sht.ring_synthesis(plan, syn, prec)
        assert float((got - want).abs().max() / want.abs().max()) < tol
