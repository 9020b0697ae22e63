"""Entries that take arrays aligned to their elements only: the same results as from 16-byte aligned
arrays."""

import pytest
import torch

from gmaster_b200 import _lib, sht, sht_tc

pytestmark = pytest.mark.gpu


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _offset(t, by=1):
    """A copy of t that starts `by` real elements after a 16-byte boundary."""
    flat = torch.view_as_real(t).reshape(-1) if t.is_complex() else t.reshape(-1)
    buf = torch.empty(flat.numel() + max(4, by), dtype=flat.dtype, device=t.device)
    out = buf[by:by + flat.numel()]
    out.copy_(flat)
    assert out.data_ptr() % 16 != 0
    return out


@pytest.mark.parametrize("nside,lmax,ncomp", [(8, 20, 1), (64, 191, 2), (64, 130, 20)])
@pytest.mark.parametrize("prec", [_lib.MIXED, _lib.FP64])
def test_fold_residual(cuda, nside, lmax, ncomp, prec):
    plan = sht.get_plan(nside, lmax)
    real = torch.float64 if prec == _lib.FP64 else torch.float32
    shape = (plan.L, plan.nlanes, ncomp, 4)
    syn, rhs = (torch.randn(shape, generator=_gen(i), dtype=real, device="cuda") for i in (1, 2))
    want = sht.fold_residual(plan, syn, rhs, prec)
    for which in range(3):
        args = [_offset(x) if i == which else x.clone() for i, x in enumerate((syn, rhs, torch.zeros_like(syn)))]
        _lib.call("gm_fold_residual", prec, nside, plan.L, ncomp, _lib.ptr(args[0]), _lib.ptr(args[1]),
                  _lib.ptr(plan.shifted), _lib.ptr(args[2]), _lib.stream_handle(plan.device))
        assert torch.equal(args[2].reshape(shape), want)


@pytest.mark.parametrize("spin,ncomp,tables,prec", [(0, 1, True, _lib.MIXED), (0, 5, True, _lib.MIXED),
                                                    (2, 2, True, _lib.MIXED), (2, 4, False, _lib.MIXED),
                                                    (0, 3, False, _lib.FP64), (3, 2, False, _lib.FP64)])
def test_legendre_passes_and_refinement(cuda, spin, ncomp, tables, prec):
    """Unaligned rhs, syn and alm, in the passes and in the Jacobi steps (to the last bits: the alms
    are sums of a few CTAs in any order)."""
    nside, lmax = 32, 90
    plan = sht.get_plan(nside, lmax)
    real = torch.float64 if prec == _lib.FP64 else torch.float32
    tol = 1e-12 if prec == _lib.FP64 else 1e-6
    ck = sht.ck_args(plan, spin, prec) if tables else None
    shape = (plan.L, plan.nlanes, ncomp, 4)
    rhs = torch.randn(shape, generator=_gen(3), dtype=real, device="cuda")
    alm = torch.randn((ncomp, plan.nelem), generator=_gen(4), dtype=torch.complex128, device="cuda")
    close = lambda a, b: float((a - b).norm()) <= tol * float(b.norm())   # noqa: E731
    want = torch.zeros_like(alm)
    sht.run_legendre(plan, spin, ncomp, prec, "ana", -1, rhs, want, ck=ck)
    got = _offset(torch.zeros_like(alm))
    sht.run_legendre(plan, spin, ncomp, prec, "ana", -1, _offset(rhs), got, ck=ck)
    assert close(torch.view_as_complex(got.clone().reshape(ncomp, plan.nelem, 2)), want)
    syn = torch.empty(shape, dtype=real, device="cuda")
    sht.run_legendre(plan, spin, ncomp, prec, "syn", -1, alm, syn, ck=ck)
    out = _offset(torch.zeros_like(syn))
    sht.run_legendre(plan, spin, ncomp, prec, "syn", -1, _offset(alm), out, ck=ck)
    assert torch.equal(out.reshape(shape), syn)

    def refine(make):
        bufs = [make(x) for x in (rhs, torch.zeros_like(rhs), torch.zeros_like(rhs), alm)]
        _lib.call("gm_refine", prec, spin, nside, lmax, ncomp, 2, _lib.ptr(plan.geom), _lib.ptr(plan.seeds),
                  _lib.ptr(bufs[0]), _lib.ptr(plan.shifted), _lib.ptr(bufs[1]), _lib.ptr(bufs[2]), _lib.ptr(bufs[3]),
                  -1, -1, *(ck if ck is not None else (None,) * 7), _lib.stream_handle(plan.device))
        return bufs[3].clone().reshape(-1)

    assert close(refine(_offset), torch.view_as_real(refine(lambda x: x.clone())).reshape(-1))


@pytest.mark.parametrize("spin,ncomp", [(0, 3), (2, 6)])
def test_batched_fold(cuda, spin, ncomp):
    """The batched fold from synthesis arrays at a 4-byte boundary; images off a 16-byte boundary are
    refused."""
    nside, lmax = 16, 47
    tp = sht_tc.get_tc_plan(nside, lmax)
    p = tp.plan
    H, nv = (2 * ncomp, 1) if spin == 0 else (ncomp, 2)
    synd = [torch.randn((p.L, p.nlanes, 2 * H), generator=_gen(i), device="cuda") for i in range(nv)]
    rhs = torch.randn((p.L, p.nlanes, ncomp, 4), generator=_gen(5), device="cuda")
    out = []
    for make in (torch.clone, _offset):
        s = [make(x) for x in synd]
        img = [torch.zeros(tp.img_bytes, dtype=torch.uint8, device="cuda") for _ in synd]
        _lib.call("gm_tc_fold", nside, lmax, spin, ncomp, _lib.ptr(s[0]), _lib.ptr(s[-1]) if spin else None,
                  _lib.ptr(rhs), _lib.ptr(p.shifted), _lib.ptr(img[0]), _lib.ptr(img[-1]) if spin else None, 64.0,
                  _lib.stream_handle(p.device))
        out.append(torch.cat(img))
    assert torch.equal(*out)
    off = torch.zeros(tp.img_bytes + 16, dtype=torch.uint8, device="cuda")[2:]
    with pytest.raises(_lib.GMError):
        _lib.call("gm_tc_fold", nside, lmax, spin, ncomp, _lib.ptr(synd[0]), _lib.ptr(synd[-1]) if spin else None,
                  _lib.ptr(rhs), _lib.ptr(p.shifted), _lib.ptr(off), _lib.ptr(img[-1]) if spin else None, 64.0,
                  _lib.stream_handle(p.device))


def test_ring_synthesis_fold_refuses_what_it_cannot_read(cuda):
    plan = sht.get_plan(8, 23)
    syn = torch.randn((plan.L, plan.nlanes, 1, 4), generator=_gen(6), device="cuda")
    maps = torch.empty(plan.npix, dtype=torch.float64, device="cuda")
    work = torch.empty(int(_lib.load().gm_ring_fold_bytes(_lib.MIXED, 8)), dtype=torch.uint8, device="cuda")
    scratch, nbytes = sht._ring_scratch(plan, _lib.MIXED)

    def call(s, m, w):
        _lib.call("gm_ring_synthesis_fold", _lib.MIXED, 8, plan.L, 1, _lib.ptr(s), _lib.ptr(plan.tw), _lib.ptr(plan.shifted),
                  _lib.ptr(m), _lib.ptr(w), work.numel(), _lib.ptr(scratch), nbytes, 0, 0, _lib.stream_handle(plan.device))

    call(syn, maps, work)
    for args in ((_offset(syn), maps, work), (syn, _offset(maps), work), (syn, maps, _offset(work, 8))):
        with pytest.raises(_lib.GMError):
            call(*args)
