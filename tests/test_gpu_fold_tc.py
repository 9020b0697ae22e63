"""Ring fold of the batched path (k_fold_tc) against the one-field fold on the same operands: the
images hold img_scale times the residual right-hand sides as f16 hi + lo.  Ring lengths below and
above the band limit, item counts that fill a warp in part.

Bound: single-precision sums of at most L / 4 aliases and the f16 split (2^-22): 2e-6 of the
largest value."""

import numpy as np
import pytest
import torch

from gmaster_b200 import _lib, sht, sht_tc

pytestmark = pytest.mark.gpu


def _row_offsets(nlanes):
    """Byte offset of (row r, lane j) in one order's image planes (MN-major, 128-byte swizzle)."""
    r, j = np.arange(128)[:, None], np.arange(nlanes)[None]
    k = j % 128
    off = (k >> 3) * 2048 + (r >> 6) * 1024 + (k & 7) * 128 + ((((r & 63) >> 3) ^ (k & 7)) << 4) + (r & 7) * 2
    return off + (j // 128) * 2 * 32768


@pytest.mark.parametrize("nside,lmax", [(4, 7), (16, 47), (64, 100), (128, 383)])
@pytest.mark.parametrize("spin,ncomp", [(0, 1), (0, 5), (0, 32), (2, 2), (2, 34), (2, 64)])
def test_images_match_one_field_fold(cuda, spin, ncomp, nside, lmax):
    tp = sht_tc.get_tc_plan(nside, lmax)
    p = tp.plan
    gen = torch.Generator(device="cuda")
    gen.manual_seed(ncomp + lmax)
    syn = torch.randn((p.L, p.nlanes, ncomp, 4), generator=gen, dtype=torch.float32, device="cuda")
    rhs = torch.randn((p.L, p.nlanes, ncomp, 4), generator=gen, dtype=torch.float32, device="cuda")
    syn[:, -1, :, 2:] = 0
    rhs[:, -1, :, 2:] = 0
    c = torch.view_as_complex(syn.unflatten(3, (2, 2)).contiguous())        # (L, lane, comp, N/S)
    if spin == 0:
        rows = [torch.cat([c[..., 0], c[..., 1]], 2)]
    else:   # a: [P_N | M_S], b: [M_N | P_S]
        P, M = c[:, :, 0::2] + 1j * c[:, :, 1::2], c[:, :, 0::2] - 1j * c[:, :, 1::2]
        rows = [torch.cat([P[..., 0], M[..., 1]], 2), torch.cat([M[..., 0], P[..., 1]], 2)]
    synd = [torch.view_as_real(x.contiguous()).flatten(2).contiguous() for x in rows]   # (L, lane, 2H)
    img = [torch.zeros(tp.img_bytes, dtype=torch.uint8, device="cuda") for _ in rows]
    scale = 64.0
    _lib.call("gm_tc_fold", nside, lmax, spin, ncomp, _lib.ptr(synd[0]), _lib.ptr(synd[1]) if spin else None,
              _lib.ptr(rhs), _lib.ptr(p.shifted), _lib.ptr(img[0]), _lib.ptr(img[1]) if spin else None, scale,
              _lib.stream_handle(p.device))
    # the one-field fold in double precision, as Sum / Diff, back to north and south
    full = torch.stack([rhs[..., 0] + rhs[..., 2], rhs[..., 1] + rhs[..., 3], rhs[..., 0] - rhs[..., 2],
                        rhs[..., 1] - rhs[..., 3]], 3).double().contiguous()
    res = sht.fold_residual(p, syn.double(), full, _lib.FP64)
    g = torch.view_as_complex(torch.stack([res[..., :2] + res[..., 2:], res[..., :2] - res[..., 2:]], 3) / 2)
    if spin == 0:
        want = [torch.cat([g[..., 0], g[..., 1]], 2)]
    else:
        P, M = g[:, :, 0::2] + 1j * g[:, :, 1::2], g[:, :, 0::2] - 1j * g[:, :, 1::2]
        want = [torch.cat([P[..., 0], M[..., 1]], 2), torch.cat([M[..., 0], P[..., 1]], 2)]
    off = torch.from_numpy(_row_offsets(p.nlanes).astype(np.int64) // 2).cuda()
    for im, w in zip(img, want):
        w = torch.view_as_real(w.contiguous()).flatten(2)                   # (L, lane, 2H)
        planes = im.view(torch.float16).reshape(p.L, -1)
        R2 = w.shape[2]
        hi = planes[:, off[:R2].T.reshape(-1)].reshape(w.shape).double()
        lo = planes[:, (off[:R2] + 16384).T.reshape(-1)].reshape(w.shape).double()
        assert float(((hi + lo) / scale - w).abs().max() / w.abs().max()) < 2e-6
        assert int((planes[:, off[R2:].reshape(-1)] != 0).sum()) == 0 if R2 < 128 else True
