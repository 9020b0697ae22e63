"""Performance cases of the pseudo-C_ell estimator: the calls a user of the package makes.

Kinds of case (the ``"kind"`` entry):

* ``field``       -- ``NmtField`` of one spin-0 map or one spin-2 (Q, U) pair: masking and the
                     analysis with its Jacobi iterations; returns the alms.
* ``synthesis``   -- ``alm2map`` of one field (simulations, purification, smoothing).
* ``sims``        -- ``fields_from_maps``: a Monte-Carlo batch of fields sharing one mask.
* ``estimate``    -- ``compute_coupled_cell`` and ``decouple_cell`` of a field (or, with
                     ``nsims`` > 1, the batched forms), the workspace being at hand.
* ``workspace``   -- ``NmtWorkspace.from_fields`` for new masks: coupling blocks, binned
                     matrix and its factorisation, and the first bandpowers through it.
* ``covariance``  -- ``NmtCovarianceWorkspace.gaussian_covariance`` of bandpowers.
* ``apodize``     -- ``mask_apodization`` of a binary mask with holes.
* ``mc``          -- ``mc_bandpowers``: the whole estimator for a batch of TQU simulations
                     that start in pinned host memory.

``exact`` restates every kind in double precision with plain torch operations: direct
harmonic sums from the recurrences of the Wigner-d rows and library FFTs, couplings by
Gauss-Legendre quadrature, distances by comparing all pairs of pixels.
"""

import itertools
import math

import numpy as np
import torch

import gmaster_b200 as nmt

DEVICE = "cuda"


# ------------------------------------------------------------------------------- cases

def listed():
    return [
        # one small spectrum through a workspace that is at hand: latency and launches only
        {"name": "estimate_qu_n64", "kind": "estimate", "nside": 64, "lmax": 191, "spin": 2,
         "nlb": 8, "nsims": 1},
        # the bandpowers of a Monte-Carlo batch of polarisation fields
        {"name": "estimate_qu_n256_x32", "kind": "estimate", "nside": 256, "lmax": 767, "spin": 2,
         "nlb": 16, "nsims": 32},
        # a low-resolution temperature map in double precision, lmax below 3 nside - 1
        {"name": "field_t_n128_fp64", "kind": "field", "nside": 128, "lmax": 300, "spin": 0,
         "n_iter": 3, "precision": "fp64"},
        # an ordinary polarisation field with the defaults
        {"name": "field_qu_n512", "kind": "field", "nside": 512, "lmax": 1535, "spin": 2,
         "n_iter": 3, "precision": "mixed"},
        # a survey-resolution temperature field, the benchmark's Nside
        {"name": "field_t_n2048", "kind": "field", "nside": 2048, "lmax": 6143, "spin": 0,
         "n_iter": 3, "precision": "mixed"},
        # the (Q, U) maps of one simulation
        {"name": "synthesis_qu_n1024", "kind": "synthesis", "nside": 1024, "lmax": 3071, "spin": 2,
         "precision": "mixed"},
        # a small map in double precision with an odd band limit
        {"name": "synthesis_t_n256_fp64", "kind": "synthesis", "nside": 256, "lmax": 701, "spin": 0,
         "precision": "fp64"},
        # a Monte-Carlo batch of polarisation simulations
        {"name": "sims_qu_n512_x32", "kind": "sims", "nside": 512, "lmax": 1535, "spin": 2,
         "nsims": 32, "n_iter": 3},
        # a new 2x2 workspace: couplings, binning, factorisation
        {"name": "workspace_qu_n512", "kind": "workspace", "nside": 512, "lmax": 1535, "spin": 2,
         "nlb": 10},
        # the Gaussian covariance of polarisation bandpowers
        {"name": "covariance_qu_n512", "kind": "covariance", "nside": 512, "lmax": 1535, "spin": 2,
         "nlb": 16},
        # apodisation of a survey mask with point-source holes
        {"name": "apodize_n1024", "kind": "apodize", "nside": 1024, "aposize": 1.0, "apotype": "C1",
         "holes": 100},
        # the whole estimator from maps in host memory
        {"name": "mc_n256_x16", "kind": "mc", "nside": 256, "nlb": 16, "nsims": 16, "n_iter": 3},
    ]


def _log_uniform(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def _lmax(rng, nside):
    """A band limit between 1.5 nside and 3 nside - 1 (odd and even alike)."""
    return rng.randint(3 * nside // 2, 3 * nside - 1)


def draw(rng):
    kind = rng.choices(["field", "synthesis", "sims", "estimate", "workspace", "covariance",
                        "apodize", "mc"], [4, 2, 2, 2, 2, 1, 1, 1])[0]
    case = {"kind": kind}
    if kind == "field":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        spin = rng.choice([0, 2])
        nside = rng.choice([32, 64, 128, 256, 512] + ([1024] if precision == "mixed" else []))
        case.update(nside=nside, lmax=_lmax(rng, nside), spin=spin, n_iter=rng.choice([0, 3, 3]),
                    precision=precision)
    elif kind == "synthesis":
        nside = rng.choice([32, 64, 128, 256, 512, 1024])
        case.update(nside=nside, lmax=_lmax(rng, nside), spin=rng.choice([0, 2]),
                    precision=rng.choice(["mixed", "mixed", "fp64"]))
    elif kind == "sims":
        nside = rng.choice([64, 128, 256, 512])
        case.update(nside=nside, lmax=_lmax(rng, nside), spin=rng.choice([0, 2]),
                    nsims=_log_uniform(rng, 3, 32), n_iter=3)
    elif kind == "estimate":
        nside = rng.choice([32, 64, 128, 256])
        lmax = _lmax(rng, nside)
        case.update(nside=nside, lmax=lmax, spin=rng.choice([0, 2]), nlb=rng.randint(4, 20),
                    nsims=rng.choice([1, 1, _log_uniform(rng, 2, 32)]))
    elif kind == "workspace":
        nside = rng.choice([32, 64, 128, 256, 512])
        case.update(nside=nside, lmax=_lmax(rng, nside), spin=rng.choice([0, 2]),
                    nlb=rng.randint(4, 20))
    elif kind == "covariance":
        nside = rng.choice([64, 128, 256, 512])
        case.update(nside=nside, lmax=_lmax(rng, nside), spin=rng.choice([0, 2]),
                    nlb=rng.randint(8, 24))
    elif kind == "apodize":
        nside = rng.choice([128, 256, 512])
        case.update(nside=nside, aposize=round(rng.uniform(1.0, 3.0), 2),
                    apotype=rng.choice(["C1", "C2"]), holes=rng.randint(0, 100))
    else:
        case.update(nside=rng.choice([64, 128, 256]), nlb=rng.randint(8, 24),
                    nsims=_log_uniform(rng, 4, 24), n_iter=3)
    return case


# ------------------------------------------------------------------------------- inputs

def _rings(nside):
    """cos(theta), phi0, pixels and first pixel of the HEALPix rings (float64 / int64)."""
    i = np.arange(1, 4 * nside)
    north = np.where(i > 2 * nside, 4 * nside - i, i)
    cap = north < nside
    z = np.where(cap, 1.0 - north.astype(np.float64) ** 2 / (3.0 * nside ** 2),
                 (2.0 * nside - north) * 2.0 / (3.0 * nside))
    z = np.where(i > 2 * nside, -z, z)
    nphi = np.where(cap, 4 * north, 4 * nside)
    shifted = cap | ((north - nside) % 2 == 0)
    phi0 = np.where(shifted, np.pi / nphi, 0.0)
    offset = np.concatenate([[0], np.cumsum(nphi)[:-1]])
    return z, phi0, nphi, offset


def _pixel_vectors(nside):
    """(npix, 3) float64 unit vectors of the pixel centres on the GPU."""
    z, phi0, nphi, offset = _rings(nside)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE)  # noqa: E731
    ring = torch.repeat_interleave(torch.arange(4 * nside - 1, device=DEVICE), dev(nphi))
    k = torch.arange(12 * nside ** 2, device=DEVICE) - dev(offset)[ring]
    phi = dev(phi0)[ring] + 2 * np.pi * k / dev(nphi)[ring]
    zz = dev(z)[ring]
    s = torch.sqrt((1 - zz) * (1 + zz))
    return torch.stack([s * torch.cos(phi), s * torch.sin(phi), zz], 1)


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _pole(seed):
    r = np.random.default_rng(int(seed))
    v = np.array([0.4, 0.3, 1.0]) + 0.2 * r.normal(size=3)
    return torch.from_numpy(v / np.linalg.norm(v)).to(DEVICE)


def _mask(nside, seed):
    """A smooth Galactic cut about a tilted pole: zero within 15 degrees of its equator,
    one beyond 25, a C2 taper between (f_sky about 0.66)."""
    lat = torch.asin((_pixel_vectors(nside) @ _pole(seed)).clamp(-1, 1)).abs()
    x = ((lat - math.radians(15.0)) / math.radians(10.0)).clamp(0, 1)
    return 0.5 * (1 - torch.cos(math.pi * x))


def _maps(nside, n, seed):
    """(n, npix) float64 maps: white noise over smooth large-scale patterns."""
    g = _generator(seed)
    out = torch.randn((n, 12 * nside ** 2), generator=g, device=DEVICE, dtype=torch.float64)
    v = _pixel_vectors(nside)
    for k in (1, 3, 7):
        d = torch.randn((3, n), generator=g, device=DEVICE, dtype=torch.float64)
        out += (torch.cos(k * (v @ d)) / k).T
    return out


def _alms(lmax, spin, seed):
    """(nmaps, nelem) complex128 Gaussian alms with C_l = 1 / (l + 10)^2 (healpy packing)."""
    n = 1 if spin == 0 else 2
    g = _generator(seed)
    ell, m = _ell_m(lmax)
    a = torch.randn((n, ell.shape[0]), generator=g, device=DEVICE, dtype=torch.complex128)
    a = torch.where(m == 0, a.real * math.sqrt(2.0) + 0j, a) / (ell + 10.0)
    return torch.where(ell >= spin, a, torch.zeros_like(a))


def _ell_m(lmax):
    m = torch.repeat_interleave(torch.arange(lmax + 1, device=DEVICE),
                                torch.arange(lmax + 1, 0, -1, device=DEVICE))
    start = m * (2 * lmax + 1 - m) // 2
    return torch.arange(m.shape[0], device=DEVICE) - start, m


def _binary_mask(case, seed):
    """One where |latitude| > 20 degrees about a tilted pole, with circular holes."""
    v = _pixel_vectors(case["nside"])
    mask = ((v @ _pole(seed)).abs() > math.sin(math.radians(20.0))).to(torch.float64)
    r = np.random.default_rng(int(seed) + 1)
    for _ in range(case["holes"]):
        c = r.normal(size=3)
        radius = math.radians(r.uniform(0.2, 0.6))
        mask[v @ torch.from_numpy(c / np.linalg.norm(c)).to(DEVICE) > math.cos(radius)] = 0.0
    return mask


def _spectra(lmax, spin, seed):
    """Best-guess spectra of one field with itself: [TT] or [EE, EB, BE, BB]."""
    r = np.random.default_rng(int(seed))
    ell = np.arange(lmax + 1)
    base = (1.0 + 0.2 * np.sin(ell / 30.0 + r.uniform(0, 6))) / (ell + 10.0) ** 2
    rows = [base] if spin == 0 else [base, 0.02 * base, 0.02 * base, 0.1 * base]
    return torch.from_numpy(np.stack(rows)).to(DEVICE)


def _field_inputs(case, seed):
    """Mask and maps (nsims, nmaps, npix) of the cases that work on fields."""
    nm = 1 if case["spin"] == 0 else 2
    ns = case.get("nsims", 1)
    maps = _maps(case["nside"], ns * nm, seed).reshape(ns, nm, -1)
    return _mask(case["nside"], seed), maps


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": dict(case)}
    if kind in ("field", "sims"):
        st["mask"], st["maps"] = _field_inputs(case, seed)
    elif kind == "synthesis":
        st["alm"] = _alms(case["lmax"], case["spin"], seed)
        st["minfo"] = nmt.NmtMapInfo(None, (12 * case["nside"] ** 2,))
        st["ainfo"] = nmt.NmtAlmInfo(case["lmax"])
    elif kind == "estimate":
        mask, maps = _field_inputs(case, seed)
        kw = {"lmax": case["lmax"], "lmax_mask": case["lmax"], "precision": "fp64"}
        st["fields"] = [nmt.NmtField(mask, m, n_iter=0, lite=True, **kw) for m in maps]
        st["w"] = nmt.NmtWorkspace.from_fields(st["fields"][0], st["fields"][0],
                                               nmt.NmtBin.from_lmax_linear(case["lmax"], case["nlb"]))
    elif kind in ("workspace", "covariance"):
        mask = _mask(case["nside"], seed)
        f = nmt.NmtField(mask, None, spin=case["spin"], lmax=case["lmax"], lmax_mask=case["lmax"],
                         precision="fp64")
        f.get_mask_alms()
        st["f"], st["bins"] = f, nmt.NmtBin.from_lmax_linear(case["lmax"], case["nlb"])
        st["cl"] = _spectra(case["lmax"], case["spin"], seed)
        if kind == "covariance":
            st["w"] = nmt.NmtWorkspace.from_fields(f, f, st["bins"])
            st["cw"] = nmt.NmtCovarianceWorkspace.from_fields(f, f)
    elif kind == "apodize":
        st["mask"] = _binary_mask(case, seed)
    else:
        nside = case["nside"]
        mask = _mask(nside, seed)
        maps = _maps(nside, 3 * case["nsims"], seed).reshape(case["nsims"], 3, -1)
        st["mask"] = mask
        st["t"] = maps[:, 0].contiguous().cpu().pin_memory()
        st["qu"] = maps[:, 1:].contiguous().cpu().pin_memory()
        f0 = nmt.NmtField(mask, None, spin=0, precision="fp64")
        f2 = nmt.NmtField(mask, None, spin=2, precision="fp64")
        b = nmt.NmtBin.from_nside_linear(nside, case["nlb"])
        st["w"] = nmt.workspaces_from_fields([(f0, f0), (f0, f2), (f2, f2)], b)
    return st


# ------------------------------------------------------------------------------- the pass

def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "field":
        return nmt.NmtField(st["mask"], st["maps"][0], n_iter=case["n_iter"], lmax=case["lmax"],
                            precision=case["precision"], lite=True).get_alms()
    if kind == "sims":
        fields = nmt.fields_from_maps(st["mask"], st["maps"], n_iter=case["n_iter"],
                                      lmax=case["lmax"], precision="mixed")
        return [f.get_alms() for f in fields]
    if kind == "synthesis":
        return nmt.alm2map(st["alm"], case["spin"], st["minfo"], st["ainfo"],
                           precision=case["precision"])
    if kind == "estimate":
        fields, w = st["fields"], st["w"]
        if case["nsims"] == 1:
            cl = nmt.compute_coupled_cell(fields[0], fields[0])
            return [cl, w.decouple_cell(cl)]
        cls = nmt.compute_coupled_cells(fields, fields)
        return list(cls) + [torch.stack(nmt.decouple_cells(w, cls))]
    if kind == "workspace":
        w = nmt.NmtWorkspace.from_fields(st["f"], st["f"], st["bins"])
        return [w.mcm_blocks, w.mcm_binned, w.decouple_cell(st["cl"])]
    if kind == "covariance":
        cl = st["cl"]
        return st["cw"].gaussian_covariance(cl, cl, cl, cl, st["w"])
    if kind == "apodize":
        return nmt.mask_apodization(st["mask"], case["aposize"], apotype=case["apotype"])
    bps = nmt.mc_bandpowers(st["mask"], st["t"], st["qu"], *st["w"], n_iter=case["n_iter"],
                            precision="mixed")
    return [torch.stack(b) for b in bps]


# ------------------------------------------------------------------------------- work

def _sht_flops(nside, lmax, spin, nfields, passes):
    """One complex multiply-add per (l, m, northern lane) and map; both row variants for
    spin 2."""
    L = lmax + 1
    if spin == 0:
        return 4.0 * 2 * nside * L * (L + 1) / 2 * nfields * passes
    return 4.0 * (4 * nside - 1) * L * L * nfields * passes


def work(case):
    kind = case["kind"]
    if kind == "apodize":
        npix = 12 * case["nside"] ** 2
        return {"bytes": 16.0 * npix, "flops": 20.0 * npix}
    nside = case["nside"]
    lmax = case.get("lmax", 3 * nside - 1)
    L, npix, spin = lmax + 1, 12 * nside ** 2, case.get("spin", 0)
    nm = 1 if spin == 0 else 2
    nelem = L * (L + 1) // 2
    ns = case.get("nsims", 1)
    if kind in ("field", "sims"):
        return {"bytes": 8.0 * npix * (nm * ns + 1) + 16.0 * nelem * nm * ns,
                "flops": _sht_flops(nside, lmax, spin, ns, 1 + 2 * case["n_iter"])}
    if kind == "synthesis":
        return {"bytes": 8.0 * npix * nm + 16.0 * nelem * nm,
                "flops": _sht_flops(nside, lmax, spin, 1, 1)}
    if kind == "mc":
        nb = (lmax - 1) // case["nlb"]
        passes = 1 + 2 * case["n_iter"]
        return {"bytes": 8.0 * npix * (3 * ns + 1) + 8.0 * nb * 7 * ns + 8.0 * 21 * nb * nb,
                "flops": _sht_flops(nside, lmax, 0, ns, passes) + _sht_flops(nside, lmax, 2, ns, passes)}
    ncls = nm * nm
    nb = (lmax - 1) // case["nlb"]
    n = ncls * nb
    if kind == "estimate":
        return {"bytes": ns * (16.0 * nelem * nm + 8.0 * ncls * (L + nb)) + 8.0 * n * n,
                "flops": ns * (4.0 * nelem * ncls + 2.0 * n * n)}
    blocks = 1 if spin == 0 else 2
    if kind == "workspace":
        # the l3 sums of every pair l1 <= l2 (one multiply-add each per block), the LU
        triples = L * L * (L + 2) / 3.0
        return {"bytes": 8.0 * blocks * L * L + 8.0 * n * n,
                "flops": 2.0 * blocks * triples + 2.0 / 3.0 * n ** 3}
    # covariance: the kernels read once, the triangular solves of both sides
    return {"bytes": 8.0 * blocks * L * L + 16.0 * n * n,
            "flops": 4.0 * ncls * ncls * L * L + 4.0 * n ** 3}


# ------------------------------------------------------------------------------- tolerance

def tolerance(case):
    """Largest relative errors of another correct implementation at the same precision.
    Mixed transforms carry single-precision rows and sums: 1e-6 to 3.5e-6 off the exact sums
    up to Nside 1024.  Double precision: recurrences over thousands of rows (1e-14 to 1e-12),
    coupling sums and the solves behind them (to 2e-12)."""
    kind = case["kind"]
    if kind in ("sims", "mc") or case.get("precision") == "mixed":
        return {"rel": 2e-5}
    if kind in ("field", "synthesis", "apodize"):
        return {"rel": 1e-11}
    return {"rel": 2e-11}


# ------------------------------------------------------------------------------- exact

def _wigner_rows(x, lmax, orders, sp, block):
    """Normalised rows sqrt((2l+1)/4pi) d^l_{m,sp}(theta) at x = cos(theta) for the orders
    m = 0..orders-1 (``orders`` an int) or one order m (a one-element list): yields
    (l of the first row, table (norders, rows, npoints)), float64, by the three-term
    recurrence in l with a power-of-two scale per element."""
    one = isinstance(orders, list)
    ms = torch.tensor(orders if one else list(range(orders)), dtype=torch.float64, device=DEVICE)
    M, s = ms.shape[0], float(sp)
    a = abs(sp)
    half = torch.sqrt((1 - x) / 2).clamp_min(1e-300), torch.sqrt((1 + x) / 2).clamp_min(1e-300)
    lsin, lcos = torch.log2(half[0]), torch.log2(half[1])
    v = torch.zeros((M, x.shape[0]), dtype=torch.float64, device=DEVICE)
    vp, e = torch.zeros_like(v), torch.zeros_like(v)
    scale = torch.ones_like(v)
    l0 = torch.clamp(ms, min=a)
    start = int(l0[0])
    # d^l0_{m,sp}: l0 = m: (-1)^(m-sp) sqrt(C(2m, m+sp)) cos^(m+sp) sin^(m-sp); l0 = a > m:
    # sp = +a: sqrt(C(2a, a+m)) cos^(a+m) sin^(a-m); sp = -a: (-1)^(m+a) sqrt(C(2a, a-m)) cos^(a-m) sin^(a+m)
    top = ms >= a
    lo = torch.where(top, ms + s, torch.full_like(ms, float(a)) + (ms if sp >= 0 else -ms))
    hi = torch.where(top, ms - s, torch.full_like(ms, float(a)) - (ms if sp >= 0 else -ms))
    sign = torch.where(top, 1 - 2 * torch.remainder(ms - s, 2),
                       torch.ones_like(ms) if sp >= 0 else 1 - 2 * torch.remainder(ms + a, 2))
    norm = 0.5 * (_log2_binomial(2 * l0, lo)) + 0.5 * torch.log2((2 * l0 + 1) / (4 * math.pi))
    table, first = None, 0
    for l in range(lmax + 1):
        if table is None:
            first = l
            rows = min(block, lmax + 1 - l)
            table = torch.zeros((M, rows, x.shape[0]), dtype=torch.float64, device=DEVICE)
        lo_m = 0 if one else min(l, M)        # orders below lo_m (or all, if one) advance
        n_adv = (1 if l > start else 0) if one else (lo_m if l > a else 0)
        if n_adv:
            m = ms[:n_adv, None]
            den = torch.sqrt((l * l - m * m) * (l * l - s * s))
            al = math.sqrt((2.0 * l + 1) * (2.0 * l - 1)) * l / den
            c = m * s / ((l - 1.0) * l) if l > 1 else torch.zeros_like(m)
            l1 = l - 1.0
            num = torch.sqrt(((l1 * l1 - m * m) * (l1 * l1 - s * s)).clamp_min(0))
            be = math.sqrt((2.0 * l + 1) / (2.0 * l - 3)) * l * num / (l1 * den) if l > 1 else torch.zeros_like(m)
            new = torch.addcmul(al * (x[None] - c) * v[:n_adv], -be, vp[:n_adv])
            vp[:n_adv] = v[:n_adv]
            v[:n_adv] = new
        for k in ([0] if one and l == start else [] if one else
                  list(range(min(a + 1, M))) if l == a else [l] if a < l < M else []):
            f = norm[k] + lo[k] * lcos + hi[k] * lsin
            e[k] = torch.floor(f)
            v[k] = sign[k] * torch.exp2(f - e[k])
            vp[k] = 0
            scale[k] = torch.exp2(e[k])
        if l % 16 == 0:
            big = (v.abs() > 2.0 ** 100) & (e < 0)
            fac = torch.where(big, 2.0 ** -100, 1.0)
            v *= fac
            vp *= fac
            e += torch.where(big, 100.0, 0.0)
            scale = torch.exp2(e)
        have = M if one else min(l + 1, M)
        table[:have, l - first] = v[:have] * scale[:have]
        if l - first + 1 == table.shape[1]:
            yield first, table
            table = None


def _log2_binomial(n, k):
    """log2 C(n, k) of whole-valued tensors, summed exactly enough for 1e-13 results."""
    n_np, k_np = n.cpu().numpy().astype(int), k.cpu().numpy().astype(int)
    out = []
    for a, b in zip(n_np, k_np):
        c = math.comb(int(a), int(b)) if a <= 600 else None
        if c is None:
            # C(2m, m -+ s) from C(2m, m), whose logarithm follows from Stirling's series
            m, d = int(a) // 2, abs(int(b) - int(a) // 2)
            ser = -1 / (8 * m) + 1 / (192 * m ** 3) - 1 / (640 * m ** 5)
            val = 2.0 * m - 0.5 * math.log2(math.pi * m) + ser / math.log(2.0)
            for q in range(d):
                val += math.log2((m - q) / (m + 1 + q))
            out.append(val)
        else:
            shift = max(0, c.bit_length() - 60)
            out.append(math.log2(c >> shift) + shift)
    return torch.tensor(out, dtype=torch.float64, device=DEVICE)


class _Sphere:
    """Direct spherical-harmonic sums of HEALPix maps in double precision."""

    def __init__(self, nside, lmax):
        self.nside, self.lmax, self.L = nside, lmax, lmax + 1
        z, phi0, nphi, offset = _rings(nside)
        self.x = torch.from_numpy(z).to(DEVICE)
        self.nring = 4 * nside - 1
        m = np.arange(self.L)
        self.phase = torch.exp(-1j * torch.from_numpy(np.outer(phi0, m)).to(DEVICE))   # (nring, L)
        self.groups = []
        for n in np.unique(nphi):
            rings = np.nonzero(nphi == n)[0]
            pix = offset[rings][:, None] + np.arange(n)[None]
            self.groups.append((int(n), torch.from_numpy(rings).to(DEVICE), torch.from_numpy(pix).to(DEVICE)))
        self.m = torch.from_numpy(m).to(DEVICE)
        self.block = max(1, min(64, int(1.0e8 // (self.L * self.nring))))

    def ring_sums(self, maps):
        """(n, npix) -> (L, nring, n) complex: w sum_pix f e^{-i m phi}."""
        out = torch.empty((self.L, self.nring, maps.shape[0]), dtype=torch.complex128, device=DEVICE)
        w = 4 * math.pi / (12 * self.nside ** 2)
        for n, rings, pix in self.groups:
            f = torch.fft.fft(maps[:, pix], dim=2)                       # (n, rings, nphi)
            out[:, rings] = (f[:, :, self.m % n] * self.phase[rings] * w).permute(2, 1, 0)
        return out

    def ring_maps(self, g):
        """(L, nring, n) complex orders m >= 0 of real maps -> (n, npix)."""
        out = torch.empty((g.shape[2], 12 * self.nside ** 2), dtype=torch.float64, device=DEVICE)
        for n, rings, pix in self.groups:
            c = g[:, rings].permute(2, 1, 0) * self.phase[rings].conj()  # (n, rings, L)
            f = torch.zeros((c.shape[0], c.shape[1], n), dtype=torch.complex128, device=DEVICE)
            f.index_add_(2, self.m % n, c)
            f.index_add_(2, (-self.m[1:]) % n, c[:, :, 1:].conj())
            out[:, pix] = (torch.fft.ifft(f, dim=2) * n).real
        return out

    def _rows(self, sp):
        return _wigner_rows(self.x, self.lmax, self.L, sp, self.block)

    def _analyse(self, g, sp):
        """sum over rings of row * g: (L_m, nring, n) complex -> (L_m, L_l, n) complex."""
        gr = torch.view_as_real(g).flatten(2)                            # (L, nring, 2n)
        out = torch.zeros((self.L, self.L, gr.shape[2]), dtype=torch.float64, device=DEVICE)
        for l, tab in self._rows(sp):
            h = min(self.L, l + tab.shape[1])
            out[:h, l:l + tab.shape[1]] = torch.bmm(tab[:h], gr[:h])
        return torch.view_as_complex(out.unflatten(2, (-1, 2)))

    def _synthesise(self, a, sp):
        ar = torch.view_as_real(a).flatten(2)
        out = torch.zeros((self.L, self.nring, ar.shape[2]), dtype=torch.float64, device=DEVICE)
        for l, tab in self._rows(sp):
            h = min(self.L, l + tab.shape[1])
            out[:h] += torch.bmm(tab[:h].transpose(1, 2), ar[:h, l:l + tab.shape[1]])
        return torch.view_as_complex(out.unflatten(2, (-1, 2)))

    def analysis(self, maps, spin):
        """(n, npix) -> (L_m, L_l, n); spin 2: maps Q, U, Q, U, ... and alms E, B, E, B, ..."""
        g = self.ring_sums(maps)
        if spin == 0:
            return self._analyse(g, 0)
        p = self._analyse(g[..., 0::2] + 1j * g[..., 1::2], -2)
        q = self._analyse(g[..., 0::2] - 1j * g[..., 1::2], 2)
        return torch.stack([-(p + q) / 2, 1j * (p - q) / 2], 3).flatten(2)

    def synthesis(self, alm, spin):
        if spin == 0:
            return self.ring_maps(self._synthesise(alm, 0))
        e, b = alm[..., 0::2], alm[..., 1::2]
        p = self._synthesise(-(e + 1j * b), -2)
        q = self._synthesise(-(e - 1j * b), 2)
        return self.ring_maps(torch.stack([(p + q) / 2, (p - q) / 2j], 3).flatten(2))

    def map2alm(self, maps, spin, n_iter):
        alm = self.analysis(maps, spin)
        for _ in range(n_iter):
            alm = alm - self.analysis(self.synthesis(alm, spin) - maps, spin)
        ell, m = _ell_m(self.lmax)
        return alm[m, ell].T.contiguous()                                # (n, nelem)

    def unpack(self, packed):
        ell, m = _ell_m(self.lmax)
        out = torch.zeros((self.L, self.L, packed.shape[0]), dtype=torch.complex128, device=DEVICE)
        out[m, ell] = packed.T
        return out


def _pcl(a, b, lmax):
    ell, m = _ell_m(lmax)
    w = torch.where(m == 0, 1.0, 2.0)
    rows = []
    for x in a:
        for y in b:
            c = torch.zeros(lmax + 1, dtype=torch.float64, device=DEVICE)
            rows.append(c.index_add_(0, ell, w * (x * y.conj()).real))
    return torch.stack(rows) / (2 * torch.arange(lmax + 1, dtype=torch.float64, device=DEVICE) + 1)


def _gauss_legendre(n):
    k = torch.arange(1, n + 1, dtype=torch.float64, device=DEVICE)
    x = torch.cos(math.pi * (k - 0.25) / (n + 0.5)) * (1 - (n - 1) / (8.0 * n ** 3))
    for it in range(4):
        p0, p1 = torch.ones_like(x), x.clone()
        for j in range(2, n + 1):
            p0, p1 = p1, ((2 * j - 1) * x * p1 - (j - 1) * p0) / j
        dp = n * (x * p1 - p0) / (x * x - 1)
        if it < 3:
            x = x - p1 / dp
    return x, 2 / ((1 - x * x) * dp * dp)


def _couplings(window, lmax):
    """(4, L, L) blocks TT, TE, M+, M- of a mask spectrum, divided by 2 l2 + 1."""
    n = (2 * lmax + window.shape[0] - 1) // 2 + 2
    x, w = _gauss_legendre(n)

    def rows(lm, m, sp):
        r = torch.cat([t[0] for _, t in _wigner_rows(x, lm, [m], sp, 64)])
        return r / torch.sqrt((2 * torch.arange(lm + 1, dtype=torch.float64, device=DEVICE) + 1) / (4 * math.pi))[:, None]

    lw = window.shape[0] - 1
    ell = torch.arange(lw + 1, dtype=torch.float64, device=DEVICE)
    xi = ((2 * ell + 1) / (4 * math.pi) * window) @ rows(lw, 0, 0)
    wx = 0.5 * w * xi
    p00, p02, p22, p2m = (rows(lmax, *q) for q in ((0, 0), (0, 2), (2, 2), (2, -2)))
    quad = lambda d: (d * wx) @ d.T  # noqa: E731
    even, odd = quad(p22), quad(p2m)
    return torch.stack([quad(p00), quad(p02), (even + odd) / 2, (even - odd) / 2])


def _slots(spin1, spin2):
    """(block, row, column, sign) of the coupling matrix of a spin pair."""
    if spin1 != spin2:
        return 2, [(1, 0, 0, 1.0), (1, 1, 1, 1.0)]
    if spin1 == 0:
        return 1, [(0, 0, 0, 1.0)]
    return 4, ([(2, c, c, 1.0) for c in range(4)]
               + [(3, c, 3 - c, -1.0 if c in (1, 2) else 1.0) for c in range(4)])


def _binning(lmax, nlb):
    """(nbands, L) averaging operator of bands of nlb multipoles from l = 2."""
    nb = (lmax - 1) // nlb
    B = torch.zeros((nb, lmax + 1), dtype=torch.float64, device=DEVICE)
    for b in range(nb):
        B[b, 2 + b * nlb:2 + (b + 1) * nlb] = 1.0 / nlb
    return B


def _binned_matrix(blocks, lmax, nlb, spin1, spin2):
    B = _binning(lmax, nlb)
    T = (B > 0).to(torch.float64).T
    col = 2 * torch.arange(lmax + 1, dtype=torch.float64, device=DEVICE) + 1
    ncls, slots = _slots(spin1, spin2)
    nb = B.shape[0]
    out = torch.zeros((nb, ncls, nb, ncls), dtype=torch.float64, device=DEVICE)
    for k, r, c, sign in slots:
        out[:, r, :, c] = sign * (B @ (blocks[k] * col) @ T)
    return out.reshape(nb * ncls, nb * ncls)


def _bandpowers(matrix, cl, lmax, nlb):
    B = _binning(lmax, nlb)
    rhs = (B @ cl.T).reshape(-1)
    return torch.linalg.solve(matrix, rhs).reshape(B.shape[0], cl.shape[0]).T


def _odd_factor(o1, o2, i1, i2):
    """Coupling of the outputs (o1, o2) of a pair of spin-2 fields to its inputs (i1, i2): 0
    for the parity-even K+K+ (o = i), +-1 for K+K- (one component changed, with the sign of
    E~ = K+ E + i K- B, B~ = K+ B - i K- E), None for both changed (K-K- joins no other)."""
    if o1 == i1 and o2 == i2:
        return 0
    if o1 != i1 and o2 != i2:
        return None
    first = o1 != i1
    return (1 if first else -1) * (1 if (o1 if first else o2) == 0 else -1)


def _exact_covariance(case, seed):
    lmax, nlb, spin = case["lmax"], case["nlb"], case["spin"]
    mask = _mask(case["nside"], seed)
    sphere = _Sphere(case["nside"], lmax)
    a = sphere.map2alm(torch.stack([mask, mask * mask]), 0, 3)
    wl, ww = _pcl(a[:1], a[:1], lmax)[0], _pcl(a[1:], a[1:], lmax)[0]
    matrix = _binned_matrix(_couplings(wl, lmax), lmax, nlb, spin, spin)
    xi = _couplings(ww, lmax)
    cl = _spectra(lmax, spin, seed)
    B = _binning(lmax, nlb)
    nb = B.shape[0]

    def term(p, q, kernel):
        sym = (torch.outer(cl[p], cl[q]) + torch.outer(cl[q], cl[p])) / 2
        return B @ (sym * kernel) @ B.T

    if spin == 0:
        cov = 2 * term(0, 0, xi[0])
    else:
        cov = torch.zeros((nb, 4, nb, 4), dtype=torch.float64, device=DEVICE)
        cache = {}

        def get(p, q, k):
            key = (min(p, q), max(p, q), k)
            if key not in cache:
                cache[key] = term(p, q, xi[k])
            return cache[key]

        r2 = range(2)
        for ia, ib, ic, idd in itertools.product(r2, repeat=4):
            out = 0
            for jc, jd in ((ic, idd), (idd, ic)):   # <a1 b1><a2 b2>, <a1 b2><a2 b1>
                for p, q, r, t in itertools.product(r2, repeat=4):
                    f, g = _odd_factor(ia, jc, p, q), _odd_factor(ib, jd, r, t)
                    if f is None or g is None or (f == 0) != (g == 0):
                        continue
                    sign, k = (1.0, 2) if f == 0 else (-float(f * g), 3)
                    out = out + sign * get(2 * p + q, 2 * r + t, k)
            cov[:, 2 * ia + ib, :, 2 * ic + idd] = out
        cov = cov.reshape(4 * nb, 4 * nb)
    half = torch.linalg.solve(matrix, cov)
    return torch.linalg.solve(matrix, half.T).T


def _exact_apodize(case, seed):
    if case["nside"] > 512:
        return None
    mask = _binary_mask(case, seed)
    v = _pixel_vectors(case["nside"])
    bad, good = torch.nonzero(mask <= 0)[:, 0], torch.nonzero(mask > 0)[:, 0]
    vb = v[bad].T.contiguous()
    d2 = torch.empty(good.shape[0], dtype=torch.float64, device=DEVICE)
    step = max(1, int(4e8 // max(1, bad.shape[0])))
    for s in range(0, good.shape[0], step):
        q = v[good[s:s + step]]
        near = v[bad[torch.argmax(q @ vb, 1)]]
        d2[s:s + step] = ((q - near) ** 2).sum(1)
    threshold = 1 - math.cos(math.radians(case["aposize"]))
    x = torch.sqrt(0.5 * d2 / threshold)
    taper = x - torch.sin(2 * math.pi * x) / (2 * math.pi) if case["apotype"] == "C1" else 0.5 * (1 - torch.cos(math.pi * x))
    out = mask.clone()
    out[good] *= torch.where(d2 < 2 * threshold, taper, torch.ones_like(x))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "apodize":
        return _exact_apodize(case, seed)
    if case["nside"] > 1024:
        return None   # the direct sums take minutes at Nside 2048
    if kind == "covariance":
        return _exact_covariance(case, seed)
    nside = case["nside"]
    lmax = case.get("lmax", 3 * nside - 1)
    sphere = _Sphere(nside, lmax)
    if kind == "synthesis":
        return sphere.synthesis(sphere.unpack(_alms(lmax, case["spin"], seed)), case["spin"])
    if kind == "field":
        mask, maps = _field_inputs(case, seed)
        return sphere.map2alm(maps[0] * mask, case["spin"], case["n_iter"])
    if kind == "sims":
        mask, maps = _field_inputs(case, seed)
        alm = sphere.map2alm((maps * mask).flatten(0, 1), case["spin"], case["n_iter"])
        return list(alm.reshape(case["nsims"], -1, alm.shape[1]))
    spin = case.get("spin", 0)
    mask = _mask(nside, seed)
    mask_alm = sphere.map2alm(mask[None], 0, 3)
    blocks = _couplings(_pcl(mask_alm, mask_alm, lmax)[0], lmax)
    if kind == "workspace":
        col = 2 * torch.arange(lmax + 1, dtype=torch.float64, device=DEVICE) + 1
        matrix = _binned_matrix(blocks, lmax, case["nlb"], spin, spin)
        used = torch.zeros_like(blocks)
        for k in ([0] if spin == 0 else [2, 3]):
            used[k] = blocks[k] * col
        return [used, matrix, _bandpowers(matrix, _spectra(lmax, spin, seed), lmax, case["nlb"])]
    if kind == "estimate":
        _, maps = _field_inputs(case, seed)
        ns = case["nsims"]
        alm = sphere.map2alm((maps * mask).flatten(0, 1), spin, 0)
        alm = alm.reshape(ns, -1, alm.shape[1])
        matrix = _binned_matrix(blocks, lmax, case["nlb"], spin, spin)
        cls = [_pcl(a, a, lmax) for a in alm]
        bps = torch.stack([_bandpowers(matrix, c, lmax, case["nlb"]) for c in cls])
        return [cls[0], bps[0]] if ns == 1 else cls + [bps]
    ns = case["nsims"]
    maps = _maps(nside, 3 * ns, seed).reshape(ns, 3, -1) * mask
    t = sphere.map2alm(maps[:, 0], 0, case["n_iter"])
    p = sphere.map2alm(maps[:, 1:].flatten(0, 1), 2, case["n_iter"]).reshape(ns, 2, -1)
    out = []
    for s1, s2, a, b in ((0, 0, t[:, None], t[:, None]), (0, 2, t[:, None], p), (2, 2, p, p)):
        matrix = _binned_matrix(blocks, lmax, case["nlb"], s1, s2)
        out.append(torch.stack([_bandpowers(matrix, _pcl(a[i], b[i], lmax), lmax, case["nlb"])
                                for i in range(ns)]))
    return out
