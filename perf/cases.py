"""Performance cases: the work that a user of this package has it do, through its public
entry points, over the sizes, windows and options that phase-linking runs use.

Every case is a dict with a ``kind`` and its sizes; ``listed()`` names the fixed ones,
``draw(rng)`` gives further ones of the same ranges.  ``prepare`` makes the inputs from a
seed, ``run`` is one pass, ``work`` the bytes and operations that the pass cannot do
without, and ``exact`` the same outputs in float64 by plain torch (``None`` for whole
numbers, masks and cases too large for it).

The scenes: circular-Gaussian speckle with the exponential-decay coherence model
(gamma0 0.7, gamma_inf 0.1, tau 36 days, 12 days apart) on parcels of different
backscatter, some of them built-up (bright, stable, phase noise 0.3 rad: the persistent
scatterers), under a deformation bump of 3 rad.
"""

import math

import numpy as np
import torch

import dolphin_gb300 as dp

PARCEL = 40  # side of a parcel of constant backscatter


# ------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------
def _case(kind, n, rows, cols, hy=5, hx=11, sy=1, sx=1, shp="glrt", evd=False, radius=0, name=None):
    c = dict(kind=kind, n=n, rows=rows, cols=cols, hy=hy, hx=hx, sy=sy, sx=sx, shp=shp, evd=evd, radius=radius)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest whole chain (PS, GLRT neighbours, phase linking) on device tensors: the
        # 10-date 128 x 128 stack with an 11 x 11 window, bound by launches and latency
        _case("chain", 10, 128, 128, 5, 5, name="chain_small"),
        # the production block: 30 dates, 1024 x 1024 with its half-window halo, PS, GLRT, EMI,
        # CRLB, as the block loop of a 4096 x 4096 frame calls it 16 times
        _case("chain", 30, 1034, 1046, name="chain_block"),
        # multilooked outputs (strides 3 x 6, rectangular windows), an odd number of dates (20 and
        # a compressed SLC), phase linking alone
        _case("link", 21, 1536, 2304, sy=3, sx=6, shp="rect", name="link_strided"),
        # the EVD estimator on a ragged block of one 15-date ministack
        _case("link", 15, 501, 777, evd=True, name="link_evd"),
        # the deepest ministack of the batch workload, 45 dates, 11 x 11 window
        _case("link", 45, 500, 512, 5, 5, name="link_deep"),
        # the drop-in on host arrays, as an existing workflow calls it: numpy in, numpy out
        _case("host", 12, 256, 320, 5, 5, name="host_dropin"),
        # several ministacks of uneven depth in one batch (8, 15, 24, 36 dates, 256 x 250 each)
        _case("batch", 36, 256, 250, 5, 5, name="batch_uneven"),
        # amplitude dispersion and PS selection of a 30-date half frame
        _case("ps", 30, 2048, 4096, name="ps_frame"),
        # GLRT neighbour masks of two blocks
        _case("shp", 30, 1024, 2048, name="glrt_masks"),
        # KS neighbour masks, the other SHP test, on 20 dates
        _case("shp", 20, 512, 512, shp="ks", name="ks_masks"),
        # the similarity raster after a ministack: median, radius 7
        _case("similarity", 30, 1400, 1500, shp="median", radius=7, name="similarity_median"),
        # the sequential estimator: two ministacks of 10 dates with a compressed SLC between
        # them, 512 x 512 blocks, every output raster
        _case("sequential", 20, 1024, 1024, name="sequential"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


WINDOWS = ((5, 11), (5, 5), (7, 7), (3, 6))


def draw(rng):
    kind = rng.choice(["chain", "link", "link", "link", "host", "batch", "ps", "shp", "shp", "compress", "similarity",
                       "sequential"])
    hy, hx = rng.choice(WINDOWS)
    aspect = math.exp(rng.uniform(-0.7, 0.7))

    def size(lo, hi):
        px = _log_int(rng, lo, hi)
        rows = max(40, int(math.sqrt(px * aspect)))
        return rows, max(40, px // rows)

    if kind in ("chain", "link"):
        n = rng.randint(5, 45)
        sy, sx = (1, 1) if kind == "chain" else rng.choice([(1, 1), (1, 1), (2, 2), (3, 6), (1, 3)])
        # the solve grows with n cubed: no more of it than the 30-date block has
        top = min(1000000, int(1.0e6 * (27.0 / n) ** 3))
        rows, cols = size(6000, top)
        if sy * sx > 1:
            rows, cols = min(rows * sy, 3000), min(cols * sx, 3000)
        return _case(kind, n, rows, cols, hy, hx, sy, sx, rng.choice(["glrt", "glrt", "rect"]) if kind == "link" else "glrt",
                     evd=kind == "link" and rng.random() < 0.25)
    if kind == "host":
        n = rng.randint(6, 24)
        rows, cols = size(4000, 120000)
        return _case(kind, n, rows, cols, hy, min(hx, 7), shp=rng.choice(["glrt", "rect"]))
    if kind == "batch":
        n = rng.randint(16, 45)
        rows, cols = size(6000, 90000)
        return _case(kind, n, rows, cols, hy, hx)
    if kind == "ps":
        rows, cols = size(6000, 6000000)
        return _case(kind, rng.randint(8, 60), rows, cols)
    if kind == "shp":
        shp = rng.choice(["glrt", "glrt", "ks"])
        sy, sx = rng.choice([(1, 1), (1, 1), (3, 6)])
        rows, cols = size(6000, 1500000 if shp == "glrt" else 300000)
        if sy * sx > 1:
            rows, cols = min(rows * sy, 2000), min(cols * sx, 2000)
        return _case(kind, rng.randint(8, 40), rows, cols, hy, hx, sy, sx, shp)
    if kind == "compress":
        sy, sx = rng.choice([(1, 1), (3, 6), (2, 2)])
        rows, cols = size(20000, 4000000)
        return _case(kind, rng.randint(5, 30), rows, cols, sy=sy, sx=sx)
    if kind == "similarity":
        rows, cols = size(10000, 1500000)
        return _case(kind, rng.randint(8, 30), rows, cols, shp=rng.choice(["median", "median", "max"]),
                     radius=rng.choice([7, 7, 11]))
    rows, cols = size(60000, 800000)
    sy, sx = rng.choice([(1, 1), (1, 1), (2, 2)])
    return _case("sequential", rng.randint(8, 24), rows, cols, 5, 5, sy, sx)


# ------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------
def _coherence(n):
    t = 12.0 * np.arange(n)
    g = 0.6 * np.exp(-np.abs(t[:, None] - t[None, :]) / 36.0) + 0.1
    np.fill_diagonal(g, 1.0)
    return g


def _scene(n, rows, cols, seed):
    """(n, rows, cols) complex64 CUDA stack."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))

    def normal(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    pr, pc = -(-rows // PARCEL), -(-cols // PARCEL)
    level = torch.exp(0.6 * normal(pr, pc))
    urban = torch.rand((pr, pc), generator=g, device="cuda") < 0.08

    def spread(x):
        return x.repeat_interleave(PARCEL, 0).repeat_interleave(PARCEL, 1)[:rows, :cols]

    level, urban = spread(level), spread(urban)
    r = torch.arange(rows, device="cuda", dtype=torch.float32)[:, None] - rows // 2
    c = torch.arange(cols, device="cuda", dtype=torch.float32)[None, :] - cols // 2
    bump = 3.0 * torch.exp(-(r * r + c * c) / (2.0 * (max(rows, cols) / 8.0) ** 2))
    chol = torch.from_numpy(np.linalg.cholesky(_coherence(n))).to("cuda", torch.float32)
    out = torch.empty((n, rows, cols), dtype=torch.complex64, device="cuda")
    step = max(1, (1 << 21) // cols)
    for a in range(0, rows, step):
        b = min(rows, a + step)
        w = normal(2, n, (b - a) * cols).mul_(math.sqrt(0.5))
        x = torch.matmul(chol, w).reshape(2, n, b - a, cols)
        amp = torch.exp(0.3 * normal(n, b - a, cols)) * level[a:b]
        z = torch.complex(x[0], x[1]) * amp
        point = torch.polar(4.0 * level[a:b] * (1.0 + 0.15 * normal(n, b - a, cols)), 0.3 * normal(n, b - a, cols))
        z = torch.where(urban[a:b], point, z)
        frac = torch.linspace(0.0, 1.0, n, device="cuda")[:, None, None]
        out[:, a:b] = z * torch.polar(torch.ones_like(frac * bump[a:b]), frac * bump[a:b])
    return out


def _batch_depths(n):
    return [max(8, n // 4), max(8, 5 * n // 12), 2 * n // 3, n]


def prepare(case, seed):
    c = dict(case)
    kind, n, rows, cols = c["kind"], c["n"], c["rows"], c["cols"]
    hw, st = dp.HalfWindow(c["hy"], c["hx"]), dp.Strides(c["sy"], c["sx"])
    s = dict(c=c, hw=hw, st=st)
    if kind == "batch":
        stacks = [_scene(d, rows, cols, seed * 8 + i) for i, d in enumerate(_batch_depths(n))]
        s["batch"] = dp.PhaseLinkBatch(stacks, hw, alpha=0.001, forms={}, graph=False)
        return s
    z = _scene(n, rows, cols, seed)
    if kind == "ps":
        s["mag"] = z.abs()
        return s
    if kind == "similarity":
        s["z"] = torch.polar(torch.ones_like(z.real), torch.angle(z * z[:1].conj()))
        return s
    if kind == "shp" and c["shp"] == "ks":
        s["mag"] = z.abs()
        return s
    if kind == "chain":
        s["z"] = z
        return s
    mean, disp, ps = dp.calc_ps_block(z.abs(), 0.25, n)
    var = (disp * mean) ** 2
    s.update(mean=mean, var=var, ps=ps)
    if kind == "shp":
        return s
    if kind == "sequential":
        s.update(z=z, disp=disp)
        return s
    if kind == "compress":
        ph = torch.angle(z[:, c["sy"] // 2::c["sy"], c["sx"] // 2::c["sx"]])[:, :rows // c["sy"], :cols // c["sx"]]
        s.update(z=z, pl=torch.polar(torch.ones_like(ph), 0.8 * ph).contiguous())
        return s
    nb = None
    if c["shp"] == "glrt":
        nb = dp.estimate_neighbors(halfwin_rowcol=hw, alpha=0.001, strides=st, mean=mean, var=var, nslc=n)
    s.update(z=z, nb=nb)
    if kind == "host":
        for k in ("z", "mean"):
            s[k] = s[k].cpu().numpy()
        s["ps"] = ps.cpu().numpy().astype(bool)
        s["nb"] = None if nb is None else nb.cpu().numpy().astype(bool)
    return s


# ------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------
def run(s):
    c, hw, st = s["c"], s["hw"], s["st"]
    kind, n = c["kind"], c["n"]
    if kind == "chain":
        z = s["z"]
        mean, disp, ps = dp.calc_ps_block(z.abs(), 0.25, n)
        nb = dp.estimate_neighbors(halfwin_rowcol=hw, alpha=0.001, mean=mean, var=(disp * mean) ** 2, nslc=n)
        return tuple(dp.run_phase_linking(z, hw, ps_mask=ps, neighbor_arrays=nb, avg_mag=mean))
    if kind in ("link", "host"):
        return tuple(dp.run_phase_linking(s["z"], hw, st, use_evd=c["evd"], ps_mask=s["ps"], neighbor_arrays=s["nb"],
                                          avg_mag=s["mean"]))
    if kind == "batch":
        return [tuple(o) for o in s["batch"].run()]
    if kind == "ps":
        return dp.calc_ps_block(s["mag"], 0.25, n)
    if kind == "shp":
        if c["shp"] == "ks":
            return dp.estimate_neighbors(halfwin_rowcol=hw, alpha=0.05, strides=st, amp_stack=s["mag"],
                                         method=dp.ShpMethod.KS)
        return dp.estimate_neighbors(halfwin_rowcol=hw, alpha=0.001, strides=st, mean=s["mean"], var=s["var"], nslc=n)
    if kind == "compress":
        return dp.compress(s["z"], s["pl"], slc_mean=s["mean"], reference_idx=0), s["mean"]  # the mean is updated in place
    if kind == "similarity":
        f = dp.median_similarity if c["shp"] == "median" else dp.max_similarity
        return f(s["z"], c["radius"])
    out = dp.run_wrapped_phase_sequential(
        s["z"], ministack_size=-(-n // 2), half_window=hw, strides=st, ps_mask=s["ps"], amp_mean=s["mean"],
        amp_dispersion=s["disp"], shp_method=dp.ShpMethod.GLRT, shp_alpha=0.001, shp_nslc=n)
    return dict(pl_slcs=out.pl_slcs, crlb=out.crlb, closure=out.closure_phases, comp_slcs=out.comp_slcs,
                temp_coh=out.temp_coh, shp_counts=[x.to(torch.int32) for x in out.shp_counts],
                similarity=out.similarity, amp_dispersion=out.amp_dispersion, eigenvalues=out.eigenvalues,
                estimator=out.estimator)


# ------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------
def _circle(radius):
    """Half-heights of the columns -h .. h of the filled midpoint circle of radius h = radius - 1."""
    h = radius - 1
    top = [0] * (h + 1)
    x, y, d = h, 0, 1 - h
    while x >= y:
        for a, b in ((x, y), (y, x)):
            top[a] = max(top[a], b)
        y += 1
        if d <= 0:
            d += 2 * y + 1
        else:
            x -= 1
            d += 2 * (y - x) + 1
    for a in range(h - 1, -1, -1):
        top[a] = max(top[a], top[a + 1])
    return [top[abs(a)] for a in range(-h, h + 1)]


def _link_work(n, rows, cols, out_px, w, masks):
    flops = out_px * (4.0 * w * n * (n + 1) + 3.0 * n**3 + 56.0 * n**2)
    nbytes = 8.0 * n * rows * cols + out_px * ((w if masks else 0) + 12.0 * n + 4.0 * (n - 2) + 13.0) + 5.0 * rows * cols
    return nbytes, flops


def work(case):
    c = case
    kind, n, rows, cols = c["kind"], c["n"], c["rows"], c["cols"]
    px, w = rows * cols, (2 * c["hy"] + 1) * (2 * c["hx"] + 1)
    out_px = (rows // c["sy"]) * (cols // c["sx"])
    if kind in ("chain", "link", "host"):
        # in a chain the masks, the mean and the PS mask are intermediate
        b, f = _link_work(n, rows, cols, out_px, w, c["shp"] == "glrt" and kind != "chain")
        if kind == "chain":
            b -= 5.0 * px
            f += 8.0 * px * w + 6.0 * n * px
    elif kind == "batch":
        b = f = 0.0
        for d in _batch_depths(n):
            b1, f1 = _link_work(d, rows, cols, px, w, False)
            b, f = b + b1 - 5.0 * px, f + f1 + 8.0 * px * w + 6.0 * d * px
    elif kind == "ps":
        b, f = px * (4.0 * n + 9.0), px * 6.0 * n
    elif kind == "shp":
        if c["shp"] == "ks":
            b, f = 4.0 * n * px + out_px * w, out_px * w * 2.0 * n
        else:
            b, f = 8.0 * px + out_px * w, out_px * w * 8.0
    elif kind == "compress":
        # the given mean is read and written
        b, f = px * (8.0 * n + 16.0) + out_px * 8.0 * n, px * 14.0 * n
    elif kind == "similarity":
        k = sum(2 * h + 1 for h in _circle(c["radius"])) - 1
        b, f = px * (8.0 * n + 4.0), px * (4.0 * k * n + 2.0 * k)
    else:
        m = -(-n // 2)
        b = f = 0.0
        for d in (m, n - m + 1):
            b1, f1 = _link_work(d, rows, cols, out_px, w, False)
            b, f = b + b1 + px * 12.0, f + f1 + out_px * w * 8.0 + px * 20.0 * d + out_px * 4.0 * 136 * d
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------------
# the same in float64
# ------------------------------------------------------------------------------------
def _exact_link(z, hw, st, nb, ps, mag, evd):
    n, rows, cols = z.shape
    hy, hx = hw
    sy, sx = st
    orow, ocol = rows // sy, cols // sx
    wy, wx = 2 * hy + 1, 2 * hx + 1
    dev = z.device
    zt = z.to(torch.complex128).permute(1, 2, 0).reshape(rows * cols, n).contiguous()
    pix = orow * ocol
    cpx = torch.empty((n, pix), dtype=torch.complex128, device=dev)
    crlb = torch.zeros((n, pix), dtype=torch.float64, device=dev)
    tco = torch.empty(pix, dtype=torch.float64, device=dev)
    eig = torch.empty(pix, dtype=torch.float64, device=dev)
    clo = torch.empty((pix, max(n - 2, 0)), dtype=torch.float64, device=dev)
    eye = torch.eye(n, dtype=torch.float64, device=dev)
    low = torch.tril(torch.ones(n, n, dtype=torch.bool, device=dev), -1)
    step = max(256, (1 << 27) // (16 * n * max(wy * wx, 4 * n)))
    for a in range(0, pix, step):
        p = torch.arange(a, min(pix, a + step), device=dev)
        r0 = (sy // 2 + (p // ocol) * sy - hy).clamp(0, rows - wy)
        c0 = (sx // 2 + (p % ocol) * sx - hx).clamp(0, cols - wx)
        q = ((r0[:, None, None] + torch.arange(wy, device=dev)[None, :, None]) * cols + c0[:, None, None]
             + torch.arange(wx, device=dev)[None, None, :]).reshape(len(p), -1)
        x = zt[q]
        if nb is not None:
            x = x * nb.reshape(pix, -1)[p].to(torch.float64)[:, :, None]
        num = torch.bmm(x.transpose(1, 2), x.conj())
        amp = num.diagonal(dim1=1, dim2=2).real
        den = torch.sqrt(amp[:, :, None] * amp[:, None, :])
        cov = torch.where(den > 1e-6, num / den.clamp_min(1e-300), torch.zeros_like(num))
        gam = cov.abs()
        chol, info = torch.linalg.cholesky_ex(gam + 1e-6 * eye)
        ok = (info == 0) & torch.isfinite(chol).flatten(1).all(1)
        ginv = torch.cholesky_inverse(torch.where(ok[:, None, None], chol, eye))
        power = cov * gam
        emi = ok if not evd else torch.zeros_like(ok)
        mat = torch.where(emi[:, None, None], ginv * cov, power)
        it = torch.where(emi[:, None, None], torch.linalg.inv_ex(torch.where(emi[:, None, None], mat - 0.99 * eye,
                                                                             eye.to(mat.dtype)))[0], power)
        for _ in range(9):  # 512 steps of the (inverse) iteration by squaring
            it = it / it.abs().amax((1, 2), keepdim=True).clamp_min(1e-300)
            it = torch.bmm(it, it)
        v = it.sum(2)
        v = v / torch.linalg.vector_norm(v, dim=1, keepdim=True)
        eig[p] = (v.conj() * torch.bmm(mat, v[:, :, None])[:, :, 0]).sum(1).real
        v = v * torch.exp(-1j * torch.angle(v[:, :1]))
        u = torch.exp(1j * torch.angle(v))
        cpx[:, p] = u.T
        t = torch.exp(1j * torch.angle(cov)) * u[:, None, :] * u.conj()[:, :, None]
        tco[p] = t[:, low].mean(1).abs()
        fim = 2.0 * math.sqrt(hy * hx) * (gam * ginv - eye)
        fim = fim[:, 1:, 1:] + 1e-6 * eye[1:, 1:]
        d = torch.linalg.inv_ex(fim)[0].diagonal(dim1=1, dim2=2)
        crlb[1:, p] = torch.where(ok[:, None], d, torch.full_like(d, math.nan)).sqrt().T
        i = torch.arange(n - 2, device=dev)
        clo[p] = torch.angle(cov[:, i, i + 1] * cov[:, i + 1, i + 2] * cov[:, i, i + 2].conj())
    # persistent scatterers: the phase of the brightest one in the look window, coherence 1
    look = torch.arange(rows * cols, device=dev).reshape(rows, cols)[:orow * sy, :ocol * sx]
    look = look.reshape(orow, sy, ocol, sx).permute(0, 2, 1, 3).reshape(pix, sy * sx)
    psl = ps.reshape(-1).bool()[look]
    best = torch.where(psl, mag.reshape(-1)[look], torch.full((1,), -math.inf, device=dev))
    at = look.gather(1, best.argmax(1, keepdim=True))[:, 0]
    has = psl.any(1)
    zp = zt[at].T
    zp = torch.exp(1j * (torch.angle(zp) - torch.angle(zp[:1])))
    cpx = torch.where(has, zp, cpx)
    tco = torch.where(has, torch.ones_like(tco), tco)
    return (cpx.reshape(n, orow, ocol), tco.reshape(orow, ocol), None, eig.reshape(orow, ocol), None,
            crlb.reshape(n, orow, ocol), clo.reshape(orow, ocol, -1))


def _exact_similarity(z, radius, kind):
    n, rows, cols = z.shape
    h = radius - 1
    half = _circle(radius)
    out = torch.empty((rows, cols), dtype=torch.float64, device=z.device)
    step = max(1, (1 << 25) // (cols * sum(2 * k + 1 for k in half)))
    cc = torch.arange(cols, device=z.device)
    for a in range(0, rows, step):
        b = min(rows, a + step)
        r = torch.arange(a, b, device=z.device)
        own = torch.exp(1j * torch.angle(z[:, a:b].to(torch.complex128)))
        vals = []
        for dc in range(-h, h + 1):
            for dr in range(-half[dc + h], half[dc + h] + 1):
                if dr == 0 and dc == 0:
                    continue
                rq, cq = (r + dr).clamp(0, rows - 1), (cc + dc).clamp(0, cols - 1)
                q = torch.exp(1j * torch.angle(z[:, rq][:, :, cq].to(torch.complex128)))
                v = (own * q.conj()).real.mean(0)
                self_ = (rq == r)[:, None] & (cq == cc)[None, :]  # a clipped offset that reaches the pixel itself
                vals.append(torch.where(self_, torch.full_like(v, math.nan), v))
        v = torch.stack(vals)
        if kind == "max":
            out[a:b] = torch.where(torch.isnan(v), torch.full_like(v, -math.inf), v).amax(0)
        else:
            out[a:b] = torch.nanquantile(v.reshape(v.shape[0], -1), 0.5, dim=0).reshape(b - a, cols)
    return out


def exact(case, seed):
    c = case
    kind, n, rows, cols = c["kind"], c["n"], c["rows"], c["cols"]
    w = (2 * c["hy"] + 1) * (2 * c["hx"] + 1)
    out_px = (rows // c["sy"]) * (cols // c["sx"])
    if kind in ("chain", "link", "host"):
        if out_px * (4.0 * w * n * n + 20.0 * n**3) > 3e11:
            return None
        s = prepare(dict(c, kind="link"), seed)
        return _exact_link(s["z"], s["hw"], s["st"], s["nb"], s["ps"], s["mean"], c["evd"])
    if kind == "ps":
        x = prepare(c, seed)["mag"].to(torch.float64)
        mean = x.mean(0)
        return mean, x.var(0, unbiased=False).sqrt() / mean, None
    if kind == "compress":
        s = prepare(c, seed)
        z, pl = s["z"].to(torch.complex128), s["pl"].to(torch.complex128)
        pl = pl * pl[:1].conj()
        up = torch.zeros_like(z)
        rep = pl.repeat_interleave(rows // pl.shape[1], 1).repeat_interleave(cols // pl.shape[2], 2)
        up[:, :rep.shape[1], :rep.shape[2]] = rep
        ph = torch.angle((z * up.conj()).sum(0))
        m = torch.where(ph == 0, torch.full_like(ph, math.nan), s["mean"].to(torch.float64))
        return torch.polar(m.nan_to_num(), ph) + torch.where(torch.isnan(m), m, torch.zeros_like(m)), m
    if kind == "similarity":
        if rows * cols * n > 7e7 * (1 if c["radius"] < 9 else 0.4):
            return None
        return _exact_similarity(prepare(c, seed)["z"], c["radius"], c["shp"])
    return None
