"""Performance cases of the reconstruction path, through its public entry
points: single frames in both arithmetic forms (resident device planes in and
out), a batch of uneven frames, a gradient evaluation, the allocation-free DC
stage, and a whole decode step from host buffers to the bytes of a PPM file.

``listed`` gives the fixed cases, ``draw`` further ones of the same ranges,
``prepare`` what a program has in hand before the call, ``run`` one pass,
``work`` the bytes and operations a pass cannot do without, and ``exact`` the
result in 64-bit arithmetic (a restatement in plain torch, without this
package's code).

Frames are synthetic, of the reference encoder's kind: its scalars, quant
field, DC and coefficient statistics on the generator images, and its
transform mix at butteraugli distance 0.5, 1 or 3 (or a broad mix that gives
every transform type a share). They are generated on the GPU from the seed.
"""

import math

import numpy as np
import torch

from pik_b200 import layout, native

DEV = "cuda" if torch.cuda.is_available() else "cpu"

# Shares of 8x8 cells per transform type. d05 / d1 / d3: what the reference
# encoder picks on the generator images at that distance; broad: every type.
MIXES = {
    "d05": {"DCT32X32": 0.22, "DCT16X16": 0.72, "DCT": 0.058,
            "DCT4X4": 0.001, "DCT2X2": 0.001},
    "d1": {"DCT16X16": 0.90, "DCT": 0.09, "DCT4X4": 0.004, "DCT2X2": 0.006},
    "d3": {"DCT32X32": 0.89, "DCT16X16": 0.08, "DCT": 0.03},
    "broad": {"DCT32X32": 0.18, "DCT16X16": 0.22, "DCT": 0.36,
              "DCT4X4": 0.08, "DCT2X2": 0.04, "IDENTITY": 0.03,
              "LINES": 0.02, "DCT_NOHF": 0.04, "DCT4X4_NOHF": 0.03},
}
DISTANCE = {"d05": 0.5, "d1": 1.0, "d3": 3.0, "broad": 1.0}


def listed():
    f = dict(kind="frame", w=0, h=0, form="split_bf16", mix="d1", epf=True,
             gaborish=2, hf=True, srgb8=False)
    return [
        # A small preview: the launches' latency is what counts.
        dict(f, name="thumb_256x256_fp32", w=256, h=256, form="fp32",
             mix="broad"),
        # A ragged size with part groups, part tiles and part blocks.
        dict(f, name="odd_1030x530_split", w=1030, h=530, mix="broad"),
        # A full-HD frame in the default form, with the 8-bit output that a
        # viewer shows beside the linear planes.
        dict(f, name="hd_1920x1080_fp32_srgb8", w=1920, h=1080, form="fp32",
             srgb8=True),
        # The headline workload's size, mix and form.
        dict(f, name="uhd_3840x2160_split", w=3840, h=2160),
        # The same in the default form.
        dict(f, name="uhd_3840x2160_fp32", w=3840, h=2160, form="fp32"),
        # A strongly compressed photo of odd size: 32x32 transforms mostly.
        dict(f, name="photo_3001x2003_fp32_d3", w=3001, h=2003, form="fp32",
             mix="d3"),
        # Without the adaptive filter and the HF prediction, strongest
        # gaborish: the options a fast encoder switches off.
        dict(f, name="plain_2048x1536_split", w=2048, h=1536, mix="broad",
             epf=False, hf=False, gaborish=4),
        # The largest: a high-quality very large frame.
        dict(f, name="huge_8192x8192_split", w=8192, h=8192, mix="d05"),
        # Many images of uneven sizes decoded together.
        dict(kind="batch", name="batch_24_split", count=24, lo=256, hi=1536,
             form="split_bf16", mix="broad"),
        # One gradient evaluation of an encoder's tuning loop.
        dict(kind="adjoint", name="adjoint_1024x1024_split", w=1024, h=1024,
             form="split_bf16", mix="d1"),
        # The DC stage alone, for callers that must not allocate.
        dict(kind="dc", name="dc_4096x4096", w=4096, h=4096),
        # What a decoder program does per image, from the entropy decoder's
        # host buffers to the bytes of the PPM file it writes.
        dict(kind="decode", name="decode_1280x720_ppm", w=1280, h=720,
             form="fp32", mix="d1"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frame"] * 6 + ["batch", "adjoint", "dc", "decode"])
    form = rng.choice(["fp32", "split_bf16"])
    mix = rng.choice(sorted(MIXES))
    if kind == "frame":
        return dict(kind=kind, w=size(64, 5000), h=size(64, 5000), form=form,
                    mix=mix, epf=rng.random() < 0.85,
                    gaborish=rng.choice([0, 1, 2, 2, 3, 4]),
                    hf=rng.random() < 0.85, srgb8=rng.random() < 0.4)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 24), lo=size(64, 256),
                    hi=size(300, 1536), form=form, mix=mix)
    if kind == "adjoint":
        return dict(kind=kind, w=size(64, 1536), h=size(64, 1024), form=form,
                    mix=mix)
    if kind == "dc":
        return dict(kind=kind, w=size(64, 4096), h=size(64, 4096))
    return dict(kind=kind, w=size(64, 2048), h=size(64, 1280), form=form,
                mix=mix)


# ---------------------------------------------------------------------------
# Inputs.


def _place(rng, acs, size, code, share):
    """Places `share` of the cells as aligned size x size transforms."""
    by, bx = acs.shape
    ny, nx = by // size, bx // size
    if not ny or not nx or share <= 0:
        return
    v = acs[:ny * size, :nx * size].reshape(ny, size, nx, size)
    free = np.flatnonzero((v == 0xFF).all(axis=(1, 3)))
    n = min(len(free), int(share * by * bx / size ** 2))
    pick = rng.choice(free, n, replace=False)
    y, x = pick // nx * size, pick % nx * size
    for i in range(size):
        for j in range(size):
            acs[y + i, x + j] = (code << 4) | (i * size + j)


def _first_cells(acs):
    """(y, x) of the first cell of the transform that covers each cell."""
    t, b = acs >> 4, (acs & 15).astype(np.int64)
    cov = np.where(t == 5, 4, np.where(t == 4, 2, 1))
    y, x = np.indices(acs.shape)
    return y - b // cov, x - b % cov


def _coarse(rng, shape, cell, amp):
    c = rng.normal(0.0, amp, (shape[0] // cell + 2, shape[1] // cell + 2))
    return np.repeat(np.repeat(c, cell, 0), cell, 1)[:shape[0], :shape[1]]


def _frame(w, h, seed, mix, epf=True, gaborish=2, hf=True):
    """A frame's side information (host) and its AC (device, int16)."""
    rng = np.random.default_rng([seed, w, h])
    by, bx = -(-h // 8), -(-w // 8)
    ty, tx = -(-h // 64), -(-w // 64)
    shares = dict(MIXES[mix])
    acs = np.full((by, bx), 0xFF, np.uint8)
    _place(rng, acs, 4, 5, shares.pop("DCT32X32", 0.0))
    _place(rng, acs, 2, 4, shares.pop("DCT16X16", 0.0))
    free = acs == 0xFF
    codes = np.array([layout.ACS_TYPES[k] << 4 for k in shares], np.uint8)
    p = np.array(list(shares.values()))
    cut = np.cumsum(p / p.sum())
    acs[free] = codes[np.minimum(np.searchsorted(cut, rng.random(free.sum())),
                                 len(codes) - 1)]
    # Quant field at distance 1: about 10 in flat regions (the 40% that the
    # adaptive filter smooths), about 21 in textured ones.
    flat = _coarse(rng, (by, bx), 8, 1.0) < -0.25
    qf = np.where(flat, 10.0, 21.0) / DISTANCE[mix] * np.exp(
        rng.normal(0.0, 0.08, (by, bx)))
    qf = np.clip(np.round(qf), 4, 64).astype(np.int32)
    fy, fx = _first_cells(acs)
    qf = qf[fy, fx]
    dc = np.empty((3, by, bx), np.int16)
    for c, (mean, sd) in enumerate(((-10., 20.), (240., 48.), (0., 27.))):
        v = mean + _coarse(rng, (by, bx), 16, 0.8 * sd) + rng.normal(
            0.0, 0.3 * sd, (by, bx))
        dc[c] = np.clip(np.round(v), -2000, 2000)
    # AC: sparse, its magnitude falling with the frequency in 8-point units;
    # 11% of the Y coefficients and under 1% of the others are non-zero at
    # distance 1.
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 7919 + w * 31 + h)
    a = torch.from_numpy(acs).to(DEV)
    cov = torch.ones_like(a, dtype=torch.int32)
    cov[(a >> 4) == 4] = 2
    cov[(a >> 4) == 5] = 4
    pos = (a & 15).int()[..., None] * 64 + torch.arange(64, device=DEV)
    n = 8 * cov[..., None]
    freq = (pos // n + pos % n).float() * (8.0 / n)
    ac = torch.empty((3, by, bx * 64), dtype=torch.int16, device=DEV)
    for c, amp in enumerate((0.5, 3.4, 0.45)):
        mean = (amp / DISTANCE[mix]) * torch.exp(freq * (-1 / 2.9))
        u = torch.rand(freq.shape, generator=g, device=DEV).clamp_min_(1e-12)
        mag = torch.floor(-torch.log(u) * mean)
        sign = torch.rand(freq.shape, generator=g, device=DEV) < 0.5
        v = torch.where(sign, mag, -mag).clamp_(-2000, 2000)
        ac[c] = v.reshape(by, bx * 64).to(torch.int16)
    f = layout.Frame(
        xsize=w, ysize=h, gaborish=gaborish, predict_lf=1, predict_hf=int(hf),
        have_ar=int(epf), epf_enable_adaptive=1, epf_sigma=0,
        epf_use_sharpened=0, global_scale=3065, quant_dc=16, ytox_dc=130,
        ytob_dc=120, ytox_map=rng.integers(98, 129, (ty, tx)).astype(np.int32),
        ytob_map=np.full((ty, tx), 120, np.int32), ac_strategy=acs,
        raw_quant_field=qf, ar_sigma_lut_ids=np.zeros((by, bx), np.uint8),
        quantized_dc=dc, quantized_ac=np.zeros((3, 1, 64), np.int16))
    return f, ac


def _case_frame(case, seed):
    return _frame(case["w"], case["h"], seed, case["mix"],
                  case.get("epf", True), case.get("gaborish", 2),
                  case.get("hf", True))


def _batch_sizes(case):
    rng = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    return [tuple(int(v) for v in rng.integers(case["lo"], case["hi"] + 1, 2))
            for _ in range(case["count"])]


def _target(f, seed):
    """The XYB image an encoder tunes towards: here the frame's own DC, one
    value per 8x8 block, with noise."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 104729 + 1)
    mul = torch.from_numpy(f.dequant_table[f.dequant_offsets.ravel()[:3]])
    mul = mul.double() * (65536 / f.global_scale / f.quant_dc)
    q = torch.from_numpy(f.quantized_dc).double() * mul[:, None, None]
    x = q[0] + q[1] * ((f.ytox_dc - 128) / 256)
    b = q[2] + q[1] * (f.ytob_dc / 128)
    t = torch.stack([x, q[1], b]).float().to(DEV)
    t = t.repeat_interleave(8, 1).repeat_interleave(8, 2)
    t = t[:, :f.ysize, :f.xsize].contiguous()
    noise = torch.randn(t.shape, generator=g, device=DEV)
    return t + 0.01 * noise


def _begin(ctx, f, ac):
    ctx.begin(f)
    ctx.set_ac_device(_planes(ac), ac.shape[2])


def _planes(ac):
    return [ac[c].data_ptr() for c in range(3)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dc":
        f, _ = _frame(case["w"], case["h"], seed, "d1")
        by, bx = f.blocks
        return dict(kind=kind, f=f, bx=bx, by=by,
                    q=torch.from_numpy(f.quantized_dc).to(DEV),
                    mul=f.dequant_table[f.dequant_offsets.ravel()[:3]],
                    out=torch.empty((3, by, bx), device=DEV))
    if kind == "batch":
        b = native.Batch(case["count"], form=case["form"])
        acs, outs = [], []
        for i, (w, h) in enumerate(_batch_sizes(case)):
            f, ac = _frame(w, h, seed * 1000 + i, case["mix"])
            _begin(b.frames[i], f, ac)
            acs.append(ac)
            outs.append(torch.empty((3, h, w), device=DEV))
        return dict(kind=kind, b=b, ac=acs, outs=outs,
                    ptrs=[o.data_ptr() for o in outs],
                    strides=[o.shape[2] for o in outs])
    f, ac = _case_frame(case, seed)
    ctx = native.Context(0, form=case["form"])
    s = dict(kind=kind, f=f, ac=ac, ctx=ctx, w=f.xsize,
             lin=torch.empty((3, f.ysize, f.xsize), device=DEV))
    if kind == "decode":
        f.quantized_ac = ac.cpu().numpy()
        return s
    _begin(ctx, f, ac)
    if kind == "frame":
        s["rgb"] = (torch.empty((f.ysize, f.xsize, 3), dtype=torch.uint8,
                                device=DEV) if case["srgb8"] else None)
    else:
        by, bx = f.blocks
        s.update(target=_target(f, seed),
                 loss=torch.empty(1, dtype=torch.float64, device=DEV),
                 g_ac=torch.empty((3, by, bx * 64), device=DEV),
                 g_qf=torch.empty((by, bx), device=DEV))
    return s


def run(s):
    kind = s["kind"]
    if kind == "frame":
        # The decoder hands over the frame's AC planes and reconstructs.
        ctx, rgb = s["ctx"], s["rgb"]
        ctx.set_ac_device(_planes(s["ac"]), s["ac"].shape[2])
        ctx.reconstruct_device(s["lin"].data_ptr(), s["w"],
                               rgb.data_ptr() if rgb is not None else 0,
                               3 * s["w"])
        return s["lin"] if rgb is None else (s["lin"], rgb)
    if kind == "batch":
        s["b"].reconstruct_device(s["ptrs"], s["strides"])
        return s["outs"]
    if kind == "adjoint":
        ctx = s["ctx"]
        ctx._check(ctx.L.pikgpu_adjoint(
            ctx.h, s["target"].data_ptr(), s["loss"].data_ptr(),
            s["g_ac"].data_ptr(), s["g_qf"].data_ptr(), 1))
        return s["loss"], s["g_ac"], s["g_qf"]
    if kind == "dc":
        f = s["f"]
        native.dc_reconstruct_noalloc(
            s["q"].data_ptr(), s["bx"], s["by"], f.global_scale, f.quant_dc,
            s["mul"], f.ytox_dc, f.ytob_dc, s["out"].data_ptr(),
            torch.cuda.current_stream().cuda_stream)
        return s["out"]
    # decode: a new image each time, as a decoder program meets them.
    ctx = s["ctx"]
    ctx.begin(s["f"])
    ctx.set_ac()
    ctx.reconstruct_device(s["lin"].data_ptr(), s["w"])
    ppm = ctx.encode_pnm(8)
    return s["lin"], np.frombuffer(ppm, np.uint8)


def work(case):
    """Bytes per pixel: 6 of int16 AC, 0.28 of DC and side information in;
    12 of linear RGB out (and 3 of sRGB). Operations: two separable
    transforms (32 multiply-adds a pixel and channel each way), and the
    filter's neighbourhood (56 neighbours: 12 differences and three
    multiply-adds per channel) on the share of the frame it filters."""
    kind = case["kind"]
    if kind == "dc":
        px = -(-case["w"] // 8) * -(-case["h"] // 8)
        return {"bytes": px * 3 * (2 + 4), "flops": px * 56 * 3 * 27}
    if kind == "batch":
        px = sum(w * h for w, h in _batch_sizes(case))
    else:
        px = case["w"] * case["h"]
    by, fl = 18.28, 3 * 2 * 32
    if case.get("epf", True):
        fl += 0.4 * (56 * 3 * 27 + 3 * 4 * 32)
    if case.get("srgb8"):
        by += 3
    if kind == "decode":
        by += 3
    if kind == "adjoint":  # target in; both gradients out; twice the work
        by, fl = 6.28 + 12 + 12 + 0.07, 2 * fl
    return {"bytes": px * by, "flops": px * fl}


# ---------------------------------------------------------------------------
# The result in 64 bits: a restatement in plain torch. The filter's integer
# decisions (guide bytes, sigma per block) are taken here again, from 64-bit
# values, so that a value on a rounding boundary may fall the other way.

LINES_P = [[6, 7, 15], [5, 14, 23], [40, 49, 58], [48, 56, 57],
           [4, 13, 22, 31], [3, 12, 30, 39], [24, 33, 51, 60],
           [32, 41, 50, 59], [2, 11, 20, 29, 38, 47],
           [1, 10, 19, 37, 46, 55], [8, 17, 26, 44, 53, 62],
           [16, 25, 34, 43, 52, 61], [0, 9, 18, 27, 36, 45, 54, 63]]
LINES_C = [[6, 7, 15], [5, 14, 23], [40, 49, 58], [48, 56, 57],
           [4, 13, 22, 31], [3, 12, 21, 30], [24, 33, 42, 51],
           [32, 41, 50, 59], [2, 11, 20, 29, 38, 47],
           [10, 19, 28, 37, 46, 55], [17, 26, 35, 44, 53, 62],
           [16, 25, 34, 43, 52, 61], [18, 27, 36, 45, 54, 39, 60, 63]]
LINES_DC = [[0, 8, 9, 16, 17, 18, 25, 26, 27, 34, 35, 36, 43, 44, 45, 52, 53,
             54, 61, 62, 63],
            [24, 32, 33, 40, 41, 42, 48, 49, 50, 51, 56, 57, 58, 59, 60],
            [3, 4, 5, 6, 7, 12, 13, 14, 15, 21, 22, 23, 30, 31, 39],
            [1, 2, 10, 11, 19, 20, 28, 29, 37, 38, 46, 47, 55]]
HADAMARD = np.array([[1, 1, 1, 1], [1, 1, -1, -1], [1, -1, 1, -1],
                     [1, -1, -1, 1]], float)
DC4 = [0, 1, 8, 9]


def _scales(n):
    k = np.arange(n)
    alpha = np.where(k == 0, math.sqrt(0.5), 1.0)
    i = math.sqrt(2 / n) * alpha * np.cos(k * math.pi / (2 * n))
    d = 1 / (n * i)
    return (d, i, alpha) if n == 8 else (i, d, alpha)


def _mats(n):
    """Inverse (pixel x frequency) and forward (frequency x pixel)."""
    d, i, alpha = _scales(n)
    k = np.arange(n)
    c = np.cos(np.outer(np.arange(n) + 0.5, k) * math.pi / n)
    s = n * math.sqrt(2 / n) * alpha
    return c * (s * d), (c * (s * i)).T / n


def _norms(n):
    v = []
    for k in range(n):
        p = 1.0
        if k not in (0, n // 2):
            tz = (k & -k).bit_length() - 1
            for j in range(int(math.log2(n)) - 1 - tz):
                p *= math.cos(math.pi / (1 << (j + 3)))
        v.append(p)
    return np.array(v)


def _total(n, m):
    """DCT total scale and its inverse, for m x m low frequencies."""
    d, i, _ = _scales(n)
    l1 = _norms(n)
    t, q = (d / l1)[:m], (i * l1)[:m]
    return n * np.outer(t, t), n * np.outer(q, q)


def _kron(m):
    """P = m C^T m^T on row-major vectors."""
    n = m.shape[0]
    return np.einsum("vl,uk->vukl", m, m).reshape(n * n, -1)


def _lf_forward(dctn, n):
    """2x2-cell values of a block -> its low frequencies."""
    _, f = _mats(n)
    return (_total(n, n)[0] * _total(dctn, n)[1]).ravel()[:, None] * _kron(f)


def _lf_inverse(dctn, lf, n):
    a, _ = _mats(n)
    keep = np.zeros((n, n))
    keep[:lf, :lf] = 1
    s = _total(n, n)[1] * _total(dctn, n)[0] * keep
    return _kron(a) * s.ravel()[None, :]


def _sub4(m):
    """The four interleaved 4x4 transforms: maps 64 -> 64 of DCT4X4 after
    (inverse) or before (forward) the Hadamard of the four DCs."""
    out = np.zeros((64, 64))
    for y in range(2):
        for x in range(2):
            px = [(4 * y + i) * 8 + 4 * x + j for i in range(4)
                  for j in range(4)]
            co = [(y + 2 * i) * 8 + x + 2 * j for i in range(4)
                  for j in range(4)]
            out[np.ix_(px, co)] = m
    return out


def _with_hadamard(m, scale, first):
    h = np.eye(64)
    h[np.ix_(DC4, DC4)] = HADAMARD * scale
    return m @ h if first else h @ m


def _t8(i):
    return (i & 7) * 8 + (i >> 3)


def _inverse8(t):
    if t in (0, 7):
        return _kron(_mats(8)[0])
    if t in (3, 8):
        return _with_hadamard(_sub4(_kron(_mats(4)[0])), 1.0, True)
    if t == 2:
        m = np.eye(64)
        for s in (2, 4, 8):
            h, step = s // 2, np.eye(64)
            for y in range(h):
                for x in range(h):
                    src = [y * 8 + x, y * 8 + h + x, (y + h) * 8 + x,
                           (y + h) * 8 + h + x]
                    dst = [2 * y * 8 + 2 * x, 2 * y * 8 + 2 * x + 1,
                           (2 * y + 1) * 8 + 2 * x,
                           (2 * y + 1) * 8 + 2 * x + 1]
                    step[dst] = 0
                    step[np.ix_(dst, src)] = HADAMARD
            m = step @ m
        return m
    if t == 1:
        m = np.zeros((64, 64))
        dc = np.zeros((4, 64))
        dc[:, DC4] = HADAMARD
        for y in range(2):
            for x in range(2):
                co = [[(y + 2 * i) * 8 + x + 2 * j for j in range(4)]
                      for i in range(4)]
                ctr = dc[2 * y + x].copy()
                for k in np.ravel(co)[1:]:
                    ctr[k] -= 1 / 16
                for i in range(4):
                    for j in range(4):
                        p = (4 * y + i) * 8 + 4 * x + j
                        m[p] = ctr
                        if (i, j) == (0, 0):
                            m[p, (y + 2) * 8 + x + 2] += 1
                        elif (i, j) != (1, 1):
                            m[p, co[i][j]] += 1
        return m
    m = np.zeros((64, 64))  # LINES
    for p, c in zip(LINES_P, LINES_C):
        n = len(p)
        for k in range(n):
            s = (1 / n if k == 0 else 2 / n) / _lines_fwd(n, k)
            for j in range(n):
                m[_t8(p[j]), _t8(c[k])] = s * math.cos(
                    k * (j + 0.5) * math.pi / n)
    signs = [[1, 1, 1, 1], [1, -1, 1, -1], [1, 1, -1, -1], [1, -1, -1, 1]]
    for region, sg in zip(LINES_DC, signs):
        for v in region:
            m[_t8(v), [0, 8, 1, 9]] += sg
    for p, a, b in ((21, 12, 30), (28, 19, 37), (35, 26, 44), (42, 33, 51)):
        m[p] = (m[a] + m[b]) / 2
    return m


def _lines_fwd(n, k):
    return 1 / n if k == 0 else 2 / n if n in (3, 6) else 2 / n / 2 ** 0.5


def _forward8(t):
    if t in (0, 7):
        return _kron(_mats(8)[1])
    if t in (3, 8):
        return _with_hadamard(_sub4(_kron(_mats(4)[1]).T).T, 0.25, False)
    if t == 2:
        return np.linalg.inv(_inverse8(2))
    if t == 1:
        m = np.zeros((64, 64))
        for y in range(2):
            for x in range(2):
                px = [(4 * y + i) * 8 + 4 * x + j for i in range(4)
                      for j in range(4)]
                for i in range(4):
                    for j in range(4):
                        c = (y + 2 * i) * 8 + x + 2 * j
                        src = px[0] if (i, j) == (1, 1) else px[4 * i + j]
                        if (i, j) == (0, 0):
                            m[c, px] = 1 / 16
                        else:
                            m[c, src] += 1
                            m[c, px[5]] -= 1
        return _with_hadamard(m, 0.25, False)
    m = np.zeros((64, 64))  # LINES
    res, dcs = np.eye(64), np.zeros((4, 64))
    for r, region in enumerate(LINES_DC):
        q = [_t8(v) for v in region]
        dcs[r, q] = 1 / len(q)
        res[np.ix_(q, q)] -= 1 / len(q)
    m[0] = dcs.sum(0) / 4
    m[8] = (dcs[0] - dcs[1] + dcs[2] - dcs[3]) / 4
    m[1] = (dcs[0] + dcs[1] - dcs[2] - dcs[3]) / 4
    m[9] = (dcs[0] - dcs[1] - dcs[2] + dcs[3]) / 4
    for p, c in zip(LINES_P, LINES_C):
        n = len(p)
        for k in range(n):
            m[_t8(c[k])] = sum(
                _lines_fwd(n, k) * math.cos(k * (j + 0.5) * math.pi / n) *
                res[_t8(p[j])] for j in range(n))
    return m


def _mirror(i, n):
    i = np.asarray(i) % (2 * n)
    return np.where(i < n, i, 2 * n - 1 - i)


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def _pad(img, n):
    h, w = img.shape[-2:]
    y = _t(_mirror(np.arange(-n, h + n), h))
    x = _t(_mirror(np.arange(-n, w + n), w))
    return img[..., y[:, None], x[None, :]]


def _sym3(img, w0, w1, w2):
    p = _pad(img, 1)
    v = p[..., :-2, :] + p[..., 2:, :]
    m = p[..., 1:-1, :]
    out = w0 * m[..., 1:-1]
    out = out + w1 * (v[..., 1:-1] + m[..., :-2] + m[..., 2:])
    return out + w2 * (v[..., :-2] + v[..., 2:])


def _gaborish(img, s):
    if not s:
        return img
    b1, b2 = ((0.056007960760453189, 0.045899074552453879) if s == 1 else
              (0.75 * 0.13959942428275746, 0.75 * 0.074240717189152386)
              if s == 2 else
              tuple(v * (0.875 if s == 3 else 1.0) for v in
                    (0.11501538179658321, 0.089979079587015454)))
    m = 1 / (1 + 4 * (b1 + b2))
    return _sym3(img, m, b1 * m, b2 * m)


def _weight_bits(mul, sad):
    t = np.minimum(sad, 507) * 64 * np.int64(mul)
    return ((t & 0xFFFF0000) + 0x3F800000).astype(np.uint32).view(np.float32)


def _mul_table():
    t = np.zeros(673, np.int32)
    mul = -32768
    for s in range(16, 673, 4):
        while mul < 0 and not _weight_bits(mul, np.array([s >> 2]))[0] > 0.5:
            mul += 1
        t[s] = mul
    for s in range(16, 672, 4):
        step = np.float32(t[s + 4] - t[s]) / np.float32(4)
        for i in range(1, 4):
            t[s + i] = int(np.float32(t[s]) + np.float32(i) * step)
    return t


SIGMA_LUT = np.array(
    [1.9815775622811198, 1.9715084740908622, 1.6819963065873933,
     1.2146133632942862, 1.0395364091521881, 0.93552327583169714,
     0.68568655651684773, 0.51174440217871964, 0.36397262821018583,
     0.31621830414136975, 0.30262954326557712, 0.246314237855494,
     0.21617524864418683, 0.10, 0.05, 0.0], np.float32)
AR_SCALE = np.ones(9, np.float32)
AR_SCALE[[5, 4, 3, 8, 2]] = [1.2282996852328099, 1.1423171621463439, 1.2, 1.2,
                             1.0098134203870499]


def _sigma(qf, acs, stretch):
    f32 = np.float32
    q = qf.astype(f32) * AR_SCALE[acs >> 4] * f32(0.039324273)
    pos = (q - f32(0.022156)) * f32(29.435892)
    i = np.clip(pos.astype(np.int64), 0, 14)
    fr = pos - i.astype(f32)
    u = fr * SIGMA_LUT[i + 1] + (f32(1) - fr) * SIGMA_LUT[i]
    u = np.where(q <= f32(0.022156), SIGMA_LUT[0],
                 np.where(q >= f32(0.531738), SIGMA_LUT[15], u))
    s = (u * f32(stretch) + f32(0.5182760822018414)).astype(np.int32)
    return np.minimum(s, 672)


def _epf(img, src, qf, acs):
    """The adaptive filter of `img` with the guide from `src`; the guide and
    the sigma are held fixed where a gradient is taken. Also returns which
    blocks it filters."""
    with torch.no_grad():
        lo, hi = float(src.min()), float(src.max())
        rng = np.float32(hi) - np.float32(lo)
        mul = 1.0 if rng == 0 else float(np.float32(255) / rng)
        sig = _sigma(qf, acs, np.float32(1) if rng == 0
                     else np.float32(255) / rng)
        g = ((_pad(src, 6) - lo) * mul).to(torch.int32) & 255
        g = g.to(torch.int16)
        table = _mul_table().astype(np.int64)
        px = _t(np.maximum(sig, 0)).repeat_interleave(8, 0)
        px = px.repeat_interleave(8, 1)
        m64 = _t(table * 64)[px].to(torch.int32)
        on = px >= 16
    h, w = img.shape[-2:]
    p = _pad(img, 6)
    num, den = torch.zeros_like(img), 0
    centre = g[:, 5:h + 7, 5:w + 8]
    for cy in range(-3, 4):
        for cx in range(-3, 5):
            with torch.no_grad():
                o = g[:, 5 + cy:h + 7 + cy, 5 + cx:w + 8 + cx]
                d = (centre - o).abs()
                r = d[:, :h] + d[:, 1:h + 1] + d[:, 2:h + 2]
                sad = (r[:, :, :w] + r[:, :, 1:w + 1] + r[:, :, 2:w + 2] +
                       r[:, :, 3:w + 3])
                sad = sad.amax(0).int().clamp_max(507)
                bits = ((sad * m64) & -65536) + 0x3F800000
                wt = bits.view(torch.float32)
                wt = torch.where(wt >= 0.05, wt, 0.0).double()
            num = num + wt * p[:, 6 + cy:h + 6 + cy, 6 + cx:w + 6 + cx]
            den = den + wt
    return torch.where(on, num / den, img), sig >= 16


class _Exact:
    """One frame in 64 bits. `ac`: the device's int16 AC."""

    def __init__(self, f, ac):
        self.f = f
        self.by, self.bx = f.blocks
        self.igs = 65536.0 / f.global_scale
        self.iqd = self.igs / f.quant_dc
        self.off = f.dequant_offsets.reshape(-1, 7, 3)
        self.table = _t(f.dequant_table.astype(np.float64))
        self.mul_dc = [float(f.dequant_table[self.off[0, 0, c]]) * self.iqd
                       for c in range(3)]
        self.first = {}  # type -> (y, x) of the first cells
        blk0 = (f.ac_strategy & 15) == 0
        for t in range(9):
            ys, xs = np.nonzero(blk0 & (f.ac_strategy >> 4 == t))
            if len(ys):
                self.first[t] = (_t(ys), _t(xs))
        self.kind = f.ac_strategy >> 4
        self.kind = np.where(self.kind == 7, 0,
                             np.where(self.kind == 8, 3, self.kind))
        self.qf = _t(f.raw_quant_field).double()
        self.q_ac = ac

    def matrix(self, c):
        """The dequantisation matrix of every cell (By, Bx, 64)."""
        o = self.off[0][self.kind, c].astype(np.int64)
        o = o + (self.f.ac_strategy & 15).astype(np.int64) * 64
        return self.table[_t(o)[..., None] + torch.arange(64, device=DEV)]

    def dc(self):
        f = self.f
        q = _t(f.quantized_dc).double()
        y = q[1] * self.mul_dc[1]
        dc = torch.stack([(f.ytox_dc - 128) / 256 * y + q[0] * self.mul_dc[0],
                          y, f.ytob_dc / 128 * y + q[2] * self.mul_dc[2]])
        ph, pw = -(-self.by // 8) * 8, -(-self.bx // 8) * 8
        iy = torch.arange(ph, device=DEV).clamp_max(self.by - 1)
        ix = torch.arange(pw, device=DEV).clamp_max(self.bx - 1)
        pad = dc[:, iy[:, None], ix[None, :]]
        z = np.zeros((ph // 8, pw // 8), np.int32)
        den, _ = _epf(pad, pad, z + f.quant_dc // 2, z)
        den = den[:, :self.by, :self.bx]
        half = torch.tensor(self.mul_dc, device=DEV,
                            dtype=torch.float64)[:, None, None] / 2
        return torch.maximum(dc - half, torch.minimum(den, dc + half))

    def dequant(self, qf):
        f, by, bx = self.f, self.by, self.bx
        ob = (0.05465007330715401, 0.07005449891748593, 0.049935103337343655)
        d = []
        for c in range(3):
            q = self.q_ac[c].reshape(by, bx, 64).double()
            a = torch.where(q.abs() >= 1.5,
                            q - 0.145 / torch.where(q == 0, 1.0, q),
                            torch.sign(q) * (1 - ob[c]))
            d.append(a * self.matrix(c) * (self.igs / qf)[..., None])

        def per_cell(m):
            m = np.repeat(np.repeat(m, 8, 0), 8, 1)[:by, :bx]
            return _t(m)[..., None]
        d[0] = d[0] + per_cell((f.ytox_map - 128) / 256) * d[1]
        d[2] = d[2] + per_cell(f.ytob_map / 128) * d[1]
        return torch.stack(d).reshape(3, by, bx * 64)

    def cells(self, t, per):
        """Index arrays of type t's blocks over an image of `per` x `per`
        values per cell: (n, cov per, 1) rows and (n, 1, cov per) columns."""
        ys, xs = self.first[t]
        a = torch.arange(layout.ACS_COVER[t] * per, device=DEV)
        return ((ys * per)[:, None, None] + a[None, :, None],
                (xs * per)[:, None, None] + a[None, None, :])

    def coef_index(self, t):
        ys, xs = self.first[t]
        cov = layout.ACS_COVER[t]
        r = ys[:, None, None] + torch.arange(cov, device=DEV)[None, :, None]
        q = (xs * 64)[:, None, None] + torch.arange(
            64 * cov, device=DEV)[None, None, :]
        return r, q

    def to_pixels(self, t, co):
        """(3, n, (8 cov)^2) coefficients -> (3, n, 8 cov, 8 cov)."""
        n = 8 * layout.ACS_COVER[t]
        if n == 8:
            return (co @ _t(_inverse8(t)).T).reshape(*co.shape[:2], 8, 8)
        a = _t(_mats(n)[0])
        return a @ co.reshape(*co.shape[:2], n, n).transpose(-1, -2) @ a.T

    def from_pixels(self, t, px):
        n = 8 * layout.ACS_COVER[t]
        if n == 8:
            return px.reshape(*px.shape[:2], 64) @ _t(_forward8(t)).T
        b = _t(_mats(n)[1])
        return (b @ px.transpose(-1, -2) @ b.T).reshape(*px.shape[:2], n * n)

    def lf(self, dc, ac):
        """LF prediction and update of `ac`; also the groups' pred2x2 as
        a list of (y0, x0, gys, gxs, image)."""
        f = self.f
        ac = ac.clone()
        preds = []
        up8 = _t(_lf_inverse(8, 1, 2)[:, :1])
        for y0 in range(0, self.by, 64):
            for x0 in range(0, self.bx, 64):
                gys, gxs = min(64, self.by - y0), min(64, self.bx - x0)
                g = dc[:, _t(_mirror(np.arange(y0 - 1, y0 + gys + 1),
                                     self.by))[:, None],
                       _t(_mirror(np.arange(x0 - 1, x0 + gxs + 1),
                                  self.bx))[None, :]]
                a = np.zeros((gys + 2, gxs + 2), np.uint8)
                a[1:-1, 1:-1] = f.ac_strategy[y0:y0 + gys, x0:x0 + gxs]
                llf = g.clone()
                tmp = torch.zeros((3, 2 * gys + 4, 2 * gxs + 4),
                                  dtype=torch.float64, device=DEV)
                blocks = []
                for t in range(9):
                    ys, xs = np.nonzero(a == t << 4)
                    if not len(ys):
                        continue
                    cov = layout.ACS_COVER[t]
                    ys, xs = _t(ys), _t(xs)

                    def idx(per):
                        k = torch.arange(cov * per, device=DEV)
                        return ((ys * per)[:, None, None] + k[None, :, None],
                                (xs * per)[:, None, None] + k[None, None, :])
                    i1, i2 = idx(1), idx(2)
                    blocks.append((t, cov, ys, xs, i1, i2))
                    v = g[:, i1[0], i1[1]].reshape(3, len(ys), cov * cov)
                    if cov > 1:
                        v = v @ _t(_lf_forward(8 * cov, cov)).T
                        m = np.zeros((2 * cov, 2 * cov), int)
                        m[:cov, :cov] = 1
                        up = _t(_lf_inverse(8 * cov, cov, 2 * cov)
                                [:, m.ravel() == 1])
                    else:
                        up = (up8 if t in (0, 6, 7) else
                              torch.ones_like(up8))
                    s = (3, len(ys), cov, cov)
                    llf[:, i1[0], i1[1]] = v.reshape(s)
                    s = (3, len(ys), 2 * cov, 2 * cov)
                    tmp[:, i2[0], i2[1]] = (v @ up.T).reshape(s)
                lf = _sym3(tmp, 0.41459272584128337, 0.25489157325704559,
                           0.046449679523692139)
                pred = torch.zeros_like(tmp)
                for t, cov, ys, xs, i1, i2 in blocks:
                    n2 = (2 * cov) ** 2
                    s = (3, len(ys), 2 * cov, 2 * cov)
                    if cov == 1 and t not in (0, 6, 7):
                        fw, inv = _t(HADAMARD / 4), _t(HADAMARD)
                    else:
                        fw = _t(_lf_forward(8 * cov, 2 * cov))
                        inv = _t(_lf_inverse(8 * cov, 2 * cov, 2 * cov))
                    v = lf[:, i2[0], i2[1]].reshape(3, len(ys), n2) @ fw.T
                    v = v.reshape(s)
                    corner = llf[:, i1[0], i1[1]]
                    # Ring cells predict from the DC alone, the group's own
                    # blocks from their updated low frequencies.
                    inner = ((ys > 0) & (xs > 0) & (ys <= gys) & (xs <= gxs))
                    k = (inner.nonzero()[:, 0])
                    by, bx = y0 + ys[k] - 1, x0 + xs[k] - 1
                    n = torch.arange(2 * cov, device=DEV)
                    lin = n[:, None] * (8 * cov) + n[None, :]
                    row = by[:, None, None] + (lin // (64 * cov))[None]
                    col = (bx * 64)[:, None, None] + (lin % (64 * cov))[None]
                    new = v.clone()
                    new[:, :, :cov, :cov] = corner
                    own = new[:, k] + torch.where(
                        ((n[:, None] < cov) & (n[None, :] < cov)), 0.0,
                        ac[:, row, col])
                    ac[:, row, col] = own
                    new = new.index_copy(1, k, own)
                    pred[:, i2[0], i2[1]] = (
                        new.reshape(3, len(ys), n2) @ inv.T).reshape(s)
                preds.append((y0, x0, gys, gxs, pred))
        return ac, preds

    def upsampled(self, preds):
        s = 2.0007879236394901
        k = np.exp(-np.arange(-4, 5) ** 2 / (2 * s * s))
        k /= k.sum()
        taps = np.zeros((3, 4))
        for i in range(4):
            taps[0, i] = k[:4 - i].sum()
            taps[1, i] = k[4 - i:8 - i].sum()
            taps[2, i] = k[8 - i:].sum()
        taps = _t(taps)
        rows = {}
        for y0, x0, gys, gxs, p in preds:
            p = p[:, 1:-1, 1:-1]
            v = sum(p[:, :, i:i + 2 * gxs, None] * taps[i] for i in range(3))
            v = v.reshape(3, 2 * gys + 2, 8 * gxs)
            v = sum(v[:, i:i + 2 * gys, None] * taps[i][:, None]
                    for i in range(3))
            rows.setdefault(y0, []).append(v.reshape(3, 8 * gys, 8 * gxs))
        return torch.cat([torch.cat(r, 2) for r in rows.values()], 1)

    def idct(self, ac, preds):
        f = self.f
        up = self.upsampled(preds) if f.predict_hf else None
        out = torch.zeros((3, 8 * self.by, 8 * self.bx), dtype=torch.float64,
                          device=DEV)
        for t in self.first:
            n, cov = 8 * layout.ACS_COVER[t], layout.ACS_COVER[t]
            r, q = self.coef_index(t)
            co = ac[:, r, q].reshape(3, len(r), n * n)
            py, px = self.cells(t, 8)
            if f.predict_hf and t in (0, 3, 4, 5):
                keep = torch.ones((n, n), dtype=torch.float64, device=DEV)
                keep[:2 * cov, :2 * cov] = 0
                co = co + self.from_pixels(t, up[:, py, px]) * keep.ravel()
            out[:, py, px] = self.to_pixels(t, co)
        return out

    def clamp(self, orig, filt, qf, active):
        """The correction of each filtered block, limited coefficient by
        coefficient to half a quantisation step."""
        out = orig.clone()
        for t, (ys, xs) in self.first.items():
            n, cov = 8 * layout.ACS_COVER[t], layout.ACS_COVER[t]
            cy = ys[:, None] + torch.arange(cov, device=DEV)
            cx = xs[:, None] + torch.arange(cov, device=DEV)
            on = active[cy[:, :, None], cx[:, None, :]].flatten(1).any(1)
            if not bool(on.any()):
                continue
            py, px = (v[on] for v in self.cells(t, 8))
            ys, xs = ys[on], xs[on]
            base = orig[:, py, px]
            b = self.from_pixels(t, filt[:, py, px] - base)
            ratio = torch.ones_like(b[0])
            for c in range(3):
                o = int(self.off[0][{7: 0, 8: 3}.get(t, t), c])
                step = self.table[o:o + n * n] * (self.igs / qf[ys, xs])[:, None]
                m = self.mul_dc[c]
                s = _t(_total(n, cov)[1] if cov > 1 else np.ones((1, 1))) * m
                k = torch.arange(cov, device=DEV)
                step = step.index_copy(
                    1, (k[:, None] * n + k[None, :]).ravel(),
                    s.reshape(1, -1).expand(len(ys), -1))
                lim = torch.minimum(torch.maximum(b[c], -step / 2), step / 2)
                zero = b[c] == 0
                r = torch.where(zero, 0.0, lim / torch.where(zero, 1.0, b[c]))
                ratio = torch.where(r < ratio, r, ratio)
            out[:, py, px] = base + self.to_pixels(t, b * ratio)
        return out

    def pre_opsin(self, ac, qf):
        f = self.f
        a, preds = self.lf(self.dc(), ac)
        px = self.idct(a, preds)
        if f.have_ar:
            filt, act = _epf(px, _gaborish(px, f.gaborish).detach(),
                             f.raw_quant_field, f.ac_strategy)
            px = self.clamp(px, filt, qf, _t(act))
        return _gaborish(px, f.gaborish)[:, :f.ysize, :f.xsize]

    def linear(self):
        v = self.pre_opsin(self.dequant(self.qf), self.qf)
        m = np.array([[0.29956550340058319, 0.63373087833825936,
                       0.077705617820981968],
                      [0.22158691104574774, 0.68491388044116142,
                       0.096254234043612538],
                      [0.20062661225219422, 0.070366199217588729,
                       0.5571760754215358]]) / 255
        bias = np.array([0.26786006338144885, 0.24494032763907073,
                         0.14255999980363571]) / 255
        g = torch.stack([v[1] + v[0], v[1] - v[0], v[2]]) ** 3
        g = g - _t(bias)[:, None, None]
        return torch.einsum("ij,jhw->ihw", _t(np.linalg.inv(m)), g)


def exact(case, seed):
    kind = case["kind"]
    if kind == "dc":
        f, ac = _frame(case["w"], case["h"], seed, "d1")
        return _Exact(f, ac).dc()
    if kind == "batch":
        outs = []
        for i, (w, h) in enumerate(_batch_sizes(case)):
            outs.append(_Exact(*_frame(w, h, seed * 1000 + i,
                                       case["mix"])).linear())
        return outs
    if case["w"] * case["h"] > 3e7:
        return None  # tens of gigabytes of 64-bit planes
    f, ac = _case_frame(case, seed)
    e = _Exact(f, ac)
    if kind == "frame":
        return (e.linear(), None) if case["srgb8"] else e.linear()
    if kind == "decode":
        return e.linear(), None
    d = e.dequant(e.qf).requires_grad_(True)
    rel = torch.ones_like(e.qf, requires_grad=True)  # qf / qf0
    per_coef = rel.repeat_interleave(64, 1)
    pre = e.pre_opsin(d / per_coef, e.qf * rel)
    loss = ((pre - _target(f, seed).double()) ** 2).sum()
    loss.backward()
    return (loss.detach().reshape(1), d.grad, rel.grad / e.qf)
