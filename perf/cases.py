"""Performance cases of the framework: what its users have it do, through its public entry points.

The kinds of work, each over a range of scanner sizes:

  osem         one frame already on the device: uniform start image, OSEM iterations, image back
               (the inner loop of every reconstruction; f32, bf16 and fp16 stored terms, the reference's
               and the exact-adjoint back projector, PSF and MAP)
  dynamic      the frames of a dynamic study in one batch, uneven iteration counts, every image back
  reconstruct  one frame from pinned host sinograms to the host image in one call
  pair         the function-level projector interface on host arrays (FP, BP, rotate-back of one view pair)
  pair_device  back projection of one view pair in device buffers, without allocation
  listmode     l64 words on the device to sinograms (a whole stream or one timed frame), and the span-9
               trues of a span-3 prompts + delayed histogram

Inputs are a water cylinder with six hot spheres (line integrals in closed form), attenuation, lognormal
normalisation, Gaussian scatter, flat randoms and Poisson prompts; listmode events follow the cylinder's
expected prompts.  `exact` restates the reconstruction in plain torch in 64 bits: the float32 sample
positions and interpolation weights of the scanner's tables, everything else in double.
"""
import ctypes
import math

import numpy as np
import torch

import hrrt_reconstruction_b200 as H
from hrrt_reconstruction_b200 import listmode_synth

STORAGE = {"f32": H.STORE_F32, "bf16": H.STORE_16, "f16": H.STORE_F16}
F = np.float32
_sinf = ctypes.CDLL("libm.so.6").sinf  # the C library's, as the program that made the tables calls it
_sinf.restype, _sinf.argtypes = ctypes.c_float, [ctypes.c_float]
MU_WATER = 0.0096  # /mm

# HRRT model 999 (the benchmark's scanner) and the small scanner of the tests
HRRT = dict(rings=104, bins=256, views=288, radius=234.5, maxdel=67, subsets=16)
SMALL = dict(rings=24, bins=64, views=96, radius=58.625, maxdel=13, subsets=16)


def _osem(name, scanner, span, storage="f32", adjoint=False, psf=False, map=False, iterations=1):
    return dict(name=name, kind="osem", **scanner, span=span, storage=storage, adjoint=adjoint, psf=psf, map=map,
                iterations=iterations)


def listed():
    return [
        # the benchmark's study: one pass over the 16 subsets at the scanner's full resolution
        _osem("osem_span3", HRRT, 3),
        # the routine span, with the 16-bit stored terms
        _osem("osem_span9_bf16", HRRT, 9, storage="bf16"),
        # the matched projector pair
        _osem("osem_span9_adjoint", HRRT, 9, adjoint=True),
        # resolution modelling (-B) with the one-step-late prior (-b 1,beta) from the fifth subset on
        _osem("osem_span9_psf_map", HRRT, 9, psf=True, map=True),
        # a small scanner, two iterations: launches and their gaps count
        _osem("osem_small_span3", SMALL, 3, iterations=2),
        # between the two, with sizes that fill no tile
        _osem("osem_ragged_span9", dict(rings=59, bins=148, views=160, radius=134.5, maxdel=38, subsets=10), 9,
              storage="f16"),
        # a short dynamic study
        dict(name="dynamic_span9_f16", kind="dynamic", **HRRT, span=9, storage="f16", frames=5),
        # file to image: upload, sensitivity and one iteration behind it
        dict(name="reconstruct_span9", kind="reconstruct", **HRRT, span=9, storage="f32", iterations=1),
        # a program that calls the projectors view by view, on the small scanner: the smallest calls
        dict(name="pair_small_span3", kind="pair", **SMALL, span=3),
        # a real-time loop back-projecting one view pair at a time
        dict(name="pair_device_span3", kind="pair_device", **HRRT, span=3),
        # a long frame: prompts and delayed at span 3, then the span-9 trues
        dict(name="listmode_span3_long", kind="listmode", span=3, events=100_000_000, per_ms=1000, duration=0,
             trues=False, fold=True),
        # a short timed frame of trues at span 9, cut by its time tags
        dict(name="listmode_span9_short", kind="listmode", span=9, events=1_000_000, per_ms=100, duration=7,
             trues=True, fold=False),
    ]


def _draw_scanner(rng, lo=0.25, hi=1.0):
    """A scanner between the small one and the HRRT, in proportion."""
    s = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    span = rng.choice([3, 3, 5, 7, 9, 9])
    rings = max(24 if span < 7 else 32, 4 * round(26 * s) - rng.choice([0, 1]))  # padded planes: whole groups of 8
    views = 16 * max(5, round(18 * s))
    subsets = rng.choice([n for n in (4, 6, 8, 9, 10, 12, 16, 18) if views % (2 * n) == 0])
    return dict(rings=rings, bins=4 * max(16, round(64 * s)), views=views, radius=round(234.5 * s, 3),
                maxdel=int(rings * 0.64), subsets=subsets, span=span)


def draw(rng):
    kind = rng.choice(["osem", "osem", "osem", "dynamic", "reconstruct", "pair", "pair_device", "listmode", "listmode"])
    if kind == "listmode":
        span = rng.choice([3, 9])
        events = int(math.exp(rng.uniform(math.log(3e4), math.log(1e8))))
        per_ms = rng.choice([50, 200, 1000])
        seconds = events // (per_ms * 1000)
        trues = rng.random() < 0.5
        return dict(kind=kind, span=span, events=events, per_ms=per_ms,
                    duration=rng.randint(1, seconds) if seconds > 1 and rng.random() < 0.5 else 0, trues=trues,
                    fold=span == 3 and not trues and rng.random() < 0.5)
    storage = rng.choice(["f32", "f32", "bf16", "f16"])
    if kind == "osem":
        adjoint = rng.random() < 0.2
        return dict(kind=kind, **_draw_scanner(rng, hi=0.8 if adjoint else 1.0), storage=storage, adjoint=adjoint,
                    psf=rng.random() < 0.2, map=rng.random() < 0.2, iterations=1)
    if kind == "dynamic":
        return dict(kind=kind, **_draw_scanner(rng, hi=0.6), storage=storage, frames=rng.randint(2, 6))
    if kind == "reconstruct":
        return dict(kind=kind, **_draw_scanner(rng, hi=0.6), storage=storage, iterations=rng.randint(1, 2))
    if kind == "pair":
        return dict(kind=kind, **_draw_scanner(rng, hi=0.5))
    return dict(kind=kind, **_draw_scanner(rng))


# ---------------------------------------------------------------------------
# The scanner's tables, in the single precision of the reference's program
# ---------------------------------------------------------------------------
class Scanner:
    def __init__(self, case):
        self.rings, self.N, self.V = case["rings"], case["bins"], case["views"]
        self.R, self.span, self.subsets = F(case["radius"]), case["span"], case["subsets"]
        size = F(1.21875)
        self.size, ring = size, F(2) * size
        self.nz = 2 * self.rings - 1
        self.zp = (self.nz + 3) // 4 * 4
        self.c = self.N // 2
        self.G = (case["maxdel"] - (self.span - 1) // 2) // self.span
        self.zs = self.span - 1
        self.z_min, self.z_max, self.npskip = 6, min(200, self.nz - 3), 3
        self.eps1, self.eps2, self.eps3, self.image_max = 5e-2, 1e-2, 1e-10, 1e4
        # segments 0, +1, -1, +2, ... as the files hold them: (first plane, last plane, offset)
        self.seg, off = [], 0
        for s in range(2 * self.G + 1):
            g = (s + 1) // 2
            lo = 0 if g == 0 else (self.span + 1) // 2 + (g - 1) * self.span
            hi = 2 * self.rings - 2 - lo
            self.seg.append((lo, hi, off))
            off += hi - lo + 1
        self.planes = off
        two_r = F(2) * self.R

        def angle(d):  # sine and cosine of an axial difference d (mm)
            t = np.sqrt(d * d + two_r * two_r)
            return d / t, two_r / t
        self.tan, self.rescale, self.bp_scale = [None], [None], [F(1) * self.span * ring / two_r]
        self.tan_bp = [None]
        for g in range(1, self.G + 1):
            sn, cs = angle(F(g * self.span) * ring)
            lo, hi, _ = self.seg[2 * g]
            n = hi - lo + 1
            t, r = np.full(n, sn / cs, F), np.full(n, size / abs(cs), F)
            for k in range(self.zs):
                mean_rd = self.span * g - (self.span - 1) // 2 + (k + 1) // 2
                v, u = angle(F(mean_rd) * ring)
                t[[k, n - 1 - k]] = v / u
                r[[k, n - 1 - k]] = size / abs(u)
            self.tan.append(t)  # per plane, of the segment with planes rising along the rotated rows
            self.rescale.append(r)
            self.tan_bp.append(sn / cs)
            self.bp_scale += [cs * cs * cs * F(self.span) * ring / two_r] * 2
        i = (np.arange(self.N) - self.c).astype(F)
        r2 = i[None, :] * size * i[None, :] * size + i[:, None] * size * i[:, None] * size
        fov = np.sqrt(r2) <= F(0.95) * size * F(self.N) / F(2)
        self.fov = fov  # [x][y]
        self.cyl0 = np.where(fov.any(1), fov.argmax(1), 0)
        self.cyl1 = np.where(fov.any(1), self.N - fov[:, ::-1].argmax(1), 0)
        half = self.V // 2
        v = np.arange(half)
        dpsi = F(math.pi) / F(self.V)
        self.sin = np.array([_sinf(float(F(k) * dpsi)) for k in v], F)
        self.sin[0] = 0
        self.cos = np.sqrt(1.0 - (self.sin * self.sin).astype(np.float64)).astype(F)

    def order(self):
        """The subset order: each time the remaining subset furthest from the last."""
        S, done = self.subsets, [0]
        while len(done) < S:
            best, far = 0, 0
            for j in range(S):
                d = min(abs(j - done[-1]), S - abs(j - done[-1]))
                if j not in done and d > far:
                    best, far = j, d
            done.append(best)
        return done

    def views(self, subset):
        return [subset + self.subsets * k for k in range(self.V // self.subsets // 2)]

    def geometry(self):
        return H.hrrt_geometry(span=self.span, nrings=self.rings, nelements=self.N, nangles=self.V,
                               ring_radius=float(self.R), plane_sep=1.21875, binsize=1.21875,
                               maxdel=self.G * self.span + (self.span - 1) // 2, subsets=self.subsets)

    @property
    def shape(self):
        return self.planes, self.V, self.N


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _chords(sc, radius, centre, out, gain):
    """out += gain * the length of every line of response inside a sphere (finite `centre` z) or a z cylinder
    (centre None), mm; flat-file layout on the device."""
    dev, size = out.device, float(sc.size)
    psi = torch.arange(sc.V, device=dev, dtype=torch.float32) * (math.pi / sc.V)
    u = (torch.arange(sc.N, device=dev, dtype=torch.float32) - sc.c) * size
    x, y = (0.0, 0.0) if centre is None else (float(centre[0]), float(centre[1]))
    du = u[None, :] - (x * torch.cos(psi) + y * torch.sin(psi))[:, None]
    w = -x * torch.sin(psi) + y * torch.cos(psi)
    for s, (lo, hi, off) in enumerate(sc.seg):
        g = (s + 1) // 2
        t = 0.0 if g == 0 else float(sc.tan_bp[g]) * (-1.0 if s % 2 else 1.0)
        cos2 = 1.0 / (1.0 + t * t)
        z = (torch.arange(lo, hi + 1, device=dev, dtype=torch.float32) - (sc.nz - 1) / 2) * size
        block = out[off:off + hi - lo + 1]
        if centre is None:
            length = 2.0 * (radius * radius - du * du).clamp_(min=0).sqrt() / math.sqrt(cos2)
            inside = (z.abs() <= radius).float()
            block += gain * inside[:, None, None] * length[None]
        else:
            dz = float(centre[2]) - (z[:, None, None] + (w * t)[None, :, None])
            block += gain * 2.0 * (radius * radius - (du * du)[None] - dz * dz * cos2).clamp_(min=0).sqrt()


def _study(sc, seed, device, counts_per_bin=0.64, sphere_gain=3.0, shared=None):
    """Device sinograms of one frame: prompts int16, randoms, norm, atten, scatter float32.  `shared`: the
    norm and attenuation of the study's earlier frames."""
    gen = torch.Generator(device=device)
    gen.manual_seed(int(seed))
    rng = np.random.default_rng(seed)
    s = sc.N * float(sc.size) / 312.0  # the phantom scaled to the bore
    zl = min(100.0 * s, 0.42 * sc.nz * float(sc.size))
    trues = torch.zeros(sc.shape, device=device)
    _chords(sc, 100.0 * s, None, trues, 1.0)
    if shared is None:
        atten = torch.exp_(MU_WATER * trues)
        norm = torch.empty(sc.shape, device=device).normal_(generator=gen).mul_(0.1).exp_()
    else:
        norm, atten = shared
    for r in (5.0, 7.5, 10.0, 12.5, 15.0, 18.0):
        rho, phi = 70.0 * s * math.sqrt(rng.random()), 2 * math.pi * rng.random()
        _chords(sc, r * s, (rho * math.cos(phi), rho * math.sin(phi), (2 * rng.random() - 1) * 0.8 * zl), trues,
                sphere_gain)
    trues /= norm * atten
    k = counts_per_bin * trues.numel() / 1.5 / float(trues.sum(dtype=torch.float64))
    trues *= k
    u = (torch.arange(sc.N, device=device) - sc.N / 2) / (sc.N / 4)
    scatter = (0.15 * float(trues.mean(dtype=torch.float64)) * 1.6) * torch.exp(-0.5 * u * u)
    scatter = scatter.expand(sc.shape).contiguous()
    randoms = torch.full(sc.shape, 0.25 * counts_per_bin, device=device)
    mean = trues.add_(randoms).add_(scatter / norm)
    prompts = torch.poisson(mean, generator=gen).clamp_(max=32767).to(torch.int16)
    return dict(prompts=prompts, randoms=randoms, norm=norm, atten=atten, scatter=scatter)


_pool = {}


def _host(tensors, keep=False):
    """Pinned host copies (numpy); of a pool that the next call overwrites unless `keep`."""
    out = {}
    for name, t in tensors.items():
        if keep:
            h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
        else:
            if name not in _pool or _pool[name].numel() < t.numel():
                _pool[name] = torch.empty(t.numel(), dtype=t.dtype, pin_memory=True)
            h = _pool[name][:t.numel()].view(t.shape)
        h.copy_(t)
        out[name] = h.numpy()
    return out


def _image_out(sc):
    return torch.empty((sc.nz, sc.N, sc.N), dtype=torch.float32, pin_memory=True).numpy()


def _pair_inputs(sc, seed):
    rng = np.random.default_rng(seed)
    img = rng.random((sc.N, sc.N, sc.zp), dtype=F) + F(0.5)
    img *= sc.fov[:, :, None]
    img[:, :, sc.nz:] = 0
    rows = rng.random((2 * sc.planes, sc.N), dtype=F) * F(2)
    rows[:, 0] = 0
    corr = rng.random((sc.N, sc.N, sc.zp), dtype=F) * sc.fov[:, :, None]
    return dict(image=img, rows=rows, corr=corr.astype(F), view=int(rng.integers(0, sc.V // 2)))


_streams = []


def _stream():
    """The program's own stream for the calls on device buffers."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


BETA = 0.004  # MAP: of the sensitivity of an unattenuated line (far from where the update divides by nothing)


def _frames(case):
    """Counts a bin and iterations of a dynamic study's frames: short early ones, long late ones."""
    n = case["frames"]
    return [(0.01 * 60.0 ** (f / max(n - 1, 1)), 1 + f % 3) for f in range(n)]


def prepare(case, seed):
    dev = torch.device("cuda")
    kind = case["kind"]
    if kind == "listmode":
        words = _words(case, seed, dev)
        lm = H.Listmode(case["span"])
        n = lm.sino_size
        sino = torch.zeros(n, dtype=torch.int16, device=dev)
        delayed = None if case["trues"] else torch.zeros(n, dtype=torch.int16, device=dev)
        fold = torch.zeros(2209 * 288 * 256, dtype=torch.int16, device=dev) if case["fold"] else None
        return dict(case=case, lm=lm, words=words, sino=sino, delayed=delayed, fold=fold, stream=_stream())
    sc = Scanner(case)
    ctx = H.Context(sc.geometry())
    assert ctx.sino_shape == sc.shape and ctx.image_shape == (sc.N, sc.N, sc.zp)
    st = dict(case=case, ctx=ctx)
    if kind == "pair":
        return st | _pair_inputs(sc, seed)
    if kind == "pair_device":
        inp = _pair_inputs(sc, seed)
        rows = torch.from_numpy(inp["rows"]).to(dev)
        return st | dict(rows=rows, out=torch.empty(ctx.image_shape, device=dev), view=inp["view"], stream=_stream())
    if kind == "dynamic":
        first, batch, shared = None, None, None
        for f, (counts, iterations) in enumerate(_frames(case)):
            t = _study(sc, seed * 100 + f, dev, counts_per_bin=counts, sphere_gain=1.0 + f, shared=shared)
            shared = shared or (t["norm"], t["atten"])
            h = _host(t)
            if batch is None:
                batch = ctx.batch(case["frames"], norm=h["norm"], atten=h["atten"], storage=STORAGE[case["storage"]])
            batch.set_frame(f, h["prompts"], h["randoms"], h["scatter"], iterations)
        return st | dict(batch=batch, out=[_image_out(sc) for _ in range(case["frames"])])
    t = _study(sc, seed, dev)
    if kind == "reconstruct":
        return st | _host(t, keep=True) | dict(out=_image_out(sc))
    h = _host(t)
    if case["adjoint"]:
        ctx.set_backprojector(H.BP_ADJOINT)
    if case["psf"]:
        ctx.set_psf(True)
    ctx.upload_inputs(h["prompts"], h["randoms"], h["norm"], h["atten"], h["scatter"], storage=STORAGE[case["storage"]])
    ctx.sensitivity()
    if case["map"]:
        ctx.set_map(1, _beta(sc, case), 5)
    return st | dict(out=_image_out(sc))


def _beta(sc, case):
    """The prior's weight against a sensitivity of the size this scanner has."""
    samples = sc.V / sc.subsets * sum((hi - lo + 1) / sc.nz for lo, hi, _ in sc.seg)
    return BETA * 0.5 * samples * (1.0 if case["adjoint"] else float(sc.bp_scale[0]))


def _words(case, seed, dev):
    hrrt = Scanner(dict(HRRT, span=3))
    e = torch.zeros((hrrt.planes, 1, 256), device=dev)
    u = (torch.arange(256, device=dev) - 128) * 1.21875
    length = 2 * (100.0 ** 2 - u * u).clamp(min=0).sqrt()
    shape = length * torch.exp(-MU_WATER * length)
    for lo, hi, off in hrrt.seg:
        z = (torch.arange(lo, hi + 1, device=dev) - 103) * 1.21875
        e[off:off + hi - lo + 1, 0] = (z.abs() <= 100).float()[:, None] * shape[None]
    e += 0.25 * e.mean()
    e = e.expand(hrrt.planes, 288, 256)
    if case["span"] == 9:
        # the acceptance weights are looked up in the span that the words are histogrammed in
        nine = Scanner(dict(HRRT, span=9))
        e = e[:1].amax().expand(1, 1, 1) * torch.ones((nine.planes, 1, 256), device=dev) * shape / shape.max()
        e = (e + 0.25 * e.mean()).expand(nine.planes, 288, 256)
    return listmode_synth.synth_words(case["events"], e, seed=seed, span=case["span"], events_per_ms=case["per_ms"],
                                      chunk=1 << 24, device=dev)


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "osem":
        ctx = st["ctx"]
        ctx.init_image()
        stats = ctx.osem(case["iterations"])
        return [ctx.get_image(out=st["out"]), stats.sum_image]
    if kind == "dynamic":
        st["batch"].run()
        return [st["batch"].get_image(f, out=st["out"][f])[0] for f in range(case["frames"])]
    if kind == "reconstruct":
        out, stats = st["ctx"].reconstruct(st["prompts"], st["randoms"], st["norm"], st["atten"], st["scatter"],
                                           storage=STORAGE[case["storage"]], iterations=case["iterations"],
                                           out=st["out"])
        return [out, stats.sum_image]
    if kind == "pair":
        ctx, view = st["ctx"], st["view"]
        fp = ctx.fp_pair(st["image"], view)
        bp = ctx.bp_pair(st["rows"], view)
        return [fp, bp, ctx.rotate_add(bp, view, st["corr"])]
    stream = st["stream"]
    if kind == "pair_device":
        rc = H.lib.hrrt_bp_pair_noalloc(st["ctx"]._h, ctypes.c_void_p(st["rows"].data_ptr()), st["view"],
                                        ctypes.c_void_p(st["out"].data_ptr()), ctypes.c_void_p(stream.cuda_stream))
        if rc != 0:
            raise H.HrrtError(f"bp_pair_noalloc: {rc}")
        return st["out"]
    lm, words, delayed = st["lm"], st["words"], st["delayed"]
    with torch.cuda.stream(stream):
        st["sino"].zero_()
        if delayed is not None:
            delayed.zero_()
    lm.reset_clock()
    stats = lm.histogram_device(words.data_ptr(), words.numel(), st["sino"].data_ptr(),
                                delayed.data_ptr() if delayed is not None else None,
                                mode=H.LM_TRUES if case["trues"] else H.LM_PROMPTS_AND_DELAYED,
                                duration=case["duration"], stream=stream.cuda_stream)
    out = [st["sino"], {k: v for k, v in stats.items() if k != "ms"}]
    if delayed is not None:
        out.append(delayed)
    if st["fold"] is not None:
        lm.trues_span9_device(st["sino"].data_ptr(), delayed.data_ptr(), st["fold"].data_ptr(),
                              stream=stream.cuda_stream)
        out.append(st["fold"])
    return out


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "listmode":
        planes = 6367 if case["span"] == 3 else 2209
        sinos = 1 if case["trues"] else 2
        words = 2 * (case["events"] + case["events"] // case["per_ms"])
        if case["duration"]:
            words = min(words, 2 * case["duration"] * 1000 * (case["per_ms"] + 1))
        b = 4 * words + 2 * sinos * planes * 288 * 256
        if case["fold"]:
            b += 2 * 2209 * 288 * 256
        return {"bytes": b, "flops": 12 * case["events"]}
    sc = Scanner(case)
    bins = sc.planes * sc.V * sc.N
    vol = 4 * sc.N * sc.N * sc.nz
    # every FOV column of every view meets every plane once, a linear interpolation each way
    samples = sc.V * sc.planes * int(sc.fov.sum())
    if kind in ("pair", "pair_device"):
        rows = 4 * 2 * sc.planes * sc.N
        one = 4 * samples * 2 / sc.V
        if kind == "pair_device":
            return {"bytes": rows + vol, "flops": one}
        return {"bytes": 2 * rows + 5 * vol, "flops": 2 * one + 8 * vol / 4}
    term = 4 if case["storage"] == "f32" else 2
    if kind == "dynamic":
        total = sum(it for _, it in _frames(case))
        return {"bytes": bins * (2 + term) * total + vol * (sc.subsets + 2 * case["frames"]), "flops": 8 * samples * total}
    it = case["iterations"]
    if kind == "reconstruct":
        # the inputs come over the host link once; the sensitivity is a back projection of every view
        return {"bytes": bins * 18 + vol, "flops": 8 * samples * it + 4 * samples}
    flops = 8 * samples * it
    if case["psf"]:
        flops += it * sc.subsets * 2 * 3 * 13 * 2 * vol / 4
    if case["map"]:
        flops += it * sc.subsets * 18 * 20 * vol / 4
    return {"bytes": it * (bins * (2 + term) + vol * sc.subsets) + 2 * vol, "flops": flops}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
class Exact:
    """The projectors as matrices over (rotated row, plane), applied to every column quad of a set of view
    pairs at once."""

    def __init__(self, sc, dev):
        self.sc, self.dev = sc, dev
        c, nz, zp, zs = sc.c, sc.nz, sc.zp, sc.zs
        self.rows = np.arange(1, c)  # rotated rows below the centre; row N - y mirrors row y
        self.fp, self.bp = [None], [None]
        Y = len(self.rows)
        for g in range(1, sc.G + 1):
            lo, hi, _ = sc.seg[2 * g]
            n = hi - lo + 1
            w1, w2 = torch.zeros((n, Y, zp), dtype=torch.float64), torch.zeros((n, Y, zp), dtype=torch.float64)
            e1, e2 = torch.zeros((n, Y, zp), dtype=torch.float64), torch.zeros((n, Y, zp), dtype=torch.float64)
            a = np.arange(n)
            for yi, y in enumerate(self.rows):
                # forward: per plane the positions on row y and on its mirror, in single precision; the middle
                # planes take the position of the first of them
                near = (a + lo).astype(F) + F(y - c) * sc.tan[g]
                far = (a + lo).astype(F) + F(c - y) * sc.tan[g]
                z1, z2 = near.astype(np.int64), far.astype(np.int64)
                f1, f2 = near - z1.astype(F), far - z2.astype(F)
                if z1[0] >= 0 and z2[n - 1] <= nz - 1:
                    mid = slice(zs, n - zs)
                    z1[mid], z2[mid] = z1[zs] + a[mid] - zs, z2[zs] + a[mid] - zs
                    f1[mid], f2[mid] = f1[zs], f2[zs]
                    for w, z, fa, fb in ((w1, z1, f2, f1), (w2, z2, f1, f2)):
                        # sample z takes the other side's fraction, sample z + 1 its own
                        for dz, f in ((0, fa), (1, fb)):
                            k = z + dz < zp
                            w[a[k], yi, z[k] + dz] += torch.from_numpy(f[k].astype(np.float64))
                # backward: voxel plane z reads the segment at z + shift, row y (e1) and its mirror (e2)
                for e, yy in ((e1, y), (e2, sc.N - y)):
                    u = -F(yy - c) * sc.tan_bp[g]
                    shift = int(np.floor(u))
                    f = abs(u) - F(int(abs(u)))
                    f = float(F(1) - f) if u < 0 else float(f)
                    if u < 0:
                        shift = -int(abs(u)) - 1
                    for dz, wt in ((0, 1.0 - f), (1, f)):
                        z = a + lo - shift - dz
                        k = (z >= 0) & (z < nz)
                        e[a[k], yi, z[k]] += wt
            self.fp.append([w.reshape(n, Y * zp).to(dev) for w in (w1, w2)])
            self.bp.append([e.reshape(n, Y * zp).to(dev) for e in (e1, e2)])
        self.xs = np.arange(1, c + 1)
        ok = (self.rows[None, :] >= sc.cyl0[self.xs][:, None]) & (sc.cyl0 != sc.cyl1)[self.xs][:, None]
        self.ok = torch.from_numpy(ok).to(dev)  # [x][row]
        self.okc = torch.from_numpy((sc.cyl0 != sc.cyl1)[self.xs]).to(dev)
        self.fov = torch.from_numpy(sc.fov).to(dev)

    def _points(self, views, a, b):
        """Corner columns and weights of rotated-grid points (a, b), every view: [view, *a.shape]."""
        sc = self.sc
        cs, sn = (v[np.asarray(views)].reshape((-1,) + (1,) * a.ndim) for v in (sc.cos, sc.sin))
        fa, fb, fc = (a - sc.c).astype(F)[None], (b - sc.c).astype(F)[None], F(sc.c)
        x = fa * cs - fb * sn + fc
        y = fa * sn + fb * cs + fc
        out = (x < 0) | (x > F(sc.N - 2)) | (y < 0)
        ix, iy = np.where(out, 0, x).astype(np.int64), np.where(out, 0, y).astype(np.int64)
        out |= (ix + 1) * sc.N + iy + 1 >= sc.N * sc.N
        x1, y1 = (x - ix).astype(np.float64), (y - iy).astype(np.float64)
        base = np.where(out, 0, ix * sc.N + iy)
        w = np.stack([(1 - x1) * (1 - y1), x1 * (1 - y1), y1 * (1 - x1), y1 * x1]) * ~out
        idx = np.stack([base, base + sc.N, base + 1, base + sc.N + 1]) * ~out
        return torch.from_numpy(idx).to(self.dev), torch.from_numpy(w).to(self.dev)

    def _sample(self, img, views, a, b):
        idx, w = self._points(views, a, b)
        return sum(img[idx[k]] * w[k][..., None] for k in range(4))

    def _lanes(self):
        x, y = np.broadcast_arrays(self.xs[:, None], self.rows[None, :])
        N = self.sc.N
        near = [(x, y), (N - x, y), (N - y, x), (N - y, N - x)]
        far = [(x, N - y), (N - x, N - y), (y, x), (y, N - x)]
        cx = self.xs
        cc = np.full_like(cx, self.sc.c)
        return near, far, [(cx, cc), (N - cx, cc), (cc, cx), (cc, N - cx)]

    def forward(self, img, views):
        """[pair][x][4 lanes][plane] estimates of an [N][N][zp] image."""
        sc = self.sc
        img = img.reshape(sc.N * sc.N, sc.zp)
        near, far, mid = self._lanes()
        P, X, Y = len(views), len(self.xs), len(self.rows)
        T = [torch.empty((P, X, 4, Y, sc.zp), dtype=torch.float64, device=self.dev) for _ in range(2)]
        C = torch.empty((P, X, 4, sc.zp), dtype=torch.float64, device=self.dev)
        for l in range(4):
            T[0][:, :, l] = self._sample(img, views, *near[l]) * self.ok[None, :, :, None]
            T[1][:, :, l] = self._sample(img, views, *far[l]) * self.ok[None, :, :, None]
            C[:, :, l] = self._sample(img, views, *mid[l])
        out = torch.empty((P, X, 4, sc.planes), dtype=torch.float64, device=self.dev)
        out[..., :sc.nz] = ((T[0].sum(3) + T[1].sum(3) + C) * float(sc.size))[..., :sc.nz]
        T = [t.view(P * X * 4, Y * sc.zp) for t in T]
        for g in range(1, sc.G + 1):
            w1, w2 = self.fp[g]
            scale = torch.from_numpy(sc.rescale[g].astype(np.float64)).to(self.dev)
            for s, (t1, t2) in ((2 * g, T), (2 * g - 1, T[::-1])):
                lo, hi, off = sc.seg[s]
                v = (t1 @ w1.T + t2 @ w2.T).view(P, X, 4, -1)
                out[..., off:off + hi - lo + 1] = (v + C[..., lo:hi + 1]) * scale
        return out * self.okc[None, :, None, None]

    def _unquad(self, q):
        """The bin a quad's lanes 1 and 3 share with 0 and 2 at the centre counts once."""
        q = q.clone()
        if self.xs[-1] == self.sc.c:
            q[:, -1, 1::2] = 0
        return q * self.okc[None, :, None, None]

    def adjoint(self, q, views):
        """The transpose of forward: [N][N][zp] from [pair][x][4][plane]."""
        sc = self.sc
        q = self._unquad(q)
        P, X, Y = len(views), len(self.xs), len(self.rows)
        q0 = q[..., :sc.nz] * float(sc.size)
        T = [torch.zeros((P * X * 4, Y, sc.zp), dtype=torch.float64, device=self.dev) for _ in range(2)]
        C = torch.zeros((P, X, 4, sc.zp), dtype=torch.float64, device=self.dev)
        for t in T:
            t[..., :sc.nz] += q0.reshape(-1, 1, sc.nz)
        C[..., :sc.nz] += q0
        for g in range(1, sc.G + 1):
            scale = torch.from_numpy(sc.rescale[g].astype(np.float64)).to(self.dev)
            for s, (t1, t2) in ((2 * g, T), (2 * g - 1, T[::-1])):
                lo, hi, off = sc.seg[s]
                v = (q[..., off:off + hi - lo + 1] * scale)
                C[..., lo:hi + 1] += v
                v = v.reshape(P * X * 4, -1)
                t1.view(P * X * 4, -1).addmm_(v, self.fp[g][0])
                t2.view(P * X * 4, -1).addmm_(v, self.fp[g][1])
        near, far, mid = self._lanes()
        img = torch.zeros((sc.N * sc.N, sc.zp), dtype=torch.float64, device=self.dev)

        def back(points, values):
            idx, w = self._points(views, *points)
            for k in range(4):
                img.index_add_(0, idx[k].reshape(-1), (values * w[k][..., None]).reshape(-1, sc.zp))
        for l in range(4):
            for t, pts in zip(T, (near, far)):
                back(pts[l], t.view(P, X, 4, Y, sc.zp)[:, :, l] * self.ok[None, :, :, None])
            back(mid[l], C[:, :, l] * self.okc[None, :, None])
        img[:, sc.nz:] = 0
        return img.view(sc.N, sc.N, sc.zp)

    def backward(self, q, views):
        """The voxel-driven back projection into the rotated frame of every pair: [pair][N][N][zp]."""
        sc, N, c = self.sc, self.sc.N, self.sc.c
        q = q * self.okc[None, :, None, None]
        P, X, Y = len(views), len(self.xs), len(self.rows)
        S = [torch.zeros((P * X * 4, Y, sc.zp), dtype=torch.float64, device=self.dev) for _ in range(2)]
        M = torch.zeros((P, X, 4, sc.zp), dtype=torch.float64, device=self.dev)
        M[..., :sc.nz] = q[..., :sc.nz]
        for s in S:
            s[..., :sc.nz] += q[..., :sc.nz].reshape(-1, 1, sc.nz)
        for g in range(1, sc.G + 1):
            for s, (s1, s2) in ((2 * g, S), (2 * g - 1, S[::-1])):
                lo, hi, off = sc.seg[s]
                v = q[..., off:off + hi - lo + 1]
                M[..., lo:hi + 1] += v
                v = v.reshape(P * X * 4, -1)
                s1.view(P * X * 4, -1).addmm_(v, self.bp[g][0])
                s2.view(P * X * 4, -1).addmm_(v, self.bp[g][1])
        out = torch.zeros((P, N, N, sc.zp), dtype=torch.float64, device=self.dev)
        near, far, mid = self._lanes()
        for l in range(4):
            x = slice(0, X - 1) if l % 2 and self.xs[-1] == c else slice(0, X)
            for s, pts in zip(S, (near, far)):
                a, b = (torch.from_numpy(np.ascontiguousarray(i[x])).to(self.dev) for i in pts[l])
                out[:, a, b] += s.view(P, X, 4, Y, sc.zp)[:, x, l] * self.ok[None, x, :, None]
            a, b = (torch.from_numpy(np.ascontiguousarray(i[x])).to(self.dev) for i in mid[l])
            out[:, a, b] += M[:, x, l]
        return out

    def rotate(self, buf, view):
        """The rotate-back of one pair's [N][N][zp] frame."""
        sc, N = self.sc, self.sc.N
        cs, sn, h = sc.cos[view], F(-sc.sin[view]), F(N // 2)
        x0 = F(-N / 2) * cs + h * sn + h
        y0 = F(-N / 2) * sn - h * cs + h
        X, ys = np.arange(N).astype(F), sc.cyl0.astype(F)
        px, py = x0 - ys * sn + X * cs, y0 + ys * cs + X * sn
        ax, ay = np.zeros((N, N), F), np.zeros((N, N), F)
        for k in range(N):  # the positions step along y in single precision
            y = sc.cyl0 + k
            m = y < sc.cyl1
            ax[np.arange(N)[m], y[m]], ay[np.arange(N)[m], y[m]] = px[m], py[m]
            px, py = px - sn, py + cs
        ix, iy = ax.astype(np.int64), ay.astype(np.int64)
        out = (ix < 0) | (ix > N - 2) | (iy < 0) | (iy > N - 2) | ~sc.fov
        ix, iy = np.where(out, 0, ix), np.where(out, 0, iy)
        x1, y1 = (ax - ix.astype(F)).astype(np.float64) * ~out, (ay - iy.astype(F)).astype(np.float64) * ~out
        buf = buf.reshape(N * N, sc.zp)
        res = 0
        for dx, dy, w in ((0, 0, (1 - x1) * (1 - y1)), (1, 0, x1 * (1 - y1)), (0, 1, y1 * (1 - x1)), (1, 1, y1 * x1)):
            i = torch.from_numpy(((ix + dx) * N + iy + dy) * ~out).to(self.dev)
            res = res + buf[i] * torch.from_numpy(w * ~out).to(self.dev)[..., None]
        return res

    def correct(self, q, views, adjoint):
        """The correction image of a subset's quads (segment weights applied here for the reference's)."""
        if adjoint:
            return self.adjoint(q, views)
        sc = self.sc
        weight = torch.empty(sc.planes, dtype=torch.float64, device=self.dev)
        for s, (lo, hi, off) in enumerate(sc.seg):
            weight[off:off + hi - lo + 1] = float(sc.bp_scale[s])
        back = self.backward(q * weight, views)
        return sum(self.rotate(back[p], v) for p, v in enumerate(views))

    def quads(self, sino, views):
        """[pair][x][4][plane] of a flat [plane][view][bin] sinogram."""
        sc = self.sc
        v = torch.tensor(views, device=self.dev)
        x = torch.from_numpy(self.xs).to(self.dev)
        lanes = [sino[:, w][:, :, b] for w, b in ((v, x), (v, sc.N - x), (v + sc.V // 2, x), (v + sc.V // 2, sc.N - x))]
        return torch.stack(lanes, 0).permute(2, 3, 0, 1).to(torch.float64).contiguous()

    def blur(self, img):
        """The PSF of the HRRT's default kernel: x, then y, then z, each renormalised over what it saw."""
        sc = self.sc
        sig = [F(f) / F(np.sqrt(8 * np.log(2)) * 1.21875) for f in (0.9 * np.sqrt(8 * np.log(2)), 2.5 * np.sqrt(8 * np.log(2)))]
        size = 2 * int(1.5 * 2.5 * np.sqrt(8 * np.log(2)) * np.sqrt(np.log(10) / np.log(2)) / 1.21875 / 2) + 1
        h = (size - 1) // 2
        i = np.arange(-h, h + 1)
        k = np.exp(-0.5 * (i / sig[0].astype(np.float64)) ** 2) + float(F(0.05)) * np.exp(-0.5 * (i / sig[1].astype(np.float64)) ** 2)
        k = k.astype(F)
        k = (k / F(k.sum(dtype=F))).astype(np.float64)
        cols = torch.from_numpy((np.arange(sc.N)[:, None] >= sc.cyl0[None, :]) & (np.arange(sc.N)[:, None] < sc.cyl1[None, :])).to(self.dev)
        fov = self.fov.double()
        planes = torch.zeros(sc.zp, dtype=torch.float64, device=self.dev)
        planes[sc.z_min:sc.z_max] = 1

        def along(v, seen, dim):
            v = v * seen
            acc, norm = torch.zeros_like(v), torch.zeros_like(seen)
            for m in range(-h, h):  # the last tap is not used
                n = v.shape[dim]
                src, dst = slice(max(0, m), min(n, n + m)), slice(max(0, -m), min(n, n - m))
                acc.narrow(dim, dst.start, dst.stop - dst.start).add_(v.narrow(dim, src.start, src.stop - src.start), alpha=k[m + h])
                norm.narrow(dim, dst.start, dst.stop - dst.start).add_(seen.narrow(dim, src.start, src.stop - src.start), alpha=k[m + h])
            return torch.where(norm > 0, acc / norm.clamp(min=1e-300), torch.zeros_like(acc))
        v = along(img, cols.double()[..., None].expand_as(img).clone(), 0) * fov[..., None]
        v = along(v, fov[..., None].expand_as(v).clone(), 1) * fov[..., None]
        v = along(v, planes[None, None].expand_as(v).clone(), 2) * fov[..., None]
        v[..., sc.nz:] = 0
        return v

    def prior(self, img):
        """Green's prior: tanh of the differences to the 18 neighbours."""
        sc = self.sc
        seen = img[self.fov][:, :sc.nz]
        delta = max(float(seen.max()), 0.0) * 1.2 / 20
        c = img[1:-1, 1:-1, 1:sc.nz - 1]
        face, edge = 0, 0
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dz in (-1, 0, 1):
                    far = abs(dx) + abs(dy) + abs(dz)
                    if far in (1, 2):
                        n = img[1 + dx:sc.N - 1 + dx, 1 + dy:sc.N - 1 + dy, 1 + dz:sc.nz - 1 + dz]
                        t = torch.tanh((c - n) / delta)
                        face, edge = (face + t, edge) if far == 1 else (face, edge + t)
        out = torch.zeros_like(img)
        out[1:-1, 1:-1, 1:sc.nz - 1] = face + math.sqrt(0.5) * edge
        return out * self.fov[..., None]


def _prepared(sc, study):
    """prompts, additive and multiplicative terms of a frame, 64 bits, flat layout."""
    norm = study["norm"].double()
    for lo, hi, off in sc.seg:
        n = hi - lo + 1
        norm[off:off + sc.npskip] = 0
        norm[off + n - sc.npskip:off + n] = 0
    atten = study["atten"].double()
    den = norm * atten.clamp(min=1)
    mult = torch.where((norm > 0) & (den > sc.eps2), 1 / den.clamp(min=1e-300), torch.zeros_like(den))
    add = study["randoms"].double().mul_(norm).add_(study["scatter"]).mul_(atten)
    return study["prompts"].float() * (norm != 0), add, mult


def _reconstruction(sc, ex, study, iterations, sens, adjoint=False, psf=False, beta=0.0):
    """The frame's image [N][N][zp] and its last sum."""
    p, a, m = _prepared(sc, study)
    if not sens:
        for s in range(sc.subsets):
            back = ex.correct(ex.quads(m, sc.views(s)), sc.views(s), adjoint)
            back = ex.blur(back) if psf else back
            sens.append(torch.where(back.abs() > sc.eps1, 1 / back, torch.zeros_like(back)))
            sens[-1][..., sc.nz:] = 0
    del m
    img = torch.zeros((sc.N, sc.N, sc.zp), dtype=torch.float64, device=ex.dev)
    img[..., sc.z_min:sc.z_max] = ex.fov[..., None].double()
    done = 0
    for _ in range(iterations):
        for s in sc.order():
            views = sc.views(s)
            den = ex.forward(ex.blur(img) if psf else img, views) + ex.quads(a, views)
            q = ex.quads(p, views)
            q = torch.where(q == 0, q, torch.where(den > sc.eps3, q / den, torch.ones_like(q)))
            corr = ex.correct(q, views, adjoint)
            corr = ex.blur(corr) if psf else corr
            if beta and done >= 5:
                new = img * (corr / (beta * ex.prior(img) + 1 / sens[s])).clamp(0.1, 100)
            else:
                new = img * (corr.clamp(0.01, 100) * sens[s])
            img = torch.where(ex.fov[..., None], new.clamp(max=sc.image_max), img)
            done += 1
        total = float(img[ex.fov][:, sc.z_min:sc.z_max].sum())
        img = torch.where(img < 1e-16, torch.zeros_like(img), img)
    return img, total


def _saved(sc, ex, img):
    return (img * ex.fov[..., None])[..., :sc.nz].permute(2, 1, 0).contiguous().cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "listmode":
        return None  # whole numbers
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    sc = Scanner(case)
    ex = Exact(sc, dev)
    if kind in ("osem", "reconstruct"):
        opt = {k: case.get(k, False) for k in ("adjoint", "psf")}
        beta = _beta(sc, case) if case.get("map") else 0.0
        img, total = _reconstruction(sc, ex, _study(sc, seed, dev), case["iterations"], [], beta=beta, **opt)
        return [_saved(sc, ex, img), total]
    if kind == "dynamic":
        sens, shared, out = [], None, []
        for f, (counts, iterations) in enumerate(_frames(case)):
            t = _study(sc, seed * 100 + f, dev, counts_per_bin=counts, sphere_gain=1.0 + f, shared=shared)
            shared = shared or (t["norm"], t["atten"])
            out.append(_saved(sc, ex, _reconstruction(sc, ex, t, iterations, sens)[0]))
        return out
    inp = _pair_inputs(sc, seed)
    view, rows = inp["view"], torch.from_numpy(inp["rows"]).to(dev).double().view(2, sc.planes, sc.N)
    sino = torch.zeros((sc.planes, sc.V, sc.N), dtype=torch.float64, device=dev)
    sino[:, view], sino[:, view + sc.V // 2] = rows[0], rows[1]
    weight = torch.empty(sc.planes, dtype=torch.float64, device=dev)
    for s, (lo, hi, off) in enumerate(sc.seg):
        weight[off:off + hi - lo + 1] = float(sc.bp_scale[s])
    back = ex.backward(ex.quads(sino, [view]) * weight, [view])[0]
    if kind == "pair_device":
        return back
    est = ex.forward(torch.from_numpy(inp["image"]).to(dev).double(), [view])[0].permute(1, 2, 0)  # [4][plane][x]
    x = torch.from_numpy(ex.xs).to(dev)
    fp = torch.zeros((2, sc.planes, sc.N), dtype=torch.float64, device=dev)
    for l in range(4):
        fp[l // 2][:, sc.N - x if l % 2 else x] = est[l]
    corr = torch.from_numpy(inp["corr"]).to(dev).double() + ex.rotate(back, view)
    return [t.cpu().numpy() for t in (fp.view(2 * sc.planes, sc.N), back, corr)]
