"""The performance cases of the renderer: what a user's program has it do, through its public
entry points, from an interactive preview to a converged 1080p frame and the learned estimator.

A case is a dict of plain values whose "op" names the work:

  draw     Sim.draw_to_bins on a warmed-up simulation (the chaos game; the reference's main loop
           draws 128 passes per call and reads the drawn count back)
  preview  what an edited genome costs: warmup, clear, 128 passes, density estimation + tonemap
  batch    Batch.run of several genomes and their images
  tail     density_tonemap of a rendered histogram (the image tail of a frame)
  density  density_estimate alone, also at radii beyond the default
  filter   density_estimate, then the tonemap with flam3's spatial filter (what a flam3 file with
           a `filter` attribute takes when it is supersampled)
  conv     one 3x3 convolution layer of the learned estimator
  gemm     one BF16 matrix product
  infer    the learned estimator's image of a frame's features
  train    one training step of the learned estimator, with the gradients read back

listed() are the sizes of this repository's own workloads (bench.py, learned.py); draw() spreads
the same kinds of work over their ranges, odd and ragged sizes among them.
"""
import math

import numpy as np
import torch

import refrakt_gb300 as R

DE_CURVE = 0.4
GAMMA, BRIGHTNESS, VIBRANCY = 2.2, 4.0, 1.0

# name -> (synthesiser kind, seed, number of xforms, final xform, parametric variations forced,
# approximate FP32 operations of one point's formulas)
GENOMES = {
    "small": (R.SYNTH_SMALL, 0, 0, False, False, 50),
    "frame": (R.SYNTH_RANDOM, 1, 8, True, True, 60),
    "contract": (R.SYNTH_CONTRACT, 4, 0, False, False, 30),
    "spacefill": (R.SYNTH_SPACEFILL, 5, 0, False, False, 50),
    "rich": (R.SYNTH_RANDOM, 103, 5, False, False, 60),
}

# the learned estimator's layers: (upsampled or only inputs, skip inputs, outputs, level)
CHANNELS = (32, 48, 64, 96)


def listed():
    return [
        # the small workload of bench.py: few walkers, so most of the chip idles
        dict(name="draw_small", op="draw", genome="small", w=512, h=512, walkers=65536, slots=2048, passes=256),
        # the headline frame's chaos game: 152 x 4 CTAs of 4096 walkers on the 1080p x 2 grid
        dict(name="draw_1080p", op="draw", genome="frame", w=3840, h=2160, walkers=2490368, slots=4096, passes=128),
        # a poster: a histogram several times larger than L2
        dict(name="draw_8k", op="draw", genome="spacefill", w=8192, h=8192, walkers=2490368, slots=4096, passes=32),
        # an edit in an interactive session: 640 x 360, 128 passes of 262,144 walkers
        dict(name="preview_360p", op="preview", genome="rich", w=640, h=360, walkers=262144, passes=128, radius=9),
        # the learned path's data generation: short runs of several genomes at 512 x 512
        dict(name="batch_8x512", op="batch", items=8, w=512, h=512, spp=64, first=200),
        # the 1080p frame's image tail at supersample 2, converged
        dict(name="tail_1080p", op="tail", w=3840, h=2160, ss=2, radius=9, min_radius=0, spp=1000, k2=0.0),
        # a wide estimator on a half-resolution histogram
        dict(name="density_r20", op="density", w=960, h=540, radius=20, min_radius=0, spp=50),
        # a flam3 file's own filter on the 1080p frame at supersample 2
        dict(name="filter_1080p", op="filter", w=3840, h=2160, ss=2, radius=9, min_radius=0, spp=250, shape=0,
             filter=1.0),
        # the decoder convolution at full resolution: 48 upsampled + 32 skip channels to 32
        dict(name="conv_decoder", op="conv", n=1, h=1080, w=1920, ca=48, cb=32, out=32, up=True, relu=True, f32=False),
        # a general product
        dict(name="gemm_4096", op="gemm", m=4096, n=4096, k=4096, f32=True, splits=1),
        # the learned path's 1080p frame
        dict(name="infer_1080p", op="infer", n=1, h=1080, w=1920),
        # the training step of learned.py: 16 crops of 256 x 256
        dict(name="train_16x256", op="train", n=16, h=256, w=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(("draw", "draw", "preview", "batch", "tail", "density", "filter", "conv", "gemm", "infer", "train"))
    if op == "draw":
        g = rng.choice(sorted(GENOMES))
        slots = rng.choice((1024, 2048, 4096, 4096))
        return dict(op=op, genome=g, w=_log(rng, 200, 3840), h=_log(rng, 150, 2160),
                    walkers=slots * _log(rng, 8, 2490368 // slots), slots=slots, passes=_log(rng, 16, 128))
    if op == "preview":
        return dict(op=op, genome=rng.choice(("small", "rich", "frame")), w=_log(rng, 160, 960), h=_log(rng, 90, 540),
                    walkers=4096 * _log(rng, 16, 152), passes=rng.choice((64, 128)), radius=rng.choice((5, 9, 11)))
    if op == "batch":
        return dict(op=op, items=rng.randint(2, 10), w=8 * rng.randint(24, 64), h=8 * rng.randint(24, 64),
                    spp=rng.choice((16, 32, 64)), first=200 + rng.randint(0, 7))
    if op == "tail":
        ss = rng.choice((1, 2, 2, 4))
        return dict(op=op, w=ss * _log(rng, 160, 3840 // ss), h=ss * _log(rng, 90, 2160 // ss), ss=ss,
                    radius=rng.choice((5, 9, 9, 11)), min_radius=rng.choice((0, 0, 1)), spp=_log(rng, 16, 1000),
                    k2=rng.choice((0.0, 0.0, 0.02)))
    if op == "density":
        return dict(op=op, w=_log(rng, 160, 960), h=_log(rng, 90, 540), radius=rng.choice((3, 9, 13, 16, 20)),
                    min_radius=rng.choice((0, 0, 2)), spp=_log(rng, 16, 500))
    if op == "filter":
        ss = rng.choice((2, 3, 4))
        return dict(op=op, w=ss * _log(rng, 160, 3840 // ss), h=ss * _log(rng, 90, 2160 // ss), ss=ss, radius=9,
                    min_radius=0, spp=_log(rng, 16, 500), shape=rng.choice((0, 1, 2, 3)),
                    filter=rng.choice((0.5, 0.75, 1.0)))
    if op == "conv":
        up = rng.random() < 0.5
        lv = rng.randint(0, 2)
        c = CHANNELS[lv]
        ca, cb = (CHANNELS[lv + 1], c) if up else (c, 0)
        h, w = _log(rng, 64, 1080), _log(rng, 64, 1920)
        return dict(op=op, n=1, h=h - h % 2, w=w - w % 2, ca=ca, cb=cb, out=c, up=up, relu=True, f32=rng.random() < 0.3)
    if op == "gemm":
        return dict(op=op, m=_log(rng, 128, 4096), n=_log(rng, 32, 4096), k=8 * _log(rng, 8, 512),
                    f32=rng.random() < 0.7, splits=1)
    if op == "infer":
        return dict(op=op, n=1, h=8 * rng.randint(16, 135), w=8 * rng.randint(16, 240))
    n = rng.randint(1, 16)
    return dict(op=op, n=n, h=8 * rng.randint(8, 32), w=8 * rng.randint(8, 32))


# ---- inputs -----------------------------------------------------------------------------------

_compiler = None


def _genome(name, w, h):
    global _compiler
    if _compiler is None:
        _compiler = R.FlameCompiler()
    kind, seed, n, final, forced, _ = GENOMES[name]
    return R.Flame.synthesize(_compiler, kind, seed, w, h, n_xforms=n, final_xform=final, force_parametric=forced)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _histogram(case, seed):
    """A flame-like histogram [h, w, 4]: a Poisson sample of a filament density with a long tail
    (bright cores, sparse fringes, empty background), mean `spp` points per bin, each point of
    opacity 1 with a palette colour that varies slowly over the plane."""
    w, h = case["w"], case["h"]
    g = _gen(seed)
    par = torch.rand(8, 6, generator=g, device="cuda").tolist()
    y = torch.linspace(-1, 1, h, device="cuda")[:, None]
    x = torch.linspace(-w / h, w / h, w, device="cuda")[None, :]
    rate = torch.zeros(h, w, device="cuda")
    for a, b, c, d, e, f in par:  # eight curved filaments
        th = 6.2831853 * a
        u = math.cos(th) * x + math.sin(th) * y
        v = -math.sin(th) * x + math.cos(th) * y
        s = v - (b - 0.5) - 0.3 * torch.sin((2 + 4 * c) * u + 6.2831853 * d)
        width = 0.01 + 0.04 * e
        rate += (0.2 + f) / (1 + (s / width) ** 2) ** 2 * torch.exp(-2 * (u * u + v * v))
    rate *= case["spp"] / float(rate.mean())
    hits = torch.poisson(rate, generator=g)
    t = 0.5 + 0.5 * torch.sin(3 * x + 2 * y + 6.2831853 * par[0][0])
    pal = torch.stack([0.1 + 0.9 * t, 0.9 - 0.6 * t, 0.3 + 0.5 * torch.cos(2 * t), torch.ones_like(t)], -1)
    return (hits[..., None] * pal).contiguous()


def _features(case, seed):
    """Input features of the learned estimator, [n, h, w, 8] bf16: log density, its colour, the
    plain image and the run's level (denoiser_features' layout)."""
    n, h, w = case["n"], case["h"], case["w"]
    out = torch.empty(n, h, w, 8, dtype=torch.bfloat16, device="cuda")
    for i in range(n):
        b = _histogram(dict(w=w, h=h, spp=64), seed * 1009 + i)
        a = b[..., 3]
        l = torch.log10(1 + a * (w * h / float(a.sum())))
        s = l / a.clamp_min(1)
        img = (b[..., :3] * s[..., None]).clamp(0, 1) ** (1 / GAMMA)
        out[i] = torch.cat([l[..., None], b[..., :3] * s[..., None], img, torch.full_like(l, 0.6)[..., None]], -1)
    return out


def _params(layers, seed):
    """He-scaled weights of a network in training: the output layer small, so that the image stays near its base."""
    r = np.random.default_rng(seed)
    parts = []
    for L in layers:
        k = L["taps"] * (L["in_a"] + L["in_b"])
        std = math.sqrt(2.0 / k) * (1.0 if L["relu"] else 0.05)
        parts += [r.normal(0, std, L["out"] * k), r.normal(0, 0.02, L["out"])]
    return np.concatenate(parts).astype(np.float32)


def _unet_layers():
    """The layer table that Denoiser.layers() reports, restated for exact()."""
    c, L, prev, cin, skip = CHANNELS, [], -1, 8, []
    for l in range(4):
        L.append(dict(in_a=cin, in_b=0, out=c[l], taps=9, upsample=0, relu=1, src_a=prev, src_b=-1))
        L.append(dict(in_a=c[l], in_b=0, out=c[l], taps=9, upsample=0, relu=1, src_a=len(L) - 1, src_b=-1))
        skip.append(len(L) - 1)
        prev, cin = -100 - (l + 1), c[l]
    low = skip[3]
    for l in (2, 1, 0):
        L.append(dict(in_a=c[l + 1], in_b=c[l], out=c[l], taps=9, upsample=1, relu=1, src_a=low, src_b=skip[l]))
        L.append(dict(in_a=c[l], in_b=0, out=c[l], taps=9, upsample=0, relu=1, src_a=len(L) - 1, src_b=-1))
        low = len(L) - 1
    L.append(dict(in_a=c[0], in_b=0, out=3, taps=1, upsample=0, relu=0, src_a=low, src_b=-1))
    return L


def _conv_inputs(case, seed):
    g = _gen(seed)
    n, h, w, ca, cb = case["n"], case["h"], case["w"], case["ca"], case["cb"]
    ha, wa = (h // 2, w // 2) if case["up"] else (h, w)
    relu = lambda *s: torch.randn(*s, generator=g, device="cuda").clamp_min(0).to(torch.bfloat16)  # noqa: E731
    xa = relu(n, ha, wa, ca)
    xb = relu(n, h, w, cb) if cb else None
    k = 9 * (ca + cb)
    wt = (torch.randn(case["out"], k, generator=g, device="cuda") * math.sqrt(2.0 / k)).to(torch.bfloat16)
    bias = torch.randn(case["out"], generator=g, device="cuda") * 0.05
    return xa, xb, wt, bias


def _gemm_inputs(case, seed):
    g = _gen(seed)
    a = torch.randn(case["m"], case["k"], generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(case["n"], case["k"], generator=g, device="cuda").to(torch.bfloat16)
    return a, b


def _target(case, seed):
    g = _gen(seed + 77)
    n, h, w = case["n"], case["h"], case["w"]
    return torch.rand(n, h, w, 3, generator=g, device="cuda")


# ---- the work ---------------------------------------------------------------------------------


def prepare(case, seed):
    op, s = case["op"], {"case": case}
    if op in ("draw", "preview"):
        w, h = case["w"], case["h"]
        s["flame"] = f = _genome(case["genome"], w, h)
        i = f.info()
        f.set_view(i["center"], i["scale"], float(seed % 360))
        s["sim"] = sim = R.Sim(case["walkers"], cta_slots=case.get("slots", 4096), seed=seed)
        sim.set_bad_value_reset(True)
        s["bins"] = torch.zeros(h, w, 4, device="cuda")
        s["hits"] = torch.zeros(h, w, dtype=torch.int32, device="cuda")
        if op == "draw":
            sim.warmup(f, 19)
        else:
            s["image"] = torch.zeros(h, w, 4, device="cuda")
    elif op == "batch":
        global _compiler
        _compiler = _compiler or R.FlameCompiler()
        w, h, n = case["w"], case["h"], case["items"]
        items = []
        for k in range(n):
            q = case["first"] + k
            f = R.Flame.synthesize(_compiler, R.SYNTH_RANDOM, q, w, h, n_xforms=2 + q % 11, final_xform=True)
            f.set_estimator(9, 0, DE_CURVE)
            items.append((f, w, h, w * h * case["spp"], seed * 1000 + k))
        s["batch"] = R.Batch(items, cta_slots=4096, image_f32=True, bad_value_reset=True)
        s["images"] = [torch.zeros(h, w, 4, device="cuda") for _ in range(n)]
    elif op in ("tail", "density", "filter"):
        s["bins"] = _histogram(case, seed)
        ss = case.get("ss", 1)
        if op in ("density", "filter"):
            s["de"] = torch.zeros_like(s["bins"])
        s["image"] = torch.zeros(case["h"] // ss, case["w"] // ss, 4, device="cuda")
    elif op == "conv":
        s["xa"], s["xb"], s["wt"], s["bias"] = _conv_inputs(case, seed)
        rows = case["n"] * case["h"] * case["w"]
        s["c"] = torch.zeros(rows, case["out"], dtype=torch.float32 if case["f32"] else torch.bfloat16, device="cuda")
    elif op == "gemm":
        s["a"], s["b"] = _gemm_inputs(case, seed)
        s["c"] = torch.zeros(case["m"], case["n"], dtype=torch.float32 if case["f32"] else torch.bfloat16, device="cuda")
    else:
        n, h, w = case["n"], case["h"], case["w"]
        s["net"] = R.Denoiser(n * h * w)
        s["net"].set_params(_params(s["net"].layers(), seed))
        s["feats"] = _features(case, seed)
        if op == "infer":
            s["out"] = torch.zeros(n, h, w, 3, device="cuda")
        else:
            s["target"] = _target(case, seed)
    return s


def run(s):
    c = s["case"]
    op = c["op"]
    if op == "draw":
        drawn = s["sim"].draw_to_bins(s["flame"], s["bins"], s["hits"], c["w"], c["h"], c["passes"])
        return {"rgba": s["bins"], "hits": s["hits"], "drawn": drawn}
    if op == "preview":
        s["sim"].warmup(s["flame"], 19)
        s["bins"].zero_()
        s["hits"].zero_()
        s["sim"].draw_to_bins(s["flame"], s["bins"], s["hits"], c["w"], c["h"], c["passes"], sync=False)
        R.density_tonemap(s["bins"], c["w"], c["h"], c["radius"], 0, DE_CURVE, 1, GAMMA, BRIGHTNESS, VIBRANCY, 0.0,
                          out_f32=s["image"])
        return {"image": s["image"], "hits": s["hits"]}
    if op == "batch":
        s["batch"].run()
        for i, img in enumerate(s["images"]):
            s["batch"].image_f32(i, img)
        return s["images"]
    if op == "tail":
        R.density_tonemap(s["bins"], c["w"], c["h"], c["radius"], c["min_radius"], DE_CURVE, c["ss"], GAMMA, BRIGHTNESS,
                          VIBRANCY, c["k2"], out_f32=s["image"])
        return s["image"]
    if op in ("density", "filter"):
        R.density_estimate(s["bins"], c["w"], c["h"], c["radius"], c["min_radius"], DE_CURVE, s["de"])
        if op == "density":
            return s["de"]
        R.tonemap_filter(s["de"], c["w"], c["h"], c["ss"], c["filter"], c["shape"], GAMMA, BRIGHTNESS, VIBRANCY, 0.0,
                         out_f32=s["image"])
        return s["image"]
    if op == "conv":
        R.conv3x3_bf16(s["xa"], s["wt"], s["c"], xb=s["xb"], up=c["up"],
                       mode=R.GEMM_STORE_F32 if c["f32"] else R.GEMM_STORE_BF16, bias=None if c["f32"] else s["bias"],
                       relu=c["relu"] and not c["f32"])
        return s["c"]
    if op == "gemm":
        R.gemm_bf16(s["a"], s["b"], s["c"], mode=R.GEMM_STORE_F32 if c["f32"] else R.GEMM_STORE_BF16, splits=c["splits"])
        return s["c"]
    if op == "infer":
        s["net"].infer(s["feats"], s["out"])
        return s["out"]
    loss = s["net"].train_step(s["feats"], s["target"], 1e-4)
    return {"loss": loss, "gradients": s["net"].gradients()}


def _unet_macs():
    """Multiply-adds of one forward pass per level-0 pixel (the levels have 1, 1/4, 1/16, 1/64 of the pixels)."""
    level = [l for l in range(4) for _ in range(2)] + [2, 2, 1, 1, 0, 0, 0]
    return sum(L["out"] * L["taps"] * (L["in_a"] + L["in_b"]) / 4.0 ** l for L, l in zip(_unet_layers(), level))


def work(case):
    op = case["op"]
    if op in ("draw", "preview"):
        bins, steps = case["w"] * case["h"], case["walkers"] * case["passes"]
        # the histogram read and written, walkers and RNG states in and out
        return {"bytes": 40.0 * bins + 64.0 * case["walkers"], "flops": float(GENOMES[case["genome"]][5]) * steps}
    if op == "batch":
        bins = case["items"] * case["w"] * case["h"]
        return {"bytes": 16.0 * bins, "flops": 60.0 * bins * case["spp"]}
    if op in ("tail", "density", "filter"):
        bins, ss = case["w"] * case["h"], case.get("ss", 1)
        out = bins / ss ** 2 if op != "density" else bins
        # per bin: its radius and its own disc's centre at least; per pixel the tonemap
        return {"bytes": 16.0 * bins + 16.0 * out, "flops": 20.0 * bins + 40.0 * out}
    if op == "conv":
        rows, cin = case["n"] * case["h"] * case["w"], case["ca"] + case["cb"]
        a = case["ca"] / (4.0 if case["up"] else 1.0) + case["cb"]
        return {"bytes": rows * (2.0 * a + case["out"] * (4.0 if case["f32"] else 2.0)),
                "flops": 18.0 * rows * cin * case["out"]}
    if op == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2.0 * (m + n) * k + (4.0 if case["f32"] else 2.0) * m * n, "flops": 2.0 * m * n * k}
    px = case["n"] * case["h"] * case["w"]
    if op == "infer":
        return {"bytes": px * (16.0 + 12.0), "flops": 2.0 * _unet_macs() * px}
    return {"bytes": px * (16.0 + 12.0), "flops": 6.0 * _unet_macs() * px}


# ---- what the outputs are in 64 bits ------------------------------------------------------------


def _f32(v):
    return float(np.float32(v))


def _density64(bins, radius, min_radius):
    """Every bin spreads over its disc: radius max(min, min(R, int(R / a^curve))), weights
    (1 - d^2) (2/pi) / r^2 with d = |offset| / (r + 1/2), inside 4 |offset|^2 <= (2r + 1)^2."""
    b = bins.double()
    a = b[..., 3]
    r = torch.zeros_like(a, dtype=torch.int64)
    for k in range(1, radius + 1):  # int(R / a^curve) >= k  <=>  a <= (R / k)^(1 / curve)
        r += (a <= (radius / k) ** (1.0 / _f32(DE_CURVE))).long()
    r = r.clamp_min(min_radius)
    r = torch.where(a > 0, r, torch.full_like(r, -1))
    big = max(radius, min_radius)
    h, w = a.shape
    out = torch.zeros_like(b)
    rr = torch.arange(big + 1, device=b.device, dtype=torch.float64)
    for dy in range(-big, big + 1):
        for dx in range(-big, big + 1):
            d2 = dx * dx + dy * dy
            wt = (1 - d2 / (rr + 0.5) ** 2) * 0.63661977236 / rr.clamp_min(1) ** 2
            wt = torch.where(4 * d2 <= (2 * rr + 1) ** 2, wt, torch.zeros_like(wt))
            wt[0] = 1.0 if d2 == 0 else 0.0
            wt = torch.cat([wt, wt.new_zeros(1)])  # the last entry serves the empty bins (index -1)
            y0, y1, x0, x1 = max(0, -dy), h - max(0, dy), max(0, -dx), w - max(0, dx)
            if y1 <= y0 or x1 <= x0:
                continue
            src = b[y0:y1, x0:x1] * wt[r[y0:y1, x0:x1]][..., None]
            out[y0 + dy:y1 + dy, x0 + dx:x1 + dx] += src
    return out


def _finish64(v):
    a = v[..., 3:4]
    ig = 1.0 / _f32(GAMMA)
    vib = _f32(VIBRANCY)
    rgb = v[..., :3]
    z = torch.where(a > 0, a ** ig / a, torch.zeros_like(a))
    rgb = (rgb ** ig * (1 - vib) + z * rgb * vib).clamp(0, 1)
    return torch.cat([torch.where(a > 0, rgb, torch.zeros_like(rgb)), torch.ones_like(a)], -1)


def _log64(de, k2):
    a = de[..., 3:4]
    k = _f32(k2) if k2 > 0 else a.numel() / float(a.sum())
    return torch.where(a > 0, de * (0.5 * _f32(BRIGHTNESS) * torch.log1p(a * k) / math.log(10.0) / a), torch.zeros_like(de))


def _filter_taps(ss, radius, shape):
    support = (1.5, 0.5, 1.0, 1.0)[shape]
    fw = 2.0 * support * ss * _f32(radius)
    n = int(fw) + 1
    n += (n ^ ss) & 1
    t = []
    for i in range(n):
        x = ((2.0 * i + 1.0) / n - 1.0) * support * n / fw
        q = abs(x)
        t.append((math.exp(-2 * x * x) * math.sqrt(2 / math.pi), float(q <= 0.5), max(0.0, 1 - q),
                  (2 * q - 3) * q * q + 1 if q < 1 else 0.0)[shape])
    return [v / sum(t) for v in t]


def _unet64(params, feats, grad):
    x0 = feats.double().permute(0, 3, 1, 2)
    acts, ws, o = [], [], 0
    for L in _unet_layers():
        cin, k = L["in_a"] + L["in_b"], 3 if L["taps"] == 9 else 1
        nw = L["out"] * L["taps"] * cin
        p = torch.from_numpy(params).to(feats.device)
        w = p[o:o + nw].to(torch.bfloat16).double().view(L["out"], k, k, cin).permute(0, 3, 1, 2).contiguous()
        b = p[o + nw:o + nw + L["out"]].double()
        o += nw + L["out"]
        w.requires_grad_(grad)
        b.requires_grad_(grad)
        ws.append((w, b))
        s = L["src_a"]
        if s == -1:
            x = x0
        elif s <= -100:  # the pooled output of the level above
            x = torch.nn.functional.avg_pool2d(acts[2 * (-100 - s - 1) + 1], 2)
        else:
            x = acts[s]
        if L["upsample"]:
            x = x.repeat_interleave(2, 2).repeat_interleave(2, 3)
        if L["in_b"]:
            x = torch.cat([x, acts[L["src_b"]]], 1)
        y = torch.nn.functional.conv2d(x, w, b, padding=k // 2)
        acts.append(torch.relu(y) if L["relu"] else y)
    return x0.permute(0, 2, 3, 1)[..., 4:7] + acts[-1].permute(0, 2, 3, 1), ws


def exact(case, seed):
    op = case["op"]
    if op in ("draw", "preview", "batch"):
        return None  # chaotic trajectories: no 64-bit run follows them
    if op in ("tail", "density", "filter"):
        de = _density64(_histogram(case, seed), case["radius"], case["min_radius"])
        if op == "density":
            return de
        v = _log64(de, case.get("k2", 0.0))
        h, w, ss = case["h"], case["w"], case["ss"]
        if op == "tail":
            return _finish64(v.view(h // ss, ss, w // ss, ss, 4).mean((1, 3)))
        taps = _filter_taps(ss, case["filter"], case["shape"])
        pad = (len(taps) - ss) // 2
        v = torch.nn.functional.pad(v, (0, 0, pad, pad + ss, pad, pad + ss))
        cols = sum(t * v[:, i:i + w:ss] for i, t in enumerate(taps))
        return _finish64(sum(t * cols[i:i + h:ss] for i, t in enumerate(taps)))
    if op == "conv":
        xa, xb, wt, bias = _conv_inputs(case, seed)
        x = xa.double().permute(0, 3, 1, 2)
        if case["up"]:
            x = x.repeat_interleave(2, 2).repeat_interleave(2, 3)
        if xb is not None:
            x = torch.cat([x, xb.double().permute(0, 3, 1, 2)], 1)
        c = case["ca"] + case["cb"]
        k = wt.double().view(-1, 9, c).permute(0, 2, 1).reshape(-1, c, 3, 3)
        y = torch.nn.functional.conv2d(x, k, None if case["f32"] else bias.double(), padding=1)
        y = torch.relu(y) if case["relu"] and not case["f32"] else y
        return y.permute(0, 2, 3, 1).reshape(-1, case["out"])
    if op == "gemm":
        a, b = _gemm_inputs(case, seed)
        return a.double() @ b.double().t()
    params = _params(_unet_layers(), seed)
    feats = _features(case, seed)
    if op == "infer":
        with torch.no_grad():
            return _unet64(params, feats, False)[0].clamp(0, 1)
    pred, ws = _unet64(params, feats, True)
    loss = (pred - _target(case, seed).double()).abs().mean()
    loss.backward()
    g = [q for w, b in ws for q in (w.grad.permute(0, 2, 3, 1).reshape(-1), b.grad)]
    return {"loss": float(loss.detach()), "gradients": torch.cat(g).cpu().numpy()}
