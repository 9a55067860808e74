"""Performance cases: what a user of the restoration library has it do.

Every case goes through a public entry point: the host mirror of the solver
(`compute`), `Artefact.process` from JPEG bytes, `process_jpeg(s)`, the
device-resident solves of the C ABI, the learned start and the warm-start
network's own prediction and training step. Sizes run from a thumbnail to the
6000x4000 image of the benchmark, with the iteration counts the library
defaults to (50), the benchmark's long run (100) and the learned start's 8.

Inputs are synthetic photographs-like images (blurred noise, rectangles,
gratings) made on the GPU from the seed and quantised with the IJG tables.
`exact` restates the solver and the network in float64 torch.
"""
import ctypes as C
import math

import numpy as np
import torch

from artefact_b200 import Artefact, JpegSource, ValueCollection, compute, process_jpeg, synth
from artefact_b200 import _native as N
from artefact_b200 import warmstart as WS
from artefact_b200.api import Coefficient, Context, Jpeg, process_jpegs

WEIGHT, PWEIGHT = 0.3, 0.001  # the library's defaults
SAMPLING = {"gray": [(1, 1)], "4:4:4": [(1, 1)] * 3, "4:2:2": [(1, 1), (2, 1), (2, 1)],
            "4:2:0": [(1, 1), (2, 2), (2, 2)]}


def listed():
    return [
        # A thumbnail restored by one call on host data: launches and latency.
        dict(name="thumbnail_host", kind="host", w=96, h=64, sub="4:2:0", quality=60, iterations=50, f32=False),
        # A ragged gray scan with float32 coefficients, as jpeg/zune.rs hands them over.
        dict(name="gray_ragged_host_f32", kind="host", w=518, h=389, sub="gray", quality=50, iterations=50, f32=True),
        # A web photo whose size fills no tile evenly, 4:2:2, result kept on the GPU.
        dict(name="web_422_device", kind="device", w=1000, h=667, sub="4:2:2", quality=50, iterations=50),
        # The headline workload: a video-sized frame, coefficients and planes in HBM.
        dict(name="frame_1080p_420_device", kind="device", w=1920, h=1080, sub="4:2:0", quality=75, iterations=50),
        # The largest: a camera image at full chroma and 100 iterations.
        dict(name="camera_24mp_444_device", kind="device", w=6000, h=4000, sub="4:4:4", quality=30, iterations=100),
        # One file from bytes to RGB, decode included: what the command line of the reference does.
        dict(name="file_1080p_420_rgb", kind="file", w=1920, h=1080, sub="4:2:0", quality=75, iterations=50),
        # Components restored separately with their own iteration counts, to RGB.
        dict(name="separate_640_420_rgb", kind="separate", w=640, h=480, sub="4:2:0", quality=40, iterations=50),
        # A folder of mixed photos solved as one batch to RGB.
        dict(name="batch_12_photos_rgb", kind="batch_rgb", count=12, small=256, large=1600, quality=60, iterations=50),
        # Many small images on the GPU in one batch (contact sheets, tiles).
        dict(name="batch_48_tiles_device", kind="batch_device", count=48, small=64, large=320, quality=50,
             iterations=50),
        # The learned start with its short refinement, in place of the 50 plain iterations.
        dict(name="learned_1080p_420_device", kind="learned", w=1920, h=1080, quality=50, iterations=8),
        # The per-component network alone: the luma of a frame.
        dict(name="predict_1080p_luma", kind="predict", count=1, w=1920, h=1080, quality=50),
        # Gradients of one joint training step on a batch of crops, at the start of a training run.
        dict(name="train_joint_16x256", kind="train", count=16, w=256, h=256, quality=50),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds, over their ranges of size, sampling and quality."""
    kind = rng.choice(["host", "device", "device", "device", "file", "separate", "batch_rgb", "batch_device",
                       "learned", "predict", "train"])
    q = rng.randint(20, 90)
    sub = rng.choice(["gray", "4:4:4", "4:2:2", "4:2:0", "4:2:0"])
    if kind == "host":
        return dict(kind=kind, w=_log(rng, 24, 900), h=_log(rng, 24, 900), sub=sub, quality=q, iterations=50,
                    f32=rng.random() < 0.5)
    if kind == "device":
        return dict(kind=kind, w=_log(rng, 200, 4200), h=_log(rng, 200, 3000), sub=sub, quality=q,
                    iterations=rng.choice([30, 50, 100]))
    if kind in ("file", "separate"):
        return dict(kind=kind, w=_log(rng, 200, 1920), h=_log(rng, 200, 1080),
                    sub=rng.choice(["4:4:4", "4:2:2", "4:2:0"]), quality=q, iterations=50)
    if kind == "batch_rgb":
        return dict(kind=kind, count=rng.randint(4, 16), small=256, large=_log(rng, 400, 1400), quality=q,
                    iterations=50)
    if kind == "batch_device":
        return dict(kind=kind, count=rng.randint(8, 96), small=64, large=_log(rng, 160, 640), quality=q,
                    iterations=50)
    if kind == "learned":
        return dict(kind=kind, w=16 * _log(rng, 16, 160), h=16 * _log(rng, 16, 100), quality=q, iterations=8)
    if kind == "predict":
        return dict(kind=kind, count=rng.randint(1, 4), w=8 * _log(rng, 16, 240), h=8 * _log(rng, 16, 135), quality=q)
    return dict(kind=kind, count=rng.randint(2, 16), w=16 * rng.randint(6, 16), h=16 * rng.randint(6, 16), quality=q)


# ------------------------------------------------------------------- inputs

LUMA = [16, 11, 10, 16, 24, 40, 51, 61, 12, 12, 14, 19, 26, 58, 60, 55, 14, 13, 16, 24, 40, 57, 69, 56,
        14, 17, 22, 29, 51, 87, 80, 62, 18, 22, 37, 56, 68, 109, 103, 77, 24, 35, 55, 64, 81, 104, 113, 92,
        49, 64, 78, 87, 103, 121, 120, 101, 72, 92, 95, 98, 112, 100, 103, 99]
CHROMA = [17, 18, 24, 47, 99, 99, 99, 99, 18, 21, 26, 66, 99, 99, 99, 99, 24, 26, 56, 99, 99, 99, 99, 99,
          47, 66, 99, 99, 99, 99, 99, 99] + [99] * 32


def _table(quality, chroma):
    scale = 5000 // quality if quality < 50 else 200 - 2 * quality
    return np.array([min(255, max(1, (v * scale + 50) // 100)) for v in (CHROMA if chroma else LUMA)], np.float32)


def _blur(img, sigma=4.0):
    r = int(3 * sigma)
    k = [math.exp(-0.5 * (d / sigma) ** 2) for d in range(-r, r + 1)]
    for dim in (-1, -2):
        n = img.shape[dim]
        idx = torch.arange(-r, n + r, device=img.device).clamp(0, n - 1)
        p = img.index_select(dim, idx)
        out = torch.zeros_like(img)
        for i, v in enumerate(k):
            out += p.narrow(dim, i, n) * (v / sum(k))
        img = out
    return img


def _channel(h, w, seed):
    """One channel of the generator, float32 in 0..255 on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    n = _blur(torch.randn(1, h, w, generator=g, device="cuda"))[0]
    img = n / n.std().clamp(min=1e-6) * 25.0 + 128.0
    for _ in range(20):
        level, cx, cy = rng.uniform(0, 255), rng.uniform(0, w), rng.uniform(0, h)
        rw, rh = rng.uniform(0.03, 0.3) * w, rng.uniform(0.03, 0.3) * h
        x0, x1, y0, y1 = int(max(cx - rw, 0)), int(min(cx + rw, w)), int(max(cy - rh, 0)), int(min(cy + rh, h))
        if x1 > x0 and y1 > y0:
            img[y0:y1, x0:x1] = 0.3 * img[y0:y1, x0:x1] + 0.7 * level
    yy = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    xx = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    for _ in range(3):
        t, period, phase = rng.uniform(0, np.pi), rng.uniform(6, 40), rng.uniform(0, 2 * np.pi)
        img += 20.0 * torch.sin(2 * np.pi * (xx * np.cos(t) + yy * np.sin(t)) / period + phase)
    return img.round().clamp(0, 255)


def _dct(dtype):
    m = [[(math.sqrt(1 / 8) if u == 0 else 0.5) * math.cos((2 * y + 1) * u * math.pi / 16) for y in range(8)]
         for u in range(8)]
    return torch.tensor(m, dtype=dtype, device="cuda")


def _blocks(plane):
    h, w = plane.shape
    return plane.reshape(h // 8, 8, w // 8, 8).transpose(1, 2)


def _plane(blocks):
    bh, bw = blocks.shape[:2]
    return blocks.transpose(1, 2).reshape(bh * 8, bw * 8)


def _components(w, h, sub, quality, seed):
    """(sh, sv, int16 blocks [bh][bw][8][8] on the GPU, table) of each component, and the rounded size."""
    samp = SAMPLING[sub]
    mw, mh = 8 * max(s[0] for s in samp), 8 * max(s[1] for s in samp)
    W, H = (w + mw - 1) // mw * mw, (h + mh - 1) // mh * mh
    if sub == "gray":
        planes = [_channel(h, w, seed * 3) - 128.0]
    else:
        r, g, b = (_channel(h, w, seed * 3 + k) for k in range(3))
        planes = [0.299 * r + 0.587 * g + 0.114 * b - 128.0, -0.168736 * r - 0.331264 * g + 0.5 * b,
                  0.5 * r - 0.418688 * g - 0.081312 * b]
    D = _dct(torch.float32)
    out = []
    for c, ((sh, sv), p) in enumerate(zip(samp, planes)):
        iy = torch.arange(H, device="cuda").clamp(max=h - 1)
        ix = torch.arange(W, device="cuda").clamp(max=w - 1)
        p = p[iy][:, ix].reshape(H // sv, sv, W // sh, sh).mean(dim=(1, 3)).round()
        q = _table(quality, c > 0)
        X = D @ _blocks(p) @ D.T
        co = (X / torch.from_numpy(q).cuda().reshape(8, 8)).round().to(torch.int16).contiguous()
        out.append((sh, sv, co, q))
    return out, W, H


def _coefficients(comps, f32=False):
    """Host Coefficient objects, as a decoder hands them to the solver."""
    out = []
    for sh, sv, co, q in comps:
        bh, bw = co.shape[:2]
        a = co.reshape(-1).cpu().numpy()
        out.append(Coefficient(bw * 8, bh * 8, bw, bh, sh, sv, a.astype(np.float32) if f32 else a, q.copy()))
    return out


def _batch(case, seed):
    """(w, h, sub, seed) of each image of a batch: sizes spread over its range, odd ones among them."""
    rng = np.random.default_rng(seed + 77)
    shape = np.random.default_rng(case["count"] * 1000 + case["large"])  # the same sizes for every seed
    n = case["count"]
    return [(int(shape.integers(case["small"], case["large"] + 1)), int(shape.integers(case["small"], case["large"] + 1)),
             ["4:2:0", "4:4:4"][int(shape.integers(2))], int(rng.integers(1 << 20))) for _ in range(n)]


class _Device:
    """Channels of one image with coefficients and result planes in HBM."""

    def __init__(self, comps, W, H, planes=None):
        self.n, self.W, self.H, self.pitch = len(comps), W, H, (W + 31) // 32 * 32
        self.comps = comps
        self.ch = (N.ArtChannel * self.n)()
        for a, (sh, sv, co, q) in zip(self.ch, comps):
            bh, bw = co.shape[:2]
            a.rounded_px_w, a.rounded_px_h, a.block_w, a.block_h = bw * 8, bh * 8, bw, bh
            a.samp_h, a.samp_v, a.coef_type, a.dct_coefs = sh, sv, N.ART_COEF_I16, co.data_ptr()
            a.quant_table = q.ctypes.data_as(C.POINTER(C.c_float))
        self.outs = [torch.zeros(H, self.pitch, device="cuda") for _ in comps] if planes is None else planes
        self.ptrs = (C.c_void_p * self.n)(*[o.data_ptr() for o in self.outs])


def _batch_planes(sizes, dtype=torch.float32):
    """One buffer for the result planes of a batch on the GPU, and each image's views of it."""
    at, views = 0, []
    for W, H, n in sizes:
        pitch = (W + 31) // 32 * 32
        views.append((at, n, H, pitch))
        at += n * H * pitch
    buf = torch.zeros(at, dtype=dtype, device="cuda")
    return buf, [list(buf[o:o + n * H * p].view(n, H, p)) for o, n, H, p in views]


def _initial():
    """Parameters a joint training run starts from: He weights, the head drawn for all twelve outputs."""
    p = WS.init_params(0)
    rng, n = np.random.default_rng(1), 16 * 9 * 32
    at = p.size - n - 16
    p[at:at + 12 * 9 * 32] = rng.standard_normal(12 * 9 * 32) * 0.05 * math.sqrt(2.0 / (9 * 32))
    return p


def _crops(case, seed):
    """Coefficient images, tables and targets of a batch of 4:2:0 training crops."""
    B, w, h = case["count"], case["w"], case["h"]
    cy, cc, tg = [], [], []
    for b in range(B):
        comps, W, H = _components(w, h, "4:2:0", case["quality"], seed * 64 + b)
        cy.append(_plane(comps[0][2]))
        cc.append(torch.stack([_plane(c[2]) for c in comps[1:]]))
        # Targets of a converged solve lie within a few levels of the smooth decode.
        tg.append(torch.stack([torch.nn.functional.interpolate(
            _blur(_decode(c[2], c[3], torch.float32)[None], 1.0)[None], size=(H, W), mode="nearest")[0, 0]
            for c in comps]))
    q = lambda chroma: torch.from_numpy(_table(case["quality"], chroma)).cuda()
    return (torch.stack(cy).contiguous(), torch.stack(cc).contiguous(), q(False).repeat(B, 1).contiguous(),
            q(True).repeat(B, 2, 1).contiguous(), torch.stack(tg, dim=1).contiguous())


# -------------------------------------------------------------- prepare, run


def prepare(case, seed):
    k = case["kind"]
    st = dict(case=case)
    if k == "host":
        comps, W, H = _components(case["w"], case["h"], case["sub"], case["quality"], seed)
        st.update(coefs=_coefficients(comps, case["f32"]), W=W, H=H)
    elif k == "device":
        comps, W, H = _components(case["w"], case["h"], case["sub"], case["quality"], seed)
        st.update(img=_Device(comps, W, H), ctx=Context(0))
    elif k == "file":
        st.update(data=synth.make_jpeg(case["w"], case["h"], case["quality"], case["sub"], False, seed))
    elif k == "separate":
        comps, W, H = _components(case["w"], case["h"], case["sub"], case["quality"], seed)
        st.update(jpeg=Jpeg(3, case["w"], case["h"], _coefficients(comps)))
    elif k == "batch_rgb":
        st.update(ctx=Context(0), jpegs=[Jpeg(3, w, h, _coefficients(_components(w, h, sub, case["quality"], s)[0]))
                                         for w, h, sub, s in _batch(case, seed)])
    elif k == "batch_device":
        made = [_components(w, h, sub, case["quality"], s) for w, h, sub, s in _batch(case, seed)]
        out, planes = _batch_planes([(W, H, len(comps)) for comps, W, H in made])
        imgs = [_Device(*m, planes=p) for m, p in zip(made, planes)]
        arr = (N.ArtImage * len(imgs))()
        for a, d in zip(arr, imgs):
            a.nchannel, a.max_rounded_px_w, a.max_rounded_px_h, a.out_pitch = d.n, d.W, d.H, d.pitch
            a.channels, a.weight = C.cast(d.ch, C.POINTER(N.ArtChannel)), WEIGHT
            a.pweight = (C.c_float * 3)(PWEIGHT, PWEIGHT, PWEIGHT)
            a.out_planes = C.cast(d.ptrs, C.POINTER(C.c_void_p))
        st.update(ctx=Context(0), imgs=imgs, arr=arr, out=out)
    elif k == "learned":
        comps, W, H = _components(case["w"], case["h"], "4:2:0", case["quality"], seed)
        st.update(img=_Device(comps, W, H), ctx=Context(0), net=WS.WarmStartNet.load(WS.DEFAULT_JOINT_WEIGHTS))
        st["ctx"].set_joint_warm_start(st["net"])
    elif k == "predict":
        co = torch.stack([_plane(_components(case["w"], case["h"], "gray", case["quality"], seed * 8 + b)[0][0][2])
                          for b in range(case["count"])]).contiguous()
        q = torch.from_numpy(_table(case["quality"], False)).cuda().repeat(case["count"], 1).contiguous()
        st.update(net=WS.WarmStartNet.load(), coef=co, q=q, out=torch.zeros(co.shape, device="cuda"))
    else:
        st.update(net=WS.WarmStartNet(_initial()), crops=_crops(case, seed))
    return st


def _solve_device(st, opts=None):
    d, case = st["img"], st["case"]
    N.check(N.lib().art_context_compute_device(st["ctx"].handle, d.n, d.ch, WEIGHT, (C.c_float * 3)(*[PWEIGHT] * 3),
                                               case["iterations"], d.W, d.H, d.ptrs, d.pitch, opts,
                                               C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return [o[:, :d.W] for o in d.outs]


def _refinement(k):
    """The schedule the learned start is used with: large steps that shrink, two small ones to settle."""
    return dict(step=1, decay=0.9, tail=min(2, k - 1) if k <= 12 else 0, tail_step=100)


def run(st):
    case = st["case"]
    k, its = case["kind"], case.get("iterations", 0)
    if k == "host":
        return compute(len(st["coefs"]), st["coefs"], WEIGHT, [PWEIGHT] * 3, its, st["W"], st["H"], st["W"] * st["H"])
    if k == "device":
        return _solve_device(st)
    if k == "file":
        return Artefact().source(JpegSource.Buffer(st["data"])).iterations(its).process()
    if k == "separate":
        return process_jpeg(st["jpeg"], [WEIGHT] * 3, [PWEIGHT] * 3,
                            ValueCollection.ForEach([its, its // 2, its // 2]).to_slice(), True)
    if k == "batch_rgb":
        return process_jpegs(st["jpegs"], [WEIGHT] * 3, [PWEIGHT] * 3, [its] * 3, False, context=st["ctx"])
    if k == "batch_device":
        N.check(N.lib().art_context_compute_batch_device(st["ctx"].handle, len(st["imgs"]), st["arr"], its, None,
                                                         C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return st["out"]
    if k == "learned":
        s = _refinement(its)
        o = N.ArtOptions()
        o.init_mode, o.device, o.step_iterations = N.ART_INIT_LEARNED, -1, s["step"]
        o.tail_iterations, o.tail_step_iterations, o.step_decay = s["tail"], s["tail_step"], s["decay"]
        return _solve_device(st, C.byref(o))
    if k == "predict":
        return st["net"].predict(st["coef"], st["q"], out=st["out"])
    # lr 0: the library leaves the gradients to the program's own optimiser
    loss = st["net"].train_step_joint(*st["crops"], lr=0.0)
    return dict(loss=loss, gradients=st["net"].gradients())


# ----------------------------------------------------------------------- work


def _pixels(case):
    """Component samples and full-resolution channel samples of one pass."""
    k = case["kind"]
    if k in ("batch_rgb", "batch_device"):
        items = [(w, h, sub) for w, h, sub, _ in _batch(case, 0)]
    elif k in ("learned", "train"):
        items = [(case["w"], case["h"], "4:2:0")] * case.get("count", 1)
    elif k == "predict":
        items = [(case["w"], case["h"], "gray")] * case["count"]
    else:
        items = [(case["w"], case["h"], case["sub"])]
    comp = sum(w * h / (sh * sv) for w, h, s in items for sh, sv in SAMPLING[s])
    full = sum(w * h * len(SAMPLING[s]) for w, h, s in items)
    real = sum(w * h for w, h, s in items)
    return comp, full, real


NET = [(16, 32, 0), (32, 64, 1), (64, 96, 2), (96, 128, 3), (224, 96, 2), (160, 64, 1), (96, 32, 0), (32, 16, 0)]


def work(case):
    comp, full, real = _pixels(case)
    k, its = case["kind"], case.get("iterations", 0)
    net = sum(2.0 * 9 * ci * co / 4 ** lv for ci, co, lv in NET) / 4.0 * real  # per full-resolution sample of the luma
    # One iteration: about 40 operations a sample for the gradient, 5 for the
    # step, and three 8x8 transforms of about 10 a component sample.
    solve = its * (45.0 * full + 30.0 * comp)
    if k == "separate":
        solve = its * (45.0 * real + 30.0 * real) + its // 2 * (45.0 * (full - real) + 30.0 * (comp - real))
    if k in ("file", "separate", "batch_rgb"):
        return dict(bytes=2.0 * comp + 3.0 * real, flops=solve)
    if k == "learned":
        return dict(bytes=2.0 * comp + 4.0 * full, flops=solve + net)
    if k == "predict":
        return dict(bytes=2.0 * comp + 4.0 * full, flops=net)
    if k == "train":
        return dict(bytes=2.0 * comp + 4.0 * full, flops=3.0 * net)
    return dict(bytes=(4.0 if case.get("f32") else 2.0) * comp + 4.0 * full, flops=solve)


# ---------------------------------------------------------------------- exact


def _decode(co, q, dtype=torch.float64):
    D = _dct(dtype)
    return _plane(D.T @ (co.to(dtype) * torch.from_numpy(q).cuda().to(dtype).reshape(8, 8)) @ D)


def _fista(n):
    t, fs = 1.0, []
    for _ in range(n):
        nx = (1.0 + math.sqrt(4.0 * t * t + 1.0)) / 2.0
        fs.append((t - 1.0) / nx)
        t = nx
    return fs


def _up(p, sh, sv):
    return p.repeat_interleave(sv, 0).repeat_interleave(sh, 1) if sh * sv > 1 else p


def _shift(a, dy, dx):
    """b[y, x] = a[y - dy, x - dx], zero where that lies outside."""
    b = torch.zeros_like(a)
    H, W = a.shape
    b[max(dy, 0):H + min(dy, 0), max(dx, 0):W + min(dx, 0)] = a[max(-dy, 0):H + min(-dy, 0), max(-dx, 0):W + min(-dx, 0)]
    return b


def _gradient(ys, weight):
    """TV and second-order TGV gradients of all channels (compute_step_tv.rs:29-93, compute_step_tv2.rs:32-136)."""
    n = len(ys)
    atv, atgv = 1.0 / math.sqrt(n), weight / math.sqrt(2.0) / math.sqrt(n)
    d, n1, n2 = [], 0.0, 0.0
    for y in ys:
        dx, dy = torch.zeros_like(y), torch.zeros_like(y)
        dx[:, :-1] = y[:, 1:] - y[:, :-1]
        dy[:-1] = y[1:] - y[:-1]
        gxx, gyx, gyy, gxy = (torch.zeros_like(y) for _ in range(4))
        gxx[:, 1:] = dx[:, 1:] - dx[:, :-1]
        gyx[:, 1:] = dy[:, 1:] - dy[:, :-1]
        gyy[1:] = dy[1:] - dy[:-1]
        gxy[1:] = dx[1:] - dx[:-1]
        s = 0.5 * (gxy + gyx)
        n1 = n1 + dx * dx + dy * dy
        n2 = n2 + gxx * gxx + 2.0 * s * s + gyy * gyy
        d.append((dx, dy, gxx, gyy, s))
    i1 = torch.where(n1 > 0, atv * n1.clamp(min=1e-300).rsqrt(), 0.0)
    i2 = torch.where(n2 > 0, atgv * n2.clamp(min=1e-300).rsqrt(), 0.0)
    out = []
    for dx, dy, gxx, gyy, s in d:
        a, b, u, v, w = i1 * dx, i1 * dy, i2 * (s + gxx), i2 * (gyy + s), i2 * s
        g = -(a + b) - 2.0 * (u + v - w)
        g += _shift(a + u, 0, 1) + _shift(u, 0, -1) + _shift(b + v, 1, 0) + _shift(v, -1, 0)
        g -= _shift(w, 1, -1) + _shift(w, -1, 1)
        out.append(g)
    return out


def _project(xp, comp, alpha):
    """Projected plane and the DCT-distance gradient of its clamped coefficients (compute_projection.rs:8-122)."""
    sh, sv, co, q = comp
    D, q = _dct(torch.float64), torch.from_numpy(q).cuda().double().reshape(8, 8)
    H, W = xp.shape
    mean = xp.reshape(H // sv, sv, W // sh, sh).mean(dim=(1, 3)) if sh * sv > 1 else xp
    c = co.double()
    X = torch.minimum(torch.maximum(D @ _blocks(mean) @ D.T, (c - 0.5) * q), (c + 0.5) * q)
    m, P = _plane(D.T @ X @ D), alpha * _plane(D.T @ ((X - c * q) / (q * q)) @ D)
    return (xp - _up(mean, sh, sv) + _up(m, sh, sv)) if sh * sv > 1 else m, _up(P, sh, sv)


def _solve64(comps, W, H, its, weight=WEIGHT, pweight=PWEIGHT, start=None, sched=None):
    weight, pweight = float(np.float32(weight)), float(np.float32(pweight))
    alpha = pweight * 2.0 * 255.0 * math.sqrt(2.0)
    s = sched or dict(step=its, decay=1.0, tail=0, tail_step=0)
    decay, k1 = float(np.float32(s["decay"])), its - min(s["tail"], its)
    radius = math.sqrt(W * H) / 2.0
    if start is None:
        xs = [_up(_decode(co, q), sh, sv) for sh, sv, co, q in comps]
        Ps = [0.0] * len(comps)
    else:
        xs, Ps = map(list, zip(*[_project(p, c, alpha) for p, c in zip(start, comps)]))
    ys = list(xs)
    f1, f2 = _fista(k1), _fista(its - k1)
    for i in range(its):
        if i < k1:
            step, f = radius / math.sqrt(1.0 + s["step"]) * decay ** i, f1[i + 1] if i + 1 < k1 else 0.0
        else:
            step, f = radius / math.sqrt(1.0 + s["tail_step"]), f2[i - k1 + 1] if i + 1 < its else 0.0
        for c, g in enumerate(_gradient(ys, weight)):
            g = g + Ps[c]
            n = g.norm()
            xp = ys[c] - step / n * g if n > 0 else ys[c]
            x, Ps[c] = _project(xp, comps[c], alpha)
            ys[c], xs[c] = x + f * (x - xs[c]), x
    return xs


def _network64(params, feat):
    """The encoder-decoder on feat [B][16][H0][W0] (float64, differentiable)."""
    F, o, at = torch.nn.functional, {}, 0
    for name, ci, co in WS.LAYERS:
        w = params[at:at + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        o[name] = (w, params[at + co * 9 * ci:at + co * 9 * ci + co])
        at += co * 9 * ci + co

    def conv(x, name):
        w, b = o[name]
        xp, r = F.pad(x, (1, 1, 1, 1)), 0.0
        for t in range(9):  # plain matrix products: float64 convolutions have no fast path
            r = r + torch.einsum("bchw,nc->bnhw", xp[:, :, t // 3:t // 3 + x.shape[2], t % 3:t % 3 + x.shape[3]],
                                 w[:, :, t // 3, t % 3])
        r = r + b[None, :, None, None]
        return r if name == "head" else r.relu()

    up = lambda x: F.interpolate(x, scale_factor=2, mode="nearest")
    e1 = conv(feat, "e1")
    e2 = conv(F.avg_pool2d(e1, 2), "e2")
    e3 = conv(F.avg_pool2d(e2, 2), "e3")
    e4 = conv(F.avg_pool2d(e3, 2), "e4")
    d3 = conv(torch.cat([e3, up(e4)], 1), "d3")
    d2 = conv(torch.cat([e2, up(d3)], 1), "d2")
    d1 = conv(torch.cat([e1, up(d2)], 1), "d1")
    return conv(d1, "head")


def _cells(p):
    """[B][H][W] -> [B][4][H/2][W/2], the 2x2 cells as channels."""
    return torch.nn.functional.pixel_unshuffle(p[:, None], 2)


def _steps(q, H, W):
    return q.double().reshape(-1, 8, 8).repeat(1, H // 8, W // 8)


def _smooth_up(p):
    """[B][h][w] upsampled 2x by linear interpolation between cell centres, edges clamped."""
    return torch.nn.functional.interpolate(p[:, None], scale_factor=2, mode="bilinear", align_corners=False)[:, 0]


def _blockimage(coef, q):
    """Decoded samples of coefficient images [B][H][W] with tables [B][64]."""
    B, H, W = coef.shape
    D = _dct(torch.float64)
    X = coef.double().reshape(B, H // 8, 8, W // 8, 8).transpose(2, 3) * q.double().reshape(B, 1, 1, 8, 8)
    return (D.T @ X @ D).transpose(2, 3).reshape(B, H, W)


def _joint64(params, cy, cc, qy, qc):
    """Joint 4:2:0 network: bases [3][B][H][W] and residuals in units of 16 levels."""
    B, H, W = cy.shape
    y = _blockimage(cy, qy)
    c = [_blockimage(cc[:, k], qc[:, k]) for k in range(2)]
    sc = [_steps(qc[:, k], H // 2, W // 2) for k in range(2)]
    feat = torch.cat([_cells(y) / 128, _cells(_steps(qy, H, W)) / 64, c[0][:, None] / 128, sc[0][:, None] / 64,
                      c[1][:, None] / 128, sc[1][:, None] / 64, torch.zeros_like(_cells(y))], 1)
    r = _network64(params, feat)
    r = torch.stack([torch.nn.functional.pixel_shuffle(r[:, 4 * k:4 * k + 4], 2)[:, 0] for k in range(3)])
    return torch.stack([y, _smooth_up(c[0]), _smooth_up(c[1])]), r


def _params(path):
    return torch.from_numpy(WS.load_params(path).astype(np.float64)).cuda()


def exact(case, seed):
    k, its = case["kind"], case.get("iterations", 0)
    if k in ("file", "separate", "batch_rgb"):
        return None  # bytes
    if k in ("host", "device"):
        comps, W, H = _components(case["w"], case["h"], case["sub"], case["quality"], seed)
        out = _solve64(comps, W, H, its)
        return [o.reshape(-1) for o in out] if k == "host" else out
    if k == "batch_device":
        made = [_components(w, h, sub, case["quality"], s) for w, h, sub, s in _batch(case, seed)]
        buf, planes = _batch_planes([(W, H, len(comps)) for comps, W, H in made], torch.float64)
        for m, views in zip(made, planes):
            for v, o in zip(views, _solve64(*m, its)):
                v[:, :o.shape[1]] = o
        return buf
    if k == "learned":
        comps, W, H = _components(case["w"], case["h"], "4:2:0", case["quality"], seed)
        t = [torch.from_numpy(c[3]).cuda()[None] for c in comps]
        base, r = _joint64(_params(WS.DEFAULT_JOINT_WEIGHTS), _plane(comps[0][2])[None],
                           torch.stack([_plane(c[2]) for c in comps[1:]])[None], t[0], torch.stack(t[1:], 1))
        return _solve64(comps, W, H, its, start=list((base + 16.0 * r)[:, 0]), sched=_refinement(its))
    if k == "predict":
        st = prepare(case, seed)
        co, q = st["coef"], st["q"]
        B, H, W = co.shape
        y, s = _blockimage(co, q), _steps(q, H, W)
        py, px = -H % 16, -W % 16
        y, s = (torch.nn.functional.pad(v, (0, px, 0, py)) for v in (y, s))
        feat = torch.cat([_cells(y) / 128, _cells(s) / 64, torch.zeros_like(_cells(y)), torch.zeros_like(_cells(y))], 1)
        r = _network64(_params(WS.DEFAULT_WEIGHTS), feat)
        return (y + 16.0 * torch.nn.functional.pixel_shuffle(r[:, :4], 2)[:, 0])[:, :H, :W].contiguous()
    cy, cc, qy, qc, target = _crops(case, seed)
    p = torch.from_numpy(_initial().astype(np.float64)).cuda().requires_grad_(True)
    base, r = _joint64(p, cy, cc, qy, qc)
    loss = ((r - (target.double() - base) / 16.0) ** 2).mean()
    loss.backward()
    return dict(loss=float(loss), gradients=p.grad)
