"""The work that users of this library give it, as cases to be timed.

A case names one kind of call and its sizes; `prepare` makes what a program
holds before the call (images on the device, a plan, a server), `run` is the
call itself through the public entry points, `work` counts the bytes and
operations it cannot do without, and `exact` is the same result in 64 bits
from plain torch.  `draw` gives further cases of the same ranges.

Kinds:
  fft       gls::fft on one image, once or as a chain of transforms
  real      gls::fft on a CV_32FC1 image (promoted to complex)
  batched   many equal images back to back
  plan      many images of individual sizes in one batch plan
  poc       gls::phaseCorrelate, one frame pair at a time
  display   the camera view: window, transform, log-magnitude, normalise
  serve     a burst of phaseCorrelate requests against resident references
  spectrum  element-wise spectrum operations, images of any size
"""
from __future__ import annotations

import math

import torch

import glscv_gb300 as gls
from glscv_gb300 import workloads

INV, SCALE, SHIFT = gls.DFT_INVERSE, gls.DFT_SCALE, gls.GLS_FFT_SHIFT
KINDS = ("fft", "real", "batched", "plan", "poc", "display", "serve", "spectrum")

_context = None


def context():
    """The program's one library context (glsCvInit)."""
    global _context
    if _context is None:
        _context = gls.Context(0)
    return _context


def listed():
    return [
        # the smallest call: a tracker's 64 x 64 patch, there and back; launches and latency
        {"name": "fft_64", "kind": "fft", "rows": 64, "cols": 64, "chain": "roundtrip"},
        # the ordinary single image: forward, then inverse with DFT_SCALE
        {"name": "fft_1024", "kind": "fft", "rows": 1024, "cols": 1024, "chain": "roundtrip"},
        # the largest single image
        {"name": "fft_4096", "kind": "fft", "rows": 4096, "cols": 4096, "chain": "roundtrip"},
        # a wide CV_32FC1 strip to its centred spectrum
        {"name": "real_512x2048", "kind": "real", "rows": 512, "cols": 2048, "chain": "shift"},
        # a stack of tiles, an odd number of them, back from their spectra
        {"name": "batched_37x256x512", "kind": "batched", "rows": 256, "cols": 512, "count": 37,
         "chain": "inverse"},
        # images of mixed sizes (128^2 .. 1024 x 2048) in one plan, forward
        {"name": "plan_mixed_160", "kind": "plan", "count": 160, "pick": 3, "rows": 0, "cols": 0,
         "chain": "forward"},
        # the benchmark's batch: 64 images of 1024^2 there and back in one plan
        {"name": "plan_1024x64", "kind": "plan", "count": 64, "pick": 0, "rows": 1024,
         "cols": 1024, "chain": "roundtrip"},
        # stabilisation: the shift between two frames, one call per pair
        {"name": "poc_1024", "kind": "poc", "rows": 1024, "cols": 1024},
        # the same on large frames
        {"name": "poc_2048", "kind": "poc", "rows": 2048, "cols": 2048},
        # the camera's spectrum view
        {"name": "display_1024", "kind": "display", "rows": 1024, "cols": 1024},
        # a burst of requests of mixed sizes at the serving loop
        {"name": "serve_12", "kind": "serve", "count": 12, "pick": 5},
        # spectrum operations on an image whose sides are no powers of two
        {"name": "spectrum_1081x1919", "kind": "spectrum", "rows": 1081, "cols": 1919},
    ]


def draw(rng):
    kind = rng.choice(KINDS)
    side = lambda lo, hi: 1 << rng.randint(lo, hi)  # noqa: E731
    if kind in ("fft", "real"):
        return {"kind": kind, "rows": side(5, 12), "cols": side(5, 12),
                "chain": rng.choice(("roundtrip", "roundtrip", "shift"))}
    if kind == "batched":
        rows, cols = side(5, 11), side(5, 11)
        most = max(2, min(400, (1 << 25) // (rows * cols)))
        return {"kind": kind, "rows": rows, "cols": cols,
                "count": int(round(math.exp(rng.uniform(math.log(2), math.log(most))))),
                "chain": rng.choice(("forward", "inverse", "roundtrip", "shift"))}
    if kind == "plan":
        if rng.random() < 0.5:
            return {"kind": kind, "count": int(round(math.exp(rng.uniform(math.log(3), math.log(160))))),
                    "pick": rng.randint(1, 9999), "rows": 0, "cols": 0,
                    "chain": rng.choice(("forward", "inverse"))}
        rows, cols = side(6, 10), side(6, 11)
        most = min(300, (1 << 26) // (rows * cols))
        return {"kind": kind, "count": int(round(math.exp(rng.uniform(math.log(2), math.log(most))))),
                "pick": 0, "rows": rows, "cols": cols, "chain": rng.choice(("forward", "roundtrip"))}
    if kind == "poc":
        return {"kind": kind, "rows": side(6, 12), "cols": side(6, 12)}
    if kind == "display":
        return {"kind": kind, "rows": side(7, 12), "cols": side(7, 12)}
    if kind == "serve":
        return {"kind": kind, "count": rng.randint(1, 12), "pick": rng.randint(1, 9999)}
    return {"kind": kind, "rows": rng.randint(33, 4096), "cols": rng.randint(33, 4096)}


# flags of the transforms that a chain runs one after another
CHAINS = {"forward": (0,), "inverse": (INV | SCALE,), "shift": (SHIFT,), "roundtrip": (0, INV | SCALE)}


def shapes_of(case):
    """(rows, cols) of every image or request of a plan or serve case."""
    if case["kind"] == "serve":
        sizes = ((512, 512), (1024, 1024), (2048, 2048))
        g = torch.Generator().manual_seed(case["pick"])
        at = torch.multinomial(torch.tensor([0.5, 0.35, 0.15]), case["count"], True, generator=g)
        return [sizes[int(i)] for i in at]
    if case["rows"]:
        return [(case["rows"], case["cols"])] * case["count"]
    return workloads.batch_sizes(case["count"], case["pick"])


# ------------------------------------------------------------------ inputs
def uniform_complex(n, gen):
    """n complex values, both parts uniform in [-1, 1), as the benchmark's images."""
    x = torch.rand(2 * n, generator=gen, device="cuda") * 2 - 1
    return torch.view_as_complex(x.view(n, 2))


def scene_pair(rows, cols, gen, noise=0.01):
    """Two frames of one scene, the second shifted by whole pixels plus a
    fraction; a spectrum that falls off as 1 / f, in [0, 1], and sensor noise
    of its own on each."""
    fy = torch.fft.fftfreq(rows, device="cuda", dtype=torch.float64)[:, None]
    fx = torch.fft.fftfreq(cols, device="cuda", dtype=torch.float64)[None, :]
    white = torch.randn(rows, cols, generator=gen, device="cuda", dtype=torch.float64)
    spec = torch.fft.fft2(white) / torch.sqrt(fx * fx + fy * fy + (4.0 / max(rows, cols)) ** 2)
    u = torch.rand(4, generator=gen, device="cuda", dtype=torch.float64).tolist()
    shift = [(0.05 + 0.15 * u[k]) * n + 0.4 * (u[2 + k] - 0.5) for k, n in enumerate((rows, cols))]
    a = torch.fft.ifft2(spec).real
    b = torch.fft.ifft2(spec * torch.exp(-2j * math.pi * (fy * shift[0] + fx * shift[1]))).real
    lo, hi = a.min(), a.max()
    out = []
    for x in (a, b):
        x = (x - lo) / (hi - lo)
        x = x + noise * torch.randn(rows, cols, generator=gen, device="cuda", dtype=torch.float64)
        out.append(x.float().contiguous())
    return out


def hann(rows, cols):
    def side(n):
        i = torch.arange(n, device="cuda", dtype=torch.float64)
        return 0.5 - 0.5 * torch.cos(2 * math.pi * i / max(n - 1, 1))
    return (side(rows)[:, None] * side(cols)[None, :]).float().contiguous()


def inputs_of(case, seed):
    """The case's input tensors, from the seed alone."""
    gen = torch.Generator("cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "plan":
        return [uniform_complex(sum(r * c for r, c in shapes_of(case)), gen)]
    if kind == "serve":
        return [(scene_pair(r, c, gen), hann(r, c)) for r, c in shapes_of(case)]
    rows, cols = case["rows"], case["cols"]
    if kind == "fft":
        return [uniform_complex(rows * cols, gen).view(rows, cols)]
    if kind == "real":
        return [torch.rand(rows, cols, generator=gen, device="cuda")]
    if kind == "batched":
        return [uniform_complex(case["count"] * rows * cols, gen).view(-1, rows, cols)]
    if kind == "poc":
        return scene_pair(rows, cols, gen) + [hann(rows, cols)]
    if kind == "display":
        return [scene_pair(rows, cols, gen)[0], hann(rows, cols)]
    return [uniform_complex(rows * cols, gen).view(rows, cols) for _ in range(2)]  # spectrum


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    kind, x = case["kind"], inputs_of(case, seed)
    s = {"kind": kind, "ctx": context(), "case": case, "x": x,
         "stream": torch.cuda.current_stream().cuda_stream}
    if kind in ("fft", "real", "batched"):
        s["flags"] = CHAINS[case["chain"]]
        s["y"] = [torch.empty(x[0].shape, dtype=torch.complex64, device="cuda") for _ in s["flags"]]
    elif kind == "plan":
        shapes = shapes_of(case)
        s["y"] = torch.empty_like(x[0])
        at, offsets = 0, []
        for r, c in shapes:
            offsets.append(8 * at)
            at += r * c
        s["plan"] = gls.Batch(s["ctx"], [x[0].data_ptr() + o for o in offsets],
                              [s["y"].data_ptr() + o for o in offsets], shapes, CHAINS[case["chain"]])
    elif kind == "display":
        s["y"] = torch.empty_like(x[0])
    elif kind == "serve":
        s["server"] = gls.Server(s["ctx"], slots=8, hbm_budget=1 << 30)
        s["requests"] = []
        for (ref, frame), window in x:
            host = torch.empty(frame.shape, dtype=torch.float32, pin_memory=True)
            host.copy_(frame)
            torch.cuda.synchronize()
            rid = s["server"].add_reference(ref.data_ptr(), window.data_ptr(), *ref.shape)
            s["requests"].append((rid, host))
        s["x"] = None
    elif kind == "spectrum":
        s["y"] = [torch.empty_like(x[0]), torch.empty_like(x[0].real), torch.empty_like(x[0].real)]
    return s


# --------------------------------------------------------------------- run
def run(state):
    kind, ctx, x, case, st = (state[k] for k in ("kind", "ctx", "x", "case", "stream"))
    if kind == "plan":
        state["plan"].execute(st)
        return state["y"]
    if kind == "serve":
        server = state["server"]
        tickets = [server.submit(rid, host.data_ptr()) for rid, host in state["requests"]]
        return [server.wait(t)[0] for t in tickets]
    rows, cols = case["rows"], case["cols"]
    if kind in ("fft", "real"):
        src, real = x[0], kind == "real"
        for dst, flags in zip(state["y"], state["flags"]):
            ctx.fft2d(src.data_ptr(), dst.data_ptr(), rows, cols, flags, st, real_input=real)
            src, real = dst, False
        return state["y"]
    if kind == "batched":
        src = x[0]
        for dst, flags in zip(state["y"], state["flags"]):
            ctx.fft2d_batched(src.data_ptr(), dst.data_ptr(), case["count"], rows, cols, flags, st)
            src = dst
        return state["y"]
    if kind == "poc":
        (dx, dy), response = ctx.phase_correlate(x[0].data_ptr(), x[1].data_ptr(), x[2].data_ptr(),
                                                 rows, cols, 5, st)
        return [dx, dy, response]
    if kind == "display":
        ctx.fft_display(x[0].data_ptr(), x[1].data_ptr(), state["y"].data_ptr(), rows, cols, 1.0, st)
        return state["y"]
    cross, mag, view = state["y"]
    ctx.mul_spectrums(x[0].data_ptr(), x[1].data_ptr(), cross.data_ptr(), rows, cols, True, st)
    ctx.mag_spectrums(cross.data_ptr(), mag.data_ptr(), rows, cols, st)
    ctx.normalize_minmax(mag.data_ptr(), view.data_ptr(), rows, cols, 0.0, 1.0, st)
    return state["y"]


# -------------------------------------------------------------------- work
def work(case):
    """Each input read once, each result written once; 5 N log2 N operations
    per transform of N pixels."""
    kind = case["kind"]
    fft = lambda n: 5.0 * n * math.log2(n)  # noqa: E731
    if kind == "plan":
        per = len(CHAINS[case["chain"]])
        px = [r * c for r, c in shapes_of(case)]
        return {"bytes": 16 * sum(px), "flops": per * sum(map(fft, px))}
    if kind == "serve":
        # the frame, the resident spectrum and the window in, five numbers out; two transforms
        px = [r * c for r, c in shapes_of(case)]
        return {"bytes": 16 * sum(px) + 40 * len(px), "flops": 2 * sum(map(fft, px))}
    n = case["rows"] * case["cols"]
    if kind in ("fft", "real", "batched"):
        per, count = len(CHAINS[case["chain"]]), case.get("count", 1)
        return {"bytes": count * n * ((4 if kind == "real" else 8) + 8 * per), "flops": count * per * fft(n)}
    if kind == "poc":
        return {"bytes": 12 * n + 24, "flops": 3 * fft(n)}
    if kind == "display":
        return {"bytes": 12 * n, "flops": fft(n)}
    # two spectra in, their product, its magnitude and the view out
    return {"bytes": 32 * n, "flops": 12 * n}


# ------------------------------------------------------------------- exact
def exact_fft(x, flags):
    """gls::fft over the last two dimensions in complex128."""
    n = x.shape[-1] * x.shape[-2]
    if flags & INV:
        y = torch.fft.ifft2(x) if flags & SCALE else torch.fft.ifft2(x) * n
    else:
        y = torch.fft.fft2(x) / n if flags & SCALE else torch.fft.fft2(x)
    return torch.fft.fftshift(y, dim=(-2, -1)) if flags & SHIFT else y


def exact_poc(a, b, window, box=5):
    """dx, dy, response, peak index and peak value in 64 bits."""
    rows, cols = a.shape
    w = window.double()
    t = torch.fft.fft2(w * a.double())
    t = t * torch.fft.fft2(w * b.double()).conj()
    mag = t.abs()
    phase = torch.where(mag > 0, t / mag.clamp_min(1e-300), torch.zeros_like(t))
    c = torch.fft.fftshift(torch.fft.ifft2(phase).real * (rows * cols))
    at = int(c.argmax())
    py, px, h = at // cols, at % cols, box // 2
    y0, y1, x0, x1 = max(py - h, 0), min(py + h, rows - 1), max(px - h, 0), min(px + h, cols - 1)
    v = c[y0:y1 + 1, x0:x1 + 1].cpu()
    total = float(v.sum())
    sx = float((v * torch.arange(x0, x1 + 1, dtype=torch.float64)[None, :]).sum())
    sy = float((v * torch.arange(y0, y1 + 1, dtype=torch.float64)[:, None]).sum())
    eps = 2.220446049250313e-16
    return [cols / 2 - sx / (total + eps), rows / 2 - sy / (total + eps), total / (rows * cols),
            float(at), float(c.flatten()[at])]


def exact(case, seed):
    kind, x = case["kind"], inputs_of(case, seed)
    if kind in ("fft", "real", "batched"):
        out, y = [], x[0].to(torch.complex128)
        for flags in CHAINS[case["chain"]]:
            y = exact_fft(y, flags)
            out.append(y)
        return out
    if kind == "plan":
        out, at = torch.empty(x[0].shape, dtype=torch.complex128, device="cuda"), 0
        for r, c in shapes_of(case):
            y = x[0][at:at + r * c].view(r, c).to(torch.complex128)
            for flags in CHAINS[case["chain"]]:
                y = exact_fft(y, flags)
            out[at:at + r * c] = y.flatten()
            at += r * c
        return out
    if kind == "serve":
        return [exact_poc(ref, frame, window) for (ref, frame), window in x]
    if kind == "poc":
        return exact_poc(*x)[:3]
    if kind == "display":
        y = torch.fft.fftshift(torch.fft.fft2(x[1].double() * x[0].double())).abs()
        y = torch.log(torch.abs(y + 1.0))
        return (y - y.min()) / (y.max() - y.min())
    a, b = (v.to(torch.complex128) for v in x)
    cross = a * b.conj()
    mag = cross.abs()
    return [cross, mag, (mag - mag.min()) / (mag.max() - mag.min())]
