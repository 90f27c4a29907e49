"""Paste jobs of the sizes this backend is used at, through its public entry points.

A case is one whole paste (or a batch of them): the solver's inputs are built
from uint8 images and then swept, as an editor, a command-line run or a
server does it.  Cases on device images go through ``reset_images`` and
``step_tensors``; cases on host images go through the processors, whose
result is the composed target on the host.

Fields of a case:
  via     "device" (CUDA images, results stay there), "host" (processor, numpy
          images in, composed target out), "solve" (sweeps to a residual
          bound) or "batch" (many jobs in one engine)
  method  "grid" or "equ"; order "jacobi" or "red_black"; precision of the
          sweep state "fp32", "fp16" or "bf16" (grid only)
  h, w    target and source size; shape / fill of the mask: "disk" (circle or
          ellipse filling that share of the image), "box" or "blob"
  gradient "src", "max" or "avg"; sweeps in all, run in `steps` equal steps
"""

from __future__ import annotations

import math

import numpy as np
import torch

from fpie_gb300.backend import EquSolver, GridSolver
from fpie_gb300.batch import BatchSolver
from fpie_gb300.process import EquProcessor, GridProcessor

_BASE = {"via": "device", "method": "grid", "order": "jacobi", "precision": "fp32",
         "shape": "disk", "fill": 0.75, "gradient": "max", "steps": 1}


def _case(**kw):
    return {**_BASE, **kw}


def listed():
    return [
        # A sticker-sized paste, first preview while it is dragged: latency only.
        _case(name="icon48_preview", h=48, w=48, gradient="src", sweeps=100),
        # The circle paste a CPU also manages (256x256, radius 96), whole run.
        _case(name="circle256_grid", h=256, w=256, gradient="src", sweeps=5000),
        # The same size as the command line runs it by default: equation
        # method, images in host memory, composed image back.
        _case(name="circle256_equ_host", via="host", method="equ", h=256, w=256, sweeps=5000),
        # An irregular selection with odd sides and an odd number of sweeps.
        _case(name="blob333x517_avg", h=333, w=517, shape="blob", gradient="avg", sweeps=777),
        # A banner: long, thin, a picture after every 100 sweeps (-p 100).
        _case(name="strip180x1500_progress", via="host", h=180, w=1500, shape="box", fill=0.97,
              sweeps=1000, steps=10),
        # The headline paste: an 800x800 square on 1024x1024, 5000 sweeps.
        _case(name="square800_grid", h=1024, w=1024, shape="box", fill=0.7817, sweeps=5000),
        # The same paste in the red-black order of the OpenMP equation solver.
        _case(name="square800_equ_rb", method="equ", order="red_black", h=1024, w=1024, shape="box",
              fill=0.7817, sweeps=1000),
        # A radius-450 circle with FP16 corrections (iterative refinement).
        _case(name="circle450_fp16", precision="fp16", h=1024, w=1024, fill=0.879, sweeps=2048),
        # A first preview of that circle from host images: mostly reset and copies.
        _case(name="circle450_preview_host", via="host", h=1024, w=1024, fill=0.879, sweeps=100),
        # A radius-1800 circle on 4096x4096: larger than L2.
        _case(name="circle1800_grid", h=4096, w=4096, fill=0.879, sweeps=512),
        # Sweeps to a residual bound, checked every 256 sweeps, state read back.
        _case(name="solve200", via="solve", h=200, w=200, sweeps=20000, tol=0.01),
        # A server's mix: 24 uneven jobs in one engine, images in and out.
        _case(name="batch24", via="batch", h=400, w=400, sweeps=2000, jobs=24),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    c = dict(_BASE)
    kind = rng.choice(["grid", "grid", "grid", "equ", "rb", "mixed", "host", "batch"])
    c["shape"] = rng.choice(["disk", "box", "blob"])
    c["fill"] = round(rng.uniform(0.5, 0.97), 3)
    c["gradient"] = rng.choice(["src", "max", "avg"])
    if kind == "batch":
        c.update(via="batch", h=log(96, 512), w=log(96, 512), sweeps=log(200, 3000), jobs=log(4, 24))
        return c
    c["h"] = log(32, 2200)
    c["w"] = min(3000, max(32, int(c["h"] * math.exp(rng.uniform(-1.2, 1.2)))))
    # At most 2e9 pixel updates: below the largest listed cases.
    c["sweeps"] = min(log(60, 6000), max(60, int(2e9 / (c["h"] * c["w"]))))
    if kind in ("equ", "rb"):
        c["method"] = "equ"
        c["order"] = "red_black" if kind == "rb" else "jacobi"
    if kind == "mixed":
        c["precision"] = rng.choice(["fp16", "bf16"])
    if kind == "host":
        c.update(via="host", method=rng.choice(["grid", "equ"]))
        c["steps"] = rng.choice([1, 4])
        c["sweeps"] -= c["sweeps"] % c["steps"]
    return c


# ---- inputs ----------------------------------------------------------------------


def _image(gen, h, w, base):
    """A photograph-like uint8 image: a smooth field plus noise of sigma 8."""
    field = torch.rand((1, 3, base, base), generator=gen, device="cuda") * 255.0
    img = torch.nn.functional.interpolate(field, size=(h, w), mode="bilinear", align_corners=True)[0]
    img = img + 8.0 * torch.randn((3, h, w), generator=gen, device="cuda")
    return img.round().clamp(0, 255).to(torch.uint8).permute(1, 2, 0).contiguous()


def _mask(gen, h, w, shape, fill):
    yy = torch.arange(h, device="cuda", dtype=torch.float64)[:, None]
    xx = torch.arange(w, device="cuda", dtype=torch.float64)[None, :]
    ry, rx = fill * h / 2, fill * w / 2
    dy, dx = (yy - h // 2), (xx - w // 2)
    if shape == "disk":
        on = (dy / ry) ** 2 + (dx / rx) ** 2 <= 1.0
    elif shape == "box":
        on = (dy.abs() < ry) & (dx.abs() < rx)
    else:  # smoothed noise over its mean, inside the box
        k = max(3, min(h, w) // 12) | 1
        noise = torch.rand((1, 1, h, w), generator=gen, device="cuda", dtype=torch.float64)
        for _ in range(2):
            noise = torch.nn.functional.avg_pool2d(noise, k, 1, k // 2, count_include_pad=False)
        on = (noise[0, 0] > noise.mean() - 0.3 * noise.std()) & (dy.abs() < ry) & (dx.abs() < rx)
    on[h // 2, w // 2] = True
    return on.to(torch.uint8) * 255


def _images(case, seed):
    """(src, mask, tgt) as CUDA uint8 tensors."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    h, w = case["h"], case["w"]
    base = min(32, max(4, min(h, w) // 16))
    return (_image(gen, h, w, base), _mask(gen, h, w, case["shape"], case["fill"]),
            _image(gen, h, w, base))


def _job_cases(case):
    """The uneven jobs of a batch: sides from 32 up to the case's, all shapes."""
    r = np.random.default_rng(case["jobs"])
    out = []
    for k in range(case["jobs"]):
        h, w = (int(round(math.exp(r.uniform(math.log(32), math.log(case[s]))))) for s in "hw")
        out.append(dict(case, h=h, w=w, shape=("disk", "box", "blob")[k % 3],
                        gradient=("src", "max", "avg")[(k // 3) % 3],
                        sweeps=int(case["sweeps"] * r.uniform(0.5, 1.5))))
    return out


def _host(images):
    return tuple(t.cpu().numpy() for t in images)


# ---- one pass ----------------------------------------------------------------------


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    if case["via"] == "batch":
        s.jobs = [(j, _host(_images(j, seed + 1000 * (k + 1)))) for k, j in enumerate(_job_cases(case))]
        s.batch = BatchSolver(8e9)
        return s
    images = _images(case, seed)
    equ, rb = case["method"] == "equ", case["order"] == "red_black"
    if case["via"] == "host":
        s.images = _host(images)
        cls = EquProcessor if equ else GridProcessor
        s.proc = cls(case["gradient"], "gb300-rb" if rb else "gb300", device_prep=True)
        return s
    s.images = images
    s.solver = EquSolver(1024, order=case["order"]) if equ else GridSolver(8, 8)
    s.solver.set_stream(torch.cuda.current_stream().cuda_stream)
    if case["precision"] != "fp32":
        s.solver.set_precision(case["precision"])
    s.err = torch.empty(3, dtype=torch.float32, device="cuda")
    return s


def run(state):
    c = state.case
    if c["via"] == "batch":
        b = state.batch
        ids = [b.add_images(*im, (0, 0), (0, 0), j["gradient"], j["sweeps"])[0] for j, im in state.jobs]
        b.run()
        res = [b.result(i) for i in ids]
        for i in ids:
            b.remove(i)
        return [r[0] for r in res], [r[1] for r in res]
    src, mask, tgt = state.images
    k = c["sweeps"] // c["steps"]
    if c["via"] == "host":
        state.proc.reset(src, mask, tgt, (0, 0), (0, 0))
        for _ in range(c["steps"]):
            out, err = state.proc.step(k)
        return out, err
    s = state.solver
    got = s.reset_images(src, mask, tgt, (0, 0), (0, 0), c["gradient"])
    if c["via"] == "solve":
        return s.solve(c["tol"], c["sweeps"], 256), s.state()
    shape = (got[0], 3) if c["method"] == "equ" else (got[1] - got[0], got[3] - got[2], 3)
    out = torch.empty(shape, dtype=torch.uint8, device="cuda")
    for _ in range(c["steps"]):
        s.step_tensors(k, out, state.err)
    return out, state.err


# ---- what a pass cannot do without, and its result in 64 bits ------------------------


def _unknowns(case):
    h, w, f = case["h"], case["w"], case["fill"]
    area = {"disk": math.pi / 4, "box": 1.0, "blob": 0.6}[case["shape"]]
    return f * f * h * w * area, min(h, f * h + 2) * min(w, f * w + 2)


def work(case):
    if case["via"] == "batch":
        each = [work(dict(j, via="device")) for j in _job_cases(case)]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    n, crop = _unknowns(case)
    # The crop of both images and the mask once; per step a picture.  Four
    # additions and a multiplication per unknown, channel and sweep.
    return {"bytes": case["h"] * case["w"] + crop * (6 + 3 * case["steps"]),
            "flops": n * 3 * 5 * case["sweeps"]}


def _exact_paste(case, images):
    """(mask, state, |residual| sums) in float64, the solver's iteration in torch."""
    src, mask, tgt = images
    on = mask >= 128
    on[0], on[-1], on[:, 0], on[:, -1] = False, False, False, False
    r, c = on.any(1).nonzero()[:, 0], on.any(0).nonzero()[:, 0]
    box = (slice(int(r[0]) - 1, int(r[-1]) + 2), slice(int(c[0]) - 1, int(c[-1]) + 2))
    on = on[box]
    s, t = (a[box].permute(2, 0, 1).double() for a in (src, tgt))
    g = torch.zeros_like(t)
    for dim in (1, 2):
        for sign in (1, -1):
            ds, dt = s - s.roll(sign, dim), t - t.roll(sign, dim)
            if case["gradient"] == "src":
                d = ds
            elif case["gradient"] == "avg":
                d = (ds + dt) / 2
            else:
                d = torch.where(ds.abs() < dt.abs(), dt, ds)
            g += d  # the rolled-in rows are outside the mask, which never touches the frame
    g *= on
    x = torch.nn.functional.pad(t, (1, 1, 1, 1))
    mid = x[:, 1:-1, 1:-1]

    def near():
        return x[:, :-2, 1:-1] + x[:, 2:, 1:-1] + x[:, 1:-1, :-2] + x[:, 1:-1, 2:]

    def residual():
        return (4 * mid - g - near()) * on

    yy, xx = (torch.arange(k, device="cuda") for k in on.shape)
    odd = (yy[:, None] + xx[None, :]) % 2 == 1
    halves = (on & odd, on & ~odd) if case["order"] == "red_black" else (on,)
    done = 0
    while done < case["sweeps"]:
        if case["via"] == "solve" and done % 256 == 0 and float(residual().abs().max()) <= case["tol"]:
            break
        for part in halves:
            mid.copy_(torch.where(part, (g + near()) * 0.25, mid))
        done += 1
    err = residual().abs().sum((1, 2))
    # A converged paste's residual is the rounding of the swept values (ulps
    # of intensities up to 255), not a figure that 64 bits reproduce.
    return mid, err if float(err.min()) > 0.01 * float(on.sum()) else None


def exact(case, seed):
    if case["via"] == "batch":
        jobs = _job_cases(case)
        errs = [_exact_paste(dict(j, via="device"), _images(j, seed + 1000 * (k + 1)))[1]
                for k, j in enumerate(jobs)]
        return ([None] * len(jobs), errs) if any(e is not None for e in errs) else None
    x, err = _exact_paste(case, _images(case, seed))
    if case["via"] == "solve":
        return None, x.permute(1, 2, 0).contiguous()
    return None if err is None else (None, err)
