"""Workloads of the transform engine, timed through its public Python entry points.

Four kinds of call, as a program that uses the engine makes them:

* ``grid``  — one N-D grid, R2C or C2C, the way the grid-owning backend drives
  it: the passes of a transform are recorded once as a group, captured, and
  each transform replays its graph and waits for it, as ParaFaFT's forward()
  and backward() return only when they are done.
* ``plane`` — a 2-D grid through the per-stage calls of a handle (memcpy or
  memcpy2d, exec_*, sync), the way ParaFaFT drives its per-stage backend.
* ``grids`` — many independent grids of uneven sizes in one group.
* ``batch`` — a batched 1-D transform through the entry point that needs no
  handle and no allocation, ordered on the caller's stream.

Every pass runs forward and backward (unnormalised) and leaves its inputs as
they were: ``spectrum`` is the forward transform of the input and ``back`` the
backward transform of that spectrum, N times the input.
"""
import math

import torch

from parafaft_b200 import native as nv

# Sides of the uneven grids (factors 2, 3, 5).
UNEVEN_SIDES = (32, 48, 60, 64, 80, 96, 120, 128, 160)


def listed():
    return [
        # The headline: a 512^3 lattice in single precision.
        {"name": "r2c_512_f32", "kind": "grid", "shape": "512x512x512", "real": True,
         "f64": False, "split": False},
        # The reference's default precision on an everyday lattice.
        {"name": "r2c_256_f64", "kind": "grid", "shape": "256x256x256", "real": True,
         "f64": True, "split": False},
        # A small lattice in a time-stepping loop: latency and launches count.
        {"name": "c2c_64_f64", "kind": "grid", "shape": "64x64x64", "real": False,
         "f64": True, "split": False},
        # The largest grid of the benchmark, 8 GiB.
        {"name": "c2c_1024_f32", "kind": "grid", "shape": "1024x1024x1024", "real": False,
         "f64": False, "split": False},
        # Any dimension: a 4-D grid in double precision.
        {"name": "c2c_4d_f64", "kind": "grid", "shape": "128x128x64x64", "real": False,
         "f64": True, "split": False},
        # Lattices whose sides are not powers of two (factors 2, 3, 5, 7).
        {"name": "r2c_ragged_f32", "kind": "grid", "shape": "300x270x350", "real": True,
         "f64": False, "split": False},
        {"name": "c2c_ragged_f64", "kind": "grid", "shape": "180x140x225", "real": False,
         "f64": True, "split": False},
        # The split-precision tensor-core option on a 512^3 grid.
        {"name": "c2c_512_split", "kind": "grid", "shape": "512x512x512", "real": False,
         "f64": False, "split": True},
        # 2-D fields through the per-stage calls: the longest axes, and odd sides
        # with the out-of-place pad.
        {"name": "plane_4096_f32", "kind": "plane", "shape": "4096x4096", "real": False,
         "f64": False},
        {"name": "plane_odd_f64", "kind": "plane", "shape": "1225x1125", "real": True,
         "f64": True},
        # 256 independent grids of uneven sizes as one batch.
        {"name": "grids_256_f32", "kind": "grids", "count": 256, "side_seed": 2024},
        # The smallest calls: short columns where the caller may not allocate.
        {"name": "batch_128_f32", "kind": "batch", "length": 128, "batch": 512, "col": True,
         "f64": False},
    ]


# ---- drawing more cases of the same ranges ---------------------------------

def _good_sizes(lo, hi):
    """Sides people pick for FFTs: 2^a 3^b 5^c 7^d, with at most one 11 or 13."""
    out = []
    for n in range(lo, hi + 1):
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m in (1, 11, 13):
            out.append(n)
    return out


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _side(rng, about, lo, hi):
    """A side near `about`: often a power of two, else any good size, odd ones too."""
    about = min(max(about, lo), hi)
    if rng.random() < 0.45:
        sizes = [1 << k for k in range(1, 13) if lo <= (1 << k) <= hi]
    else:
        sizes = [n for n in _good_sizes(lo, hi) if 0.85 * about <= n <= 1.18 * about]
        if sizes:
            return rng.choice(sizes)
        sizes = _good_sizes(lo, hi)
    return min(sizes, key=lambda n: abs(math.log(n / about)))


def draw(rng):
    kind = rng.choice(("grid", "grid", "grid", "grid", "split", "plane", "plane", "grids",
                       "batch", "batch"))
    if kind == "grid":
        dims = rng.choice((3, 3, 3, 3, 4, 5))
        points = _log_uniform(rng, 1 << 12, 1 << (27 if dims == 3 else 25 if dims == 4 else 20))
        mean = points ** (1.0 / dims)
        lo, hi = (8, 1024) if dims == 3 else (8, 160) if dims == 4 else (4, 32)
        if rng.random() < 0.4:
            shape = [_side(rng, mean, lo, hi)] * dims
        else:
            shape = [_side(rng, mean * _log_uniform(rng, 0.5, 2.0), lo, hi) for _ in range(dims)]
        return {"kind": "grid", "shape": "x".join(map(str, shape)), "real": rng.random() < 0.6,
                "f64": rng.random() < 0.5, "split": False}
    if kind == "split":
        shape = [rng.choice((256, 512)), rng.choice((256, 512)), rng.choice((256, 512, 1024))]
        return {"kind": "grid", "shape": "x".join(map(str, shape)), "real": False, "f64": False,
                "split": True}
    if kind == "plane":
        shape = [_side(rng, _log_uniform(rng, 64, 4096), 32, 4096) for _ in range(2)]
        return {"kind": "plane", "shape": "x".join(map(str, shape)), "real": rng.random() < 0.5,
                "f64": rng.random() < 0.5}
    if kind == "grids":
        return {"kind": "grids", "count": round(_log_uniform(rng, 8, 256)),
                "side_seed": rng.randrange(1 << 20)}
    length = 1 << rng.randint(4, 12)
    batch = max(1, round(_log_uniform(rng, 1 << 10, 1 << 24) / length))
    return {"kind": "batch", "length": length, "batch": batch, "col": rng.random() < 0.5,
            "f64": rng.random() < 0.5}


# ---- shapes, inputs, work --------------------------------------------------

def _shape(case):
    return tuple(int(s) for s in case["shape"].split("x"))


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uneven_shapes(case):
    """Sides of the grids, drawn from side_seed, ordered by their last side."""
    import random
    r = random.Random(case["side_seed"])
    shapes = [tuple(r.choice(UNEVEN_SIDES) for _ in range(3)) for _ in range(case["count"])]
    return sorted(shapes, key=lambda s: s[2])


def _field(shape, gen):
    """A zero-mean Gaussian random field with power spectrum P(k) ~ k^-3."""
    noise = torch.randn(shape, generator=gen, device="cuda")
    k2 = 0.0
    for d, n in enumerate(shape):
        k = (torch.fft.rfftfreq(n, 1.0 / n, device="cuda") if d == len(shape) - 1
             else torch.fft.fftfreq(n, 1.0 / n, device="cuda"))
        k2 = k2 + (k * k).reshape([-1 if i == d else 1 for i in range(len(shape))])
    amp = torch.where(k2 > 0, k2.clamp(min=1.0) ** -0.75, torch.zeros_like(k2))
    f = torch.fft.irfftn(torch.fft.rfftn(noise) * amp, s=shape)
    return f / f.std()


def _input(case, seed):
    """The input of a pass as a list of tensors (one, except for ``grids``)."""
    g = _generator(seed)
    if case["kind"] == "grids":
        return [_field(s, g) for s in _uneven_shapes(case)]
    if case["kind"] == "batch":
        n, b = case["length"], case["batch"]
        shape, real = ((n, b) if case["col"] else (b, n)), False
    else:
        shape, real = _shape(case), case["real"]
    rdt = torch.float64 if case["f64"] else torch.float32
    full = shape if real else shape + (2,)
    if case["f64"]:  # double precision grids: uniform on [-1, 1)
        x = torch.rand(full, generator=g, device="cuda", dtype=rdt).mul_(2).sub_(1)
    else:
        x = torch.randn(full, generator=g, device="cuda", dtype=rdt)
    return [x if real else torch.view_as_complex(x)]


def work(case):
    """Bytes: forward and backward each read their input once and write their
    output once. Operations: 5 N log2 N per complex transform, half for real."""
    if case["kind"] == "grids":
        total = flops = 0
        for s in _uneven_shapes(case):
            n = s[0] * s[1] * s[2]
            total += 2 * (4 * n + 8 * s[0] * s[1] * (s[2] // 2 + 1))
            flops += 2 * 2.5 * n * math.log2(n)
        return {"bytes": total, "flops": flops}
    rsize = 8 if case["f64"] else 4
    if case["kind"] == "batch":
        n = case["length"] * case["batch"]
        return {"bytes": 8 * rsize * n, "flops": 2 * 5.0 * n * math.log2(case["length"])}
    shape = _shape(case)
    n = math.prod(shape)
    if case["real"]:
        half = n // shape[-1] * (shape[-1] // 2 + 1)
        return {"bytes": 2 * rsize * (n + 2 * half), "flops": 2 * 2.5 * n * math.log2(n)}
    return {"bytes": 8 * rsize * n, "flops": 2 * 5.0 * n * math.log2(n)}


# ---- plans -----------------------------------------------------------------

def _plan_axes(h, shape, real):
    """One stage per axis that is transformed complex (all but the last for R2C)."""
    d = len(shape)
    w = shape[-1] // 2 + 1 if real else shape[-1]
    dims = shape[:-1] + (w,)
    for ax in range(d - 1):
        trail = math.prod(dims[ax + 1:])
        h.plan_c2c(ax, shape[ax], trail, trail, 1)
    rows = math.prod(shape[:-1])
    if real:
        h.plan_r2c(shape[-1], rows, 1, 2 * w)
        h.plan_c2r(shape[-1], rows, 1, 2 * w)
    else:
        h.plan_c2c(d - 1, shape[-1], rows, 1, shape[-1])
    return dims


def _axis(h, dims, ax, direction, ptr, csize):
    """Every leading slice of a strided axis, as ParaFaFT issues them."""
    slab = math.prod(dims[ax:]) * csize
    for i in range(math.prod(dims[:ax])):
        h.exec_c2c(ax, direction, ptr + i * slab)


def _forward(h, shape, real, out, src, nbytes, csize):
    dims = shape[:-1] + ((shape[-1] // 2 + 1) if real else shape[-1],)
    d = len(shape)
    if src != out:
        h.memcpy(out, src, nbytes)
    if real:
        h.exec_r2c(out)
    else:
        h.exec_c2c(d - 1, nv.FORWARD, out)
    for ax in range(d - 2, -1, -1):
        _axis(h, dims, ax, nv.FORWARD, out, csize)


def _backward(h, shape, real, out, src, nbytes, csize):
    dims = shape[:-1] + ((shape[-1] // 2 + 1) if real else shape[-1],)
    d = len(shape)
    h.memcpy(out, src, nbytes)
    for ax in range(d - 1):
        _axis(h, dims, ax, nv.BACKWARD, out, csize)
    if real:
        h.exec_c2r(out)
    else:
        h.exec_c2c(d - 1, nv.BACKWARD, out)


def _padded(x):
    """Real rows in the in-place layout: 2 * (n // 2 + 1) reals per row."""
    n = x.shape[-1]
    p = torch.zeros(x.shape[:-1] + (2 * (n // 2 + 1),), dtype=x.dtype, device=x.device)
    p[..., :n] = x
    return p


def _prepare_grid(case, seed):
    shape, real = _shape(case), case["real"]
    prec = nv.F64 if case["f64"] else nv.F32
    flags = nv.FLAG_SPLIT_TC if case["split"] else 0
    x = _input(case, seed)[0]
    if real:
        x = _padded(x)
    spec, back = torch.zeros_like(x), torch.zeros_like(x)
    nbytes = x.numel() * x.element_size()
    csize = 16 if case["f64"] else 8
    torch.cuda.synchronize()
    groups = []
    for step, out, src in ((_forward, spec, x), (_backward, back, spec)):
        h = nv.Handle(prec, len(shape), flags=flags)
        _plan_axes(h, shape, real)
        g = nv.Group([h])
        g.begin()
        step(h, shape, real, out.data_ptr(), src.data_ptr(), nbytes, csize)
        g.end()
        g.sync()
        g.capture()
        groups.append(g)
    n = shape[-1]
    outs = {"spectrum": torch.view_as_complex(spec.view(spec.shape[:-1] + (-1, 2))) if real
            else spec, "back": back[..., :n] if real else back}
    return {"kind": "grid", "groups": groups, "x": x, "spec": spec, "back_buf": back,
            "outs": outs}


def _prepare_plane(case, seed):
    shape, real = _shape(case), case["real"]
    x = _input(case, seed)[0]
    rows, n = shape
    pitch = 2 * (n // 2 + 1) if real else n
    spec = torch.zeros((rows, pitch), dtype=x.dtype, device="cuda")
    back = torch.zeros_like(spec)
    h = nv.Handle(nv.F64 if case["f64"] else nv.F32, 2)
    _plan_axes(h, shape, real)
    torch.cuda.synchronize()
    outs = {"spectrum": torch.view_as_complex(spec.view(rows, -1, 2)) if real else spec,
            "back": back[:, :n]}
    return {"kind": "plane", "h": h, "real": real, "shape": shape, "x": x, "spec": spec,
            "back_buf": back, "esize": x.element_size(), "outs": outs}


def _prepare_grids(case, seed):
    """All grids in one buffer, each grid's rows padded and its start aligned to
    256 bytes; grids of the same last side lie one after another."""
    shapes = _uneven_shapes(case)
    fields = _input(case, seed)
    starts, spans, at = [], {}, 0
    for s in shapes:
        pitch = 2 * (s[2] // 2 + 1)
        rows = -(-(s[0] * s[1]) // 32) * 32  # whole 256-byte units of any even pitch
        starts.append(at)
        lo, _ = spans.get(s[2], (at, at))
        at += rows * pitch
        spans[s[2]] = (lo, at)
    x = torch.zeros(at, device="cuda")
    for s, f, o in zip(shapes, fields, starts):
        pitch = 2 * (s[2] // 2 + 1)
        x[o:o + s[0] * s[1] * pitch].view(s[0] * s[1], pitch)[:, :s[2]] = f.view(-1, s[2])
    spec, back = torch.zeros_like(x), torch.zeros_like(x)
    torch.cuda.synchronize()
    handles = []
    for s in shapes:
        h = nv.Handle(nv.F32, 3)
        _plan_axes(h, s, True)
        handles.append(h)
    g = nv.Group(handles)
    g.begin()
    for h, s, o in zip(handles, shapes, starts):
        nbytes = 8 * s[0] * s[1] * (s[2] // 2 + 1)
        px, ps, pb = (t.data_ptr() + 4 * o for t in (x, spec, back))
        _forward(h, s, True, ps, px, nbytes, 8)
        _backward(h, s, True, pb, ps, nbytes, 8)
    g.end()
    g.sync()
    g.capture()
    outs = {}
    for n, (lo, hi) in spans.items():
        w = n // 2 + 1
        outs["spectrum_%03d" % n] = torch.view_as_complex(spec[lo:hi].view(-1, w, 2))
        outs["back_%03d" % n] = back[lo:hi].view(-1, 2 * w)[:, :n]
    return {"kind": "grids", "groups": [g], "handles": handles, "x": x, "spec": spec,
            "back_buf": back, "outs": outs}


def _prepare_batch(case, seed):
    x = _input(case, seed)[0]
    n, b = case["length"], case["batch"]
    return {"kind": "batch", "x": x, "outs": {"spectrum": torch.zeros_like(x),
                                              "back": torch.zeros_like(x)},
            "args": (n, b, b, 1) if case["col"] else (n, b, 1, n),
            "prec": nv.F64 if case["f64"] else nv.F32}


def prepare(case, seed):
    return {"grid": _prepare_grid, "plane": _prepare_plane, "grids": _prepare_grids,
            "batch": _prepare_batch}[case["kind"]](case, seed)


def run(state):
    outs = state["outs"]
    if state["kind"] == "batch":
        stream = torch.cuda.current_stream().cuda_stream
        nv.c2c_noalloc(state["prec"], nv.FORWARD, *state["args"], state["x"], outs["spectrum"],
                       stream)
        nv.c2c_noalloc(state["prec"], nv.BACKWARD, *state["args"], outs["spectrum"],
                       outs["back"], stream)
    elif state["kind"] == "plane":
        h, (rows, n), e = state["h"], state["shape"], state["esize"]
        x, spec, back = (state[k].data_ptr() for k in ("x", "spec", "back_buf"))
        nbytes = state["spec"].numel() * e
        if state["real"]:  # forward(real, complex): the pad copy comes first
            h.memcpy2d(spec, 2 * (n // 2 + 1) * e, x, n * e, n * e, rows)
            _forward(h, (rows, n), True, spec, spec, nbytes, 2 * e)
        else:
            _forward(h, (rows, n), False, spec, x, nbytes, e)
        h.sync()
        _backward(h, (rows, n), state["real"], back, spec, nbytes, 2 * e if state["real"] else e)
        h.sync()
    else:
        for g in state["groups"]:
            g.replay()
            g.sync()
    return outs


# ---- what run() returns, in 64 bits ----------------------------------------

def exact(case, seed):
    xs = [x.to(torch.complex128 if x.is_complex() else torch.float64)
          for x in _input(case, seed)]
    if case["kind"] == "grids":
        outs = {}
        for n in sorted({s[2] for s in _uneven_shapes(case)}):
            spec, back = [], []
            for s, x in zip(_uneven_shapes(case), xs):
                if s[2] != n:
                    continue
                rows = s[0] * s[1]
                gap = -rows % 32
                spec += [torch.fft.rfftn(x).reshape(rows, -1),
                         torch.zeros(gap, n // 2 + 1, dtype=torch.complex128, device="cuda")]
                back += [(x * x.numel()).reshape(rows, n),
                         torch.zeros(gap, n, dtype=torch.float64, device="cuda")]
            outs["spectrum_%03d" % n] = torch.cat(spec)
            outs["back_%03d" % n] = torch.cat(back)
        return outs
    x = xs[0]
    if case["kind"] == "batch":
        return {"spectrum": torch.fft.fft(x, dim=0 if case["col"] else 1),
                "back": x * case["length"]}
    return {"spectrum": torch.fft.rfftn(x) if case["real"] else torch.fft.fftn(x),
            "back": x * x.numel()}
