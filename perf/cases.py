"""Performance cases of the stencil solver, through its public entry points.

Three kinds of work that a user's program has the library do:

* ``solve``: one grid on the device, T steps, through a kept plan (``Plan.run``);
* ``host``:  one grid in pinned host buffers, copies included (``Plan.run_host``);
* ``batch``: many problems of mixed dimension, size, shape and T in one call
  (``Batch.execute``), inputs and outputs on the device.

The ranges: 1-D grids of 2^12 .. 2^26 cells, 2-D sides of 64 .. 8192, 3-D sides of 32 ..
512, T of 1 .. 128, all nine shapes, both boundaries, every arithmetic form.  Sizes with a
name elsewhere in the repository (Heat-1D 2^20, Box2D9P 4096^2, Box2D25P 8192^2, Box3D27P
512^3, the mixed batch) are the benchmark's; the small ones are of the tests' kind.
"""
import math

import numpy as np
import torch

import flashfftstencil_b200 as ffs

# shape -> (dimension, radius, star: only taps on the axes)
SHAPES = {
    "Heat-1D": (1, 1, False), "1D5P": (1, 2, False), "1D7P": (1, 3, False),
    "Heat-2D": (2, 1, True), "Star2D9P": (2, 2, True), "Box2D9P": (2, 1, False), "Box2D25P": (2, 2, False),
    "Heat-3D": (3, 1, True), "Box3D27P": (3, 1, False),
}
BY_DIM = {d: [s for s, v in SHAPES.items() if v[0] == d] for d in (1, 2, 3)}


def _solve(name, shape, T, boundary, nx, ny=1, nz=1, form="auto", weights="positive", kind="solve"):
    return {"name": name, "kind": kind, "shape": shape, "nx": nx, "ny": ny, "nz": nz, "T": T, "boundary": boundary,
            "form": form, "weights": weights}


def listed():
    return [
        # the smallest calls: a few tens of microseconds, launches and host work count
        _solve("line-10000", "1D5P", 16, "periodic", 10_000),
        _solve("plate-300x260", "Heat-2D", 12, "fixed", 300, 260),
        _solve("block-100x90x70", "Heat-3D", 10, "periodic", 100, 90, 70),
        # a long line in one fused pass (the 1-D benchmark problem)
        _solve("heat-1d-2^20", "Heat-1D", 64, "fixed", 1 << 20),
        # a few steps between two uses of the grid (output, coupling), odd sides
        _solve("star-1999x2047-few", "Star2D9P", 4, "periodic", 1999, 2047),
        # the headline: a large plate with drawn weights and a held ring
        _solve("box-4096", "Box2D9P", 32, "fixed", 4096, 4096),
        # the largest plate and the longest fused run, weights of both signs
        _solve("box25-8192", "Box2D25P", 128, "periodic", 8192, 8192, weights="signed"),
        # the large volume
        _solve("box27-512", "Box3D27P", 16, "fixed", 512, 512, 512),
        # ordinary plate and volume in the matrix forms that a caller may ask for by name
        _solve("box-1536x1024-fp64", "Box2D9P", 24, "fixed", 1536, 1024, form="fp64"),
        _solve("box27-128-ozaki", "Box3D27P", 16, "fixed", 128, 128, 128, form="ozaki"),
        # the headline grid from and to pinned host memory
        _solve("host-4096", "Box2D9P", 32, "fixed", 4096, 4096, kind="host"),
        # many independent problems in one call
        {"name": "batch-96", "kind": "batch", "count": 96, "mix": 1, "form": "auto"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["solve", "host", "batch"], [0.8, 0.1, 0.1])[0]
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(16, 96), "mix": rng.randrange(1 << 20), "form": "auto"}
    dim = rng.choices([1, 2, 3], [0.2, 0.5, 0.3])[0]
    shape = rng.choice(BY_DIM[dim])
    form = "auto" if kind == "host" else rng.choices(["auto", "fp64", "ozaki", "bf16x3"], [0.76, 0.1, 0.07, 0.07])[0]
    if dim == 1 and form in ("ozaki", "bf16x3"):  # tensor-core forms are 2-D and 3-D
        form = "fp64"
    lo, hi = {1: (1 << 12, 1 << 26), 2: (64, 8192), 3: (32, 512)}[dim]
    if form != "auto":  # the matrix forms do several times the work per cell: up to a quarter of the side
        hi = {1: 1 << 22, 2: 2048, 3: 128}[dim]
    first = _log_int(rng, lo, hi)
    sides = [first] + [max(lo, min(hi, int(first * rng.uniform(0.6, 1.6)))) for _ in range(dim - 1)]
    if rng.random() < 0.3:  # whole multiples of 32, as programs often have
        sides = [max(lo, s // 32 * 32) for s in sides]
    sides += [1] * (3 - dim)
    cells = sides[0] * sides[1] * sides[2]
    limit = {1: 4e9, 2: 8e9, 3: 2e9}[dim] if form == "auto" else {1: 2e8, 2: 2e8, 3: 3e7}[dim]
    T = max(1, min(_log_int(rng, 1, 128), int(limit // cells)))
    weights = "signed" if rng.random() < 0.25 and not SHAPES[shape][2] else "positive"
    return {"kind": kind, "shape": shape, "nx": sides[0], "ny": sides[1], "nz": sides[2], "T": T,
            "boundary": rng.choice(["fixed", "periodic"]), "form": form, "weights": weights}


def _weights(shape, rng, kind):
    """Dense weights of a shape, dx fastest: uniform and summing to 1, or normal and scaled to a spectral radius of 1."""
    dim, r, star = SHAPES[shape]
    K = 2 * r + 1
    w = rng.standard_normal((K,) * dim) if kind == "signed" else rng.random((K,) * dim)
    if star:
        axes = np.abs(np.indices((K,) * dim) - r)
        w = np.where((axes > 0).sum(axis=0) <= 1, w, 0.0)
    if kind == "signed":
        return w / np.abs(np.fft.fftn(w, s=({1: 4096, 2: 512, 3: 64}[dim],) * dim)).max()
    return w / w.sum()


def _grid(shape, rng_seed, signed):
    g = torch.Generator(device="cuda").manual_seed(rng_seed)
    x = torch.rand(shape, generator=g, dtype=torch.float64, device="cuda")
    return (2.0 * x - 1.0) if signed else x


def _mix(case):
    """The problems of a batch: 60 % 2-D, 30 % 1-D, 10 % 3-D, sizes log-uniform, T uniform in 1 .. 64."""
    rng = np.random.default_rng(case["mix"])
    problems = []
    for i in range(case["count"]):
        u = rng.random()
        if u < 0.6:
            shape = ["Heat-2D", "Star2D9P", "Box2D9P"][rng.integers(3)]
            lo, hi, n = 64, 2048, 2
        elif u < 0.9:
            shape = ["1D5P", "1D7P"][rng.integers(2)]
            lo, hi, n = 1 << 12, 1 << 20, 1
        else:
            shape = ["Heat-3D", "Box3D27P"][rng.integers(2)]
            lo, hi, n = 32, 256, 3
        ext = tuple(int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(n))
        problems.append((shape, ext, int(rng.integers(1, 65)), ["fixed", "periodic"][rng.integers(2)]))
    return problems


def _extents(case):
    return (case["nx"], case["ny"], case["nz"])[: SHAPES[case["shape"]][0]]


def _plan(shape, ext, T, w, boundary, form):
    dim, r, _ = SHAPES[shape]
    return ffs.Plan(dim, shape, ext, T, weights=w, radius=r, boundary=boundary, form=form)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        plans, ins, outs = [], [], []
        problems = _mix(case)
        cells = [math.prod(ext) for _, ext, _, _ in problems]
        pad = [(c + 31) // 32 * 32 for c in cells]  # each problem starts on a 256-byte boundary
        flat_in = _grid((sum(pad),), seed, False)
        flat_out = torch.zeros_like(flat_in)
        at = 0
        for (shape, ext, T, boundary), size in zip(problems, pad):
            plans.append(_plan(shape, ext, T, _weights(shape, rng, "positive"), boundary, case["form"]))
            ins.append(flat_in.data_ptr() + 8 * at)
            outs.append(flat_out.data_ptr() + 8 * at)
            at += size
        return {"kind": "batch", "batch": ffs.Batch(plans), "plans": plans, "in": flat_in, "out": flat_out, "ins": ins,
                "outs": outs}
    ext = _extents(case)
    w = _weights(case["shape"], rng, case["weights"])
    plan = _plan(case["shape"], ext, case["T"], w, case["boundary"], case["form"])
    x = _grid(tuple(reversed(ext)), seed, case["weights"] == "signed")
    if case["kind"] == "host":
        host = torch.empty(x.shape, dtype=torch.float64, pin_memory=True)
        host.copy_(x)
        back = torch.empty(x.shape, dtype=torch.float64, pin_memory=True)
        return {"kind": "host", "plan": plan, "x": host.numpy(), "out": back.numpy(), "keep": (host, back)}
    return {"kind": "solve", "plan": plan, "x": x, "out": torch.empty_like(x)}


def run(state):
    if state["kind"] == "batch":
        state["batch"].execute(state["ins"], state["outs"], stream=torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if state["kind"] == "host":
        return state["plan"].run_host(state["x"], state["out"])
    return state["plan"].run(state["x"], state["out"])


def _least(shape, ext, T):
    """(bytes, flops) that T steps of one grid cannot do without: each cell read and written once; direct steps, or one
    real transform of the grid each way and the product with the spectrum, whichever is less."""
    dim, r, star = SHAPES[shape]
    taps = 1 + 2 * r * dim if star else (2 * r + 1) ** dim
    cells = math.prod(ext)
    return 16.0 * cells, cells * min(2.0 * taps * T, 5.0 * math.log2(cells) + 3.0)


def work(case):
    todo = [(s, e, T) for s, e, T, _ in _mix(case)] if case["kind"] == "batch" else [(case["shape"], _extents(case), case["T"])]
    each = [_least(*t) for t in todo]
    return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}


def _stepped(x, w, T, boundary):
    """T direct steps of the centred correlation, in 64 bits."""
    dim, r = x.dim(), (w.shape[0] - 1) // 2
    taps = [(idx, float(w[idx])) for idx in np.ndindex(*w.shape) if w[idx] != 0.0]
    for _ in range(T):
        if boundary == "periodic":
            p = x
            for d in range(dim):
                n = x.shape[d]
                p = p.index_select(d, torch.arange(-r, n + r, device=x.device) % n)
            acc = torch.zeros_like(x)
            for idx, v in taps:
                acc.add_(p[tuple(slice(i, i + n) for i, n in zip(idx, x.shape))], alpha=v)
            x = acc
        elif all(n > 2 * r for n in x.shape):  # the ring of width r keeps its values
            acc = x.new_zeros([n - 2 * r for n in x.shape])
            for idx, v in taps:
                acc.add_(x[tuple(slice(i, n - 2 * r + i) for i, n in zip(idx, x.shape))], alpha=v)
            y = x.clone()
            y[tuple(slice(r, n - r) for n in x.shape)] = acc
            x = y
    return x


def exact(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        problems = _mix(case)
        pad = [(math.prod(ext) + 31) // 32 * 32 for _, ext, _, _ in problems]
        flat_in = _grid((sum(pad),), seed, False)
        out = torch.zeros_like(flat_in)
        at = 0
        for (shape, ext, T, boundary), size in zip(problems, pad):
            n = math.prod(ext)
            w = _weights(shape, rng, "positive")
            x = flat_in[at:at + n].reshape(tuple(reversed(ext)))
            out[at:at + n] = _stepped(x, w, T, boundary).reshape(-1)
            at += size
        return out
    w = _weights(case["shape"], rng, case["weights"])
    x = _grid(tuple(reversed(_extents(case))), seed, case["weights"] == "signed")
    y = _stepped(x, w, case["T"], case["boundary"])
    return y.cpu().numpy() if case["kind"] == "host" else y
