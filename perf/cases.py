"""The summed-area-table work whose speed is followed, as a user's program asks for it.

Every case goes through the package's public calls (`scanrow_brlt`, `brlt_scanrow`,
`scanrowcolumn`, `sat`, `scan_rows`, `scan_cols`, `scan_rows_transposed`,
`BatchPlan` and the autograd box-filter layer) on tensors that are already on the
GPU.  Images of 1-byte pixels are uniform in 0..255, f32 and f64 images uniform in
[0, 1), i32 images small signed counts, layer activations and gradients N(0, 1).

`listed()` holds the fixed cases, `draw(rng)` one more of the same ranges:

    single SATs      sides 64 .. 8192 (f64: .. 4096), packed rows or rows padded
                     to 128 bytes, the three entry points, the suffix SAT and the
                     compensated mode
    row/column scans sides 64 .. 8192, row scans also with transposed output
    batches          16 .. 512 images with sides 64 .. 4096
    box layers       1 .. 192 planes with sides 128 .. 1024, forward + backward
"""
import math
import random

import torch

import sat_gb300

_DT = {"u8": torch.uint8, "i32": torch.int32, "u32": torch.uint32, "f32": torch.float32, "f64": torch.float64}
_SIZE = {"u8": 1, "i32": 4, "u32": 4, "f32": 4, "f64": 8}


def _sat(name, entry, t_in, t_out, w, h, pitched=False, mode="plain", reverse=False):
    return {"name": name, "kind": "sat", "entry": entry, "in": t_in, "out": t_out, "width": w, "height": h,
            "pitched": pitched, "mode": mode, "reverse": reverse}


def _scan(name, entry, t_in, t_out, w, h, pitched=False):
    return {"name": name, "kind": "scan", "entry": entry, "in": t_in, "out": t_out, "width": w, "height": h,
            "pitched": pitched}


def _batch(name, images, lo, hi, sizes, pitched):
    return {"name": name, "kind": "batch", "images": images, "lo": lo, "hi": hi, "sizes": sizes, "pitched": pitched}


def _box(name, n, c, h, w, radii):
    return {"name": name, "kind": "box", "n": n, "c": c, "height": h, "width": w, "radii": radii}


def listed():
    return [
        # a thumbnail or a detection window: the call's latency is all of it
        _sat("sat_u8_333x200", "scanrow_brlt", "u8", "u32", 333, 200),
        # the image size of the reference's own command line
        _sat("sat_u8_1024", "brlt_scanrow", "u8", "u32", 1024, 1024),
        # a video frame's luminance as f32, one SAT a frame (box filters, Haar features)
        _sat("sat_f32_1920x1080", "scanrowcolumn", "f32", "f32", 1920, 1080),
        # a large 8-bit scan or satellite tile: the integer SAT
        _sat("sat_u8_8192", "scanrow_brlt", "u8", "u32", 8192, 8192),
        # the same size in f32: the benchmark's headline
        _sat("sat_f32_8192", "scanrowcolumn", "f32", "f32", 8192, 8192),
        # the suffix SAT (the SAT's gradient) of a packed image with odd sides
        _sat("sat_rev_f32_2999x3001", "sat", "f32", "f32", 2999, 3001, reverse=True),
        # the compensated f32 SAT, for sums that have to be good to the last bits
        _sat("sat_f32c_8192", "sat", "f32", "f32", 8192, 8192, mode="compensated"),
        # the f64 SAT at the benchmark's size
        _sat("sat_f64_4096", "scanrow_brlt", "f64", "f64", 4096, 4096),
        # column sums of an image (vertical integration) on their own
        _scan("cols_f32_4096", "scan_cols", "f32", "f32", 4096, 4096),
        # row scan with transposed output, the half step of a separable integral transform
        _scan("rows_t_u8_8192", "scan_rows_transposed", "u8", "u32", 8192, 8192),
        # a folder of decoded images of all sizes, packed rows as a decoder leaves them
        _batch("batch512_u8", 512, 64, 4096, 7, False),
        # a training step through a box-filter layer: means at three radii and the input's gradient
        _box("box_64x3x1024", 64, 3, 1024, 1024, "3,7,15"),
    ]


def _side(rng, lo, hi):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    # every third side is a round one, the others fall as they fall (odd ones among them)
    return max(lo, v // 64 * 64) if rng.random() < 0.33 else v


def draw(rng):
    kind = rng.choice(["sat", "sat", "sat", "sat", "sat", "scan", "scan", "batch", "box", "box"])
    if kind == "sat":
        t_in, t_out = rng.choice([("u8", "u32"), ("u8", "u32"), ("u8", "f32"), ("f32", "f32"), ("f32", "f32"),
                                  ("i32", "i32"), ("f32", "f64"), ("f64", "f64")])
        hi = 4096 if t_out == "f64" else 8192
        entry = rng.choice(["scanrow_brlt", "brlt_scanrow", "scanrowcolumn", "sat"])
        mode = "compensated" if entry == "sat" and (t_in, t_out) == ("f32", "f32") and rng.random() < 0.5 else "plain"
        c = _sat("", entry, t_in, t_out, _side(rng, 64, hi), _side(rng, 64, hi), rng.random() < 0.4, mode,
                 entry == "sat" and rng.random() < 0.5)
    elif kind == "scan":
        t_in, t_out = rng.choice([("u8", "u32"), ("f32", "f32"), ("u8", "f32")])
        c = _scan("", rng.choice(["scan_rows", "scan_cols", "scan_rows_transposed"]), t_in, t_out,
                  _side(rng, 64, 8192), _side(rng, 64, 8192), rng.random() < 0.4)
    elif kind == "batch":
        c = _batch("", _side(rng, 16, 512), 64, rng.choice([512, 1024, 4096]), rng.randrange(1000),
                   rng.random() < 0.5)
    else:
        radii = sorted(rng.sample([3, 4, 5, 7, 9, 11, 15, 21, 31], rng.choice([1, 2, 3, 4])))
        c = _box("", _side(rng, 1, 64), rng.choice([1, 3]), _side(rng, 128, 1024), _side(rng, 128, 1024),
                 ",".join(map(str, radii)))
    del c["name"]
    return c


def _sizes(case):
    """(width, height) of a batch's images, log-uniform in [lo, hi]."""
    r = random.Random(case["sizes"])
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    return [(int(round(math.exp(r.uniform(lo, hi)))), int(round(math.exp(r.uniform(lo, hi)))))
            for _ in range(case["images"])]


def _row(width, size, pitched):
    """Row length in elements: the width, or the width padded to 128 bytes."""
    return width if not pitched else (width * size + 127) // 128 * 128 // size


def _rand(shape, t, g):
    dev = torch.device("cuda")
    if t == "u8":
        return torch.randint(0, 256, shape, dtype=torch.uint8, device=dev, generator=g)
    if t == "i32":
        return torch.randint(-1000, 1000, shape, dtype=torch.int32, device=dev, generator=g)
    return torch.rand(shape, dtype=_DT[t], device=dev, generator=g)


def _image(case, g):
    w, h = case["width"], case["height"]
    return _rand((h, _row(w, _SIZE[case["in"]], case["pitched"])), case["in"], g)[:, :w]


def _box_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case["n"], case["c"], case["height"], case["width"])
    radii = [int(r) for r in case["radii"].split(",")]
    x = torch.randn(shape, device="cuda", generator=g)
    grad = torch.randn(shape[:2] + (len(radii),) + shape[2:], device="cuda", generator=g)
    return x, grad, radii


def prepare(case, seed):
    if case["kind"] == "box":
        x, grad, radii = _box_inputs(case, seed)
        return {"case": case, "layer": sat_gb300.BoxFilter(radii), "x": x.requires_grad_(True), "grad": grad}
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "batch":
        # one allocation for all images, as a loader hands them over, each on a 256-byte boundary
        def cut(t, make):
            rows = [(w, h, _row(w, _SIZE[t], case["pitched"])) for w, h in _sizes(case)]
            at, total = [], 0
            for w, h, row in rows:
                at.append(total)
                total += (row * h * _SIZE[t] + 255) // 256 * 256 // _SIZE[t]
            flat = make(total)
            return flat, [flat[a:a + row * h].view(h, row)[:, :w] for a, (w, h, row) in zip(at, rows)]

        _, images = cut("u8", lambda n: _rand((n,), "u8", g))
        flat, outs = cut("u32", lambda n: torch.zeros(n, dtype=torch.int32, device="cuda").view(torch.uint32))
        return {"case": case, "flat": _bits(flat), "plan": sat_gb300.BatchPlan(images, outs)}
    return {"case": case, "x": _image(case, g)}


def _bits(t):
    """u32 sums as the i32 tensor of the same bits: torch cannot index uint32 on the GPU."""
    return t.view(torch.int32) if t.dtype == torch.uint32 else t


def run(state):
    case = state["case"]
    if case["kind"] == "sat":
        x, t = state["x"], _DT[case["out"]]
        if case["entry"] == "sat":
            return _bits(sat_gb300.sat(x, t, mode=case["mode"], reverse=case["reverse"]))
        return _bits(getattr(sat_gb300, case["entry"])(x, t))
    if case["kind"] == "scan":
        return _bits(getattr(sat_gb300, case["entry"])(state["x"], _DT[case["out"]]))
    if case["kind"] == "batch":
        state["plan"].exec()
        return state["flat"]  # every image's SAT
    means = state["layer"](state["x"])
    (dx,) = torch.autograd.grad(means, state["x"], state["grad"])
    return {"means": means.detach(), "dx": dx}


def work(case):
    if case["kind"] == "batch":
        px = sum(w * h for w, h in _sizes(case))
        return {"bytes": px * 5, "flops": px * 2}
    px = case["width"] * case["height"]
    if case["kind"] == "box":
        px, r = px * case["n"] * case["c"], len(case["radii"].split(","))
        # x and the means' gradients in, the means and dx out
        return {"bytes": px * 4 * (2 + 2 * r), "flops": px * 8 * r}
    adds = 1 if case["kind"] == "scan" else 2
    return {"bytes": px * (_SIZE[case["in"]] + _SIZE[case["out"]]), "flops": px * adds}


def _exact_sums(x, dims, reverse):
    """Prefix (or suffix) sums along `dims` in 64 bits.  f64 values of [0, 1) are
    cut in two at 2^-26, so that both parts' sums are exact and one addition rounds."""
    parts = [x.double()]
    if x.dtype == torch.float64:
        hi = torch.floor(x * 2.0**26) * 2.0**-26
        parts = [hi, x - hi]
    done = []
    for p in parts:
        if reverse:
            p = p.flip(dims)
        for d in dims:
            p = p.cumsum(d)
        done.append(p.flip(dims) if reverse else p)
    return done[0] if len(done) == 1 else done[0] + done[1]


def _box_sums(x, r):
    """Sums over the clipped (2r+1) x (2r+1) windows of every plane of x (f64)."""
    for d in (-1, -2):
        n = x.shape[d]
        i = torch.arange(n, device=x.device)
        s = torch.cat([torch.zeros_like(x.narrow(d, 0, 1)), x.cumsum(d)], d)
        x = s.index_select(d, (i + r + 1).clamp(max=n)) - s.index_select(d, (i - r).clamp(min=0))
    return x


def _areas(h, w, r):
    def length(n):
        i = torch.arange(n, device="cuda")
        return ((i + r).clamp(max=n - 1) - (i - r).clamp(min=0) + 1).double()

    return length(h)[:, None] * length(w)[None, :]


def exact(case, seed):
    if case["kind"] == "batch" or case["out" if "out" in case else "kind"] in ("u32", "i32"):
        return None  # whole numbers
    if case["kind"] == "box":
        x, grad, radii = _box_inputs(case, seed)
        h, w = case["height"], case["width"]
        means = torch.empty(grad.shape, dtype=torch.float64, device="cuda")
        dx = torch.zeros(x.shape, dtype=torch.float64, device="cuda")
        for n in range(x.shape[0]):
            for k, r in enumerate(radii):
                area = _areas(h, w, r)
                means[n, :, k] = _box_sums(x[n].double(), r) / area
                dx[n] += _box_sums(grad[n, :, k].double() / area, r)
        return {"means": means, "dx": dx}
    x = _image(case, torch.Generator(device="cuda").manual_seed(seed))
    if case["kind"] == "sat":
        return _exact_sums(x, (1, 0), case["reverse"])
    s = _exact_sums(x, (0,) if case["entry"] == "scan_cols" else (1,), False)
    return s.t().contiguous() if case["entry"] == "scan_rows_transposed" else s
