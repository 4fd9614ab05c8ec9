"""Parity of the CUDA path (through the C ABI) with the oracle.

Integer outputs must be bit-exact against the reference's CPU integral image
(golden vectors made by running it, and the C restatement for other inputs),
including the mod-2^32 wrap.  Float outputs are compared with the FP64
oracle with the tolerances below, stated relative to SAT(|a|) computed in
FP64 (the denominator that stays meaningful under cancellation):

  plain f32       max |S - S64| / SAT(|a|)64  <= 1e-5
  compensated f32 max |S - S64| / SAT(|a|)64  <= 2e-7   (one final rounding)
  f64             max |S - S64| / SAT(|a|)64  <= 1e-13
"""
import hashlib

import numpy as np
import pytest
import torch

import sat_gb300
from sat_gb300 import _lib
from tests.util import bits, empty_pitched, to_dev, to_np

pytestmark = pytest.mark.gpu

TOL = {np.dtype(np.float32): 1e-5, np.dtype(np.float64): 1e-13}
TOL_COMP = 2e-7
ALGOS = [sat_gb300.scanrow_brlt, sat_gb300.brlt_scanrow, sat_gb300.scanrowcolumn]


def _check_float(oracle, a, s, tol, reverse=False):
    ref = oracle.sat_fp64(a, reverse=reverse)
    den = oracle.sat_fp64(a, reverse=reverse, absval=True)
    err = np.abs(s.astype(np.float64) - ref)
    mask = den > 0
    worst = float(np.max(err[mask] / den[mask])) if mask.any() else 0.0
    assert np.all(err[~mask] == 0)
    assert worst <= tol, worst
    return worst


def _check(oracle, a, out_np, out_dtype, tol=None, reverse=False):
    out_dtype = np.dtype(out_dtype)
    if out_dtype.kind in "iu":
        ref = oracle.sat_reverse(a, out_dtype) if reverse else oracle.sat_serial(a, out_dtype)
        assert np.array_equal(bits(out_np), bits(ref))
    else:
        _check_float(oracle, a, out_np, tol or TOL[out_dtype], reverse)


def test_golden_small_all_entry_points(cuda, oracle, golden):
    z, meta = golden
    for case in meta["small"]:
        a = z[case["key"] + "__in"]
        r = z[case["key"] + "__out"]
        x = to_dev(a)
        for fn in ALGOS:
            for scan in (sat_gb300.KOGGE_STONE_SCAN, sat_gb300.LF_SCAN):
                out = to_np(fn(x, torch.float32 if r.dtype == np.float32 else
                               {np.dtype(np.uint32): torch.uint32, np.dtype(np.int32): torch.int32,
                                np.dtype(np.float64): torch.float64}[r.dtype], scan_type=scan))
                if r.dtype.kind in "iu":
                    assert np.array_equal(bits(out), bits(r)), (case["key"], fn.__name__)
                else:
                    _check_float(oracle, a, out, TOL[r.dtype])
                    _check_float(oracle, a, r, TOL[r.dtype])  # the reference itself meets the same bound


def test_reference_size_1024_digests(cuda, oracle, golden):
    """The reference's smallest benchmark size (1024 x 1024, ScanRow-BRLT.cu:272-273)
    through all three entry points."""
    _, meta = golden
    for case in meta["big"]:
        ti, to = oracle.PAIRS[case["pair"]]
        a = oracle.gen(case["kind"], case["seed"], (case["h"], case["w"])).astype(ti)
        assert hashlib.sha256(a.tobytes()).hexdigest() == case["in_sha256"]
        x = to_dev(a)
        for fn in ALGOS:
            out = to_np(fn(x, {np.dtype(np.uint32): torch.uint32, np.dtype(np.float32): torch.float32,
                               np.dtype(np.float64): torch.float64}[np.dtype(to)]))
            if np.dtype(to).kind in "iu":
                assert hashlib.sha256(out.tobytes()).hexdigest() == case["out_sha256"], (case["key"], fn.__name__)
            else:
                _check_float(oracle, a, out, TOL[np.dtype(to)])


PAIR_KINDS = {np.uint8: "u8", np.int8: "i8", np.int32: "i32", np.uint32: "u32",
              np.float32: "f32u", np.float64: "f64u"}
SHAPES = [(1, 1), (1, 700), (700, 1), (2, 3), (63, 127), (64, 128), (65, 129), (127, 255),
          (129, 257), (300, 1000), (1000, 300), (517, 769)]


@pytest.mark.parametrize("cfg", [0, 1, 2, 3, 4, 5, 6])
def test_all_pairs_all_configs(cuda, oracle, cfg):
    sat_gb300.set_config(cfg)
    try:
        for name, (ti, to) in oracle.PAIRS.items():
            for i, shape in enumerate(SHAPES):
                a = oracle.gen(PAIR_KINDS[ti], 1000 + i, shape)
                out = sat_gb300.sat(to_dev(a), {np.uint32: torch.uint32, np.int32: torch.int32,
                                                np.float32: torch.float32, np.float64: torch.float64}[to])
                _check(oracle, a, to_np(out), to)
    finally:
        sat_gb300.set_config(-1)


@pytest.mark.parametrize("cfg", [0, 1, 2, 3, 4, 5, 6])
def test_reverse_all_configs(cuda, oracle, cfg):
    sat_gb300.set_config(cfg)
    try:
        for name in ("u8_u32", "i32_i32", "f32_f32", "f64_f64", "u8_f64"):
            ti, to = oracle.PAIRS[name]
            for i, shape in enumerate(SHAPES):
                a = oracle.gen(PAIR_KINDS[ti], 2000 + i, shape)
                out = sat_gb300.sat(to_dev(a), {np.uint32: torch.uint32, np.int32: torch.int32,
                                                np.float32: torch.float32, np.float64: torch.float64}[to],
                                    reverse=True)
                _check(oracle, a, to_np(out), to, reverse=True)
    finally:
        sat_gb300.set_config(-1)


def test_pitched_unaligned_and_inplace(cuda, oracle):
    # pitch > width with vector-aligned rows
    a = oracle.gen("u8", 7, (333, 555))
    src = empty_pitched(333, 555, 640, torch.uint8)
    src.copy_(to_dev(a))
    dst = empty_pitched(333, 555, 600, torch.uint32, fill=-1)
    sat_gb300.scanrowcolumn(src, torch.uint32, out=dst)
    assert np.array_equal(to_np(dst), oracle.sat_serial(a, np.uint32))
    # odd pitch: rows not 4-byte aligned -> scalar loads
    src2 = empty_pitched(333, 555, 557, torch.uint8)
    src2.copy_(to_dev(a))
    dst2 = empty_pitched(333, 555, 559, torch.uint32)
    sat_gb300.scanrow_brlt(src2, torch.uint32, out=dst2)
    assert np.array_equal(to_np(dst2), oracle.sat_serial(a, np.uint32))
    # base pointer offset by one element (misaligned for vectors, aligned for elements)
    big = torch.zeros(1 + 200 * 300, dtype=torch.uint8, device="cuda")
    view = big[1:].view(200, 300)
    b = oracle.gen("u8", 8, (200, 300))
    view.copy_(to_dev(b))
    out = sat_gb300.brlt_scanrow(view, torch.uint32)
    assert np.array_equal(to_np(out), oracle.sat_serial(b, np.uint32))
    # the padding between rows is never written
    pad = dst.as_strided((333, 45), (600, 1), dst.storage_offset() + 555)
    assert np.all(to_np(pad) == np.uint32(0xFFFFFFFF))
    # in place, f32 -> f32 on one buffer
    f = oracle.gen("f32u", 9, (400, 700))
    x = to_dev(f)
    sat_gb300.sat(x, torch.float32, out=x)
    _check(oracle, f, to_np(x), np.float32)


@pytest.mark.parametrize("pair", ["u8_u32", "u8_f64", "f32_f32", "f64_f64", "i8_i32"])
def test_aligned_pitch_ragged_width(cuda, oracle, pair):
    """16-byte aligned pitches with widths that end mid-chunk: the tensor maps
    cover the whole 16-byte chunks and the row tails go by plain accesses.
    The row padding (sentinel-filled) must stay untouched, forward and reverse."""
    ti, to = oracle.PAIRS[pair]
    ti, to = np.dtype(ti), np.dtype(to)
    kind = {"u1": "u8", "i1": "i8", "f4": "f32u", "f8": "f64u"}[ti.str[1:]]
    tin = {np.dtype(np.uint8): torch.uint8, np.dtype(np.int8): torch.int8,
           np.dtype(np.float32): torch.float32, np.dtype(np.float64): torch.float64}[ti]
    tout = {np.dtype(np.uint32): torch.uint32, np.dtype(np.int32): torch.int32,
            np.dtype(np.float32): torch.float32, np.dtype(np.float64): torch.float64}[to]
    for h, w in [(70, 17), (131, 555), (66, 1001), (40, 3), (257, 129)]:
        a = oracle.gen(kind, 40 + w, (h, w)).astype(ti)
        pin = -(-w * ti.itemsize // 64) * 64 // ti.itemsize + 16 // ti.itemsize
        pout = -(-w * to.itemsize // 64) * 64 // to.itemsize + 16 // to.itemsize
        src = empty_pitched(h, w, pin, tin)
        src.copy_(to_dev(a))
        fill = -1 if to.kind in "iu" else float("nan")
        for rev in (False, True):
            dst = empty_pitched(h, w, pout, tout, fill=fill)
            sat_gb300.sat(src, tout, reverse=rev, out=dst)
            _check(oracle, a, to_np(dst), to, reverse=rev)
            pad = dst.as_strided((h, pout - w), (pout, 1), dst.storage_offset() + w)
            padn = to_np(pad)
            if to.kind in "iu":
                assert np.all(bits(padn) == 0xFF), (h, w, rev)
            else:
                assert np.all(np.isnan(padn)), (h, w, rev)


def test_back_to_back_calls_reuse_workspace(cuda, oracle):
    rng = np.random.default_rng(0)
    outs = []
    for i in range(40):
        h, w = int(rng.integers(1, 900)), int(rng.integers(1, 900))
        a = oracle.gen("u8", 3000 + i, (h, w))
        outs.append((a, sat_gb300.scanrow_brlt(to_dev(a), torch.uint32)))
    sat_gb300.stream_check()
    for a, o in outs:
        assert np.array_equal(to_np(o), oracle.sat_serial(a, np.uint32))


def test_other_stream(cuda, oracle):
    s = torch.cuda.Stream()
    a = oracle.gen("u8", 44, (1500, 1300))
    x = to_dev(a)
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        out = sat_gb300.scanrowcolumn(x, torch.uint32)
    s.synchronize()
    sat_gb300.stream_check(s)
    assert np.array_equal(to_np(out), oracle.sat_serial(a, np.uint32))


@pytest.mark.parametrize("kind", ["f32u", "f32log"])
def test_compensated_f32(cuda, oracle, kind):
    a = oracle.gen(kind, 55, (2048, 2048))
    x = to_dev(a)
    plain = to_np(sat_gb300.sat(x, torch.float32))
    comp = to_np(sat_gb300.sat(x, torch.float32, mode="compensated"))
    ref = oracle.sat_fp64(a)
    den = oracle.sat_fp64(a, absval=True)
    e_plain = oracle.err_stats(plain, ref, den)
    e_comp = oracle.err_stats(comp, ref, den)
    assert e_plain["max_rel_abs"] <= 1e-5, e_plain
    assert e_comp["max_rel_abs"] <= TOL_COMP, e_comp
    if kind == "f32u":
        assert e_comp["max_rel"] <= 1e-6, e_comp
    # compensated reverse too
    rc = to_np(sat_gb300.sat(x, torch.float32, mode="compensated", reverse=True))
    e_rev = oracle.err_stats(rc, oracle.sat_fp64(a, reverse=True), oracle.sat_fp64(a, reverse=True, absval=True))
    assert e_rev["max_rel_abs"] <= TOL_COMP, e_rev


@pytest.mark.parametrize("kind", ["f32u", "f32log"])
def test_compensated_register_tiles_forward_and_reverse(cuda, oracle, kind):
    """Configuration 3 (the register-resident 128-row tiles, the default for
    large compensated images) forced on every edge shape and at 2048^2,
    forward and reverse: the reverse compensated SAT is the backward of the
    compensated autograd SAT."""
    sat_gb300.set_config(3)
    try:
        for i, shape in enumerate(SHAPES + [(2048, 2048)]):
            a = oracle.gen(kind, 6000 + i, shape)
            x = to_dev(a)
            for rev in (False, True):
                out = to_np(sat_gb300.sat(x, torch.float32, mode="compensated", reverse=rev))
                _check_float(oracle, a, out, TOL_COMP, reverse=rev)
    finally:
        sat_gb300.set_config(-1)


def test_compensated_u8_and_i8_inputs(cuda, oracle):
    for kind, dt in (("u8", np.uint8), ("i8", np.int8)):
        a = oracle.gen(kind, 66, (1000, 1500))
        comp = to_np(sat_gb300.sat(to_dev(a), torch.float32, mode="compensated"))
        exact = a.astype(np.int64).cumsum(0).cumsum(1)
        # integer-valued sums: compensated f32 is the exact sum rounded once
        assert np.array_equal(comp, exact.astype(np.float32))


def test_batch_plan_uneven(cuda, oracle):
    rng = np.random.default_rng(5)
    ins, outs, arrs = [], [], []
    for i in range(48):
        h = int(np.exp(rng.uniform(np.log(1), np.log(700))))
        w = int(np.exp(rng.uniform(np.log(1), np.log(700))))
        a = oracle.gen("u8", 4000 + i, (h, w))
        arrs.append(a)
        ins.append(to_dev(a))
        outs.append(torch.empty((h, w), dtype=torch.uint32, device="cuda"))
    plan = sat_gb300.BatchPlan(ins, outs)
    assert plan.info()["n_tiles"] > 48
    for rep in range(3):
        for o in outs:
            o.fill_(0)
        (plan.exec if rep != 1 else plan.launch)()
        plan.check()
        for a, o in zip(arrs, outs):
            assert np.array_equal(to_np(o), oracle.sat_serial(a, np.uint32))
    plan.close()


def test_batch_plan_stages_unaligned_inputs_each_exec(cuda, oracle):
    """Inputs whose rows TMA cannot address (packed rows of odd widths, an
    offset base) are copied into the plan's padded staging rows at every
    execution: after the caller changes its inputs in place, the next exec
    reads the new values.  Mixed with 16-byte pitched images and rows shorter
    than 16 bytes, which are not staged."""
    rng = np.random.default_rng(9)
    ins, outs, views = [], [], []
    for i in range(24):
        h, w = int(rng.integers(1, 400)), int(rng.integers(1, 900))
        if i % 3 == 0:  # 16-byte pitched rows: TMA reads them in place
            x = empty_pitched(h, w, (w + 15) // 16 * 16, torch.uint8)
        elif i % 3 == 1:  # packed rows, one byte past a 16-byte boundary
            x = torch.empty(h * w + 1, dtype=torch.uint8, device=cuda)[1:].view(h, w)
        else:  # packed rows
            x = torch.empty((h, w), dtype=torch.uint8, device=cuda)
        ins.append(x)
        outs.append(torch.empty((h, w), dtype=torch.uint32, device=cuda))
    plan = sat_gb300.BatchPlan(ins, outs)
    for rep in range(2):
        arrs = [oracle.gen("u8", 6000 + 100 * rep + i, tuple(x.shape)) for i, x in enumerate(ins)]
        for x, a in zip(ins, arrs):
            x.copy_(to_dev(a))
        plan.exec()
        plan.check()
        for a, o in zip(arrs, outs):
            assert np.array_equal(to_np(o), oracle.sat_serial(a, np.uint32)), rep
    plan.close()


@pytest.mark.parametrize("layout", ["packed", "offset"])
def test_single_image_staged_input(cuda, oracle, layout):
    """A single image of 1-byte inputs, at least 2^22 pixels, whose rows TMA
    cannot address (packed rows of an odd width, or a base one byte past a
    16-byte boundary) is copied into padded rows of the workspace by one more
    launch before the tile kernel: bit-exact against the oracle, both
    directions, and again after the input changes in place."""
    h, w = 2049, 2051
    n = h * w + 1
    for rev in (False, True):
        for rep in range(2):
            a = oracle.gen("u8", 7100 + 10 * rep + rev, (h, w))
            if layout == "packed":
                x = to_dev(a)
            else:
                x = torch.empty(n + 16, dtype=torch.uint8, device=cuda)[1:1 + h * w].view(h, w)
                x.copy_(to_dev(a))
            before = sat_gb300.launch_count()
            out = sat_gb300.sat(x, torch.uint32, reverse=rev)
            assert sat_gb300.launch_count() - before == 2  # the staging copy and the SAT
            ref = oracle.sat_reverse(a, np.uint32) if rev else oracle.sat_serial(a, np.uint32)
            assert np.array_equal(to_np(out), ref), (layout, rev, rep)


def test_reserve_then_capture_staged_call(cuda, oracle):
    """satgb_reserve sizes the stream's workspace for the staging rows too: a
    staged single-image call (packed u8 rows, 2049 x 2051) can then be captured
    in a CUDA graph, which allows no allocation, and the replay is bit-exact."""
    h, w = 2049, 2051
    a = oracle.gen("u8", 7300, (h, w))
    x = to_dev(a)
    y = torch.empty((h, w), dtype=torch.int32, device=cuda).view(torch.uint32)
    s = torch.cuda.Stream()
    L = _lib.load()
    with torch.cuda.stream(s):
        assert L.satgb_reserve(w, h, s.cuda_stream) == _lib.OK
        sat_gb300.sat(x, torch.uint32, out=y)  # descriptors encoded before the capture
        s.synchronize()
        y.zero_()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            sat_gb300.sat(x, torch.uint32, out=y)
        g.replay()
        s.synchronize()
    assert np.array_equal(to_np(y), oracle.sat_serial(a, np.uint32))


def test_batch_plan_float_and_reverse(cuda, oracle):
    rng = np.random.default_rng(6)
    ins, outs, arrs = [], [], []
    for i in range(20):
        h, w = int(rng.integers(1, 600)), int(rng.integers(1, 600))
        a = oracle.gen("f32u", 5000 + i, (h, w))
        arrs.append(a)
        ins.append(to_dev(a))
        outs.append(torch.empty((h, w), dtype=torch.float32, device="cuda"))
    for reverse in (False, True):
        plan = sat_gb300.BatchPlan(ins, outs, mode="compensated", reverse=reverse)
        plan.exec()
        plan.check()
        for a, o in zip(arrs, outs):
            _check_float(oracle, a, to_np(o), TOL_COMP, reverse=reverse)
        plan.close()


def test_autotune_records_and_results_stay_exact(cuda, oracle, tmp_path, monkeypatch):
    """satgb_autotune times every configuration on the caller's buffers, picks
    one, writes it to the tuning cache (one JSON object per line) and the
    next call with that size, which now uses it, is still bit-exact."""
    import json
    cache = tmp_path / "tune.jsonl"
    monkeypatch.setenv("SATGB_TUNE_CACHE", str(cache))
    a = oracle.gen("u8", 55, (700, 900))
    x = to_dev(a)
    y = torch.empty((700, 900), dtype=torch.int32, device=cuda).view(torch.uint32)
    best = sat_gb300.autotune(x, y)
    assert 0 <= best < len(sat_gb300.config_names())
    entries = [json.loads(line) for line in cache.read_text().splitlines()]
    mine = [e for e in entries if (e["in"], e["out"], e["wb"], e["hb"]) == (_lib.U8, _lib.U32, 10, 10)]
    assert mine and all(e["cfg"] == best for e in mine)
    out = to_np(sat_gb300.sat(x, torch.uint32))
    assert np.array_equal(bits(out), bits(oracle.sat_serial(a, np.uint32)))


def test_full_size_u8_properties_and_configs_agree(cuda):
    """8192 x 8192 u8 -> u32, the reference's largest case: the last row is
    the prefix of the column sums and the last column the prefix of the row
    sums (mod 2^32: the total of 2^26 bytes wraps), and the default tiles, the
    64-row two-CTA tiles and the 256-row direct-store tiles agree bit for bit."""
    g = torch.Generator(device=cuda).manual_seed(41)
    x = torch.randint(0, 256, (8192, 8192), dtype=torch.uint8, device=cuda, generator=g)
    s_def = sat_gb300.sat(x, torch.uint32)
    for cfg in (2, 4):
        sat_gb300.set_config(cfg)
        try:
            s2 = sat_gb300.sat(x, torch.uint32)
        finally:
            sat_gb300.set_config(-1)
        assert torch.equal(s_def.view(torch.int32), s2.view(torch.int32)), cfg
    col = x.to(torch.int64).sum(0).cumsum(0) & 0xFFFFFFFF
    row = x.to(torch.int64).sum(1).cumsum(0) & 0xFFFFFFFF
    assert torch.equal(s_def[-1].to(torch.int64), col)
    assert torch.equal(s_def[:, -1].to(torch.int64), row)


@pytest.mark.parametrize("cfg", [0, 1, 2, 3, 4, 5, 6])
def test_timeout_is_reported_and_context_survives(cuda, oracle, cfg):
    """A tile that never publishes makes its dependents hit the wait limit
    (every kernel: warp-specialized, pipelined, register-resident); the call
    reports SATGB_ERR_TIMEOUT and the next call is correct."""
    L = _lib.load()
    a = oracle.gen("u8", 77, (512, 512))
    x = to_dev(a)
    s = torch.cuda.Stream()
    try:
        sat_gb300.set_wait_limit_us(20_000)
        sat_gb300.set_config(cfg)
        assert L.satgb_debug_stall_tile(5) == 0
        with torch.cuda.stream(s):
            sat_gb300.scanrow_brlt(x, torch.uint32)
        L.satgb_debug_stall_tile(-1)
        # the next call, queued before anyone read the error, is unaffected
        with torch.cuda.stream(s):
            after = sat_gb300.scanrow_brlt(x, torch.uint32)
        with pytest.raises(sat_gb300.SatError) as ei:
            sat_gb300.stream_check(s)
        assert ei.value.status == _lib.ERR_TIMEOUT
        assert np.array_equal(to_np(after), oracle.sat_serial(a, np.uint32))
    finally:
        L.satgb_debug_stall_tile(-1)
        sat_gb300.set_wait_limit_us(2_000_000)
        sat_gb300.set_config(-1)
    with torch.cuda.stream(s):
        out = sat_gb300.scanrow_brlt(x, torch.uint32)
    sat_gb300.stream_check(s)  # the report was cleared by the check above
    assert np.array_equal(to_np(out), oracle.sat_serial(a, np.uint32))


def test_allocator_hook_failure(cuda, oracle):
    L = _lib.load()
    calls = []
    alloc = _lib._ALLOC_FN(lambda n, ctx: calls.append(n) or None)
    free = _lib._FREE_FN(lambda p, ctx: None)
    s = torch.cuda.Stream()  # fresh stream -> fresh workspace
    assert L.satgb_set_allocator(alloc, free, None) == 0
    try:
        x = to_dev(oracle.gen("u8", 1, (64, 64)))
        with torch.cuda.stream(s):
            with pytest.raises(sat_gb300.SatError) as ei:
                sat_gb300.scanrow_brlt(x, torch.uint32)
        assert ei.value.status == _lib.ERR_ALLOC
        assert calls
    finally:
        assert L.satgb_set_allocator(_lib._ALLOC_FN(), _lib._FREE_FN(), None) == 0


def test_launch_count_one_per_call(cuda, oracle):
    x = to_dev(oracle.gen("u8", 2, (1024, 1024)))
    before = sat_gb300.launch_count()
    for fn in ALGOS:
        fn(x, torch.uint32)
    assert sat_gb300.launch_count() - before == 3


@pytest.mark.slow
def test_full_size_8192_u8_u32_bit_exact(cuda, oracle):
    a = oracle.gen("u8", 8192, (8192, 8192))
    for fn in ALGOS:
        out = to_np(fn(to_dev(a), torch.uint32))
        assert np.array_equal(out, oracle.sat_serial(a, np.uint32)), fn.__name__


def _precision_8192(oracle, kind):
    a = oracle.gen(kind, 8193, (8192, 8192))
    x = to_dev(a)
    ref = oracle.sat_fp64(a)
    den = oracle.sat_fp64(a, absval=True)
    e_plain = oracle.err_stats(to_np(sat_gb300.sat(x, torch.float32)), ref, den)
    e_comp = oracle.err_stats(to_np(sat_gb300.sat(x, torch.float32, mode="compensated")), ref, den)
    print(f"\n[precision 8192^2 {kind}] plain {e_plain}  compensated {e_comp}")
    assert e_plain["max_rel_abs"] <= 1e-5, (kind, e_plain)
    return e_plain, e_comp


@pytest.mark.slow
def test_compensated_8192_uniform_within_1e6_relative(cuda, oracle):
    """U[0,1) inputs at 8192^2: every compensated SAT element is within 1e-6
    of the FP64 SAT relative to the element itself, |S - S64| / |S64|."""
    _, e_comp = _precision_8192(oracle, "f32u")
    assert e_comp["max_rel"] <= 1e-6, e_comp
    assert e_comp["max_rel_abs"] <= TOL_COMP, e_comp


@pytest.mark.slow
def test_compensated_8192_log_class_relative_to_sat_of_abs(cuda, oracle):
    """Magnitudes 10^U(-3,3) with random signs at 8192^2: sums cancel, so some
    exact elements are near 0 and no fixed-precision sum bounds the error
    relative to the element itself.  The stated bound for this class uses the
    condition-aware denominator SAT(|a|): |S - S64| / SAT(|a|)64 <= 2e-7
    (measured: about 3e-8); the relative error on elements is reported."""
    _, e_comp = _precision_8192(oracle, "f32log")
    assert e_comp["max_rel_abs"] <= TOL_COMP, e_comp


@pytest.mark.slow
def test_full_size_4096_f64(cuda, oracle):
    a = oracle.gen("f64u", 4096, (4096, 4096))
    out = to_np(sat_gb300.sat(to_dev(a), torch.float64))
    _check_float(oracle, a, out, TOL[np.dtype(np.float64)])


def test_cli_runs_reference_sizes(cuda):
    """`sat 0 1 0 4 2`: u8 -> u32 ScanRow-BRLT at 1024^2 and 2048^2, one CSV
    line per size in the reference's format."""
    import subprocess
    from sat_gb300 import build as B
    r = subprocess.run([B.cli_path(), "0", "1", "0", "4", "2", "--reps", "3"], capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, r.stderr
    lines = r.stdout.strip().splitlines()
    assert lines[0].startswith("uchar-->uint, ScanRow-BRLT, LF_SCAN")
    for i, line in enumerate(lines[1:], start=1):
        w, h, rest = line.split(", ", 2)
        assert int(w) == int(h) == 1024 * i
        assert rest.startswith("total time = ")
        assert float(rest.split(", ")[-1]) > 0


SCAN_TORCH = {np.dtype(np.uint32): torch.uint32, np.dtype(np.int32): torch.int32,
              np.dtype(np.float32): torch.float32, np.dtype(np.float64): torch.float64}


@pytest.mark.parametrize("which", ["rows", "cols"])
def test_row_and_column_scans_all_pairs(cuda, oracle, which):
    """satgb_scan_rows / satgb_scan_cols (ScanX / ScanY as separate ops) against
    IntegralRow / IntegralStride: bit-exact for integer outputs; floats within
    1e-5 (f32) / 1e-13 (f64) of the FP64 scan, relative to the scan of |a|."""
    fn = sat_gb300.scan_rows if which == "rows" else sat_gb300.scan_cols
    ref = oracle.scan_rows if which == "rows" else oracle.scan_cols
    axis = 1 if which == "rows" else 0
    for name, (ti, to) in oracle.PAIRS.items():
        for i, shape in enumerate([(1, 1), (3, 700), (700, 3), (129, 257), (517, 769), (37, 1601)]):
            a = oracle.gen(PAIR_KINDS[ti], 3000 + i, shape)
            out = to_np(fn(to_dev(a), SCAN_TORCH[np.dtype(to)]))
            if np.dtype(to).kind in "iu":
                assert np.array_equal(bits(out), bits(ref(a, to))), (which, name, shape)
            else:
                exact = np.cumsum(a.astype(np.float64), axis=axis)
                den = np.cumsum(np.abs(a.astype(np.float64)), axis=axis)
                err = np.abs(out.astype(np.float64) - exact) / np.maximum(den, 1e-300)
                assert err.max() <= TOL[np.dtype(to)], (which, name, shape, err.max())


def test_scan_rows_transposed_all_pairs(cuda, oracle):
    """satgb_scan_rows_transposed (SerielScan::TestX: IntegralImageAllRow, then
    Transpose) against the oracle's row scan, transposed: bit-exact for integer
    outputs, floats within the scans' tolerance."""
    for name, (ti, to) in oracle.PAIRS.items():
        for i, shape in enumerate([(1, 1), (3, 700), (700, 3), (33, 129), (129, 257), (517, 769), (37, 1601)]):
            a = oracle.gen(PAIR_KINDS[ti], 3500 + i, shape)
            out = to_np(sat_gb300.scan_rows_transposed(to_dev(a), SCAN_TORCH[np.dtype(to)]))
            assert out.shape == (shape[1], shape[0])
            if np.dtype(to).kind in "iu":
                assert np.array_equal(bits(out), bits(oracle.scan_rows(a, to).T)), (name, shape)
            else:
                exact = np.cumsum(a.astype(np.float64), axis=1).T
                den = np.cumsum(np.abs(a.astype(np.float64)), axis=1).T
                err = np.abs(out.astype(np.float64) - exact) / np.maximum(den, 1e-300)
                assert err.max() <= TOL[np.dtype(to)], (name, shape, err.max())


def test_scan_rows_transposed_pitched_and_full_size(cuda, oracle):
    """Pitched input and output, odd pitches (no vector loads), and an
    8192 x 8192 u8 -> u32 check: the last output row is every input row's sum
    and the output equals the transposed row scan, mod 2^32."""
    a = oracle.gen("u8", 92, (333, 555))
    src = empty_pitched(333, 555, 641, torch.uint8)
    src.copy_(to_dev(a))
    dst = empty_pitched(555, 333, 400, torch.uint32, fill=-1)
    sat_gb300.scan_rows_transposed(src, torch.uint32, out=dst)
    assert np.array_equal(to_np(dst), oracle.scan_rows(a, np.uint32).T)
    # an output pitch of 401 elements: no 16-byte output vectors
    dst = empty_pitched(555, 333, 401, torch.uint32, fill=-1)
    sat_gb300.scan_rows_transposed(src, torch.uint32, out=dst)
    assert np.array_equal(to_np(dst), oracle.scan_rows(a, np.uint32).T)
    af = oracle.gen("f32n", 93, (333, 555))
    dstf = empty_pitched(555, 333, 333, torch.float64)
    sat_gb300.scan_rows_transposed(to_dev(af), torch.float64, out=dstf)
    exact = np.cumsum(af.astype(np.float64), axis=1).T
    assert np.abs(to_np(dstf) - exact).max() <= 1e-12 * np.abs(exact).max()
    g = torch.Generator(device=cuda).manual_seed(43)
    x = torch.randint(0, 256, (8192, 8192), dtype=torch.uint8, device=cuda, generator=g)
    t = sat_gb300.scan_rows_transposed(x, torch.uint32)
    r = sat_gb300.scan_rows(x, torch.uint32)
    assert torch.equal(t.view(torch.int32), r.view(torch.int32).t())
    rows = x.to(torch.int64).sum(1) & 0xFFFFFFFF
    assert torch.equal(t[-1].to(torch.int64), rows)


def test_golden_scans(cuda, golden_scans):
    """The CUDA row, transposed-row and column scans against the reference's
    own outputs (tests/golden/scans_golden.npz): bit-exact for integer outputs;
    floats within the scans' tolerance of the reference's sequential sums."""
    z, meta = golden_scans
    fns = (("__rows", sat_gb300.scan_rows, 1), ("__rows_t", sat_gb300.scan_rows_transposed, 1),
           ("__cols", sat_gb300.scan_cols, 0))
    for case in meta:
        a = z[case["key"] + "__in"]
        x = to_dev(a)
        for suffix, fn, axis in fns:
            ref = z[case["key"] + suffix]
            out = to_np(fn(x, SCAN_TORCH[ref.dtype]))
            if ref.dtype.kind in "iu":
                assert np.array_equal(bits(out), bits(ref)), (case["key"], suffix)
            else:
                den = np.cumsum(np.abs(a.astype(np.float64)), axis=axis)
                if suffix == "__rows_t":
                    den = den.T
                err = np.abs(out.astype(np.float64) - ref.astype(np.float64)) / np.maximum(den, 1e-300)
                assert err.max() <= TOL[ref.dtype], (case["key"], suffix, err.max())


def test_scans_pitched_and_full_size(cuda, oracle):
    """Pitched u8 -> u32 rows and columns, and an 8192 x 8192 check of
    sum(row scan) == sum(column scan) == the SAT's last element, mod 2^32."""
    a = oracle.gen("u8", 91, (333, 555))
    src = empty_pitched(333, 555, 640, torch.uint8)
    src.copy_(to_dev(a))
    for fn, ref in ((sat_gb300.scan_rows, oracle.scan_rows), (sat_gb300.scan_cols, oracle.scan_cols)):
        for opitch in (600, 601):  # 601: no 16-byte output vectors
            dst = empty_pitched(333, 555, opitch, torch.uint32, fill=-1)
            fn(src, torch.uint32, out=dst)
            assert np.array_equal(to_np(dst), ref(a, np.uint32))
    # in place (f32 -> f32 into its own buffer)
    af = oracle.gen("f32n", 94, (300, 1000))
    y = to_dev(af)
    sat_gb300.scan_rows(y, torch.float32, out=y)
    exact = np.cumsum(af.astype(np.float64), axis=1)
    den = np.cumsum(np.abs(af.astype(np.float64)), axis=1)
    assert (np.abs(to_np(y).astype(np.float64) - exact) / np.maximum(den, 1e-300)).max() <= TOL[np.dtype(np.float32)]
    x = torch.randint(0, 256, (8192, 8192), dtype=torch.uint8, device=cuda)
    r = sat_gb300.scan_rows(x, torch.uint32)
    c = sat_gb300.scan_cols(x, torch.uint32)
    s = sat_gb300.sat(x, torch.uint32)
    total = int(x.to(torch.int64).sum().item()) % (1 << 32)
    assert int(r[:, -1].view(torch.int32).to(torch.int64).remainder(1 << 32).sum().item()) % (1 << 32) == total
    assert int(c[-1, :].view(torch.int32).to(torch.int64).remainder(1 << 32).sum().item()) % (1 << 32) == total
    assert int(s[-1, -1].view(torch.int32).to(torch.int64).item()) % (1 << 32) == total


@pytest.mark.slow
@pytest.mark.parametrize("pitched", [True, False])
def test_batch512_bit_exact(cuda, oracle, pitched):
    """The batch workload exactly as the bench builds it: 512 u8 images with
    widths and heights log-uniform in [64, 4096] (about 590 M pixels), rows
    pitched to 128 bytes or packed, one graph replay of the plan with its
    untuned configurations and one after the batch autotuner picked a
    configuration per size class; every image bit-exact against the oracle."""
    from bench import build_batch
    xs, ys, _ = build_batch(cuda, pitched=pitched)
    plan = sat_gb300.BatchPlan(xs, ys)
    cls = plan.classes()
    assert cls[0]["images"] > 0 and cls[1]["images"] > 0 and cls[0]["images"] + cls[1]["images"] == 512
    for rep, tuned in ((0, False), (1, True)):
        if tuned:
            chosen = plan.autotune()  # every configuration of each class, timed on these images
            assert [c["config"] for c in plan.classes()] == list(chosen)
        for y in ys:
            y.view(torch.int32).fill_(-1)
        plan.exec()
        plan.check()
        for i, (x, y) in enumerate(zip(xs, ys)):
            a = to_np(x)
            assert np.array_equal(bits(to_np(y)), bits(oracle.sat_serial(a, np.uint32))), (tuned, i)
    plan.close()


@pytest.mark.slow
def test_stress_32768_u8_u32_bit_exact(cuda, oracle):
    """32768 x 32768 u8 -> u32 (2^30 pixels; sums wrap mod 2^32 many times)
    bit-exact against the oracle."""
    a = oracle.gen("u8", 32768, (32768, 32768))
    x = to_dev(a)
    out = sat_gb300.sat(x, torch.uint32)
    del x
    got = to_np(out)
    del out
    assert np.array_equal(got, oracle.sat_serial(a, np.uint32))


@pytest.mark.slow
def test_stress_16384_compensated_f32(cuda, oracle):
    """16384 x 16384 U[0,1) through the compensated f32 SAT: within 1e-6 of
    the FP64 SAT relative to each element, and 2e-7 relative to SAT(|a|)."""
    a = oracle.gen("f32u", 16384, (16384, 16384))
    comp = to_np(sat_gb300.sat(to_dev(a), torch.float32, mode="compensated"))
    e = oracle.err_stats(comp, oracle.sat_fp64(a), oracle.sat_fp64(a, absval=True))
    print(f"\n[precision 16384^2 f32u compensated] {e}")
    assert e["max_rel"] <= 1e-6, e
    assert e["max_rel_abs"] <= TOL_COMP, e


@pytest.mark.parametrize("cfg", [0, 1, 2, 5, 6])
@pytest.mark.parametrize("shape", [(1, 1), (128, 128), (129, 129), (130, 20001), (20001, 130), (1, 70000), (70000, 1),
                                   (1025, 1153), (2300, 700), (700, 2300), (3000, 2944)])
def test_tile_orders(cuda, cfg, shape):
    """Every tile of every order (anti-diagonals of wide, tall and square tile
    grids, single rows and columns of tiles, row-major) is computed once: u8 -> u32
    bit for bit, both directions."""
    h, w = shape
    g = torch.Generator(device="cpu").manual_seed(h * 7 + w)
    x = torch.randint(0, 256, (h, w), dtype=torch.uint8, generator=g).to(cuda)
    try:
        sat_gb300.set_config(cfg)
        for rev in (False, True):
            ref = x.to(torch.int64)
            if rev:
                ref = ref.flip((0, 1))
            ref = ref.cumsum(0).cumsum(1)
            if rev:
                ref = ref.flip((0, 1))
            out = sat_gb300.sat(x, torch.uint32, reverse=rev)
            assert torch.equal(out.view(torch.int32).to(torch.int64) & 0xFFFFFFFF, ref & 0xFFFFFFFF), rev
        sat_gb300.stream_check()
    finally:
        sat_gb300.set_config(-1)


def test_staged_pixels_are_never_status_words(cuda):
    """A staged image leaves its padded rows in the stream's workspace: launches with
    more status words than the staged one had must not take pixels for published sums.  A fresh
    stream's first launches carry small tags, and where a row ends two bytes before a
    16-byte group's second half a pixel followed by zeros looks like one: every pixel value
    stands there in some row."""
    h, w = 2049, 2051
    flat = (torch.arange(h * w + 16) * 2654435761 // 65536 % 256).to(torch.uint8).to(cuda)
    x = flat[1:1 + h * w].view(h, w)
    big = torch.randint(0, 256, (4100, 8208), dtype=torch.uint8, device=cuda)
    ref = big.to(torch.int64).cumsum(0).cumsum(1)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    try:
        with torch.cuda.stream(s):
            for cfg in (0, 2, 5):
                for _ in range(3):
                    sat_gb300.set_config(6)
                    sat_gb300.sat(x, torch.uint32)
                    sat_gb300.set_config(cfg)
                    out = sat_gb300.sat(big, torch.uint32)
                    assert torch.equal(out.view(torch.int32).to(torch.int64) & 0xFFFFFFFF, ref & 0xFFFFFFFF), cfg
    finally:
        sat_gb300.set_config(-1)


@pytest.mark.parametrize("pixels", ["random", "lowest", "highest"])
@pytest.mark.parametrize("pair", [("u8", "u32"), ("u8", "f32"), ("i8", "i32"), ("i8", "f32")])
def test_packed_sums_of_one_byte_pixels(cuda, pair, pixels):
    """Configuration 5 adds 1-byte pixels packed two and four to a register: pixels of
    the type's limits, at tile edges, in more tiles than the grid has CTAs, in rows of one tile and
    columns of one tile, packed and offset rows, both directions.  Integer sums bit for bit; f32 sums
    exact while they stay below 2^24 and within 1e-5 of the largest sum beyond
    (64 x 64 tiles of sums of 128 exact rows at most: 2^-24 x 130 roundings)."""
    dt = {"u8": torch.uint8, "i8": torch.int8, "u32": torch.uint32, "i32": torch.int32, "f32": torch.float32}
    t_in, t_out = dt[pair[0]], dt[pair[1]]
    info = torch.iinfo(t_in)
    lo, hi = {"random": (info.min, info.max), "lowest": (info.min,) * 2, "highest": (info.max,) * 2}[pixels]
    g = torch.Generator(device="cpu").manual_seed(11)
    try:
        sat_gb300.set_config(5)
        for h, w, pad in [(1, 1, 0), (127, 129, 0), (128, 128, 0), (129, 127, 5), (100, 9001, 0), (9001, 100, 0),
                          (128, 40000, 0), (40000, 128, 0), (1281, 4099, 0), (2050, 2049, 15), (64, 130000, 0)]:
            x = torch.randint(lo, hi + 1, (h, w + pad), dtype=t_in, generator=g).to(cuda)[:, pad // 2: pad // 2 + w]
            for rev in (False, True):
                ref = x.to(torch.int64)
                ref = ref.flip((0, 1)) if rev else ref
                ref = ref.cumsum(0).cumsum(1)
                ref = ref.flip((0, 1)) if rev else ref
                out = sat_gb300.sat(x, t_out, reverse=rev)
                if t_out == torch.float32:
                    top = int(ref.abs().max())
                    assert (out.double() - ref.double()).abs().max().item() <= (0 if top < 2**24 else 1e-5 * top), (h, w, rev)
                else:
                    got = out.view(torch.int32).to(torch.int64)
                    assert torch.equal(got & 0xFFFFFFFF, ref & 0xFFFFFFFF), (h, w, rev)
        sat_gb300.stream_check()
    finally:
        sat_gb300.set_config(-1)


@pytest.mark.parametrize("t_in,t_out", [(torch.uint8, torch.uint32), (torch.int8, torch.int32), (torch.uint8, torch.float32)])
def test_packed_rows_through_their_map(cuda, t_in, t_out):
    """Packed 1-byte rows whose length is no multiple of 16 (2, 4, 8 or 16 rows make one), read through
    a map of whole groups of rows: every remainder of the length, image heights with and without rows
    after the last group, tile edges, one image and a plan of them, both directions, bit for bit."""
    g = torch.Generator(device="cpu").manual_seed(17)
    info = torch.iinfo(t_in)

    def same(out, ref):
        if t_out == torch.float32:
            return torch.equal(out.double(), ref.double())  # sums below 2^24: exact
        return torch.equal(out.view(torch.int32).to(torch.int64) & 0xFFFFFFFF, ref & 0xFFFFFFFF)

    try:
        sat_gb300.set_config(5)
        for rev in (False, True):
            ins, refs = [], []
            for w in list(range(15, 34)) + [40, 100, 127, 129, 130, 132, 136, 255, 257, 391]:
                for h in (1, 2, 15, 16, 17, 127, 130, 144, 151):
                    x = torch.randint(info.min, info.max + 1, (h, w), dtype=t_in, generator=g)
                    ref = x.to(torch.int64).flip((0, 1)) if rev else x.to(torch.int64)
                    ref = ref.cumsum(0).cumsum(1)
                    ins.append(x.to(cuda))
                    refs.append((ref.flip((0, 1)) if rev else ref).to(cuda))
            for x, ref in zip(ins, refs):
                assert same(sat_gb300.sat(x, t_out, reverse=rev), ref), (tuple(x.shape), rev)
            outs = [torch.empty(x.shape, dtype=t_out, device=cuda) for x in ins]
            plan = sat_gb300.BatchPlan(ins, outs, reverse=rev)
            plan.exec()
            plan.check()
            for x, out, ref in zip(ins, outs, refs):
                assert same(out, ref), (tuple(x.shape), rev)
            plan.close()
    finally:
        sat_gb300.set_config(-1)


@pytest.mark.parametrize("cfg", [5, -1])
@pytest.mark.parametrize("t", [torch.int32, torch.float32, torch.uint32])
def test_packed_rows_of_4_bytes(cuda, t, cfg):
    """Packed 4-byte rows off 16-byte boundaries (2 or 4 of them make a multiple): every remainder of
    the width, heights with and without rows after the last group, tile edges, images of many tiles,
    in place and out of place, one image and a plan, both directions.  Sums stay below 2^24: f32 is exact."""
    g = torch.Generator(device="cpu").manual_seed(23)
    bits = torch.int32 if t == torch.uint32 else t
    try:
        sat_gb300.set_config(cfg)
        for rev in (False, True):
            ins, refs = [], []
            for h, w in [(h, w) for w in (4, 5, 6, 7, 9, 127, 129, 130, 131, 133, 257, 390) for h in (1, 2, 3, 4, 95, 97, 130)] + \
                        [(1203, 1999), (2002, 1001), (700, 6001)]:
                x = torch.randint(0, 5, (h, w), generator=g).to(bits)
                ref = x.to(torch.int64).flip((0, 1)) if rev else x.to(torch.int64)
                ref = ref.cumsum(0).cumsum(1)
                ins.append(x.to(cuda))
                refs.append((ref.flip((0, 1)) if rev else ref).to(bits).to(cuda))
            for x, ref in zip(ins, refs):
                out = sat_gb300.sat(x.view(t), t, reverse=rev)
                assert torch.equal(out.view(bits), ref), (tuple(x.shape), rev)
                y = x.clone()
                sat_gb300.sat(y.view(t), t, reverse=rev, out=y.view(t))
                assert torch.equal(y, ref), (tuple(x.shape), rev, "in place")
            outs = [torch.empty_like(x) for x in ins]
            plan = sat_gb300.BatchPlan([x.view(t) for x in ins], [o.view(t) for o in outs], reverse=rev)
            plan.exec()
            plan.check()
            for out, ref in zip(outs, refs):
                assert torch.equal(out, ref), (tuple(ref.shape), rev, "plan")
            plan.close()
        sat_gb300.stream_check()
    finally:
        sat_gb300.set_config(-1)


@pytest.mark.parametrize("t_in,t_out", [(torch.uint8, torch.uint32), (torch.int8, torch.float32), (torch.int32, torch.int32),
                                        (torch.float32, torch.float32), (torch.int8, torch.float64),
                                        (torch.float64, torch.float64)])
def test_column_scan_by_strips_and_by_tiles(cuda, t_in, t_out):
    """Column scans on both sides of the choice between strips of columns and tiles: strip and
    block edges (32 columns, 256 rows), low and wide, narrow and tall, packed and padded rows, in place
    where the types allow it.  Small integers: every type's sums are exact."""
    g = torch.Generator(device="cpu").manual_seed(29)
    for h, w in [(1, 1), (1, 33), (7, 31), (8, 32), (255, 33), (256, 64), (257, 31), (511, 1000), (513, 4864), (769, 4865),
                 (1024, 1024), (3000, 37), (9000, 64), (2100, 5001), (300, 20001), (4100, 4096)]:
        for pad in (0, 3):
            x = torch.randint(0, 4, (h, w + pad), generator=g).to(t_in).to(cuda)[:, :w]
            ref = x.to(torch.int64).cumsum(0)
            bits = torch.int32 if t_out == torch.uint32 else t_out
            out = sat_gb300.scan_cols(x, t_out).view(bits)
            assert torch.equal(out, ref.to(bits)), (h, w, pad)
            if t_in == t_out:
                y = x.clone(memory_format=torch.contiguous_format)
                sat_gb300.scan_cols(y, t_out, out=y)
                assert torch.equal(y, ref.to(bits)), (h, w, pad, "in place")
    sat_gb300.stream_check()


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3e38])
def test_infinities_reach_what_their_element_reaches(cuda, value):
    """An infinity, a NaN or sums past the largest f32 change the sums that contain them and
    no other: the tile kernel of configuration 5 (aligned and packed rows) and column scans by strips and
    by tiles, against torch's sums of the same f32 image in f64, rounded to f32."""
    try:
        for h, w in [(500, 512), (601, 389), (3000, 40)]:
            x = torch.ones((h, w), device=cuda)
            x[h // 2, w // 3] = value
            x[h // 3, w // 2] = 3e38 if value == 3e38 else 1.0
            y = x.double()
            cols, sats = y.cumsum(0).float(), y.cumsum(0).cumsum(1).float()

            def same(got, want):
                if value == value and abs(value) != float("inf"):
                    return torch.allclose(got, want, rtol=1e-5, atol=0)
                return torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(0, 0, 0) == 0,
                                                                             want.nan_to_num(0, 0, 0) == 0)

            assert same(sat_gb300.scan_cols(x, torch.float32), cols), (h, w)
            sat_gb300.set_config(5)
            assert same(sat_gb300.sat(x, torch.float32), sats), (h, w)
            rev = sat_gb300.sat(x.flip((0, 1)).contiguous(), torch.float32, reverse=True).flip((0, 1))
            assert same(rev, sats), (h, w)
            sat_gb300.set_config(-1)
    finally:
        sat_gb300.set_config(-1)


@pytest.mark.parametrize("cfg", [0, 1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("t_in,t_out", [(torch.uint8, torch.uint32), (torch.float32, torch.float32)])
def test_waits_that_end_early_stay_inside_the_image(cuda, cfg, t_in, t_out):
    """With a wait limit of a microsecond and a first tile that never publishes, look-backs give up
    everywhere while stages are still being filled for the first time: every role goes on with the
    tiles its CTA was given, so nothing outside the result is written, the error is reported, and the next calls
    are right.  Fewer tiles than CTAs, about as many, and many a CTA; aligned and packed rows."""
    L = _lib.load()
    s = torch.cuda.Stream()
    guard = 1 << 16
    for h, w in [(130, 260), (1500, 1601), (2100, 4096)]:
        x = torch.ones((h, w), dtype=t_in, device=cuda)
        flat = torch.full((h * w + 2 * guard,), 7, dtype=torch.int32, device=cuda)
        out = flat[guard:-guard].view(h, w)
        ref = (torch.arange(1, h + 1, device=cuda)[:, None] * torch.arange(1, w + 1, device=cuda)[None, :]).to(torch.int32)
        torch.cuda.synchronize()
        try:
            sat_gb300.set_config(cfg)
            for rev in (False, True):
                sat_gb300.set_wait_limit_us(1)
                tiles = ((h + 31) // 32) * ((w + 63) // 64)
                for tile in (0, tiles - 1, 1):
                    assert L.satgb_debug_stall_tile(tile) == 0
                    for _ in range(5):
                        with torch.cuda.stream(s):
                            sat_gb300.sat(x, t_out, reverse=rev, out=out.view(t_out))
                try:
                    sat_gb300.stream_check(s)
                except sat_gb300.SatError as e:
                    assert e.status == _lib.ERR_TIMEOUT
                assert bool((flat[:guard] == 7).all()) and bool((flat[-guard:] == 7).all())
                L.satgb_debug_stall_tile(-1)
                sat_gb300.set_wait_limit_us(2_000_000)
                with torch.cuda.stream(s):
                    sat_gb300.sat(x, t_out, reverse=rev, out=out.view(t_out))
                sat_gb300.stream_check(s)
                got = out.view(torch.float32).to(torch.int32) if t_out == torch.float32 else out
                assert torch.equal(got, ref.flip((0, 1)) if rev else ref), (h, w, rev)
        finally:
            L.satgb_debug_stall_tile(-1)
            sat_gb300.set_wait_limit_us(2_000_000)
            sat_gb300.set_config(-1)


@pytest.mark.parametrize("first", [2, 5])
@pytest.mark.parametrize("t_in,t_out", [(torch.uint8, torch.uint32), (torch.float32, torch.float32)])
def test_autotuned_plan_is_the_plan_its_entry_makes(cuda, tmp_path, monkeypatch, first, t_in, t_out):
    """A plan of packed rows off 16-byte boundaries holds copies of them or not as the configuration it was
    tuned to needs them, whichever it was made with: the same as a new plan that takes the
    tuned entry.  Entries of such plans and of plans on 16-byte boundaries are kept apart."""
    import ctypes
    import json
    L = _lib.load()
    cache = tmp_path / "tune.jsonl"
    monkeypatch.setenv("SATGB_TUNE_CACHE", str(cache))
    g = torch.Generator(device="cpu").manual_seed(53)
    sizes = [(201, 301), (77, 1001), (1203, 1501)]
    xs = [torch.randint(0, 9, s, generator=g).to(t_in).to(cuda) for s in sizes]
    live = {}

    def alloc(n, ctx):
        live[(p := torch.cuda.caching_allocator_alloc(n, cuda, torch.cuda.current_stream()))] = n
        return p

    def free(p, ctx):
        if p:
            del live[p]
            torch.cuda.caching_allocator_delete(p)

    def copies():
        return [n for n in live.values() if n % 4096]  # (a workspace is whole pages)

    hooks = _lib._ALLOC_FN(alloc), _lib._FREE_FN(free)

    def check(plan, outs):
        for o in outs:
            o.view(torch.int32).zero_()
        plan.exec()
        plan.check()
        for x, o in zip(xs, outs):
            want = x.to(torch.int64).cumsum(0).cumsum(1)
            got = o.double().to(torch.int64) if t_out == torch.float32 else o.view(torch.int32).to(torch.int64)
            assert torch.equal(got, want)

    sat_gb300.release()
    torch.cuda.synchronize()
    assert L.satgb_set_allocator(*hooks, None) == 0
    try:
        outs = [torch.empty(s, dtype=torch.int32, device=cuda).view(t_out) for s in sizes]
        sat_gb300.set_config(first)
        plan = sat_gb300.BatchPlan(xs, outs)
        sat_gb300.set_config(-1)
        tuned = plan.autotune()
        mine = copies()
        check(plan, outs)
        plan.close()
        fresh = sat_gb300.BatchPlan(xs, outs)
        assert [c["config"] for c in fresh.classes()] == list(tuned)
        assert copies() == mine
        check(fresh, outs)
        fresh.close()
        aligned = [torch.zeros((h, 1024), dtype=t_in, device=cuda) for h, _ in sizes]
        plan = sat_gb300.BatchPlan(aligned, [torch.empty(a.shape, dtype=torch.int32, device=cuda).view(t_out) for a in aligned])
        plan.autotune()
        plan.close()
        assert not live
    finally:
        sat_gb300.set_config(-1)
        torch.cuda.synchronize()
        assert L.satgb_set_allocator(_lib._ALLOC_FN(), _lib._FREE_FN(), None) == 0
    rows = {json.loads(line)["tma"] for line in cache.read_text().splitlines() if "batch_in" in line}
    assert 1 in rows and any(r & 2 for r in rows)


@pytest.mark.parametrize("cfg", [0, 1, 2, 3, 5, 6])
@pytest.mark.parametrize("t", [torch.int32, torch.float64])
def test_stacks_keep_their_planes(cuda, cfg, t):
    """Stacks of planes through every kernel, many tiles a CTA and the plane changing from one tile of a stage to the
    next: each tile's results in its own plane, aligned and odd planes, both directions."""
    g = torch.Generator(device=cuda).manual_seed(61)
    try:
        sat_gb300.set_config(cfg)
        for n, h, w in [(700, 130, 128), (500, 127, 257), (64, 513, 387), (3, 2049, 2050)]:
            x = torch.randint(0, 9, (n, h, w), generator=g, device=cuda, dtype=torch.int32).to(t)
            for rev in (False, True):
                want = (x.flip((1, 2)) if rev else x).cumsum(1, dtype=t).cumsum(2, dtype=t)
                want = want.flip((1, 2)) if rev else want
                for _ in range(3):
                    assert torch.equal(sat_gb300.sat(x, t, reverse=rev), want), (n, h, w, rev)
        sat_gb300.stream_check()
    finally:
        sat_gb300.set_config(-1)


@pytest.mark.parametrize("t", [torch.float32, torch.int32, torch.uint32])
def test_both_kernels_of_configuration_5(cuda, t):
    """4-byte images on both sides of the choice between the deep kernel and 128-row tiles: views whose rows TMA cannot
    address, stacks of odd planes, an image of long anti-diagonals, plans with many tiles a diagonal, with a few packed images
    among aligned ones and with many, both directions.  Sums below 2^24: f32 is exact."""
    g = torch.Generator(device=cuda).manual_seed(59)
    bits = torch.int32 if t == torch.uint32 else t

    def image(*shape):
        return (torch.rand(shape, generator=g, device=cuda) < 0.05).to(bits)

    def want(x, rev):
        y = x.to(torch.int32)
        y = y.flip((-2, -1)) if rev else y
        y = y.cumsum(-2).cumsum(-1).to(bits)
        return y.flip((-2, -1)) if rev else y

    try:
        for rev in (False, True):
            for cfg, (h, w, off, pad) in [(5, (130, 200, 1, 3)), (5, (97, 129, 2, 1)), (5, (1, 1, 1, 4)), (5, (300, 2, 1, 2)),
                                          (-1, (3000, 2999, 1, 3)), (-1, (2500, 3101, 3, 2))]:
                sat_gb300.set_config(cfg)
                x = image(h, w + off + pad)[:, off:off + w]
                out = torch.full((h, w + pad), 7, dtype=bits, device=cuda)
                sat_gb300.sat(x.view(t), t, reverse=rev, out=out[:, :w].view(t))
                assert torch.equal(out[:, :w], want(x, rev)), (h, w, rev)
                assert bool((out[:, w:] == 7).all())
            sat_gb300.set_config(-1)
            x = image(2, 3071, 3073)
            assert torch.equal(sat_gb300.sat(x.view(t), t, reverse=rev).view(bits), want(x, rev)), rev
            x = image(16000, 16000)
            assert torch.equal(sat_gb300.sat(x.view(t), t, reverse=rev).view(bits), want(x, rev)), rev
            del x
            for packed in (0, 1, 2, 3, 16):
                xs = [image(1023, 1021 if i < packed else 1024) for i in range(16)] + [image(1100, 900)[:, 1:850]]
                outs = [torch.empty(x.shape, dtype=bits, device=cuda) for x in xs]
                plan = sat_gb300.BatchPlan([x.view(t) for x in xs], [o.view(t) for o in outs], reverse=rev)
                assert plan.classes()[0]["config"] == 5
                plan.exec()
                plan.check()
                for i, (x, out) in enumerate(zip(xs, outs)):
                    assert torch.equal(out, want(x, rev)), (packed, i, rev)
                plan.close()
        sat_gb300.stream_check()
    finally:
        sat_gb300.set_config(-1)


def test_plan_of_one_launch_keeps_one_table(cuda):
    """A plan whose classes share a launch holds the tile order (16 bytes a tile) of that launch and
    none of the classes' own: 64 columns of 2^20 pixels, half a million tiles, and a small image."""
    L = _lib.load()
    n, h = 64, 1 << 20
    ins = torch.ones((n, h, 1), dtype=torch.uint8, device=cuda)
    outs = torch.zeros((n, h, 1), dtype=torch.int32, device=cuda)
    small, small_out = torch.ones((50, 60), dtype=torch.uint8, device=cuda), torch.zeros((50, 60), dtype=torch.int32, device=cuda)
    pool = torch.empty(3 << 30, dtype=torch.uint8, device=cuda)  # the plans' workspaces
    at = [0]

    def alloc(size, ctx):
        p = pool.data_ptr() + at[0]
        at[0] += (size + 4095) // 4096 * 4096
        return p if at[0] <= pool.numel() else 0

    hooks = _lib._ALLOC_FN(alloc), _lib._FREE_FN(lambda p, ctx: None)

    def plan(k):
        return sat_gb300.BatchPlan([ins[i] for i in range(k)] + [small],
                                   [outs[i].view(torch.uint32) for i in range(k)] + [small_out.view(torch.uint32)])

    sat_gb300.release()
    assert L.satgb_set_allocator(*hooks, None) == 0
    try:
        first = plan(1)  # the kernels and the graph's own memory
        first.exec()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        p = plan(n)
        held = free - torch.cuda.mem_get_info()[0]
        c = p.classes()
        assert c[0]["config"] == c[1]["config"] and c[0]["tiles"] == n * (h // 128) and c[1]["tiles"] == 1
        assert held < 1.5 * 16 * c[0]["tiles"], held
        p.exec()
        p.check()
        want = torch.arange(1, h + 1, dtype=torch.int32, device=cuda)
        assert all(torch.equal(outs[i, :, 0], want) for i in range(n))
        assert int(small_out[-1, -1]) == 3000
        p.close()
        first.close()
    finally:
        torch.cuda.synchronize()
        assert L.satgb_set_allocator(_lib._ALLOC_FN(), _lib._FREE_FN(), None) == 0


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_infinities_leave_finite_sums_exact(cuda, value):
    """An infinity's sign and a NaN arrive in every sum that contains them, and every other sum is what it is without them, to the
    bit (sums of ones below 2^24): both kernels of configuration 5, aligned, packed and offset rows, both directions, and
    column scans by strips and by tiles, with and without a partial last strip."""
    def same(got, want):
        finite = want.isfinite()
        return (torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isposinf(), want.isposinf())
                and torch.equal(got.isneginf(), want.isneginf()) and torch.equal(got[finite], want[finite]))

    try:
        for h, w, off in [(500, 512, 0), (601, 389, 0), (300, 250, 1), (3000, 40, 0), (1030, 1001, 0), (8200, 100, 0)]:
            x = torch.ones((h, w + 4 * off), device=cuda)[:, off:off + w]
            for r, c in [(h // 2, w // 3), (0, 0), (h - 1, w - 1)]:
                y = x.clone() if not off else torch.ones((h, w + 4), device=cuda)[:, 1:1 + w]
                y[r, c] = value
                assert same(sat_gb300.scan_cols(y, torch.float32), y.double().cumsum(0).float()), (h, w)
                sats = y.double().cumsum(0).cumsum(1).float()
                sat_gb300.set_config(5)
                assert same(sat_gb300.sat(y, torch.float32), sats), (h, w)
                flipped = torch.ones((h, w + 4 * off), device=cuda)[:, off:off + w]
                flipped.copy_(y.flip((0, 1)))
                assert same(sat_gb300.sat(flipped, torch.float32, reverse=True).flip((0, 1)), sats), (h, w)
                sat_gb300.set_config(-1)
    finally:
        sat_gb300.set_config(-1)
