"""The branch-free arithmetic of the Kalman step (csrc/flat_math.cuh) against
the plain one on the device: the quotient, reciprocal and root bit for bit
(every mantissa for the one-operand ones), the double-based functions up to
the values within ~1e-16 of a rounding boundary, the operands that send a
step back to the plain form, and whole steps from such states."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
RCP, DIV, SQRT, SIN, COS, LOG, HYPOT, INV_DET = range(8)


def built(tmp_path_factory, name):
    out = str(tmp_path_factory.mktemp("flat") / f"lib{name}.so")
    subprocess.check_call([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode",
                           "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared",
                           "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-fmad=false",
                           os.path.join(HERE, name + ".cu"), "-o", out])
    return ctypes.CDLL(out)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    L = built(tmp_path_factory, "flat_math_check")
    p = ctypes.c_void_p
    L.flat_math_check.argtypes = [ctypes.c_int, ctypes.c_longlong, p, p, p]
    L.flat_math_seen.argtypes = [ctypes.c_int, p, ctypes.c_int, p]
    L.flat_math_step.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_uint] + [p] * 9
    return L


def check(lib, what, n, a=None, b=None):
    import torch
    counts = torch.zeros(3, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert lib.flat_math_check(what, n, None if a is None else a.data_ptr(),
                               None if b is None else b.data_ptr(), counts.data_ptr()) == 0
    c = counts.cpu().tolist()
    assert c[2] == 0, "operands outside the safe range"
    return c[0], c[1]


def operands(n, seed, lo, hi, signed=True):
    """Sizes log-uniform in [lo, hi]."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    v = torch.exp(np.log(lo) + u * (np.log(hi) - np.log(lo))).float()
    if signed:
        v = torch.where(torch.rand(n, generator=g, device="cuda") < 0.5, -v, v)
    return v


@pytest.mark.parametrize("what", [RCP, SQRT])
def test_every_mantissa(lib, what):
    # 2^24 consecutive floats from 1: all mantissas in two exponents. The
    # reciprocal's last step is exact but for a mantissa of all ones, where
    # 1 / b lies next to a rounding boundary: at most one value per exponent.
    bad, ulps = check(lib, what, 1 << 24)
    assert bad <= (2 if what == RCP else 0) and ulps <= 1


def test_quotients(lib):
    n = 1 << 26
    bad, ulps = check(lib, DIV, n, operands(n, 1, 1e-6, 1e6), operands(n, 2, 1e-6, 1e6))
    assert bad <= 2 and ulps <= 1


@pytest.mark.parametrize("what,lo,hi,signed", [(SIN, 1e-3, 6.4, True), (COS, 1e-3, 6.4, True),
                                               (SIN, 10.0, 250.0, True), (LOG, 1e-20, 1e20, False),
                                               (LOG, 0.9, 1.1, False)])
def test_functions(lib, what, lo, hi, signed):
    # Two doubles within d = 1e-15 of each other (relative) round to different
    # floats when a boundary lies between them: about 2 d / 2^-23 of the values.
    n = 1 << 24
    bad, ulps = check(lib, what, n, operands(n, 3, lo, hi, signed))
    assert bad <= 4 and ulps <= 1


@pytest.mark.parametrize("what", [HYPOT, INV_DET])
def test_two_operand_functions(lib, what):
    n = 1 << 24
    bad, ulps = check(lib, what, n, operands(n, 5, 1e-2, 1e2, what == HYPOT),
                      operands(n, 6, 1e-2, 1e2, what == HYPOT))
    assert bad <= 4 and ulps <= 1


def test_operands_outside_the_range(lib):
    import torch
    v = torch.tensor([0.0, -0.0, 1.0, -1.0, 1e-7, 1e7, 5e5, 2e-6, float("inf"), -float("inf"),
                      float("nan"), 1e-40], device="cuda")
    for wide, exp in ((0, [0, 0, 1, 1, 0, 0, 1, 1, 0, 0, 0, 0]),
                      (1, [0, 0, 1, 0, 1, 1, 1, 1, 0, 0, 0, 0])):
        ok = torch.zeros(len(v), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert lib.flat_math_seen(len(v), v.data_ptr(), wide, ok.data_ptr()) == 0
        assert ok.cpu().tolist() == exp


def step_states(barrel):
    """Toy tracks of one layer with every special value in every place it can
    take: parameters, covariance, charge and hit."""
    from mkfit_b200 import synth
    n = 40000
    gen = synth.gen_fit_event if barrel else synth.gen_fit_event_steered
    ev, layer = gen(n, seed=3), 3 if barrel else 2
    rng = np.random.default_rng(7)
    a = rng.normal(0, 1, (n, 6, 6)) * np.array([.01, .01, .05, .02, .002, .002])[None, :, None]
    d = dict(par=ev.par.copy(), err=synth.pack_sym(a @ a.transpose(0, 2, 1)).astype(np.float32),
             chg=ev.chg.copy(), hpos=ev.hit_pos[layer].copy(), herr=ev.hit_err[layer].copy())
    special = np.array([0.0, -0.0, 1e-40, 1e-30, 1e-8, -1.0, 1500.0, 1e7, 3e19, -1e30, 3e38,
                        np.inf, -np.inf, np.nan, np.pi / 2, np.pi], np.float32)
    i = 1000  # the first 1000 stay ordinary
    for name in ("par", "err", "hpos", "herr"):
        for row in d[name]:
            row[i:i + len(special)] = special
            i += len(special)
    for rows in (d["par"][:2], d["hpos"][:2], d["hpos"], d["err"], d["herr"]):
        for s in special:  # at the beam line, or the whole block special
            rows[:, i] = s
            i += 1
    for q in (0, 2, -3, 127):
        d["chg"][i] = q
        i += 1
    assert i < n
    return ev, {k: np.ascontiguousarray(v) for k, v in d.items()}, i


@pytest.mark.parametrize("barrel", [1, 0])
@pytest.mark.parametrize("grid", ["usual", "inf", "huge", "nan"])
def test_steps_from_any_state(lib, barrel, grid):
    """The fit's flat propagation and update equal the plain ones bit for bit,
    infinities and NaNs included, whether or not they go back to them. The
    double functions' results may round otherwise for about 1e-7 of the
    values (test_functions), 6 per step: at most 2 of these tracks."""
    import torch
    ev, d, n_special = step_states(barrel)
    n = len(d["chg"])
    rl, xi = np.array(ev.rl_grid), np.array(ev.xi_grid)
    if grid != "usual":
        v = np.float32(dict(inf=np.inf, huge=1e38, nan=np.nan)[grid])
        xi[::2] = v
        rl[1::4] = v
    t = {k: torch.from_numpy(v).cuda() for k, v in dict(d, rl=rl, xi=xi).items()}
    for pflags in range(4):
        out = torch.zeros((2, 55, n), device="cuda")
        back = torch.zeros((2, n), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert lib.flat_math_step(n, barrel, pflags, *(t[k].data_ptr() for k in (
            "rl", "xi", "par", "err", "chg", "hpos", "herr")), out.data_ptr(), back.data_ptr()) == 0
        flat, plain = out.cpu().numpy()
        bad = ((flat != plain) & ~(np.isnan(flat) & np.isnan(plain))).any(0)
        print(f"pflags {pflags}: {bad.sum()} of {n} tracks differ, back {back.sum(1).tolist()}")
        assert not (np.isnan(flat) != np.isnan(plain)).any()
        assert bad.sum() <= 2, np.flatnonzero(bad)[:20]
        # Both ways were taken: special states went back, ordinary ones did not.
        b = back.cpu().numpy()
        assert (b[:, 1000:n_special].sum(1) > 20).all()
        if grid == "usual":
            assert b[:, :1000].sum() == 0


@pytest.fixture(scope="module")
def adjoint_lib(tmp_path_factory):
    L = built(tmp_path_factory, "adjoint_flat_check")
    L.adjoint_flat_step.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 5
    return L


@pytest.mark.parametrize("grid", ["usual", "inf", "huge", "nan"])
def test_differentiable_steps_from_any_state(adjoint_lib, grid):
    """The same for a step of the differentiable fit and its reverse, with
    special values in the gradients that enter it too (built without
    contraction on both sides, the only thing that may tell them apart but
    for the reciprocals of a mantissa of all ones: at most 2 tracks)."""
    import torch
    ev, d, _ = step_states(1)
    n = len(d["chg"])
    rng = np.random.default_rng(8)
    inp = np.concatenate([d["par"], d["err"], d["hpos"], d["herr"], np.ones((1, n), np.float32),
                          d["chg"][None].astype(np.float32)])
    bars = rng.normal(0, 1, (27, n)).astype(np.float32) * 10.0 ** rng.integers(-4, 5, (27, 1))
    bars = bars.astype(np.float32)
    special = np.array([0.0, -0.0, 1e-40, 1e-30, 1e30, 3e38, np.inf, -np.inf, np.nan], np.float32)
    i = 2000
    for row in [inp[36]] + list(bars):
        row[i:i + len(special)] = special
        i += len(special)
    bars[:, i:i + 200] = 0
    rl, xi = np.array(ev.rl_grid), np.array(ev.xi_grid)
    if grid != "usual":
        v = np.float32(dict(inf=np.inf, huge=1e38, nan=np.nan)[grid])
        xi[::2] = v
        rl[1::4] = v
    t = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (inp, bars, rl, xi)]
    out = torch.zeros((2, 58, n), device="cuda")
    torch.cuda.synchronize()
    assert adjoint_lib.adjoint_flat_step(n, *(x.data_ptr() for x in t), out.data_ptr()) == 0
    flat, plain = out.cpu().numpy()
    assert np.isfinite(plain[:, :1000]).all() or grid != "usual"
    bad = ((flat != plain) & ~(np.isnan(flat) & np.isnan(plain))).any(0)
    print(f"{bad.sum()} of {n} tracks differ; non-finite {(~np.isfinite(plain)).any(0).sum()}")
    assert bad.sum() <= 2, (np.flatnonzero(bad)[:20], np.flatnonzero(bad).size)
