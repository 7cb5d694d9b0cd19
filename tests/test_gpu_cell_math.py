"""The short exponential and logarithm of the chemistry integrators (csrc/hf_cell.cuh) on the
GPU, against long double."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
L = np.longdouble


def evaluate(lib, x):
    xd = torch.from_numpy(x).cuda()
    outs = [torch.empty_like(xd) for _ in range(4)]
    assert lib.hf_cellmath_eval(xd.data_ptr(), xd.numel(), *[o.data_ptr() for o in outs], None) == 0
    torch.cuda.synchronize()
    return [o.cpu().numpy() for o in outs]


def ulps(got, ref):
    return np.abs((got.astype(L) - ref) / np.spacing(np.abs(ref.astype(np.float64))).astype(L)).astype(np.float64)


def test_exponentials(gpu):
    """The table entry and the result round once each, half a unit of the last place both; the
    polynomial's r^4/24 - R^2 r^2/24 (R = 0.51, r = 0.65 of a step) is 3.8e-17 of the result, 0.34
    of a unit where its mantissa is near 2: 1.35 units with what the polynomial rounds."""
    assert np.finfo(L).nmant >= 63
    rng = np.random.default_rng(4)
    step = np.log(2) / 2048
    mid = (rng.integers(-800000, 800000, 20000) + 0.5) * step  # where the reduced argument is largest
    x = np.concatenate([rng.uniform(-339.9, 339.9, 60000), rng.uniform(-40, 40, 40000), rng.uniform(-1, 1, 20000), mid,
                        np.arange(-64, 65) * np.log(2), [0.0, -0.0, 1e-300, -1e-17]])
    x = x[np.abs(x) < 339.9]
    e, ep, em, _ = evaluate(gpu.lib, x)
    up, dn = np.exp(x.astype(L)), np.exp(-x.astype(L))
    worst = [float(ulps(g, r).max()) for g, r in ((e, up), (ep, up), (em, dn))]
    assert max(worst) <= 1.35, worst


def test_logarithm(gpu):
    """m ln2 + log F rounds to half a unit of its own (at most a unit of the result), the last
    sum to half a unit; log F's table entry is off by 2^-54 at most, the FP32 bracket and its
    constants by 2.6e-8 times u^3 < 7.5e-9, 2e-16: 1.5 units + 2.7e-16."""
    rng = np.random.default_rng(6)
    x = np.concatenate([rng.uniform(0.5, 2.0, 60000), rng.uniform(150, 6000, 40000), np.exp(rng.uniform(-700, 700, 40000)),
                        1.0 + rng.uniform(-2e-3, 2e-3, 20000), 2.0 ** np.arange(-1020, 1020, dtype=np.float64)])
    l = evaluate(gpu.lib, x)[3]
    ref = np.log(x.astype(L))
    err = np.abs((l.astype(L) - ref).astype(np.float64))
    worst = float((err / (1.5 * np.spacing(np.abs(ref.astype(np.float64))) + 2.7e-16)).max())
    assert worst <= 1.0, worst


def test_library_outside_the_fast_ranges(gpu):
    x = np.array([340.5, -340.5, 700.0, 709.7, 710.0, -745.0, -800.0, np.inf, -np.inf, np.nan, 1e-310, 0.0, -1.0, 1.7e308])
    e, ep, em, l = evaluate(gpu.lib, x)
    with np.errstate(all="ignore"):
        for got, ref in ((e, np.exp(x)), (ep, np.exp(x)), (em, np.exp(-x)), (l, np.log(x))):
            fin = np.isfinite(ref) & (ref != 0)
            assert np.array_equal(np.isnan(got), np.isnan(ref))
            assert np.array_equal(got[np.isinf(ref)], ref[np.isinf(ref)])
            assert np.all(np.abs(got[fin] - ref[fin]) <= 2 * np.spacing(np.abs(ref[fin])))
