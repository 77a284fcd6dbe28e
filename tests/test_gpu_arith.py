"""The arithmetic the kernels are built on, checked on the GPU: the refined
reciprocal that replaces IEEE division, and the FP64 pipe behaviour the
kernel design assumes (documented in the package's design notes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_refined_reciprocal(cuda_lib):
    """rcp.approx seed + one cubic Newton-Raphson step is within one ulp of the
    correctly rounded 1/x (the reference divides), over 26 decades."""
    import torch
    from dadi_gb300 import _lib
    x = np.exp(np.random.default_rng(0).uniform(-30, 30, 1 << 18))
    d_x = torch.from_numpy(x).cuda()
    d_o = torch.empty_like(d_x)
    _lib.check(cuda_lib.dgb_probe_rcp(_lib.dptr(d_x), _lib.dptr(d_o), len(x),
                                      _lib.stream_handle(torch)), "rcp")
    r = d_o.cpu().numpy()
    exact = 1.0 / x
    ulps = np.abs(r.view(np.int64) - exact.view(np.int64))
    assert ulps.max() <= 1
    assert (ulps == 0).mean() > 0.99


def _pivot_inputs(kind, n):
    rng = np.random.default_rng(7)
    bits = lambda: rng.integers(0, 1 << 64, n, dtype=np.uint64).view(np.float64)
    if kind == "any bits":  # every exponent, subnormals, infinities and NaN
        return bits(), bits(), bits()
    x = np.exp(rng.uniform(-80, 80, n))
    t = rng.choice([-1.0, 1.0], n) * np.exp(rng.uniform(-600, 600, n))
    c = -rng.uniform(0, 1, n)
    if kind == "short mantissas":  # exact products, ties, mantissas next to 1 and 2
        x = np.ldexp(1 + rng.integers(-64, 64, n) * 2.0 ** -52, rng.integers(-140, 140, n))
        t = np.ldexp(1 + rng.integers(-64, 64, n) * 2.0 ** -rng.integers(5, 53, n),
                     rng.integers(-1060, 1020, n))
    if kind == "pivots":  # the sweeps' range, with the zero couplings of the boundary rows
        x, t = 1 + np.exp(rng.uniform(-20, 8, n)), t ** 0.02
        c[::7] = 0.0
    return x, t, c


@pytest.mark.parametrize("kind", ["pivots", "wide", "short mantissas", "any bits"])
def test_integer_pivot_gives_the_bits_of_the_doubles(cuda_lib, kind):
    """t * (1/x), c * (1/x), t / x and c * x on the integer pipes are, bit for
    bit, what the FP64 instructions give (rounding, signs, and every value that leaves the
    integers' range: zeros, subnormals, overflows, infinities; NaN as NaN)."""
    import torch
    from dadi_gb300 import _lib
    n = 1 << 20
    with np.errstate(all="ignore"):
        xtc = np.concatenate(_pivot_inputs(kind, n))
    d = torch.from_numpy(xtc).cuda()
    o = torch.empty(8 * n, dtype=torch.float64, device="cuda")
    _lib.check(cuda_lib.dgb_probe_pivot(_lib.dptr(d), _lib.dptr(o), n,
                                        _lib.stream_handle(torch)), "pivot")
    o = o.cpu().numpy()
    got, want = o[:4 * n], o[4 * n:]
    same = (got.view(np.int64) == want.view(np.int64)) | (np.isnan(got) & np.isnan(want))
    assert same.all()


def _same_bits(a, b):
    return (a.view(np.int64) == b.view(np.int64)) | (np.isnan(a) & np.isnan(b))


@pytest.mark.parametrize("kind", ["pivots", "wide", "short mantissas", "any bits"])
def test_integer_pivot_of_the_partitioned_rows(cuda_lib, kind):
    """The partitioned solves' three products with 1/x and the delj rows'
    product are the FP64 instructions', bit for bit."""
    import torch
    from dadi_gb300 import _lib
    n = 1 << 18
    with np.errstate(all="ignore"):
        x, t, c = _pivot_inputs(kind, n)
        d = np.roll(t, 5)
    xtcd = torch.from_numpy(np.concatenate([x, t, c, d])).cuda()
    o = torch.empty(8 * n, dtype=torch.float64, device="cuda")
    _lib.check(cuda_lib.dgb_probe_pivot3(_lib.dptr(xtcd), _lib.dptr(o), n,
                                         _lib.stream_handle(torch)), "pivot3")
    o = o.cpu().numpy()
    assert _same_bits(o[:4 * n], o[4 * n:]).all()


def test_integer_pivot_of_zeros(cuda_lib):
    """Zeros of both signs in every place, against ordinary values, the ends of
    the integers' ranges, infinities and NaN."""
    import itertools
    import torch
    from dadi_gb300 import _lib
    v = [0.0, -0.0, 1.0, -1.5, 3.7e5, -2e-7, 5e-324, 1e-310, 2.0 ** -129, 2.0 ** 128, -2.0 ** 900,
         2.0 ** -900, np.inf, -np.inf, np.nan]
    x, t, c, d = [np.ascontiguousarray(a) for a in np.array(list(itertools.product(v, repeat=4))).T]
    n = len(x)
    for call, cols in ((cuda_lib.dgb_probe_pivot, (x, t, c)),
                       (cuda_lib.dgb_probe_pivot3, (x, t, c, d))):
        a = torch.from_numpy(np.concatenate(cols)).cuda()
        o = torch.empty(8 * n, dtype=torch.float64, device="cuda")
        _lib.check(call(_lib.dptr(a), _lib.dptr(o), n, _lib.stream_handle(torch)), "pivot")
        o = o.cpu().numpy()
        assert _same_bits(o[:4 * n], o[4 * n:]).all()


def test_fp64_rate_and_idle_lanes(cuda_lib):
    """The FP64 FMA rate is positive and a warp instruction with a quarter of
    its lanes active takes as long as a full one (idle lanes are not free),
    which is why the kernels pack lines into full warps."""
    import torch
    from dadi_gb300 import _lib
    full = _lib.fp64_fma_peak_tflops(torch, active_lanes=32, target_s=0.01, repeats=2)
    quarter = _lib.fp64_fma_peak_tflops(torch, active_lanes=8, target_s=0.01, repeats=2)
    assert full > 0.1
    assert quarter < 0.5 * full
