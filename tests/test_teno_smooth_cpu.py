"""The smooth-stencil tests of the TENO5 kernels, as they read their operands,
imply that the cut-off keeps every sub-stencil.

FP64 (teno_smooth_hi): on the high words of e_k = 4 b_k + eps, hi(|tau|) <=
min hi(e_k) + 2^21 (a factor 4 in the exponent field) and max hi(e_k) below
that of 1e30, unsigned.  FP32 (teno_smooth2): tau / 4 <= e_min over the whole
range to FLT_MAX, where the cut-off's reciprocal of e_min + tau flushes to 0,
and past it: what passes with an overflowed indicator is what the cut-off keeps
whole without its non-finite watch."""
import numpy as np
import pytest

HI_1E30 = 0x46293E59


def _hi(x):
    return (np.asarray(x, np.float64).view(np.uint64) >> np.uint64(32)).astype(np.int64)


def _triples(rng, n, lo, top):
    scale = 10.0 ** rng.uniform(lo, np.log10(top), (n, 1))
    b = scale * 10.0 ** rng.uniform(-1.5, 0.7, (n, 3))
    b[rng.random((n, 3)) < 0.05] = 0.0
    return np.minimum(b, top)


@pytest.mark.parametrize("seed", range(4))
def test_fp64_high_word_test_keeps_all(seed):
    rng = np.random.default_rng(seed)
    b = _triples(rng, 200_000, -60, 1e32)
    e = b + 4e-40
    tau = np.abs(e[:, 0] - e[:, 2])
    smooth = ((_hi(tau) & 0x7FFFFFFF) <= _hi(e).min(axis=1) + 0x00200000) & (_hi(e).max(axis=1) < HI_1E30)
    assert 0.1 < smooth.mean() < 0.95
    # the cut-off itself, from tau / e_k
    g = (1.0 + tau[:, None] / e) ** 6
    keep = ~(g < 1e-5 * g.sum(axis=1, keepdims=True))
    assert keep[smooth].all()
    # with room: the largest g of a triple that passes is far from cutting another
    assert (g[smooth].max(axis=1) < 2e4).all()


def test_fp64_high_word_test_refuses_non_finite():
    for bad in (np.nan, -np.nan, np.inf):
        for k in range(3):
            e = np.ones((1, 3))
            e[0, k] = bad
            with np.errstate(invalid="ignore"):
                tau = np.abs(e[:, 0] - e[:, 2])
            ok = ((_hi(tau) & 0x7FFFFFFF) <= _hi(e).min(axis=1) + 0x00200000) & (_hi(e).max(axis=1) < HI_1E30)
            assert not ok.any()


def _fp32(b, ulp):
    """(smooth, all kept, watch quiet) of FP32 indicator triples; reciprocals
    approximate to `ulp`, subnormal results flushed."""
    f = np.float32
    tiny = f(1.17549435e-38)

    def rcp(x):
        r = (f(1) / x).astype(f)
        for _ in range(abs(ulp)):
            r = np.nextafter(r, f(np.inf) if ulp > 0 else f(0))
        return np.where(r < tiny, f(0), r)

    with np.errstate(over="ignore", under="ignore", invalid="ignore"):
        e = b + tiny
        em = np.fmin(b[:, 0], np.fmin(b[:, 1], b[:, 2])) + tiny
        tau = np.abs(b[:, 0] - b[:, 2])
        smooth = f(0.25) * tau <= em
        t = em * rcp(em + tau)
        s = tau * t
        x = np.stack([s * rcp(e[:, k]) + t for k in range(3)], axis=1).astype(f)
        y = x * x
        G = (y * y) * y
        lim = f(1e-5) * ((G[:, 0] + G[:, 1]) + G[:, 2])
        return smooth, (G >= lim[:, None]).all(axis=1), np.isfinite(lim)


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("ulp", [-2, 0, 2])
def test_fp32_test_keeps_all_up_to_flt_max(seed, ulp):
    b = _triples(np.random.default_rng(seed), 200_000, -40, 3e38).astype(np.float32)
    smooth, kept, quiet = _fp32(b, ulp)
    assert 0.1 < smooth.mean() < 0.95 and (b[smooth].min(axis=1) > 1e30).any()
    assert kept[smooth].all() and quiet[smooth].all()


@pytest.mark.parametrize("ulp", [-2, 0, 2])
def test_fp32_overflowed_indicators(ulp):
    """Every pattern of infinite and NaN members beside finite ones of any size:
    a triple that passes is kept whole by the cut-off, which reports nothing
    for it; an infinite or NaN outer member never passes.  (A middle NaN has a NaN
    beside it: it is made of the outer ones' differences.)"""
    rng = np.random.default_rng(9)
    b = _triples(rng, 200_000, -40, 3.4e38).astype(np.float32)
    b[::2] = rng.uniform(3e37, 3.4e38, b[::2].shape)
    for pattern in set(range(1, 27)) - {6}:  # base-3 digits: 0 finite, 1 inf, 2 NaN
        c = b.copy()
        for k in range(3):
            m = pattern // 3 ** k % 3
            if m:
                c[:, k] = np.inf if m == 1 else np.nan
        smooth, kept, quiet = _fp32(c, ulp)
        assert kept[smooth].all() and quiet[smooth].all()
        assert smooth.any() == (pattern == 3)
