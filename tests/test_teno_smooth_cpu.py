"""The smooth-stencil tests of the TENO5 kernels, as they read their operands,
imply that the cut-off keeps every sub-stencil.

FP64 (teno_smooth_hi): on the high words of e_k = 4 b_k + eps, hi(|tau|) <=
min hi(e_k) + 2^21 (a factor 4 in the exponent field) and max hi(e_k) below
that of 1e30.  FP32 (teno_smooth2): tau <= 4 e_min over the whole range to
FLT_MAX, where the cut-off's reciprocal of e_min + tau flushes to 0."""
import numpy as np
import pytest

HI_1E30 = 0x46293E59


def _hi(x):
    return (np.asarray(x, np.float64).view(np.int64) >> 32).astype(np.int64)


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
    for bad in (np.nan, np.inf):
        for k in range(3):
            e = np.ones((1, 3))
            e[0, k] = bad
            with np.errstate(invalid="ignore"):
                tau = np.abs(e[:, 0] - e[:, 2])
            ok = ((_hi(tau) & 0x7FFFFFFF) <= _hi(e).min(axis=1) + 0x00200000) & (_hi(e).max(axis=1) < HI_1E30)
            assert not ok.any()


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("ulp", [-2, 0, 2])
def test_fp32_test_keeps_all_up_to_flt_max(seed, ulp):
    rng = np.random.default_rng(seed)
    f = np.float32
    b = _triples(rng, 200_000, -40, 3e38).astype(f)
    tiny = f(1.17549435e-38)

    def rcp(x):  # approximate to 2 ulp, subnormal results flushed
        r = (f(1) / x).astype(f)
        for _ in range(abs(ulp)):
            r = np.nextafter(r, f(np.inf) if ulp > 0 else f(0))
        return np.where(r < tiny, f(0), r)

    with np.errstate(over="ignore", under="ignore", invalid="ignore"):
        e = b + tiny
        em = e.min(axis=1)
        tau = np.abs(b[:, 0] - b[:, 2])
        smooth = tau <= f(4) * em
        t = em * rcp(em + tau)
        s = tau * t
        x = np.stack([s * rcp(e[:, k]) + t for k in range(3)], axis=1).astype(f)
        y = x * x
        G = (y * y) * y
        lim = f(1e-5) * ((G[:, 0] + G[:, 1]) + G[:, 2])
        keep = G >= lim[:, None]
    assert 0.1 < smooth.mean() < 0.95 and (em[smooth] > 1e30).any()
    assert keep[smooth].all()
