"""FP64 WENO5 / TENO5 / WENO7 faces in differences (face_flux64): the residual of the
axis sweeps, the tiles and the oracle agree where the core can go wrong --
uniform states (all indicators zero), jumps of one cell, linear and parabolic
profiles, magnitudes from 1e-6 to 1e6 -- for each face flux.

Tolerance: a face flux is a few hundred FP64 operations on terms no larger
than the largest flux component Fmax of the field, so two evaluations differ by
at most ~1000 eps Fmax, and a residual by twice that per axis over h."""
import numpy as np
import pytest

from helpers import FLUX_OF, SCHEME_OF, from_oracle, oracle_spec, to_oracle
from sonicsolver_b200 import cases

EPS = 2.220446049250313e-16


def _state(kind, n, scale):
    x = np.arange(n) / (n - 1)
    one = np.ones(n)
    if kind == "uniform":
        rho, u, p = one, 0.3 * one, one
    elif kind == "jump":
        rho, u, p = np.where(x < 0.5, 1.0, 0.6), np.where(x < 0.5, 0.2, 0.1), np.where(x < 0.5, 1.0, 0.7)
    elif kind == "linear":
        rho, u, p = 1 + 0.2 * x, 0.1 * x, 1 + 0.1 * x
    else:
        rho, u, p = 1 + 0.2 * x * x, 0.3 * np.sin(7 * x), 1 + 0.1 * np.cos(5 * x)
    return cases.conserved(scale * rho, u, 0.5 * u, -0.25 * u, scale * p)


@pytest.mark.gpu
@pytest.mark.parametrize("recipe", ["weno5Rusanov", "weno5Roe", "teno5Rusanov", "teno5Steger", "weno5LaxFriedrichs",
                                    "weno7Rusanov"])
@pytest.mark.parametrize("kind", ["uniform", "jump", "linear", "smooth"])
@pytest.mark.parametrize("scale", [1e-6, 1.0, 1e6])
def test_residual_in_differences(recipe, kind, scale, oracle):
    scheme, flux = recipe[:5], recipe[5:]
    ny, nx = 19, 35
    line = _state(kind, nx, scale)
    q = np.broadcast_to(line, (1, ny, nx, 5)).copy()
    q[0, :, :, 2] *= 1 + 0.05 * np.arange(ny)[:, None]
    h = (1.0 / (nx - 1), 1.0 / (ny - 1), 1.0)
    case = cases.Case("f", 2, (nx, ny, 1), h, (0, 0, 0), (0, 0, 0), q, 1.4, 1.0, 0.5, recipe, "SSPRK3")
    spec = oracle_spec(case, recipe=recipe)
    want = from_oracle(spec, oracle.rhs(spec, SCHEME_OF[scheme], FLUX_OF[flux], to_oracle(spec, q)))
    rho, u, v, w, p = cases.primitive(q)
    c = np.sqrt(1.4 * p / rho)
    fmax = (np.abs(q).max() + p.max()) * (np.abs(u) + np.abs(v) + c).max()
    bound = 2 * 1000 * EPS * fmax * (1 / h[0] + 1 / h[1])
    for variant in (0, 1, 2):
        s = case.solver()
        s.variant = variant
        err = np.abs(s.residual().reshape(q.shape) - want)[:, 1:-1, 1:-1]  # the solved nodes
        assert err.max() <= bound, (variant, err.max() / bound)


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e24, 1e27])
def test_weno7_beyond_the_folded_weights(scale, oracle):
    """Differences around 1e25: the folded weights' products leave FP64 range
    and the core falls back to the point form; the residual stays the oracle's."""
    nx = 41
    q = _state("jump", nx, scale)[None, None].copy()
    h = (1.0 / (nx - 1), 1.0, 1.0)
    case = cases.Case("f", 1, (nx, 1, 1), h, (0, 0, 0), (0, 0, 0), q, 1.4, 1.0, 0.5, "weno7Rusanov", "SSPRK3")
    spec = oracle_spec(case, recipe="weno7Rusanov")
    want = from_oracle(spec, oracle.rhs(spec, SCHEME_OF["weno7"], FLUX_OF["Rusanov"], to_oracle(spec, q)))
    rho, u, v, w, p = cases.primitive(q)
    fmax = (np.abs(q).max() + p.max()) * (np.abs(u) + np.sqrt(1.4 * p / rho)).max()
    s = case.solver()
    for variant in (0, 1):
        s.variant = variant
        err = np.abs(s.residual().reshape(q.shape) - want)[..., 1:-1, :]
        assert err.max() <= 2 * 1000 * EPS * fmax / h[0]


@pytest.mark.gpu
@pytest.mark.parametrize("recipe,scale", [("weno5Rusanov", s) for s in (1e18, 4e18, 1e19)] +
                                         [("teno5Rusanov", s) for s in (1e24, 1e25, 1e26)])
def test_pair_denominators_keep_their_range(recipe, scale, oracle):
    """Differences up to where the product of the two sides' denominators leaves
    FP64 range (the scale is 3 to 4 times the differences); TENO5 on a field
    rough everywhere (beside a uniform part its sixth powers leave the range
    first, in the reference too)."""
    nx = 41
    q = _state("jump", nx, scale)
    if recipe.startswith("teno5"):
        rng = np.random.default_rng(3)
        q = cases.conserved(scale * (1 + 0.3 * rng.random(nx)), 0.1 * rng.random(nx), 0.1 * rng.random(nx),
                            0.1 * rng.random(nx), scale * (1 + 0.3 * rng.random(nx)))
    q = q[None, None].copy()
    h = (1.0 / (nx - 1), 1.0, 1.0)
    bc = (int(recipe.startswith("teno5")), 0, 0)
    case = cases.Case("f", 1, (nx, 1, 1), h, bc, bc, q, 1.4, 1.0, 0.5, recipe, "SSPRK3")
    spec = oracle_spec(case, recipe=recipe)
    want = from_oracle(spec, oracle.rhs(spec, SCHEME_OF[recipe[:5]], FLUX_OF["Rusanov"], to_oracle(spec, q)))
    rho, u, v, w, p = cases.primitive(q)
    fmax = (np.abs(q).max() + p.max()) * (np.abs(u) + np.sqrt(1.4 * p / rho)).max()
    s = case.solver()
    for variant in (0, 1):
        s.variant = variant
        err = np.abs(s.residual().reshape(q.shape) - want)[..., 1:-1, :]
        assert err.max() <= 2 * 1000 * EPS * fmax / h[0]


@pytest.mark.gpu
@pytest.mark.parametrize("dim,n", [(2, (40, 9, 1)), (2, (150, 37, 1)), (3, (33, 18, 40)), (3, (20, 70, 6)), (3, (70, 9, 33))])
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("recipe", ["weno3Roe", "weno5Rusanov", "weno7Rusanov"])
def test_sweep_segments(dim, n, bc, recipe, oracle):
    """The axis sweeps with every segment length the launch picks (2 to 16 nodes
    along y and z; ragged last segments, shorter axes than a segment) against
    the oracle's residual, FP64 1e-12 of the residual's scale."""
    from helpers import smooth_state
    q = smooth_state(dim, n, seed=5)
    h = (0.02, 0.03, 0.025)
    bcs = tuple(bc if d < dim else 0 for d in range(3))
    case = cases.Case("s", dim, n, h, bcs, bcs, q, 1.4, 1.0, 0.5, recipe, "SSPRK3")
    spec = oracle_spec(case, recipe=recipe)
    want = from_oracle(spec, oracle.rhs(spec, SCHEME_OF[recipe[:5]], FLUX_OF[recipe[5:]], to_oracle(spec, q)))
    s = case.solver()
    s.variant = 0
    got = s.residual().reshape(want.shape)
    inner = tuple(slice(1, -1) if bc == 0 and d < dim else slice(None) for d in (2, 1, 0))
    a, b = got[inner].reshape(-1, 5), want[inner].reshape(-1, 5)
    assert (np.abs(a - b).max(axis=0) / np.abs(b).max()).max() <= 1e-12
