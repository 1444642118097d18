"""2-D grids too small for the full-size tiles run one- and two-round tiles, large
ones 32 x 23 tiles."""
import numpy as np
import pytest

from sonicsolver_b200 import capi, cases


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [capi.PREC_FP64, capi.PREC_FP32_FLUX])
@pytest.mark.parametrize("recipe", ["weno3Rusanov", "weno5Roe", "teno5Rusanov", "weno7Rusanov"])
@pytest.mark.parametrize("n", [(9, 9), (16, 7), (17, 8), (33, 15), (34, 16), (255, 120), (320, 200), (640, 300), (863, 845), (1535, 1541)])
def test_small_tiles_give_the_bits_of_the_large(n, recipe, precision):
    """Grids on both sides of the tile-shape rule's lines, and of one tile's
    edge: one step of the solver (the shape the rule picks) against the batch,
    which always runs 32 x 15 tiles.  Transmissive ends on x, periodic on y."""
    rng = np.random.default_rng(n[0])
    nx, ny = n
    x, y = np.arange(nx) / nx, np.arange(ny) / ny
    X, Y = np.meshgrid(x, y, indexing="xy")
    rho = 1 + 0.2 * np.sin(2 * np.pi * (X + Y)) + 0.01 * rng.standard_normal((ny, nx))
    p = 1 + 0.1 * np.cos(2 * np.pi * Y) + 0.2 * (X > 0.5)
    q = cases.conserved(rho, 0.3 + 0.1 * Y, -0.2 + 0.1 * X, 0.05, p)[None]
    case = cases.Case("t", 2, (nx, ny, 1), (1 / nx, 1 / ny, 1.0), (0, 1, 0), (0, 1, 0), q, 1.4, 1.0, 0.4, recipe,
                      "SSPRK3")
    s = case.solver(precision=precision)
    s.advance(1e30, max_steps=2)
    b = capi.Batch((64 << 20) + 130 * nx * ny, 1, recipe=recipe, precision=precision, cfl=0.4)
    slot = b.add(case, t_end=1e30, max_steps=2)
    b.step(3)
    np.testing.assert_array_equal(s.download().reshape(q.shape), b.download(slot))
