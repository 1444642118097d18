"""The CFL minimum with its FP32 bound skips no node that counts: dt equals the
operation-by-operation FP64 maximum over all nodes to the bit, in the separate
pass (sfg_compute_dt) and in the reduction fused into a step's last stage, for
smooth and spiky fields, states far outside FP32 range, and near-vacuum nodes.
Grids of SCREEN_NODES solved nodes on take the bound; a smaller one of each
kind does not."""
import numpy as np
import pytest

from sonicsolver_b200 import capi, cases

SCREEN_NODES = 400_000  # sfg_internal.h

def _dt(q, n, h, dim, gamma, cfl):
    """RusanovEOS::deltaT in numpy, every operation rounded to FP64."""
    rho = q[..., 0]
    u = [q[..., 1 + d] / rho for d in range(3)]
    kin = (0.5 * rho) * ((u[0] * u[0] + u[1] * u[1]) + u[2] * u[2])
    e = (q[..., 4] - kin) / rho
    c = np.sqrt((gamma * (((gamma - 1.0) * rho) * e)) / rho)
    jac = 1.0 / ((h[0] * h[1]) * h[2])
    m = [(h[1] * h[2]) * jac, (h[0] * h[2]) * jac, (h[0] * h[1]) * jac]
    sr = np.abs(u[0] * m[0]) + c * m[0]
    for d in range(1, dim):
        sr = sr + (np.abs(u[d] * m[d]) + c * m[d])
    return cfl / sr.max()


def _field(kind, dim, n, seed):
    rng = np.random.default_rng(seed)
    shape = tuple(reversed(n))
    rho = 1 + 0.3 * rng.random(shape)
    u, v, w = (0.4 * rng.standard_normal(shape) if d < dim else np.zeros(shape) for d in range(3))
    p = 1 + 0.2 * rng.random(shape)
    if kind == "ties":      # many nodes within an ulp of the largest rate
        rho, p, u, v, w = np.ones(shape), np.ones(shape), np.full(shape, 0.3), np.full(shape, 0.1 * (dim > 1)), 0.0 * p
        u = u * (1 + 2.0 ** -52 * rng.integers(0, 3, shape))
    elif kind == "mild":    # rough, but a few steps stay valid
        rho, p = 1 + 0.04 * rng.random(shape), 1 + 0.04 * rng.random(shape)
        u, v, w = 0.1 * u, 0.1 * v, 0.1 * w
    elif kind == "vacuum":  # nodes with next to no pressure, fast ones among them
        p = np.where(rng.random(shape) < 0.3, 1e-9, p)
        u = np.where(rng.random(shape) < 0.05, 5.0, u)
    q = cases.conserved(rho, u, v, w, p)
    if kind == "subnormal":  # energies that FP32 holds to a bit or two, at densities it holds
        q = np.zeros(shape + (5,))
        q[..., 0], q[..., 4] = 1e-36, 1.4e-45 * (1 + 0.4 * rng.random(shape))
    elif kind == "heavy":  # sound speeds below FP32 range beside resting nodes
        q[..., 0], q[..., 1:4] = 1e36 * rho, 0.0
        q[..., 4] = 1e-9 * p
    scale = {"huge": 1e45, "tiny": 1e-45}.get(kind, 1.0)
    return np.ascontiguousarray(q * scale)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["random", "ties", "vacuum", "huge", "tiny", "subnormal", "heavy"])
@pytest.mark.parametrize("dim,n", [(1, (5000, 1, 1)), (1, (450001, 1, 1)), (2, (301, 203, 1)), (2, (1100, 900, 1)),
                                   (3, (130, 61, 47)), (3, (130, 71, 53))])
def test_compute_dt_is_the_exact_minimum(kind, dim, n):
    h = (0.013, 0.017 if dim > 1 else 1.0, 0.011 if dim > 2 else 1.0)
    bc = tuple(1 if d < dim else 0 for d in range(3))
    q = _field(kind, dim, n, dim)
    s = capi.Solver(dim, n, h, bc, bc, recipe="weno3Rusanov", cfl=0.45)
    s.upload(q)
    assert s.compute_dt() == _dt(q, n, h, dim, 1.4, 0.45)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [capi.PREC_FP64, capi.PREC_FP32_FLUX])
@pytest.mark.parametrize("dim,n,variant", [(1, (400003, 1, 1), 1), (2, (700, 620, 1), 1), (2, (700, 620, 1), 0),
                                           (3, (90, 71, 67), 0), (3, (90, 71, 67), 1)])
def test_fused_minimum_is_exact(dim, n, variant, precision):
    """Every dt of a run against the state it was taken from."""
    assert np.prod(n) >= SCREEN_NODES
    h = (0.013, 0.017 if dim > 1 else 1.0, 0.011 if dim > 2 else 1.0)
    bc = tuple(1 if d < dim else 0 for d in range(3))
    q = _field("mild", dim, n, 7 + dim)
    s = capi.Solver(dim, n, h, bc, bc, recipe="weno5Rusanov", precision=precision, cfl=0.2)
    s.variant = variant
    s.upload(q)
    _, dts = s.advance(1e30, max_steps=4, dt_capacity=4)
    for k in range(4):
        s.upload(q)
        if k:
            s.advance(1e30, max_steps=k)
        assert dts[k] == _dt(s.download().reshape(q.shape), n, h, dim, 1.4, 0.2), k


@pytest.mark.gpu
def test_fused_minimum_of_a_batched_grid_is_exact():
    n, h = (700, 620, 1), (0.013, 0.017, 1.0)
    q = _field("mild", 2, n, 9)
    case = cases.Case("b", 2, n, h, (1, 1, 0), (1, 1, 0), q, 1.4, 1e30, 0.2, "weno5Rusanov", "SSPRK3")
    s = case.solver()
    _, dts = s.advance(1e30, max_steps=4, dt_capacity=4)
    b = capi.Batch(200 * q.size + (8 << 20), 1, recipe="weno5Rusanov", cfl=0.2)
    slot = b.add(case, t_end=1e30, max_steps=4)
    b.step(5)
    assert b.status(slot)["time"] == sum(float(d) for d in dts)


@pytest.mark.gpu
@pytest.mark.parametrize("dim,n", [(2, (100, 90, 1)), (2, (1100, 900, 1)), (3, (130, 71, 53))])
def test_infinite_density_opens_no_step(dim, n):
    """The rate of a node of infinite density is 0: the run stops before its
    first step, wherever the node lies."""
    h = (0.013, 0.017, 0.011 if dim > 2 else 1.0)
    bc = tuple(1 if d < dim else 0 for d in range(3))
    q = _field("random", dim, n, 3)
    q.reshape(-1, 5)[-7, 0] = np.inf
    s = capi.Solver(dim, n, h, bc, bc, recipe="weno5Rusanov", cfl=0.45)
    s.upload(q)
    with pytest.raises(capi.SolverError) as e:
        s.advance(1e30, max_steps=3)
    assert e.value.code == capi.ERR_STATE and s.time() == (0.0, 0)
    np.testing.assert_array_equal(s.download(), q.ravel())
