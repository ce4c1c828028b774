"""The EMG solver's passes at the sizes where their partition changes: the persistent conjugate gradients (768 nodes per
block) and the stencil passes that march along z (tiles of columns, chunks of planes), by the residual of their solution
under the assembled stencil."""
import numpy as np
import pytest

from opendihu_b200 import emg as E
from opendihu_b200 import workloads as WL

pytestmark = pytest.mark.gpu


def _apply(stencil, shape, x):
    """The 27-point stencil [27, N] on x; q = (dx + 1) + 3 (dy + 1) + 9 (dz + 1)."""
    nx, ny, nz = shape
    c = stencil.reshape(27, nz, ny, nx)
    p = np.pad(x.reshape(nz, ny, nx), 1)
    y = np.zeros((nz, ny, nx))
    for q in range(27):
        dx, dy, dz = q % 3, (q // 3) % 3, q // 9
        y += c[q] * p[dz:dz + nz, dy:dy + ny, dx:dx + nx]
    return y.reshape(-1)


def _solver(shape, preconditioner, rtol):
    _, _, kw = WL.emg_box(n_fibers_x=1, n_fibers_y=1, n_nodes=101, mesh_nodes=shape, width=1.0)
    rng = np.random.default_rng(4)
    pos = kw["node_positions"]
    h = np.array([1.0, 1.0, 1.0]) / (np.array(shape) - 1)
    pos += 0.1 * h * rng.uniform(-1.0, 1.0, pos.shape)      # no two elements alike
    d = np.zeros((len(pos), 3))
    d[:, 2] = 1.0
    tight = {"relativeTolerance": rtol, "absoluteTolerance": 1e-30, "maxIterations": 5000}
    return E.StaticBidomainSolver(shape, pos, kw["sigma_i"], kw["sigma_e"], direction=d, emg_solver=tight,
                                  initial_guess_nonzero=False, preconditioner=preconditioner)


# 8 and 767 to 769 nodes: one block, full, one more; 3 x 256; the largest mesh of the persistent form and the first
# beyond it are around 113,664 nodes on 148 SMs; the march along z from 1,200,000 nodes
@pytest.mark.parametrize("shape", [(2, 2, 2), (13, 59, 2), (8, 8, 12), (769, 2, 2), (16, 16, 3), (37, 61, 50),
                                   (37, 64, 48), (37, 64, 49), (110, 101, 109)])
@pytest.mark.parametrize("concurrent", [False, True])
def test_jacobi_residual(shape, concurrent):
    if concurrent and np.prod(shape) > 113664:
        pytest.skip("takes a launch per pass either way")
    with _solver(shape, "jacobi", 1e-10) as s:
        s.set_concurrent(concurrent)     # beside other work: a launch per pass
        vm = np.random.default_rng(1).uniform(-80.0, 40.0, s.n_nodes)
        s.set_vm(vm)
        s.advanceTimeSpan()
        phi, ki, k = s.phi_e(), s.stencil(0), s.stencil(1)
    rhs = -_apply(ki, shape, vm)
    rhs -= rhs.mean()
    # the recurrence's residual is within 1e-10 |rhs|; the true one differs from it by rounding only, some
    # iterations times 1e-16 |K| |phi|
    assert np.linalg.norm(_apply(k, shape, phi) - rhs) < 1e-9 * np.linalg.norm(rhs)
    assert abs(phi.mean()) < 1e-12 * np.abs(phi).max()


# tiles that do and do not divide the grid, a single tile, more tiles than planes, a thin grid
# (here the march along z takes grids from 600,000 nodes, the last six)
@pytest.mark.parametrize("shape", [(101, 37, 29), (16, 18, 360), (2, 300, 190), (101, 97, 65), (65, 97, 97),
                                   (16, 18, 2100), (550, 560, 2), (2, 500, 610), (1100, 3, 190)])
def test_multigrid_residual(shape):
    with _solver(shape, "multigrid", 1e-8) as s:
        vm = np.random.default_rng(1).uniform(-80.0, 40.0, s.n_nodes)
        s.set_vm(vm)
        its = s.advanceTimeSpan()
        phi, ki, k = s.phi_e(), s.stencil(0), s.stencil(1)
    rhs = -_apply(ki, shape, vm)
    rhs -= rhs.mean()
    assert its < 5000
    assert np.linalg.norm(_apply(k, shape, phi) - rhs) < 2e-8 * np.linalg.norm(rhs)
