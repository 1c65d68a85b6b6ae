"""The CG's stopping tests are made by every block of the kernel that follows
(`csrc/kernels.cu`), while block 0 already leaves `done`: the threads of a block
that starts late must still agree.  When p.Ap breaks down the solve ends with x
as it was, whole: nothing of the step may be added by some warps."""

import numpy as np
import pytest
import scipy.sparse as sp


def laplacian(n):
  """A 1D chain, more rows than the blocks of one launch take at once."""
  e = np.ones(n, np.float32)
  A = sp.diags([-e[1:], 3 * e, -e[1:]], [-1, 0, 1]).tocsr().astype(np.float32)
  A.sort_indices()
  return A


@pytest.mark.gpu
@pytest.mark.parametrize('size', [1e-22, 1e-19])
def test_breakdown_leaves_x(cuda, size):
  """p.Ap below 1e-30: about n size^2 / 5."""
  from controllable_pbd_3d_gb300.mgpcg_gpu import GPUMultigridSolver
  n = 600000
  m = GPUMultigridSolver().setup(laplacian(n), [])
  b = cuda.tensor(np.where(np.arange(n) % 2 == 0, size, -size).astype(np.float32), device='cuda')
  x = cuda.full((n,), 7.0, device='cuda')
  for _ in range(100):
    m.solve(b, x)
    assert int(cuda.count_nonzero(x)) == 0


@pytest.mark.gpu
@pytest.mark.parametrize('n', [233472, 240007, 330001])
def test_dot_products_of_many_rows(cuda, n):
  """From three rounds of rows on the lanes of the dot operators take turns (3
  rounds of 1,216 blocks x 64 rows: 233,472): the iterates of a float64 CG around
  the library's own V-cycle, to the accuracy float32 vectors leave it."""
  from controllable_pbd_3d_gb300.mgpcg_gpu import GPUMultigridSolver
  from test_coarse_sweeps import EPS, matrix
  A = matrix(n, 6, n)
  agg = np.arange(n) // 20
  P = sp.csr_matrix((np.ones(n, np.float32), agg, np.arange(n + 1)), shape=(n, int(agg[-1]) + 1))
  g = GPUMultigridSolver(maxiter_cg=5, tol_cg=1e-30).setup(A, [P])
  b = np.random.default_rng(4).standard_normal(n).astype(np.float32)
  x = cuda.zeros(n, device='cuda')
  its = g.solve(cuda.tensor(b, device='cuda'), x)
  assert 1 <= its <= 5

  def m(r):
    return g.vcycle_apply(cuda.tensor(r.astype(np.float32), device='cuda')).cpu().numpy().astype(np.float64)

  A = A.astype(np.float64)
  y, r = np.zeros(n), b.astype(np.float64)
  z = m(r)
  p, rz = z, r @ z
  for _ in range(its):
    q = A @ p
    a = rz / (p @ q)
    y, r = y + a * p, r - a * q
    z = m(r)
    rz, old = r @ z, rz
    p = z + rz / old * p
  assert np.abs(x.cpu().numpy() - y).max() <= 1e3 * 8 * its * EPS * np.abs(y).max()
