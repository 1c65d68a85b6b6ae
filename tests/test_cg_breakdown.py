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
