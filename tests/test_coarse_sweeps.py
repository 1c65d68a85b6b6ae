"""The coarsest level's Jacobi sweeps on a cluster (`csrc/sweep.cu`) against
float64 sweeps: fewer rows than blocks, ragged last groups, rows without a
neighbour, long rows (eight lanes), matrices beyond the cluster's shared memory
(launches of their own), with and without the transfers around them."""

import numpy as np
import pytest
import scipy.sparse as sp

from controllable_pbd_3d_gb300.mgpcg_gpu import GPUMultigridSolver

EPS = float(np.finfo(np.float32).eps)
W = 2.0 / 3.0


def matrix(n, per_row, seed):
  """Symmetric, diagonally dominant; row lengths vary, some rows stand alone."""
  rng = np.random.default_rng(seed)
  m = n * per_row // 2
  i, j = rng.integers(0, n, m), rng.integers(0, n, m)
  keep = (i != j) & (i % 7 != 3) & (j % 7 != 3)
  i, j, v = i[keep], j[keep], -rng.random(int(keep.sum()))
  B = sp.csr_matrix((np.r_[v, v], (np.r_[i, j], np.r_[j, i])), shape=(n, n))
  B.sum_duplicates()
  d = -np.asarray(B.sum(axis=1)).ravel() + 0.1 + rng.random(n)
  A = (B + sp.diags(d)).tocsr().astype(np.float32)
  A.sort_indices()
  return A


class Sweeps:
  """Float64 sweeps and, beside them, what float32 arithmetic may be off by:
  each sweep adds (row length + 4) roundings of the sizes of its terms and
  carries the error so far through |I - w D^-1 A|, whose row sums are <= 1
  here."""

  def __init__(self):
    self.err = 0.0

  def __call__(self, A, b, x, k):
    A = A.astype(np.float64)
    dinv = 1.0 / A.diagonal()
    absA, longest = abs(A), int(np.diff(A.indptr).max())
    for _ in range(k):
      size = np.abs(x) + W * dinv * (np.abs(b) + absA @ np.abs(x))
      self.err += (longest + 4) * EPS * size.max()
      x = x + W * dinv * (b - A @ x)
    return x


@pytest.mark.gpu
@pytest.mark.parametrize('n,per_row', [(1, 1), (9, 3), (127, 5), (130, 120), (1000, 60), (3001, 30),
                                       (6000, 27), (26001, 6), (40000, 5), (70001, 3)])
def test_one_level(cuda, n, per_row):
  A = matrix(n, per_row, n)
  m = GPUMultigridSolver().setup(A, [])
  b = np.random.default_rng(1).standard_normal(n).astype(np.float32)
  s = Sweeps()
  ref = s(A, b.astype(np.float64), np.zeros(n), min(50, n))
  got = [m.vcycle_apply(cuda.tensor(b, device='cuda')).cpu().numpy() for _ in range(2)]
  assert np.array_equal(got[0], got[1])
  assert np.abs(got[0] - ref).max() <= s.err


@pytest.mark.gpu
@pytest.mark.parametrize('n,nc,per_row', [(60, 5, 6), (4000, 401, 12), (50000, 6001, 8)])
def test_two_levels(cuda, n, nc, per_row):
  A = matrix(n, per_row, n)
  rng = np.random.default_rng(2)
  agg = np.r_[np.arange(nc), rng.integers(0, nc, n - nc)]
  P = sp.csr_matrix((np.ones(n, np.float32), agg, np.arange(n + 1)), shape=(n, nc))
  m = GPUMultigridSolver().setup(A, [P])
  b = rng.standard_normal(n).astype(np.float32)
  Ac = sp.csr_matrix((m._gpu_As[1].data.cpu().numpy()[:m._gpu_As[1].nnz],
                      m._gpu_As[1].indices.cpu().numpy()[:m._gpu_As[1].nnz],
                      m._gpu_As[1].indptr.cpu().numpy()), shape=(nc, nc))
  s, c = Sweeps(), Sweeps()
  b64, P64 = b.astype(np.float64), P.astype(np.float64)
  x = s(A, b64, np.zeros(n), 2)
  r = b64 - A.astype(np.float64) @ x
  members = int(np.bincount(agg).max())
  e = c(Ac, P64.T @ r, np.zeros(nc), min(50, nc))
  # the coarse right-hand side is off by the fine residual's error, and a
  # sweep passes that on times w / diagonal
  size = np.abs(b64) + abs(A).astype(np.float64) @ np.abs(x)
  rc = (float(abs(A).sum(axis=1).max()) * s.err + int(np.diff(A.indptr).max() + 4) * EPS * size.max())
  rc = members * rc + members * EPS * (P64.T @ np.abs(r)).max()
  c.err += min(50, nc) * W * float((1.0 / Ac.diagonal()).max()) * rc
  x = x + P64 @ e
  s.err += c.err + EPS * np.abs(x).max()
  ref = s(A, b64, x, 2)
  got = m.vcycle_apply(cuda.tensor(b, device='cuda')).cpu().numpy()
  assert np.abs(got - ref).max() <= s.err
