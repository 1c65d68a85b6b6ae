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


@pytest.mark.gpu
@pytest.mark.parametrize('mode', ['fast', 'parity'])
@pytest.mark.parametrize('n_smooth', [0, 1, 2, 3])
@pytest.mark.parametrize('kw', [{}, {'smoother': 'safe'}, {'use_graph': False}, {'cg_alias': True}])
def test_iterations_of_the_cg_around(cuda, mode, n_smooth, kw):
  """The CG iteration shares its vector update and dot product with the
  V-cycle's first and last sweep: the same iterates as a float64 CG around the
  library's own V-cycle, to the accuracy float32 vectors leave it."""
  if kw.get('cg_alias') and n_smooth == 0:
    pytest.skip('no smoothing and an overwritten residual do not converge')
  from controllable_pbd_3d_gb300 import MGPBDSolverGPU, meshgen
  xr, t = meshgen.hex_grid_tets(4, 5, 3)
  x0, _ = meshgen.hex_grid_tets(4, 5, 3, jitter=0.02, seed=3)
  invm = np.ones(len(xr), np.float32)
  s = MGPBDSolverGPU(cuda.tensor(x0, device='cuda'), cuda.tensor(xr, device='cuda'),
                     cuda.tensor(invm, device='cuda'), cuda.tensor(t, device='cuda'), None,
                     [0.0, -9.8, 0.0], 1.0 / 300, mu=1e5, mode=mode, n_smooth=n_smooth,
                     maxiter_cg=6, tol_cg=1e-30, **kw)
  s.init()
  s._compute_C_and_gradC()
  s._compute_rhs_gpu()
  s._fill_A_and_update_gpu()
  gm = s._gpu_solver
  its = gm.solve(s._b_gpu, s._dlam_gpu)
  assert 1 <= its <= 6
  if kw.get('cg_alias'):
    assert bool(cuda.isfinite(s._dlam_gpu).all())
    return
  L0 = gm._gpu_As[0]
  nt = s.n_tets
  A = sp.csr_matrix((L0.data.cpu().numpy()[:L0.nnz], L0.indices.cpu().numpy()[:L0.nnz],
                     L0.indptr.cpu().numpy()), shape=(nt, nt)).astype(np.float64)
  b = s._b_gpu.cpu().numpy().astype(np.float64)

  def m(r):
    return gm.vcycle_apply(cuda.tensor(r.astype(np.float32), device='cuda')).cpu().numpy().astype(np.float64)

  x, r = np.zeros(nt), b.copy()
  z = m(r)
  p, rz = z, r @ z
  for _ in range(its):
    q = A @ p
    a = rz / (p @ q)
    x, r = x + a * p, r - a * q
    z = m(r)
    rz, old = r @ z, rz
    p = z + rz / old * p
  # a few roundings of every vector an iteration, grown by CG's own
  # sensitivity: the square root of the condition number of M A, < 1e3 here
  got = s._dlam_gpu.cpu().numpy()
  assert np.abs(got - x).max() <= 1e3 * 8 * its * EPS * np.abs(x).max()
