"""Batches of the coarse network's weights loss beyond the samples whose norms are
made at once, and beyond a grid's second axis (`csrc/mpnn.cu`)."""

import numpy as np
import pytest
import scipy.sparse as sp

EPS = float(np.finfo(np.float32).eps)


def graph(n, rng):
  from controllable_pbd_3d_gb300 import CoarseGraph
  m = 4 * n
  i, j = rng.integers(0, n, m), rng.integers(0, n, m)
  v = -rng.random(m) * (i != j)
  B = sp.csr_matrix((np.r_[v, v], (np.r_[i, j], np.r_[j, i])), shape=(n, n))
  A = (B + sp.diags(-np.asarray(B.sum(axis=1)).ravel() + 0.5)).tocsr().astype(np.float32)
  A.sum_duplicates()
  A.sort_indices()
  return CoarseGraph.from_scipy(A)


@pytest.mark.gpu
@pytest.mark.parametrize('n', [3, 300])
@pytest.mark.parametrize('times', [37, 9363])  # 259 and 65,541 samples
def test_large_batches(cuda, n, times):
  """Seven samples over and over: the loss and gradient of the seven."""
  from controllable_pbd_3d_gb300 import CoarseNet
  rng = np.random.default_rng(n)
  g = graph(n, rng)
  net = CoarseNet(seed=1)
  r = cuda.tensor(rng.standard_normal((7, n)).astype(np.float32), device='cuda')
  want = net.loss_grad(g, r), net.grad.cpu().numpy().astype(np.float64)
  loss = net.loss_grad(g, r.repeat(times, 1))
  grad = net.grad.cpu().numpy().astype(np.float64)
  # the samples' terms are added to a row one after the other, each no larger than
  # 1 / batch of 8 times the gradient: half a unit of the sum for each
  assert np.abs(grad - want[1]).max() <= 8 * (n + 256 + 7 * times / 2) * EPS * np.abs(want[1]).max()
  assert abs(loss - want[0]) <= 64 * EPS * abs(want[0])
