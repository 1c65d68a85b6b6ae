"""Batches of the coarse network's weights loss (`csrc/mpnn.cu`): eight samples
are taken at once, so the batch's loss and gradient are compared with the means
over its samples taken one by one, at row counts around the tiles."""

import numpy as np
import pytest
import scipy.sparse as sp

EPS = float(np.finfo(np.float32).eps)


@pytest.mark.gpu
@pytest.mark.parametrize('n', [1, 15, 64, 65, 257, 3001])
@pytest.mark.parametrize('batch', [1, 7, 8, 9, 17])
def test_batch_is_the_mean_of_its_samples(cuda, n, batch):
  from controllable_pbd_3d_gb300 import CoarseGraph, CoarseNet
  rng = np.random.default_rng(n)
  m = 4 * n
  i, j = rng.integers(0, n, m), rng.integers(0, n, m)
  v = -rng.random(m) * (i != j)
  B = sp.csr_matrix((np.r_[v, v], (np.r_[i, j], np.r_[j, i])), shape=(n, n))
  A = (B + sp.diags(-np.asarray(B.sum(axis=1)).ravel() + 0.5)).tocsr().astype(np.float32)
  A.sum_duplicates()
  A.sort_indices()
  g = CoarseGraph.from_scipy(A)
  net = CoarseNet(seed=1)
  r = cuda.tensor(rng.standard_normal((batch, n)).astype(np.float32), device='cuda')
  loss = net.loss_grad(g, r)
  grad = net.grad.cpu().numpy().astype(np.float64)
  one = [(net.loss_grad(g, r[k:k + 1]), net.grad.cpu().numpy().astype(np.float64)) for k in range(batch)]
  # a sum over rows and samples behind two layers of 128 products: its terms'
  # roundings, against the largest gradient of a sample; the terms may be 8
  # times the sum
  big = max(np.abs(q).max() for _, q in one)
  assert np.abs(grad - np.mean([q for _, q in one], axis=0)).max() <= 8 * (n + 256 + batch) * EPS * big
  assert abs(loss - np.mean([l for l, _ in one])) <= 64 * EPS * max(abs(l) for l, _ in one)
