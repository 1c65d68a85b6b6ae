"""The Chebyshev interval that `csrc/dcg.cu` estimates inside its kernel, where
the first Lanczos step leaves little: a soft body whose compliances make up the
spectrum, with a few constraints that stick out.  The interval has to reach them:
beyond its top the polynomial is indefinite and tells them apart a thousandfold,
so that CG needs an iteration or more for each."""

import numpy as np
import pytest

from test_dual_partition import residual, solver


@pytest.mark.gpu
@pytest.mark.parametrize('dims,edges,few,lo,hi', [((6, 7, 5), True, 1, 1e5, 1e5), ((6, 7, 5), True, 12, 1.02, 1.1),
                                                  ((19, 20, 18), False, 40, 1.02, 1.1),
                                                  ((30, 30, 30), False, 100, 1.02, 1.12),
                                                  ((30, 30, 30), False, 1, 2.0, 2.0)])
def test_few_constraints_stick_out(cuda, dims, edges, few, lo, hi):
  torch = cuda
  s = solver(torch, dims, edges)
  n4 = s.n_tets if s.constraint_types is None else int((s.constraint_types != 1).sum())
  s._compute_C_and_gradC()
  s._compute_rhs_gpu()
  g = s.gradC.cpu().numpy().astype(np.float64)
  rng = np.random.default_rng(7)
  alpha = np.full(s.n_tets, 1e4 * (g**2).sum(axis=(1, 2)).max())
  alpha[rng.choice(s.n_tets, few, replace=False)] *= np.linspace(lo, hi, few)
  s.alpha_tilde.copy_(torch.tensor(alpha.astype(np.float32)))
  s._fill_A_and_update_gpu()
  s._b_gpu.copy_(torch.tensor(rng.standard_normal(s.n_tets).astype(np.float32)))
  it = s._gpu_solver.solve(s._b_gpu, s._dlam_gpu)
  rel, floor = residual(s, n4)
  print('its', it, rel, floor)
  assert rel <= 1e-6 + floor
  # inside the interval [1e-3, 1] the polynomial of degree 8 leaves at most
  # 1 / T_8(1.002) = 0.885: a condition number of 16.4, 0.6 an iteration, 29
  # iterations to 1e-6
  assert 1 <= it <= 29
