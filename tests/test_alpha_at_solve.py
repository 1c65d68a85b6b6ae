"""The compliances that count in a dual solve are those of the alpha~ view when it
runs: changed after the fill, by a factor of each constraint's own and by one for
all, with and without a start from an earlier solution."""

import numpy as np
import pytest

from test_dual_partition import residual, solver


@pytest.mark.gpu
@pytest.mark.parametrize('dims,edges,kw', [((2, 1, 3), True, {}), ((6, 7, 5), True, {}),
                                           ((6, 7, 5), True, dict(cheb_scale='jacobi')),
                                           ((6, 7, 5), True, dict(primal=True, primal_tol=1e-2)),
                                           ((19, 20, 18), False, {}), ((6, 7, 5), False, dict(persistent=2))])
def test_alpha_changed_after_the_fill(cuda, dims, edges, kw):
  torch = cuda
  s = solver(torch, dims, edges, **kw)
  n4 = s.n_tets if s.constraint_types is None else int((s.constraint_types != 1).sum())
  s._compute_C_and_gradC()
  s._compute_rhs_gpu()
  s._fill_A_and_update_gpu()
  gen = torch.Generator('cuda').manual_seed(1)
  for change in (1.0 + torch.rand(s.n_tets, device='cuda', generator=gen), 0.5,
                 0.75 + 0.25 * torch.rand(s.n_tets, device='cuda', generator=gen)):
    s.alpha_tilde.mul_(change)
    it = s._gpu_solver.solve(s._b_gpu, s._dlam_gpu)
    assert 1 <= it < 4000
    rel, floor = residual(s, n4)
    assert rel <= 1e-6 + floor, (rel, floor)
