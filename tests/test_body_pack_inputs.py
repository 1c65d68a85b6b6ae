"""Packed bodies: compliances that say nothing about stiffness, and direct solves
beside the captured substep."""

import numpy as np
import pytest

from controllable_pbd_3d_gb300.batch import BodyBatch, random_bodies

G, DT = [0.0, -9.8, 0.0], 1.0 / 300
KW = dict(mode='fast', precond='cheb', cheb_scale='none', cheb_lo=1e-3, primal=False, rel_tol_cg=1e-6,
          tol_cg=1e-14, maxiter_cg=3000, maxiter=3, atol=1e-9, rtol=1e-9, kinematic_pins=True,
          constraints='edge_volume')


@pytest.mark.gpu
@pytest.mark.parametrize('compliance', [0.0, -1e-9, 1e39])
def test_any_compliance_is_taken(cuda, compliance):
  """Of a body but the first (which selects the model)."""
  bodies = random_bodies(3, seed=5, dims=(3, 5), compliance=(1e-6, 1e-5))
  bodies[1].compliance = compliance
  with np.errstate(over='ignore'):
    b = BodyBatch(bodies, G, DT, **KW)
    b.init()
  if compliance < 1.0:  # (1e39 is not a float32)
    b.step(0)
    assert bool(cuda.isfinite(b.x).all())


@pytest.mark.gpu
def test_direct_solves_between_substeps(cuda):
  """A solve of the whole pack after a substep that ran from its graph: the
  interval has to be that of all bodies, also of the one a hundred times
  lighter than the first."""
  from test_dual_partition import residual
  torch = cuda
  bodies = random_bodies(2, seed=6, dims=(5, 7), compliance=(1.0, 1.0))
  bodies[1].invm = bodies[1].invm * np.float32(100.0)
  b = BodyBatch(bodies, G, DT, **KW)
  b.init()
  s = b.solver
  n4 = int((s.constraint_types != 1).sum())
  for i in range(3):
    b.step(i)
    s._b_gpu.copy_(torch.randn(s.n_tets, device='cuda', generator=torch.Generator('cuda').manual_seed(i)))
    its = s._gpu_solver.solve(s._b_gpu, s._dlam_gpu)
    rel, floor = residual(s, n4)
    print('its', i, its, rel, floor)
    assert its < 3000
    assert rel <= 1e-6 + floor
