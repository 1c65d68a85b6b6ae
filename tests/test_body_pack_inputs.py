"""Packed bodies whose compliances say nothing about stiffness."""

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
