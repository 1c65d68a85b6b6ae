"""Waits of the colour kernels that run out (`csrc/local.cu`), with a limit of 0: a
warp gives up at the first poll that finds a vertex missing (or, for a tet that
lists a vertex twice and a vertex of many neighbours, at the first barrier that is
not complete), all warps end, the next call reports it once, and the handle works
again."""

import ctypes as C

import numpy as np
import pytest

from controllable_pbd_3d_gb300 import Deform3D, VBDSolver, meshgen
from controllable_pbd_3d_gb300 import _native as N


def fan(n):
  """n tets around the edge (0, 1): both have n + 1 neighbours."""
  a = 2 * np.pi * np.arange(n) / n
  x = np.concatenate([[[0, 0, -0.5], [0, 0, 0.5]], np.stack([np.cos(a), np.sin(a), 0 * a], 1)])
  t = np.stack([np.zeros(n), np.ones(n), 2 + np.arange(n), 2 + (np.arange(n) + 1) % n], 1)
  return x.astype(np.float32), t.astype(np.int32).reshape(-1)


def test_limits_are_validated():
  L = N.lib()
  for create, params, kind in ((L.mgpbd_xpbd_create, N.XpbdParams(), 'xpbd'), (L.mgpbd_vbd_create, N.VbdParams(), 'vbd')):
    params.dt = 1.0 / 300
    h = C.c_void_p()
    N.check(create(C.byref(params), C.byref(h)), kind)
    limit = getattr(L, f'mgpbd_{kind}_set_barrier_limit')
    try:
      assert [limit(h, s) for s in (-1.0, 0.0, 61.0, 4.0)] == [-1, 0, -1, 0]
      assert limit(None, 4.0) == -1
    finally:
      getattr(L, f'mgpbd_{kind}_destroy')(h)


@pytest.mark.gpu
@pytest.mark.parametrize('twice', [False, True])
def test_xpbd(cuda, twice):
  xr, t = meshgen.hex_grid_tets(9, 8, 10)
  if twice:
    t = np.concatenate([t, [0, 1, 2, 0]])
  x0 = (xr + np.random.default_rng(0).uniform(-0.005, 0.005, xr.shape)).astype(np.float32)
  dev = lambda a: cuda.tensor(a, device='cuda')  # noqa: E731

  def solver():
    x = dev(x0)
    c = Deform3D(x, dev(xr.astype(np.float32)), cuda.ones(len(xr), device='cuda'), dev(t.astype(np.int32)),
                 cuda.ones(len(t) // 4, device='cuda'), 1.0 / 300, method='graph_coloring')
    c.init_rest_status()
    c.preupdate_cons()
    return c, x

  (c, x), (ref, xr_) = solver(), solver()
  limit = N.lib().mgpbd_xpbd_set_barrier_limit
  assert limit(c._h, 0.0) == 0
  c.update_cons(3)
  with pytest.raises(N.MGPBDError, match='timed out'):
    c.synchronize()
  assert limit(c._h, 4.0) == 0
  x.copy_(dev(x0))
  c.preupdate_cons()
  c.update_cons(3)
  c.synchronize()
  ref.update_cons(3)
  ref.synchronize()
  if not twice:
    assert bool(cuda.isfinite(x).all())
  assert cuda.equal(x.view(cuda.int32), xr_.view(cuda.int32))


@pytest.mark.gpu
@pytest.mark.parametrize('many', [False, True])
@pytest.mark.parametrize('rho', [0.0, 0.9])
def test_vbd(cuda, many, rho):
  if many:
    xr, t = fan(60)
    xr = np.concatenate([xr + np.float32([4.0 * k, 0, 0]) for k in range(40)])
    t = np.concatenate([t + 62 * k for k in range(40)]).astype(np.int32)
  else:
    xr, t = meshgen.hex_grid_tets(9, 8, 10)
  xr = xr.astype(np.float32)
  x0 = (xr + np.random.default_rng(0).uniform(-0.005, 0.005, xr.shape)).astype(np.float32)
  dev = lambda a: cuda.tensor(a, device='cuda')  # noqa: E731

  def solver():
    x = dev(x0)
    s = VBDSolver(x, dev(xr), cuda.ones(len(xr), device='cuda'), dev(np.asarray(t, np.int32)), None,
                  [0.0, -9.8, 0.0], 1.0 / 300, n_iterations=5, rho=rho, method='color')
    s.init()
    s.make_prediction()
    return s, x

  (s, x), (ref, x_ref) = solver(), solver()
  limit = N.lib().mgpbd_vbd_set_barrier_limit
  before = x.clone()
  assert limit(s._h, 0.0) == 0
  s.solve()
  with pytest.raises(N.MGPBDError, match='timed out'):
    s.synchronize()
  assert limit(s._h, 4.0) == 0
  x.copy_(before)
  s.solve()
  s.synchronize()
  ref.solve()
  ref.synchronize()
  assert bool(cuda.isfinite(x).all())
  assert cuda.equal(x, x_ref)
