"""The colour kernels that wait for vertices instead of at a barrier
(`csrc/local.cu`): against the serial method over the same tets in the order of
their colours, for meshes of fewer elements than a warp, of ragged colours, of
vertices without a tet, and for several passes and calls."""

import numpy as np
import pytest

from controllable_pbd_3d_gb300 import Deform3D, meshgen
from controllable_pbd_3d_gb300 import graph_coloring as gcol

EPS = float(np.finfo(np.float32).eps)


def body(dims, seed, extra=0):
  """(rest, start, inverse masses, tets), `extra` vertices without a tet."""
  if dims == 'tet':
    xr = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], np.float32)
    t = np.arange(4, dtype=np.int32)
  else:
    xr, t = meshgen.hex_grid_tets(*dims)
  rng = np.random.default_rng(seed)
  xr = np.concatenate([xr, rng.random((extra, 3))]).astype(np.float32)
  h = 1.0 if dims == 'tet' else 1.0 / max(dims)
  x = (xr + rng.uniform(-0.05 * h, 0.05 * h, xr.shape)).astype(np.float32)
  im = (0.5 + rng.random(len(xr))).astype(np.float32)
  im[rng.random(len(xr)) < 0.1] = 0.0
  return xr, x, im, np.asarray(t, np.int32).reshape(-1, 4)


MESHES = [('tet', 0), ((1, 1, 1), 3), ((2, 1, 3), 0), ((5, 4, 3), 7), ((11, 9, 10), 0), ((25, 3, 17), 1)]


@pytest.mark.gpu
@pytest.mark.parametrize('dims,extra', MESHES)
@pytest.mark.parametrize('calls', [(1,), (3,), (2, 1)])
def test_xpbd_passes(cuda, dims, extra, calls):
  xr, x0, im, t = body(dims, 5, extra)
  order = gcol.color_elements(t.reshape(-1), len(t), 4, len(xr)).ordered_indices
  vol = (0.5 + np.random.default_rng(1).random(len(t))).astype(np.float32)
  dev = lambda a: cuda.tensor(a, device='cuda')  # noqa: E731
  out = []
  for method, p in (('graph_coloring', np.arange(len(t))), ('gauss_seidel', order)):
    x = dev(x0)
    c = Deform3D(x, dev(xr), dev(im), dev(t[p].reshape(-1)), dev(vol[p]), 1.0 / 300,
                 hydro_alpha=1e-5, devia_alpha=1e-4, method=method)
    c.init_rest_status()
    c.preupdate_cons()
    for n in calls:
      c.update_cons(n)
    lam = np.empty((2, len(t)), np.float32)
    lam[:, p] = np.stack([c.hydro_lambda.cpu().numpy(), c.devia_lambda.cpu().numpy()])
    out.append((x.cpu().numpy(), lam))
  (xa, la), (xb, lb) = out
  # a vertex is rounded four times an update, at most 24 updates a pass here
  assert np.abs(xa - xb).max() <= 4 * 24 * sum(calls) * EPS * max(1.0, np.abs(x0).max())
  assert np.abs(la - lb).max() <= 1e-3 * max(np.abs(lb).max(), 1e-30)


@pytest.mark.gpu
def test_xpbd_tet_with_a_vertex_twice(cuda):
  """Such a tet has no rest shape; the others are updated as without it."""
  xr, x0, im, t = body((2, 2, 2), 3, extra=3)
  n = len(xr)
  bad = np.array([[n - 1, n - 2, n - 3, n - 1]], np.int32)
  dev = lambda a: cuda.tensor(a, device='cuda')  # noqa: E731
  out = []
  for tets in (t, np.concatenate([t, bad])):
    x = dev(x0)
    c = Deform3D(x, dev(xr), dev(im), dev(tets.reshape(-1)), dev(np.ones(len(tets), np.float32)),
                 1.0 / 300, hydro_alpha=1e-5, devia_alpha=1e-4, method='graph_coloring')
    c.init_rest_status()
    c.preupdate_cons()
    c.update_cons(2)
    out.append(x.cpu().numpy()[:n - 3])
  assert np.array_equal(out[0], out[1])


@pytest.mark.gpu
@pytest.mark.parametrize('dims,extra', MESHES)
@pytest.mark.parametrize('iterations,rho,damping', [(1, 0.0, 0.0), (4, 0.0, 0.1), (5, 0.7, 0.1)])
def test_vbd_iterations(cuda, dims, extra, iterations, rho, damping):
  """Against the serial method on the same mesh with its vertices numbered in
  the order of their colours (without Chebyshev the two then make the same
  updates; with it too, because it follows a whole iteration)."""
  from controllable_pbd_3d_gb300 import VBDSolver
  xr, x0, im, t = body(dims, 6, extra)
  order = gcol.color_vertices(t.reshape(-1), len(t), 4, len(xr)).ordered_indices
  new = np.empty_like(order)
  new[order] = np.arange(len(order))
  dev = lambda a: cuda.tensor(a, device='cuda')  # noqa: E731
  out = []
  for method, p, tets in (('color', np.arange(len(xr)), t), ('serial', order, new[t].astype(np.int32))):
    x = dev(x0[p])
    s = VBDSolver(x, dev(xr[p]), dev(im[p]), dev(tets.reshape(-1)), None, [0.0, -9.8, 0.0], 1.0 / 300,
                  n_iterations=iterations, rho=rho, damping=damping, method=method,
                  youngs_modulus=1e4, poissons_ratio=0.3)
    s.init()
    for k in range(2):
      s.step(k)
    s.synchronize()
    y = np.empty_like(x0)
    y[p] = x.cpu().numpy()
    out.append(y)
  # the sums of a vertex's <= 32 tets round differently in the two methods, by
  # 40 roundings of its step at most, and a step is at most 1 here
  assert np.abs(out[0] - out[1]).max() <= 40 * 2 * iterations * EPS * max(1.0, np.abs(x0).max())


@pytest.mark.gpu
def test_vbd_vertex_with_many_neighbours(cuda):
  """A fan of 60 tets about one edge: more neighbours than the waiting kernel
  keeps."""
  from controllable_pbd_3d_gb300 import VBDSolver
  n = 60
  a = 2 * np.pi * np.arange(n) / n
  xr = np.concatenate([[[0, 0, -0.5], [0, 0, 0.5]], np.stack([np.cos(a), np.sin(a), 0 * a], 1)]).astype(np.float32)
  t = np.array([[0, 1, 2 + k, 2 + (k + 1) % n] for k in range(n)], np.int32)
  x0 = (xr * 1.02).astype(np.float32)
  im = np.ones(n + 2, np.float32)
  order = gcol.color_vertices(t.reshape(-1), n, 4, n + 2).ordered_indices
  new = np.empty_like(order)
  new[order] = np.arange(n + 2)
  dev = lambda v: cuda.tensor(v, device='cuda')  # noqa: E731
  out = []
  for method, p, tets in (('color', np.arange(n + 2), t), ('serial', order, new[t].astype(np.int32))):
    x = dev(x0[p])
    s = VBDSolver(x, dev(xr[p]), dev(im[p]), dev(tets.reshape(-1)), None, [0.0, -9.8, 0.0], 1.0 / 300,
                  n_iterations=3, rho=0.0, damping=0.0, method=method, youngs_modulus=1e3,
                  poissons_ratio=0.3)
    s.init()
    s.step(0)
    s.synchronize()
    y = np.empty_like(x0)
    y[p] = x.cpu().numpy()
    out.append(y)
  assert np.isfinite(out[0]).all()
  assert np.abs(out[0] - out[1]).max() <= 80 * 3 * EPS * 1.1
