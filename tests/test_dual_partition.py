"""The spatial partition of the persistent dual CG (`csrc/dcg.cu`,
`csrc/dcg_plan.cpp`): the operator it applies, on the CPU for every way a
mesh is cut, and the solves on the GPU, each against float64 arithmetic."""

import ctypes as C

import numpy as np
import pytest

from controllable_pbd_3d_gb300 import _native as N
from controllable_pbd_3d_gb300 import meshgen
from controllable_pbd_3d_gb300.edge_volume import edge_volume_system

SMEM = 231000
EPS = float(np.finfo(np.float32).eps)


def mesh(nx, ny, nz, edges):
  """(rest positions, constraints (nt, 4), first length constraint)."""
  xr, t = meshgen.hex_grid_tets(nx, ny, nz)
  if not edges:
    return xr, np.asarray(t, np.int32).reshape(-1, 4), len(t) // 4
  c, types, _, _ = edge_volume_system(t)
  return xr, np.asarray(c, np.int32).reshape(-1, 4), int((types != 1).sum())


def gradients(nt, n4, rng):
  """Random slot gradients: slot 0 minus the others of a 4-slot constraint,
  n, -n, 0, 0 of a length constraint."""
  g = rng.standard_normal((nt, 4, 3)).astype(np.float32)
  g[:n4, 0] = -g[:n4, 1] - g[:n4, 2] - g[:n4, 3]
  g[n4:, 1] = -g[n4:, 0]
  g[n4:, 2:] = 0
  return g


def apply64(c, n4, g, w, alpha, x):
  """(J W J^T + alpha~) x and sum of the terms' absolute values, float64.  A
  length constraint's slots 2 and 3 have no gradient."""
  g, x = g.astype(np.float64), x.astype(np.float64)
  u, ua = np.zeros((len(w), 3)), np.zeros((len(w), 3))
  for l in range(4):
    np.add.at(u, c[:, l], g[:, l] * x[:, None])
    np.add.at(ua, c[:, l], np.abs(g[:, l] * x[:, None]))
  u, ua = u * w[:, None], ua * w[:, None]
  y = sum((g[:, l] * u[c[:, l]]).sum(1) for l in range(4)) + alpha * x
  ya = sum((np.abs(g[:, l]) * ua[c[:, l]]).sum(1) for l in range(4)) + np.abs(alpha * x)
  return y, ya


def run_plan(xr, c, n4, prob, n_prob, n_blocks, cluster, threads, smem, g, w, alpha, x):
  y, info = np.full(len(c), np.nan), np.zeros(6, np.int32)
  rc = N.lib().mgpbd_host_partition_apply(
      c.ctypes.data, len(c), n4, len(xr), xr.ctypes.data, prob.ctypes.data if prob is not None else None,
      n_prob, n_blocks, int(cluster), threads, smem, g.ctypes.data, w.ctypes.data, alpha.ctypes.data,
      x.ctypes.data, y.ctypes.data, info.ctypes.data)
  return rc, y, info


@pytest.mark.parametrize('dims,edges', [((1, 1, 1), False), ((1, 1, 1), True), ((3, 2, 5), True),
                                        ((7, 9, 8), True), ((12, 11, 13), False)])
@pytest.mark.parametrize('n_blocks,cluster,threads', [(152, False, 512), (16, True, 512), (7, True, 128),
                                                      (1, True, 768), (13, False, 768)])
def test_plan_applies_the_operator(dims, edges, n_blocks, cluster, threads):
  rng = np.random.default_rng(7)
  xr, c, n4 = mesh(*dims, edges)
  g = gradients(len(c), n4, rng)
  w = (rng.random(len(xr)) > 0.2).astype(np.float32)
  alpha = rng.random(len(c)).astype(np.float32)
  x = rng.standard_normal(len(c)).astype(np.float32)
  rc, y, info = run_plan(xr, c, n4, None, 1, n_blocks, cluster, threads, SMEM, g, w, alpha, x)
  assert rc == 0
  ref, size = apply64(c, n4, g, w, alpha, x)
  assert np.all(np.abs(y - ref) <= 1e-13 * size + 1e-300)
  # equal shares: a block holds at most one constraint more than its share
  # of each of the cuts above it
  assert info[5] <= (4 * n4 + 2 * (len(c) - n4)) / n_blocks + 4 * 9


def test_plan_of_several_bodies_and_short_memory():
  """Bodies of uneven sizes, each cut on its own; less shared memory than the
  rows need; a constraint that lists a vertex twice; too little memory."""
  rng = np.random.default_rng(3)
  xs, cs, n4s, prob_t, prob_e = [], [], [], [], []
  off = 0
  for b, dims in enumerate([(2, 3, 2), (9, 6, 7), (1, 1, 1), (5, 5, 6)]):
    xr, c, n4 = mesh(*dims, True)
    xs.append(xr + np.float32(20 * b))
    cs.append((c[:n4] + off, c[n4:] + off))
    prob_t += [b] * n4
    prob_e += [b] * (len(c) - n4)
    off += len(xr)
  xr = np.ascontiguousarray(np.concatenate(xs))
  c = np.ascontiguousarray(np.concatenate([t for t, _ in cs] + [e for _, e in cs]).astype(np.int32))
  n4, prob = len(prob_t), np.array(prob_t + prob_e, np.int32)
  g = gradients(len(c), n4, rng)
  c[5, 2] = c[5, 1]  # a repeated slot carries no gradient
  g[5, 1] = g[5, 1] + g[5, 2]
  g[5, 2] = 0
  w = np.ones(len(xr), np.float32)
  alpha = rng.random(len(c)).astype(np.float32)
  x = rng.standard_normal(len(c)).astype(np.float32)
  ref, size = apply64(c, n4, g, w, alpha, x)
  for smem, fits, blocks in ((SMEM, True, 4), (SMEM, True, 0), (20000, True, 4), (3000, False, 4)):
    rc, y, info = run_plan(xr, c, n4, prob, 4, blocks, True, 256, smem, g, w, alpha, x)
    assert (rc == 0) == fits
    if not fits:
      assert rc == -6  # MGPBD_ERANGE
      continue
    assert np.all(np.abs(y - ref) <= 1e-13 * size + 1e-300)
    assert bool(info[0]) == (smem == SMEM)


# ---------------------------------------------------------------------------

def solver(torch, dims, edges, **kw):
  from controllable_pbd_3d_gb300 import MGPBDSolverGPU
  xr, t = meshgen.hex_grid_tets(*dims)
  x0, _ = meshgen.hex_grid_tets(*dims, jitter=0.03, seed=2)
  invm = np.ones(len(xr), np.float32)
  invm[meshgen.grid_face_vertices(*dims, axis=1, side='max')] = 0.0
  s = MGPBDSolverGPU(torch.tensor(x0, device='cuda'), torch.tensor(xr, device='cuda'),
                     torch.tensor(invm, device='cuda'), torch.tensor(t, device='cuda'), None,
                     [0.0, -9.8, 0.0], 1.0 / 300, compliance=1e-5, kinematic_pins=True,
                     constraints='edge_volume' if edges else 'arap',
                     **dict(dict(mode='fast', precond='cheb', cheb_lo=1e-3, cheb_scale='none',
                                 tol_cg=1e-12, rel_tol_cg=1e-6, maxiter_cg=4000), **kw))
  s.init()
  return s


def residual(s, n4):
  """|b - A x| / |b| in float64, and what float32 arithmetic may leave of it:
  the recurrence r -= alpha A p carries a few roundings of the terms of A x."""
  c = s.t_i.cpu().numpy().reshape(-1, 4)
  x = s._dlam_gpu.cpu().numpy()
  b = s._b_gpu.cpu().numpy().astype(np.float64)
  y, size = apply64(c, n4, s.gradC.cpu().numpy(), s.v_invm.cpu().numpy().astype(np.float64),
                    s.alpha_tilde.cpu().numpy().astype(np.float64), x)
  return np.linalg.norm(b - y) / np.linalg.norm(b), 16 * EPS * np.linalg.norm(size) / np.linalg.norm(b)


# a mesh of fewer constraints than blocks; the edges of the rule between a
# cluster and the grid (120,000 vertex entries); odd sizes; more constraints
# than the chip holds
SOLVES = [((1, 1, 1), False, {}), ((2, 1, 3), True, {}), ((13, 11, 12), True, {}),
          ((18, 18, 18), False, {}), ((18, 18, 19), False, {}), ((21, 9, 25), True, {}),
          ((46, 31, 40), True, {}),
          ((6, 7, 5), True, dict(cheb_scale='jacobi')), ((6, 7, 5), True, dict(cheb_degree=1)),
          ((19, 20, 18), True, dict(cheb_scale='jacobi', cheb_degree=2)),
          ((19, 20, 18), True, dict(cheb_degree=1))]


@pytest.mark.gpu
@pytest.mark.parametrize('dims,edges,kw', SOLVES)
@pytest.mark.parametrize('change', [None, 'alpha', 'gradient'])
def test_solve_residual(cuda, dims, edges, kw, change):
  """The solution's float64 residual.  change: compliances of the caller's own
  in the alpha~ view; gradients of the caller's own whose slot 0 is not minus
  the sum of the others."""
  torch = cuda
  if change is not None and dims[0] > 30:
    pytest.skip('one run of the largest mesh is enough')
  s = solver(torch, dims, edges, **kw)
  n4 = s.n_tets if s.constraint_types is None else int((s.constraint_types != 1).sum())
  s._compute_C_and_gradC()
  s._compute_rhs_gpu()
  if change == 'alpha':
    s.alpha_tilde.mul_(1.0 + torch.rand(s.n_tets, device='cuda', generator=torch.Generator('cuda').manual_seed(1)))
  if change == 'gradient':
    s.gradC[:n4, 0] *= 1.25
  s._fill_A_and_update_gpu()
  it = s._gpu_solver.solve(s._b_gpu, s._dlam_gpu)
  assert 1 <= it < 4000
  rel, floor = residual(s, n4)
  assert rel <= 1e-6 + floor, (rel, floor)


@pytest.mark.gpu
@pytest.mark.parametrize('dims,edges,kw', [((1, 1, 1), False, {}), ((6, 7, 5), True, dict(cheb_scale='jacobi')),
                                           ((19, 20, 18), False, {})])
def test_interval_of_one_fill(cuda, dims, edges, kw):
  """Only the first solve after a fill estimates the Chebyshev interval; the
  others of that fill use the same one: the same solution, bit for bit."""
  torch = cuda
  s = solver(torch, dims, edges, **kw)
  s._compute_C_and_gradC()
  s._compute_rhs_gpu()
  out = []
  for fill in (True, False, True):
    if fill:
      s._fill_A_and_update_gpu()
    its = s._gpu_solver.solve(s._b_gpu, s._dlam_gpu)
    out.append((its, s._dlam_gpu.cpu()))
  assert out[0][0] > 0
  for its, x in out[1:]:
    assert its == out[0][0] and torch.equal(x, out[0][1])
