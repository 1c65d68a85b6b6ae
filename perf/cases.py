"""The work that users of this package have it do, as cases that can be timed.

A case is a dict of plain values; `kind` says which entry points it goes
through:

  step   one or more `MGPBDSolverGPU.step()` substeps of one body
  batch  one `BodyBatch.step()` substep of several packed bodies
  pcg    `GPUMultigridSolver` on a caller's matrix: new values, one V-cycle,
         one PCG solve
  net    the coarse network: weights of a graph, loss and gradient
  vbd    one `VBDSolver.step()`
  xpbd   one `PbdFramework.step()` over `Deform3D`

Every pass starts from the same positions and velocities (copied into the
solver's tensors), so a pass does the same work each time.  Bodies are hex
grids of 5 tets per hex, jittered, the top face pinned, with a smooth random
velocity field, so that a substep meets a moving body and not one at rest.
"""

import functools
import math

import numpy as np
import torch

import controllable_pbd_3d_gb300 as pkg
from controllable_pbd_3d_gb300 import meshgen
from controllable_pbd_3d_gb300.mgpcg_gpu import GPUMultigridSolver

DT = 1.0 / 300.0  # 60 frames a second, 5 substeps
GRAVITY = [0.0, -9.8, 0.0]
DEV = 'cuda'

# The solver settings in use.  fast: the benchmark's step, without the start
# from the last substep's solution (each pass begins anew).  amg: the
# reference's V-cycle PCG in captured graphs.  default: what a caller of the
# reference's constructor gets.
_TO_1E6 = dict(damp=1.0, maxiter=20, atol=1e-4, rtol=1e-2, maxiter_cg=6000, tol_cg=1e-12,
               rel_tol_cg=1e-6, n_smooth=2, kinematic_pins=True)
SOLVERS = {
    'fast': dict(_TO_1E6, mode='fast', precond='cheb', cheb_degree=8, cheb_lo=1e-3,
                 cheb_scale='none'),
    'amg': dict(_TO_1E6, mode='fast', smoother='safe', precond='vcycle'),
    'default': dict(damp=0.993),
}


def _step(name, nx, ny, nz, cons, solver, substeps=1, compliance=0.0, mu=0.0):
  return {'name': name, 'kind': 'step', 'nx': nx, 'ny': ny, 'nz': nz, 'constraints': cons,
          'solver': solver, 'substeps': substeps, 'compliance': compliance, 'mu': mu}


def listed():
  return [
      # the small benchmark body (5,000 tets), a whole frame of 5 substeps:
      # an interactive scene, where launches and grid barriers count
      _step('fast_cube10_frame', 10, 10, 10, 'edge_volume', 'fast', 5, compliance=1e-6),
      # a middling body of odd sizes with the reference's ARAP constraints at
      # its default stiffness: short solves, so what surrounds them counts too
      _step('fast_arap_23x17x29', 23, 17, 29, 'arap', 'fast', mu=1e6),
      # the headline benchmark body (320,000 tets, 718,520 constraints)
      _step('fast_cube40', 40, 40, 40, 'edge_volume', 'fast', compliance=1.53e-6),
      # a large slab, as in the stiff-drag scenario: its operator is larger
      # than the chip's memories
      _step('fast_slab80x20x80', 80, 20, 80, 'edge_volume', 'fast', compliance=1.53e-6),
      # a call with the reference's own defaults: host-checked loops
      _step('default_arap_11x9x10', 11, 9, 10, 'arap', 'default', mu=3e4),
      # the plain multigrid PCG that the fast step is measured against
      _step('amg_cube14', 14, 14, 14, 'edge_volume', 'amg', compliance=1.53e-6),
      # independent bodies of uneven sizes, one captured graph per substep
      {'name': 'batch_16', 'kind': 'batch', 'bodies': 16, 'lo': 6, 'hi': 18},
      # PCG on the caller's own matrix (ragged grid, 27-point stencil)
      {'name': 'pcg_37x29x41', 'kind': 'pcg', 'nx': 37, 'ny': 29, 'nz': 41},
      # one training step's forward and backward on an aggregate graph
      {'name': 'net_24x25x23', 'kind': 'net', 'nx': 24, 'ny': 25, 'nz': 23, 'samples': 8},
      # the comparison solvers of the convergence experiment
      {'name': 'vbd_cube24', 'kind': 'vbd', 'nx': 24, 'ny': 24, 'nz': 24, 'iterations': 10,
       'rho': 0.0},
      {'name': 'xpbd_cube24', 'kind': 'xpbd', 'nx': 24, 'ny': 24, 'nz': 24, 'passes': 10},
  ]


def _log_int(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi):
  """Three sides near a common size that is log-uniform in [lo, hi]."""
  n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
  return [max(3, int(round(n * rng.uniform(0.75, 1.25)))) for _ in range(3)]


def draw(rng):
  kind = rng.choice(['fast', 'fast', 'fast', 'fast', 'default', 'amg', 'batch', 'pcg', 'net',
                     'vbd', 'xpbd'])
  if kind == 'fast':
    cons = rng.choice(['edge_volume', 'edge_volume', 'arap'])
    nx, ny, nz = _dims(rng, 6, 40)
    c = {'nx': nx, 'ny': ny, 'nz': nz, 'constraints': cons,
         'substeps': 5 if nx * ny * nz < 2500 else 1, 'compliance': 0.0, 'mu': 0.0}
    if cons == 'arap':
      c['mu'] = 10.0 ** rng.uniform(4.5, 6.0)
    else:
      c['compliance'] = 10.0 ** rng.uniform(-6.3, -4.5)
    return dict(c, kind='step', solver='fast')
  if kind == 'default':
    nx, ny, nz = _dims(rng, 5, 11)
    return {'kind': 'step', 'nx': nx, 'ny': ny, 'nz': nz, 'constraints': 'arap',
            'solver': 'default', 'substeps': 1, 'compliance': 0.0,
            'mu': 10.0 ** rng.uniform(4.0, 4.7)}
  if kind == 'amg':
    nx, ny, nz = _dims(rng, 6, 14)
    return {'kind': 'step', 'nx': nx, 'ny': ny, 'nz': nz, 'constraints': 'edge_volume',
            'solver': 'amg', 'substeps': 1, 'compliance': 10.0 ** rng.uniform(-6.0, -5.0),
            'mu': 0.0}
  if kind == 'batch':
    lo = rng.randint(4, 8)
    return {'kind': 'batch', 'bodies': _log_int(rng, 3, 24), 'lo': lo,
            'hi': lo + rng.randint(2, 9)}
  if kind == 'pcg':
    nx, ny, nz = _dims(rng, 8, 44)
    return {'kind': 'pcg', 'nx': nx, 'ny': ny, 'nz': nz}
  if kind == 'net':
    nx, ny, nz = _dims(rng, 6, 36)
    return {'kind': 'net', 'nx': nx, 'ny': ny, 'nz': nz, 'samples': rng.randint(1, 16)}
  nx, ny, nz = _dims(rng, 5, 32)
  if kind == 'vbd':
    return {'kind': 'vbd', 'nx': nx, 'ny': ny, 'nz': nz, 'iterations': rng.randint(4, 20),
            'rho': rng.choice([0.0, 0.7])}
  return {'kind': 'xpbd', 'nx': nx, 'ny': ny, 'nz': nz, 'passes': rng.randint(4, 20)}


# ---- inputs ---------------------------------------------------------------

@functools.lru_cache(maxsize=8)
def _grid(nx, ny, nz):
  """The rest grid, its tets and inverse masses (the same for every seed)."""
  xr, t = meshgen.hex_grid_tets(nx, ny, nz)
  invm = np.ones(len(xr), np.float32)
  invm[meshgen.grid_face_vertices(nx, ny, nz, axis=1, side='max')] = 0.0
  return xr, t, invm


def _body(c, seed, jitter=0.01):
  """Rest positions, start positions, velocities (float32, host), tets,
  inverse masses."""
  nx, ny, nz = c['nx'], c['ny'], c['nz']
  xr, t, invm = _grid(nx, ny, nz)
  rng = np.random.default_rng(seed)
  h = 1.0 / max(nx, ny, nz)
  x = (xr + rng.uniform(-jitter * h, jitter * h, xr.shape)).astype(np.float32)
  # a smooth velocity field of up to ~0.3 a second, zero at the pinned face
  k = rng.uniform(1.0, 4.0, (3, 3))
  ph = rng.uniform(0.0, 2.0 * math.pi, (3, 3))
  v = np.stack([sum(np.sin(k[a, b] * xr[:, b] + ph[a, b]) for b in range(3)) for a in range(3)],
               axis=1) * 0.1
  top = xr[:, 1].max()
  v = (v * (top - xr[:, 1:2])).astype(np.float32)
  v[invm == 0] = 0.0
  return xr, x, v, t, invm


def _cuda(a):
  return torch.tensor(a, device=DEV)


def _lumped(xr, t):
  """Tet volumes and lumped vertex masses, as tet meshes are loaded."""
  q = t.reshape(-1, 4)
  p = xr.astype(np.float64)[q]
  vol = np.abs(np.einsum('ij,ij->i', np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]),
                         p[:, 3] - p[:, 0])) / 6.0
  m = np.bincount(q.reshape(-1), weights=np.repeat(vol / 4.0, 4), minlength=len(xr))
  return vol.astype(np.float32), (1.0 / m).astype(np.float32)


@functools.lru_cache(maxsize=8)
def _stencil(nx, ny, nz):
  """The 27-point pattern of a grid: rows, columns (sorted by row), and the
  id of each undirected edge that a nonzero belongs to (-1: diagonal)."""
  n = nx * ny * nz
  i = torch.arange(n)
  ix, iy, iz = i % nx, (i // nx) % ny, i // (nx * ny)
  rows, cols = [], []
  for dz in (-1, 0, 1):
    for dy in (-1, 0, 1):
      for dx in (-1, 0, 1):
        jx, jy, jz = ix + dx, iy + dy, iz + dz
        ok = (jx >= 0) & (jx < nx) & (jy >= 0) & (jy < ny) & (jz >= 0) & (jz < nz)
        rows.append(i[ok])
        cols.append((jx + nx * (jy + ny * jz))[ok])
  r, c = torch.cat(rows), torch.cat(cols)
  order = torch.argsort(r * n + c)
  r, c = r[order], c[order]
  _, eid = torch.unique(torch.minimum(r, c) * n + torch.maximum(r, c), return_inverse=True)
  return r, c, eid


def _matrix(c, seed):
  """A symmetric positive definite matrix on the stencil: minus random edge
  weights, a diagonal just above the row sums.  (indptr, columns, float32
  values) on the host."""
  r, col, eid = _stencil(c['nx'], c['ny'], c['nz'])
  n = c['nx'] * c['ny'] * c['nz']
  g = torch.Generator().manual_seed(seed)
  w = -(0.1 + torch.rand(int(eid.max()) + 1, generator=g, dtype=torch.float64))[eid]
  diag = r == col
  w[diag] = 0.0
  s = torch.zeros(n, dtype=torch.float64).index_add_(0, r, -w)
  shift = 1e-3 + 1e-2 * torch.rand(n, generator=g, dtype=torch.float64)
  w[diag] = s * (1.0 + shift)
  ip = torch.zeros(n + 1, dtype=torch.int64)
  ip[1:] = torch.cumsum(torch.bincount(r, minlength=n), 0)
  return ip, r, col, w.float()


def _blocks(c):
  """Aggregates of 2 x 2 x 2 grid points: the coarse row of every row."""
  nx, ny, nz = c['nx'], c['ny'], c['nz']
  i = torch.arange(nx * ny * nz)
  bx, by = (nx + 1) // 2, (ny + 1) // 2
  return (i % nx) // 2 + bx * (((i // nx) % ny) // 2 + by * (i // (nx * ny) // 2))


class _Csr:
  """A CSR matrix with what `GPUMultigridSolver.setup` reads of scipy's."""

  def __init__(self, indptr, indices, data, shape):
    self.indptr, self.indices, self.data, self.shape = indptr, indices, data, shape

  def tocsr(self):
    return self

  def sum_duplicates(self):
    pass


def prepare(case, seed):
  return _PREPARE[case['kind']](case, seed)


def _prepare_step(c, seed):
  xr, x0, v0, t, invm = _body(c, seed)
  x = _cuda(x0)
  more = {'compliance': c['compliance']} if c['compliance'] > 0 else {'mu': c['mu']}
  s = pkg.MGPBDSolverGPU(x, _cuda(xr), _cuda(invm), _cuda(t), None, GRAVITY, DT,
                         constraints=c['constraints'], **more, **SOLVERS[c['solver']])
  s.init()
  return {'kind': 'step', 'solver': s, 'x0': _cuda(x0), 'v0': _cuda(v0),
          'substeps': c['substeps']}


def _prepare_batch(c, seed):
  # the sizes are the case's, the positions and compliances the seed's
  size = np.random.default_rng([c['bodies'], c['lo'], c['hi']])
  rng = np.random.default_rng(seed)
  bodies, shift, h = [], 0.0, 1.0 / 40
  for _ in range(c['bodies']):
    nx, ny, nz = (int(v) for v in size.integers(c['lo'], c['hi'] + 1, size=3))
    xr, t = meshgen.hex_grid_tets(nx, ny, nz, h=h, origin=(shift, 0.0, 0.0))
    invm = np.ones(len(xr), np.float32)
    invm[meshgen.grid_face_vertices(nx, ny, nz, axis=1, side='max')] = 0.0
    x0 = (xr + rng.uniform(-0.01 * h, 0.01 * h, xr.shape)).astype(np.float32)
    bodies.append(pkg.Body(xr, x0, invm, t, float(10.0 ** rng.uniform(-7.0, -5.0))))
    shift += nx * h + 0.5
  b = pkg.BodyBatch(bodies, GRAVITY, DT, constraints='edge_volume', **SOLVERS['fast'])
  b.init()
  return {'kind': 'batch', 'solver': b.solver, 'batch': b, 'x0': b.x.clone(),
          'v0': torch.zeros_like(b.x)}


def _prepare_pcg(c, seed):
  ip, _, col, val = _matrix(c, seed)
  agg = _blocks(c).numpy()
  n, nc = len(agg), int(agg.max()) + 1
  A = _Csr(ip.numpy(), col.numpy(), val.numpy(), (n, n))
  P = _Csr(np.arange(n + 1), agg, np.ones(n, np.float32), (n, nc))
  m = GPUMultigridSolver(maxiter_cg=400, tol_cg=1e-4)
  m.setup(A, [P])
  g = torch.Generator().manual_seed(seed + 1)
  b = torch.randn(n, generator=g)
  return {'kind': 'pcg', 'solver': m, 'values': _cuda(val.numpy()), 'b': b.to(DEV),
          'x': torch.zeros(n, device=DEV)}


def _prepare_net(c, seed):
  ip, r, col, val = _matrix(c, seed)
  d = torch.empty(len(ip) - 1)
  d[r[r == col]] = val[r == col]
  graph = pkg.CoarseGraph(ip.int().to(DEV), col.int().to(DEV), val.to(DEV), (1.0 / d).to(DEV))
  net = pkg.CoarseNet(seed=0)
  net.load_params(_net_params(seed))
  g = torch.Generator().manual_seed(seed + 1)
  res = torch.randn((c['samples'], len(d)), generator=g)
  return {'kind': 'net', 'net': net, 'graph': graph, 'residuals': res.to(DEV)}


def _net_params(seed):
  """Glorot-uniform weights, small biases, in the library's order."""
  rng = np.random.default_rng(seed)
  f = 64
  u = lambda k, m: rng.uniform(-1, 1, k) * math.sqrt(6.0 / m)  # noqa: E731
  return np.concatenate([u(f, 2 + f), u(f, 2 + f), u(f, 600), u(2 * f * f, 3 * f), u(f, 600),
                         u(2 * f * f, 3 * f), u(f, 600), u(f, 1 + f), u(1, 600)]).astype(np.float32)


def _local_body(c, seed):
  xr, x0, v0, t, invm = _body(c, seed, jitter=0.05)
  vol, im = _lumped(xr, t)
  im[invm == 0] = 0.0
  return xr, x0, v0, t, im, vol


VBD = dict(youngs_modulus=1e4, poissons_ratio=0.3, damping=0.05)
XPBD = dict(hydro_alpha=1e-5, devia_alpha=1e-4)


def _prepare_vbd(c, seed):
  xr, x0, v0, t, im, _ = _local_body(c, seed)
  x = _cuda(x0)
  s = pkg.VBDSolver(x, _cuda(xr), _cuda(im), _cuda(t), None, GRAVITY, DT, damp=0.993,
                    n_iterations=c['iterations'], rho=c['rho'], method='color', **VBD)
  s.init()
  return {'kind': 'vbd', 'solver': s, 'x0': _cuda(x0), 'v0': _cuda(v0)}


def _prepare_xpbd(c, seed):
  xr, x0, v0, t, im, vol = _local_body(c, seed)
  x = _cuda(x0)
  cons = pkg.Deform3D(x, _cuda(xr), _cuda(im), _cuda(t), _cuda(vol), DT, method='graph_coloring',
                      **XPBD)
  f = pkg.PbdFramework(x, GRAVITY, DT, 0.993)
  f.add_cons(cons, 0)
  f.init_rest_status(0)
  return {'kind': 'xpbd', 'framework': f, 'cons': cons, 'x0': _cuda(x0), 'v0': _cuda(v0),
          'passes': c['passes']}


_PREPARE = {'step': _prepare_step, 'batch': _prepare_batch, 'pcg': _prepare_pcg,
            'net': _prepare_net, 'vbd': _prepare_vbd, 'xpbd': _prepare_xpbd}


# ---- one pass -------------------------------------------------------------

def run(s):
  k = s['kind']
  if k in ('step', 'batch'):
    # positions: a substep's result.  (Velocities are the positions'
    # difference over dt: one float32 unit of a position is 2e-5 of them.)
    sv = s['solver']
    sv.v_p.copy_(s['x0'])
    sv.v_v.copy_(s['v0'])
    if k == 'batch':
      s['batch'].step(0)
    else:
      for i in range(s['substeps']):
        sv.step(i)
    return {'x': sv.v_p}
  if k == 'pcg':
    # what each Newton iteration asks of the solver
    m = s['solver']
    m.update_fine_matrix_data(s['values'])
    z = m.vcycle_apply(s['b'])
    m.solve(s['b'], s['x'])
    return {'z': z, 'x': s['x']}
  if k == 'net':
    net = s['net']
    loss = net.loss_grad(s['graph'], s['residuals'])
    # (the gradient is a view of memory that goes with the network: a copy)
    return {'loss': loss, 'grad': net.grad.clone(), 'weights': net.weights(s['graph'])}
  if k == 'vbd':
    sv = s['solver']
    sv.v_p.copy_(s['x0'])
    sv.v_v.copy_(s['v0'])
    sv.step(0)
    return {'x': sv.v_p, 'v': sv.v_v.clone()}
  f = s['framework']
  f.v_p.copy_(s['x0'])
  f.v_v.copy_(s['v0'])
  f.step(s['passes'])
  return {'x': f.v_p, 'v': f.v_v, 'hydro': s['cons'].hydro_lambda.clone(),
          'devia': s['cons'].devia_lambda.clone()}


# ---- what a pass cannot do without ----------------------------------------

def _counts(nx, ny, nz):
  """Vertices, tets and unique edges of the hex grid (axis edges, one
  diagonal per hex face)."""
  nv = (nx + 1) * (ny + 1) * (nz + 1)
  axis = nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
  face = nx * ny * (nz + 1) + nx * (ny + 1) * nz + (nx + 1) * ny * nz
  return nv, 5 * nx * ny * nz, axis + face


def work(c):
  """Each input read once, each output written once; the operations of one
  application of the operator (the iterations are the algorithm's)."""
  k = c['kind']
  if k in ('step', 'vbd', 'xpbd', 'batch'):
    if k == 'batch':
      size = np.random.default_rng([c['bodies'], c['lo'], c['hi']])
      dims = [[int(v) for v in size.integers(c['lo'], c['hi'] + 1, size=3)]
              for _ in range(c['bodies'])]
    else:
      dims = [[c['nx'], c['ny'], c['nz']]]
    nv, nt, ne = (sum(v) for v in zip(*(_counts(*d) for d in dims)))
    if k in ('vbd', 'xpbd'):
      # positions, velocities in and out; masses; tets, rest matrices,
      # volumes or masses; xpbd: both multipliers out
      return {'bytes': 52 * nv + (56 if k == 'vbd' else 64) * nt,
              'flops': 300 * nt * c.get('iterations', c.get('passes', 1))}
    ev = k == 'batch' or c['constraints'] == 'edge_volume'
    # positions and velocities in and out, masses, tets, rest matrices,
    # compliances; edges with their rest lengths
    return {'bytes': 52 * nv + 56 * nt + (16 * ne if ev else 0),
            'flops': c.get('substeps', 1) * (48 * nt + (20 * ne if ev else 0))}
  n = c['nx'] * c['ny'] * c['nz']
  nnz = 1
  for m in (c['nx'], c['ny'], c['nz']):
    nnz *= 3 * m - 2
  if k == 'pcg':
    return {'bytes': 8 * nnz + 16 * n, 'flops': 8 * nnz}
  s = c['samples']
  # two dense layers forward and backward, the graph products between them
  return {'bytes': 8 * nnz + 4 * n * (s + 2) + 2 * 4 * 16769,
          'flops': 3 * 2 * n * 2 * 128 * 64 + 4 * 2 * 64 * nnz + 2 * s * nnz}


# ---- the same in 64 bits ---------------------------------------------------

def exact(case, seed):
  k = case['kind']
  if k == 'step':
    return _exact_step(case, seed)
  if k == 'batch':
    return None  # dense factors of every body's every Newton system
  return {'pcg': _exact_pcg, 'net': _exact_net, 'vbd': _exact_vbd, 'xpbd': _exact_xpbd}[k](case, seed)


def _edges(q):
  e = np.concatenate([q[:, [a, b]] for a, b in
                      ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))]).astype(np.int64)
  e.sort(axis=1)
  return np.unique(e, axis=0)


def _exact_step(c, seed):
  """The Newton loop with dense solves in vertex space:
  (M + J^T alpha~^-1 J) dx = J^T alpha~^-1 b on the free vertices.  alpha~ is
  compliance / dt^2, or 1 / (mu dt^2 volume)."""
  nv = _counts(c['nx'], c['ny'], c['nz'])[0]
  if c['solver'] == 'default' or 3 * nv > 9000:
    return None  # its CG is cut off at 100 iterations; or too large
  xr, x0, v0, t, invm = _body(c, seed)
  f64 = lambda a: torch.tensor(a, dtype=torch.float64, device=DEV)  # noqa: E731
  q = torch.tensor(t.reshape(-1, 4).astype(np.int64), device=DEV)
  xr, x, v = f64(xr), f64(x0), f64(v0)
  free = torch.tensor(invm > 0, device=DEV)
  dt = float(np.float32(DT))
  g = torch.tensor([float(np.float32(a)) for a in GRAVITY], dtype=torch.float64, device=DEV)
  ds = lambda p: torch.stack([p[q[:, k]] - p[q[:, 0]] for k in (1, 2, 3)], dim=2)  # noqa: E731
  B = torch.linalg.inv(ds(xr))
  ev = c['constraints'] == 'edge_volume'
  nt, n3 = len(q), 3 * nv
  m = nt
  if ev:
    e = torch.tensor(_edges(t.reshape(-1, 4)), device=DEV)
    rest = (xr[e[:, 0]] - xr[e[:, 1]]).norm(dim=1)
    m += len(e)
  if c['compliance'] > 0:
    alpha = torch.full((m,), c['compliance'] / (dt * dt), dtype=torch.float64, device=DEV)
  else:
    alpha = 1.0 / (c['mu'] * dt * dt * torch.linalg.det(ds(xr)).abs() / 6.0)

  def cons(p):
    """Constraint values and gradients: tets (n, 4, 3), edges (m, 3)."""
    F = ds(p) @ B
    if ev:
      f = [F[:, :, k] for k in range(3)]
      P = torch.stack([torch.linalg.cross(f[1], f[2]), torch.linalg.cross(f[2], f[0]),
                       torch.linalg.cross(f[0], f[1])], dim=2)
      C = (f[0] * P[:, :, 0]).sum(1) - 1.0
    else:
      U, S, Vh = torch.linalg.svd(F)
      C = ((S - 1.0) ** 2).sum(1).sqrt()
      P = U @ torch.diag_embed((S - 1.0) / C.clamp(min=1e-300)[:, None]) @ Vh
      P[C <= 1e-6] = 0.0
    G = (P @ B.transpose(1, 2)).transpose(1, 2)
    G = torch.cat([-G.sum(1, keepdim=True), G], dim=1)
    if not ev:
      return C, G, None
    d = p[e[:, 0]] - p[e[:, 1]]
    ln = d.norm(dim=1)
    return torch.cat([C, ln - rest]), G, d / ln[:, None]

  k3 = torch.arange(3, device=DEV)
  dof = (3 * q[:, :, None] + k3).reshape(nt, 12)
  if ev:
    edof = (3 * e[:, :, None] + k3).reshape(-1, 6)
  keep = free.repeat_interleave(3)
  for _ in range(c['substeps']):
    old = x
    v = torch.where(free[:, None], v + dt * g, v)
    x = torch.where(free[:, None], x + dt * v, x)
    lam = torch.zeros(m, dtype=torch.float64, device=DEV)
    r0 = None
    for ite in range(20):
      C, G, N = cons(x)
      b = -(C + alpha * lam)
      r = float(b.norm())
      r0 = r if ite == 0 else r0
      if r < 1e-4 or (r0 > 1e-12 and r < 1e-2 * r0):
        break
      K = torch.zeros(n3 * n3, dtype=torch.float64, device=DEV)
      rhs = torch.zeros(n3, dtype=torch.float64, device=DEV)

      def add(rows, J, bb, al):
        K.index_add_(0, (rows[:, :, None] * n3 + rows[:, None, :]).reshape(-1),
                     (J[:, :, None] * J[:, None, :] / al[:, None, None]).reshape(-1))
        rhs.index_add_(0, rows.reshape(-1), (J * (bb / al)[:, None]).reshape(-1))

      add(dof, G.reshape(nt, 12), b[:nt], alpha[:nt])
      if ev:
        add(edof, torch.cat([N, -N], dim=1), b[nt:], alpha[nt:])
      K = K.view(n3, n3)[keep][:, keep] + torch.eye(int(keep.sum()), dtype=torch.float64, device=DEV)
      y = torch.zeros(n3, dtype=torch.float64, device=DEV)
      y[keep] = torch.cholesky_solve(rhs[keep][:, None], torch.linalg.cholesky(K))[:, 0]
      dx = y.view(nv, 3)
      Jy = (G * dx[q]).sum((1, 2))
      if ev:
        Jy = torch.cat([Jy, (N * (dx[e[:, 0]] - dx[e[:, 1]])).sum(1)])
      lam = lam + (b - Jy) / alpha
      cur = float((C + alpha * lam).norm())
      om = 1.0
      for _ in range(10):
        if float((cons(x + om * dx)[0] + alpha * lam).norm()) < cur:
          break
        om *= 0.5
      x = x + om * dx
    v = (x - old) / dt
  return {'x': x}


def _exact_pcg(c, seed):
  ip, r, col, val = _matrix(c, seed)
  n = len(ip) - 1
  A = torch.sparse_coo_tensor(torch.stack([r, col]), val.double(), (n, n)).coalesce().to(DEV)
  agg = _blocks(c)
  P = torch.sparse_coo_tensor(torch.stack([torch.arange(n), agg]),
                              torch.ones(n, dtype=torch.float64)).coalesce().to(DEV)
  Ac = torch.sparse.mm(torch.sparse.mm(P.t(), A), P).coalesce()
  nc = Ac.shape[0]
  diag = lambda M: torch.zeros(M.shape[0], dtype=torch.float64, device=DEV).index_add_(  # noqa: E731
      0, M.indices()[0], torch.where(M.indices()[0] == M.indices()[1], M.values(), 0.0))
  D, Dc = diag(A), diag(Ac)
  mv = lambda M, y: torch.mv(M, y)  # noqa: E731
  w = float(np.float32(2.0 / 3.0))

  def vcycle(b):
    y = torch.zeros_like(b)
    for _ in range(2):
      y = y + w * (b - mv(A, y)) / D
    rc = mv(P.t(), b - mv(A, y))
    yc = torch.zeros_like(rc)
    for _ in range(min(50, nc)):
      yc = yc + w * (rc - mv(Ac, yc)) / Dc
    y = y + mv(P, yc)
    for _ in range(2):
      y = y + w * (b - mv(A, y)) / D
    return y

  g = torch.Generator().manual_seed(seed + 1)
  b = torch.randn(n, generator=g).double().to(DEV)
  # the solution itself: the float32 solve stops short of it by its tolerance
  x, res = torch.zeros_like(b), b.clone()
  z = vcycle(res)
  p, rz = z, res @ z
  for _ in range(200):
    Ap = mv(A, p)
    a = rz / (p @ Ap)
    x, res = x + a * p, res - a * Ap
    if float(res.norm()) < 1e-12 * float(b.norm()):
      break
    z = vcycle(res)
    new = res @ z
    p, rz = z + (new / rz) * p, new
  return {'z': vcycle(b), 'x': x}


def _exact_net(c, seed):
  ip, r, col, val = _matrix(c, seed)
  n = len(ip) - 1
  f = 64
  d = torch.empty(n, dtype=torch.float64)
  d[r[r == col]] = val[r == col].double()
  s = (1.0 / d).sqrt()
  vals = (val.double() * s[r] * s[col]).to(DEV)
  Ah = torch.sparse_coo_tensor(torch.stack([r, col]).to(DEV), vals, (n, n)).coalesce()
  s = s.to(DEV)
  R = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, r.to(DEV), vals.abs())
  a1 = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, r.to(DEV), vals)
  p = torch.tensor(_net_params(seed), dtype=torch.float64, device=DEV, requires_grad=True)
  w1s, w1n, b1, W2, b2, W3, b3, wo, bo = torch.split(
      p, [f, f, f, 2 * f * f, f, 2 * f * f, f, f, 1])
  H = torch.relu(w1s + a1[:, None] * w1n + b1)
  H = torch.relu(torch.cat([H, torch.sparse.mm(Ah, H)], 1) @ W2.view(2 * f, f) + b2)
  H = torch.relu(torch.cat([H, torch.sparse.mm(Ah, H)], 1) @ W3.view(2 * f, f) + b3)
  w = 1.9 / R * torch.sigmoid(H @ wo + bo)
  g = torch.Generator().manual_seed(seed + 1)
  res = torch.randn((c['samples'], n), generator=g).double().to(DEV)
  u = res * s
  u = u / u.square().mean(1, keepdim=True).sqrt()
  v = w * u
  loss = ((0.5 * v * torch.sparse.mm(Ah, v.t()).t() - v * u).sum(1) / n).mean()
  loss.backward()
  return {'loss': float(loss.detach()), 'grad': p.grad, 'weights': w.detach()}


def _groups(colors):
  colors = np.asarray(colors)
  return [torch.tensor(np.flatnonzero(colors == k), device=DEV) for k in range(colors.max() + 1)]


def _low_zero(mask):
  return (~mask & (mask + 1)).bit_length() - 1


def _rest64(xr, q):
  """Rest matrices (columns p_k - p_3, k = 0..2) inverted, and volumes."""
  D = torch.stack([xr[q[:, k]] - xr[q[:, 3]] for k in range(3)], dim=2)
  return torch.linalg.inv(D), torch.linalg.det(D).abs() / 6.0


def _f_cof(x, q, B):
  F = torch.stack([x[q[:, k]] - x[q[:, 3]] for k in range(3)], dim=2) @ B
  f = [F[:, :, k] for k in range(3)]
  cof = torch.stack([torch.linalg.cross(f[1], f[2]), torch.linalg.cross(f[2], f[0]),
                     torch.linalg.cross(f[0], f[1])], dim=2)
  return F, cof, (f[0] * cof[:, :, 0]).sum(1)


def _exact_vbd(c, seed):
  xr, x0, v0, t, im, _ = _local_body(c, seed)
  qn = t.reshape(-1, 4)
  nv = len(xr)
  # greedy colours in index order: a vertex avoids those of its neighbours
  nb = np.unique(np.concatenate([qn[:, [a, b]] for a in range(4) for b in range(4) if b < a]
                                + [qn[:, [b, a]] for a in range(4) for b in range(4) if b < a]), axis=0)
  nb = nb[nb[:, 1] < nb[:, 0]]
  first = np.searchsorted(nb[:, 0], np.arange(nv + 1)).tolist()
  other, colors = nb[:, 1].tolist(), [0] * nv
  for i in range(nv):
    m = 0
    for j in range(first[i], first[i + 1]):
      m |= 1 << colors[other[j]]
    colors[i] = _low_zero(m)
  f64 = lambda a: torch.tensor(a, dtype=torch.float64, device=DEV)  # noqa: E731
  q = torch.tensor(qn.astype(np.int64), device=DEV)
  x, v, w = f64(x0), f64(v0), f64(im)
  B, vol = _rest64(f64(xr), q)
  E, nu = VBD['youngs_modulus'], VBD['poissons_ratio']
  mu, lam = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
  dt = float(np.float32(DT))
  h2, kd = dt * dt, VBD['damping']
  old = x.clone()
  x = x + v * dt + f64(GRAVITY) * dt * dt
  xt = x.clone()
  ent_v, order = torch.sort(q.reshape(-1), stable=True)
  ptr = torch.searchsorted(ent_v, torch.arange(nv + 1, device=DEV))
  groups = []
  for g in _groups(colors):
    g = g[w[g] > 0]
    cnt = ptr[g + 1] - ptr[g]
    owner = torch.repeat_interleave(torch.arange(len(g), device=DEV), cnt)
    start = torch.cumsum(cnt, 0) - cnt
    pos = ptr[g][owner] + torch.arange(len(owner), device=DEV) - start[owner]
    groups.append((g, owner, order[pos] // 4, order[pos] % 4))
  Bv = torch.cat([B, -B.sum(1, keepdim=True)], dim=1)  # rows: b of each vertex
  om, eye = 1.0, torch.eye(3, dtype=torch.float64, device=DEV)
  for n in range(c['iterations']):
    if c['rho'] > 0 and n >= 1:
      om = 2 / (2 - c['rho'] ** 2) if n == 1 else 4 / (4 - c['rho'] ** 2 * om)
    prev = x.clone()
    for g, owner, tet, loc in groups:
      F, cof, J = _f_cof(x, q[tet], B[tet])
      b = Bv[tet, loc]
      s = lam * (J - 1.0)
      pb = ((mu * F + s[:, None, None] * cof) @ b[:, :, None])[:, :, 0]
      qv = (cof @ b[:, :, None])[:, :, 0]
      V = vol[tet]
      mh = (1.0 / w[g] / h2)[:, None]
      fo = mh * (xt[g] - x[g]) - (kd / dt) * (x[g] - old[g])
      fo = fo.index_add(0, owner, -V[:, None] * pb)
      H = (mh[:, :, None] + kd / dt) * eye
      H = H.index_add(0, owner, V[:, None, None] * (
          (mu * b.square().sum(1))[:, None, None] * eye + lam * qv[:, :, None] * qv[:, None, :]))
      x[g] += torch.linalg.solve(H, fo)
    if c['rho'] > 0 and n >= 1:
      x = torch.where((w > 0)[:, None], x + om * (x - prev), x)
  return {'x': x, 'v': 0.993 * (x - old) / dt}


def _exact_xpbd(c, seed):
  xr, x0, v0, t, im, vol = _local_body(c, seed)
  # greedy colours in index order: a tet avoids those at its vertices
  used, colors = [0] * len(xr), []
  for a, b, d, e in t.reshape(-1, 4).tolist():
    k = _low_zero(used[a] | used[b] | used[d] | used[e])
    colors.append(k)
    for i in (a, b, d, e):
      used[i] |= 1 << k
  f64 = lambda a: torch.tensor(a, dtype=torch.float64, device=DEV)  # noqa: E731
  q = torch.tensor(t.reshape(-1, 4).astype(np.int64), device=DEV)
  x, v, w, m = f64(x0), f64(v0), f64(im), f64(vol)
  B, _ = _rest64(f64(xr), q)
  dt = float(np.float32(DT))
  old = x.clone()
  x = x + v * dt + f64(GRAVITY) * (dt * dt)
  lh, ld = torch.zeros(len(q), dtype=torch.float64, device=DEV), torch.zeros(len(q), dtype=torch.float64, device=DEV)
  full = lambda G: torch.cat([G, -G.sum(1, keepdim=True)], dim=1)  # noqa: E731
  groups = _groups(colors)
  for _ in range(c['passes']):
    for g in groups:
      qg, Bg, wg = q[g], B[g], w[q[g]]
      F, cof, J = _f_cof(x, qg, Bg)
      gH = full((cof @ Bg.transpose(1, 2)).transpose(1, 2))
      gD = full((2 * F @ Bg.transpose(1, 2)).transpose(1, 2))
      dot = lambda a, b: (wg * (a * b).sum(2)).sum(1)  # noqa: E731
      CH, CD = J - 1.0, F.square().sum((1, 2)) - 3.0
      SH, SD, X = dot(gH, gH), dot(gD, gD), dot(gD, gH)
      aH, aD = XPBD['hydro_alpha'] / (dt * dt * m[g]), XPBD['devia_alpha'] / (dt * dt * m[g])
      dH = (X * (CD + aD * ld[g]) - (CH + aH * lh[g]) * (aD + SD)) / ((aH + SH) * (aD + SD) - X * X)
      dD = -(CD + aD * ld[g] + X * dH) / (aD + SD)
      x[qg.reshape(-1)] += (wg[:, :, None] * (gH * dH[:, None, None] + gD * dD[:, None, None])).reshape(-1, 3)
      lh[g] += dH
      ld[g] += dD
  return {'x': x, 'v': 0.993 * (x - old) / dt, 'hydro': lh, 'devia': ld}
