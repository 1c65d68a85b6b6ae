"""Which warps of the coarse sweeps' kernel (`csrc/sweep.cu`) may wait for its
barriers.  A block has three, reused every three sweeps and tested by one bit
of parity, so a warp that a phase does not need can miss it: on the CPU, a model
of the barriers in which one warp at a time is kept from running; on the GPU,
thousands of sweeps in blocks with fewer rows than warps, or none; and waits that
run out (a limit of 0: a block gives up at the first poll that finds a phase
incomplete, and all blocks end within their first sweeps)."""

import numpy as np
import pytest

from controllable_pbd_3d_gb300 import _native as N
from test_coarse_sweeps import Sweeps, matrix


class Bar:
  """An mbarrier: one arrival and as many stores as expected end a phase."""

  def __init__(self):
    self.done = 0       # phases that have ended
    self.arrived = False
    self.pending = 0    # stores expected less stores landed

  def step(self):
    if self.arrived and self.pending == 0:
      self.done += 1
      self.arrived = False

  def arrive(self, stores):
    self.arrived = True
    self.pending += stores
    self.step()

  def land(self):
    self.pending -= 1
    self.step()

  def passed(self, parity):
    return self.done % 2 != parity


def warp(bars, block, wid, tasks, sweeps):
  """One warp's waits: yields False where it cannot go on yet.  tasks[b]: the
  tasks of block b, one a warp, each read by all blocks with tasks."""
  slot = to = 0
  parity = 0
  total = sum(tasks)
  for s in range(1, sweeps + 1):
    slot, to = to, (to + 1) % 3
    if wid == 0 and s < sweeps:
      bars[block][to].arrive(total if tasks[block] else 0)
    if s > 1:
      while not bars[block][slot].passed(parity):
        yield False
      if slot == 0:
        parity ^= 1
    if wid < tasks[block] and s < sweeps:
      for b in range(len(tasks)):
        if tasks[b]:
          bars[b][to].land()
    yield True


def stuck(tasks, warps, sweeps, rule, starved):
  """Whether some warp never ends when `starved` runs only once all others
  cannot go on."""
  bars = [[Bar() for _ in range(3)] for _ in tasks]
  run = {(b, w): warp(bars, b, w, tasks, sweeps)
         for b in range(len(tasks)) for w in range(warps) if rule(w, tasks[b])}
  while run:
    moved = False
    for k in sorted(run, key=lambda k: k == starved):
      if k == starved and moved:
        continue
      try:
        moved = next(run[k]) or moved
      except StopIteration:
        del run[k]
        moved = True
    if not moved:
      return True
  return False


@pytest.mark.parametrize('tasks', [[2, 0], [3, 1, 2], [1, 0, 0], [4, 4]])
def test_only_warps_with_rows_may_wait(tasks):
  warps, sweeps = 4, 12
  every = [(b, w) for b in range(len(tasks)) for w in range(warps)]

  def with_rows(w, t):
    return w < t

  assert not any(stuck(tasks, warps, sweeps, with_rows, k) for k in every)
  # a warp without rows, kept from running, never ends
  idle = [(b, w) for b, w in every if w >= tasks[b]]
  for k in idle:
    if k[1] > 0:
      assert stuck(tasks, warps, sweeps, lambda w, t: True, k)


@pytest.mark.gpu
@pytest.mark.parametrize('n,per_row', [(1, 1), (16, 3), (17, 4), (100, 6), (255, 5), (300, 40), (1100, 9)])
def test_many_sweeps_of_few_rows(cuda, monkeypatch, n, per_row):
  from controllable_pbd_3d_gb300.mgpcg_gpu import GPUMultigridSolver
  sweeps = 3001
  default = N.default_params

  def params():
    p = default()
    p.coarse_sweeps = sweeps
    return p

  monkeypatch.setattr(N, 'default_params', params)
  A = matrix(n, per_row, n)
  m = GPUMultigridSolver().setup(A, [])
  b = np.random.default_rng(2).standard_normal(n).astype(np.float32)
  s = Sweeps()
  ref = s(A, b.astype(np.float64), np.zeros(n), sweeps)
  bt = cuda.tensor(b, device='cuda')
  got = [m.vcycle_apply(bt).cpu().numpy() for _ in range(10)]
  for g in got[1:]:
    assert np.array_equal(got[0], g)
  assert np.abs(got[0] - ref).max() <= s.err


@pytest.mark.gpu
def test_a_wait_that_runs_out_is_reported_later_by_the_vcycle(cuda):
  from controllable_pbd_3d_gb300.mgpcg_gpu import GPUMultigridSolver
  m = GPUMultigridSolver().setup(matrix(3001, 30, 5), [])
  b = cuda.tensor(np.random.default_rng(3).standard_normal(3001).astype(np.float32), device='cuda')
  want = m.vcycle_apply(b).clone()
  L = N.lib()
  for again in (lambda: m.vcycle_apply(b), lambda: m.solve(b, cuda.zeros_like(b)),
                lambda: N.check(L.mgpbd_synchronize(m._h), 'mgpbd_synchronize')):
    assert L.mgpbd_set_barrier_limit(m._h, 0.0) == 0
    got = m.vcycle_apply(b)
    cuda.cuda.synchronize()
    assert bool(cuda.isnan(got).any())
    assert L.mgpbd_set_barrier_limit(m._h, 4.0) == 0
    with pytest.raises(N.MGPBDError, match='timed out') as e:
      again()
    assert e.value.code == -2
    assert cuda.equal(m.vcycle_apply(b), want)


@pytest.mark.gpu
@pytest.mark.parametrize('kw', [dict(mode='fast'), dict(mode='parity'), dict(mode='fast', use_graph=False)])
def test_a_wait_that_runs_out_ends_the_solve(cuda, kw):
  from controllable_pbd_3d_gb300 import MGPBDSolverGPU, meshgen
  xr, t = meshgen.hex_grid_tets(7, 8, 6)
  x0, _ = meshgen.hex_grid_tets(7, 8, 6, jitter=0.02, seed=3)

  def solver():
    x = cuda.tensor(x0, device='cuda')
    s = MGPBDSolverGPU(x, cuda.tensor(xr, device='cuda'),
                       cuda.tensor(np.ones(len(xr), np.float32), device='cuda'), cuda.tensor(t, device='cuda'),
                       None, [0.0, -9.8, 0.0], 1.0 / 300, mu=1e5, maxiter=2, **kw)
    s.init()
    s.step(0)
    return s, x

  (s, x), (ref, x_ref) = solver(), solver()
  L = N.lib()
  assert L.mgpbd_set_barrier_limit(s._h, 0.0) == 0
  s.make_prediction()
  before = x.clone()
  with pytest.raises(N.MGPBDError, match='timed out') as e:
    s.solve(1)
  assert e.value.code == -2
  assert L.mgpbd_set_barrier_limit(s._h, 4.0) == 0
  with cuda.no_grad():
    x.copy_(before)
  s.solve(1)
  s.update_vel()
  ref.step(1)
  assert s.stats()['status'] == ref.stats()['status']
  assert cuda.equal(x, x_ref)
