"""What the host side of the partitioned dual CG takes and refuses
(`csrc/dcg_plan.cpp`, `csrc/capi.cu`), on the CPU."""

import numpy as np
import pytest

from controllable_pbd_3d_gb300 import meshgen
from test_dual_partition import apply64, run_plan

SMEM = 230000


def pack(n_bodies=2, n=3):
  """Tets of n_bodies grids side by side, a body each."""
  xs, cs, prob = [], [], []
  for b in range(n_bodies):
    xr, t = meshgen.hex_grid_tets(n, n, n, origin=(2.0 * b, 0.0, 0.0))
    cs.append(np.asarray(t, np.int32).reshape(-1, 4) + sum(len(x) for x in xs))
    prob.append(np.full(len(cs[-1]), b, np.int32))
    xs.append(xr)
  x = np.concatenate(xs).astype(np.float32)
  c = np.ascontiguousarray(np.concatenate(cs), np.int32)
  rng = np.random.default_rng(0)
  g = rng.standard_normal((len(c), 4, 3)).astype(np.float32)
  return (x, c, len(c), np.concatenate(prob), g, np.ones(len(x), np.float32),
          rng.random(len(c)).astype(np.float32), rng.standard_normal(len(c)).astype(np.float32))


@pytest.mark.parametrize('blocks', [4, 0])
@pytest.mark.parametrize('bad', [-1, 2, 2**30])
def test_a_body_that_is_not_there_is_refused(blocks, bad):
  xr, c, n4, prob, g, w, alpha, x = pack()
  assert run_plan(xr, c, n4, prob, 2, blocks, True, 256, SMEM, g, w, alpha, x)[0] == 0
  prob[len(prob) // 2] = bad
  assert run_plan(xr, c, n4, prob, 2, blocks, True, 256, SMEM, g, w, alpha, x)[0] == -1


@pytest.mark.parametrize('bad', [-1, 2**30])
def test_a_vertex_that_is_not_there_is_refused(bad):
  xr, c, n4, prob, g, w, alpha, x = pack()
  c[5, 3] = bad
  assert run_plan(xr, c, n4, prob, 2, 4, True, 256, SMEM, g, w, alpha, x)[0] == -1


def test_bodies_that_share_a_vertex_are_refused():
  xr, c, n4, prob, g, w, alpha, x = pack()
  c[-1, 2] = c[0, 0]
  assert run_plan(xr, c, n4, prob, 2, 4, True, 256, SMEM, g, w, alpha, x)[0] == -1


@pytest.mark.parametrize('bad', [np.nan, np.inf, 3e38])
def test_rest_positions_that_are_not_finite(bad):
  """They are only where the mesh is cut: any place will do, and it takes no
  longer (ordered by NaN, 100,000 constraints took 15 s)."""
  import time
  xr, t = meshgen.hex_grid_tets(27, 27, 27)
  c = np.ascontiguousarray(np.asarray(t, np.int32).reshape(-1, 4))
  rng = np.random.default_rng(1)
  g = rng.standard_normal((len(c), 4, 3)).astype(np.float32)
  w = np.ones(len(xr), np.float32)
  alpha = rng.random(len(c)).astype(np.float32)
  x = rng.standard_normal(len(c)).astype(np.float32)
  for part in (slice(None), slice(0, 40)):
    xx = xr.astype(np.float32)
    xx[part] = bad
    t0 = time.perf_counter()
    rc, y, _ = run_plan(xx, c, len(c), None, 1, 152, False, 512, SMEM, g, w, alpha, x)
    assert time.perf_counter() - t0 < 5.0
    assert rc == 0
    ref, size = apply64(c, len(c), g, w, alpha, x)
    assert np.all(np.abs(y - ref) <= 1e-13 * size)
