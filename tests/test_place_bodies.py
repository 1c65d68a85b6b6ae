"""How packed bodies share the SMs (`dcg_place_bodies` in csrc/dcg_plan.cpp), on
the CPU: with and without their softness, on each kind of cluster, for values
that a caller's masses and compliances may give it."""

import numpy as np
import pytest

from controllable_pbd_3d_gb300 import _native as N


def places(entries, softness, n16, n8, n4):
  entries = np.ascontiguousarray(entries, np.float64)
  n = len(entries)
  if softness is not None:
    softness = np.ascontiguousarray(softness, np.float64)
  count, cluster, blocks = (np.zeros(1, np.int32) for _ in range(3))
  out = []
  while not out or len(out) < count[0]:
    first, size = np.full(n, -1, np.int32), np.full(n, -1, np.int32)
    N.check(N.lib().mgpbd_host_place_bodies(
        n, entries.ctypes.data, softness.ctypes.data if softness is not None else None, n16, n8, n4, len(out),
        count.ctypes.data, cluster.ctypes.data, blocks.ctypes.data, first.ctypes.data, size.ctypes.data),
            'mgpbd_host_place_bodies')
    out.append((int(cluster[0]), int(blocks[0]), first, size))
  return out


def check(all_, kinds):
  assert all_
  for cluster, blocks, first, size in all_:
    assert cluster in kinds
    assert blocks > 0 and blocks % cluster == 0
    used = np.zeros(blocks, int)
    for f, s in zip(first, size):
      assert s in (4, 8, 16) and s <= cluster
      assert 0 <= f and f % cluster + s <= cluster  # within one cluster
      used[f:f + s] += 1
    assert used.max() == 1


@pytest.mark.parametrize('n', [1, 2, 3, 9, 16, 24, 130])
@pytest.mark.parametrize('resident', [(9, 18, 36), (2, 0, 0), (0, 18, 0), (0, 0, 36), (0, 3, 7)])
@pytest.mark.parametrize('known', [False, True])
def test_arrangements(n, resident, known):
  rng = np.random.default_rng(n)
  entries = 36 * rng.integers(2, 19, n).astype(float)**3
  softness = 10.0**rng.uniform(-4, 2, n) if known else None
  check(places(entries, softness, *resident), [c for c, r in zip((16, 8, 4), resident) if r])


def test_stiff_bodies_have_more_of_the_chip():
  """Equal bodies, more than the chip takes at once: those that need most
  iterations are not on fewer blocks than the others."""
  softness = np.array([1e-4] * 6 + [10.0] * 18)
  _, _, _, size = places(np.full(24, 36 * 12.0**3), softness, 9, 18, 36)[0]
  assert size[:6].min() >= size[6:].max()


@pytest.mark.parametrize('bad', [np.nan, np.inf, 0.0, 1e300, 1e-300])
@pytest.mark.parametrize('which', [slice(0, 1), slice(None)])
def test_any_softness(bad, which):
  softness = np.full(5, 0.1)
  softness[which] = bad
  check(places([1e3, 2e4, 5e4, 1e5, 3e5], softness, 9, 18, 36), (16, 8, 4))


def test_bodies_without_entries():
  check(places([0.0, 0.0, 36.0], [0.1, 0.1, 0.1], 9, 18, 36), (16, 8, 4))
  check(places([0.0, 0.0], None, 9, 18, 36), (16, 8, 4))
