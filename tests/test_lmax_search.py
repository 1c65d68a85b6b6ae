"""The largest-eigenvalue search of the Chebyshev interval (csrc/cheb_dev.cuh) on
the CPU: it shrinks an interval around the largest eigenvalue by the signs of the
leading minors, which are made by the kernels' own code (`all_below`), and
returns its upper end."""

import ctypes as C

import numpy as np
import pytest

from controllable_pbd_3d_gb300 import _native as N

EPS = float(np.finfo(np.float64).eps)


def lmax(a, b):
  a = np.ascontiguousarray(a, np.float64)
  b = np.ascontiguousarray(b, np.float64)
  out = C.c_double()
  N.check(N.lib().mgpbd_host_lanczos_lmax(a.ctypes.data, b.ctypes.data, len(a), C.byref(out)),
          'mgpbd_host_lanczos_lmax')
  return out.value


def check(a, b):
  """The width the search stops at; the minors are those of a tridiagonal whose
  entries are off by a few roundings; and minors that leave the range: all k
  factors below (1e-308)^(1/k) of the scale."""
  k = len(a)
  b = b[:k - 1]
  want = float(np.linalg.eigvalsh(np.diag(a) + np.diag(b, 1) + np.diag(b, -1)).max())
  r = np.r_[np.abs(b), 0.0] + np.r_[0.0, np.abs(b)]
  s = max(abs((a - r).min()), abs((a + r).max()))
  got = lmax(a, np.r_[b, 0.0])
  tol = 1e-12 * max(1.0, abs((a + r).max())) + 32 * EPS * s
  assert want - 32 * EPS * s <= got <= want + tol + s * 1e-308**(1.0 / k), (got, want)


@pytest.mark.parametrize('k', [1, 2, 3, 7, 23, 24, 31, 32])
@pytest.mark.parametrize('seed', range(4))
def test_random(k, seed):
  rng = np.random.default_rng([k, seed])
  scale = 10.0 ** rng.uniform(-6, 12)
  check(rng.uniform(-2.0, 10.0, k) * scale, rng.uniform(-1.0, 1.0, k) * scale * 10.0 ** rng.uniform(-6, 1))


@pytest.mark.parametrize('k', [24, 32])
@pytest.mark.parametrize('rows', [1, 2, 5, 23])
def test_trailing_zero_rows(k, rows):
  """A Lanczos process that ended after `rows` steps."""
  rng = np.random.default_rng(rows)
  a, b = np.zeros(k), np.zeros(k)
  a[:rows] = rng.uniform(1.0, 4.0, rows)
  b[:rows - 1] = rng.uniform(0.1, 1.0, rows - 1)
  check(a, b)


@pytest.mark.parametrize('k', [24, 32])
@pytest.mark.parametrize('spread', [0.0, 1e-14, 1e-12, 1e-9, 1e-6, 1e-3])
def test_clustered(k, spread):
  """Eigenvalues within `spread` of one another: small minors."""
  rng = np.random.default_rng(k)
  check(3.0 + spread * rng.random(k), np.full(k, spread / 8))
  a = np.full(k, 3.0)
  a[k // 2] += 2.0
  check(a, np.full(k, spread))


def test_negative_and_not_finite():
  check(np.array([-3.0, -1.0, -2.0]), np.array([0.5, 0.25, 0.0]))
  check(np.zeros(24), np.zeros(24))
  assert np.isnan(lmax([1.0, np.inf], [0.0, 0.0]))
  assert np.isnan(lmax([1.0, 2.0], [np.inf, 0.0]))
  out = C.c_double()
  a = np.ones(33)
  assert N.lib().mgpbd_host_lanczos_lmax(a.ctypes.data, a.ctypes.data, 33, C.byref(out)) == -1
  assert N.lib().mgpbd_host_lanczos_lmax(a.ctypes.data, a.ctypes.data, 0, C.byref(out)) == -1


@pytest.mark.parametrize('seed', range(3))
def test_lanczos_of_a_known_spectrum(seed):
  """24 steps as the kernels make them, q.q summed and not taken as 1."""
  rng = np.random.default_rng(seed)
  n = 400
  ev = np.concatenate([np.linspace(1e-3, 1.0, n - 1), [3.7]])
  Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
  A = (Q * ev) @ Q.T
  q, prev, beta = rng.random(n) + 0.5, np.zeros(n), 0.0
  q /= np.linalg.norm(q)
  a, b = [], []
  for _ in range(24):
    w = A @ q - beta * prev
    alpha = (q @ w) / (q @ q)
    beta = float(np.sqrt(w @ w - (2 * (q @ w) - alpha * (q @ q)) * alpha))
    a.append(alpha)
    b.append(beta)
    prev, q = q, (w - alpha * q) / beta
  check(np.array(a), np.array(b))
  assert abs(lmax(a, b) - 3.7) <= 1e-6 * 3.7
