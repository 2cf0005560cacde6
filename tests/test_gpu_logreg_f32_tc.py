"""The FP32 logistic-regression kernel whose gradient products run on the
tensor cores (csrc/logreg_f32.cu) against 64-bit arithmetic, at the edges of
its row limit (4096), its tiles (32 and 64 rows, odd and even counts of them,
128 chains, 16 and 64 features) and its FP16 form of X, and the columns and
labels that stay with the CUDA cores instead.

Bounds.  z, a chain of d FMAs, is off by d 2^-24 of sum_d |x q| at most, which
moves a residual by a quarter of that; ex2.approx and rcp.approx move it by
2^-22.  The FP16 pairs keep 2^-24 of R and of X (2^-23 in root mean square for a
column that is accepted), and the truncated sums of a tile and the FP32 sums
over tiles and splits lose less than 2^-20 of the sum of magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


@pytest.fixture(scope='module')
def pg():
  if not torch.cuda.is_available():
    pytest.skip('no CUDA device')
  import probability_gb300 as pg
  return pg


def _check(pg, X, y, q):
  lp, g = pg.LogisticRegression(X, y).log_prob_and_grad(q)
  x, t, b = X.double(), y.double()[:, None], q.double()
  n, d = X.shape
  z = x @ b.T
  mag = x.abs() @ b.abs().T
  lp64 = (t * z - torch.nn.functional.softplus(z, threshold=1e9)).sum(0) - 0.5 * (b * b).sum(1) \
      - 0.5 * d * np.log(2 * np.pi)
  g64 = (t - torch.sigmoid(z)).T @ x - b
  dr = 2.0 ** -22 + d * 2.0 ** -26 * mag                # [N, C]
  top = max(1.0, float((y - 0.5).abs().max()) + 0.5)    # largest residual
  rms = (x * x).mean(0).sqrt()
  bound_g = dr.T @ x.abs() + 2.0 ** -20 * (top * x.abs().sum(0) + b.abs()) + n * 2.0 ** -23 * rms
  terms = torch.nn.functional.softplus(z.abs()) + 0.5 * z.abs()
  bound_l = (2.0 ** -22 * terms + d * 2.0 ** -24 * mag).sum(0) + 2.0 ** -40 * lp64.abs() + 1e-6
  assert torch.isfinite(lp).all() and torch.isfinite(g).all()
  assert ((lp - lp64).abs() <= bound_l).all()
  assert ((g - g64).abs() <= bound_g).all()


def _data(n, d, c, seed):
  g = torch.Generator('cuda').manual_seed(seed)
  X = torch.randn(n, d, generator=g, device='cuda')
  X[:, 0] = 1.0
  y = (torch.rand(n, generator=g, device='cuda') < 0.4).float()
  return X, y, torch.randn(c, d, generator=g, device='cuda') / d ** 0.5


@pytest.mark.parametrize('n,d,c', [(4095, 30, 9), (4096, 1, 1), (4097, 15, 127), (4127, 16, 128),
                                   (4128, 17, 129), (4129, 48, 5), (4160, 49, 300), (9728, 63, 40),
                                   (9729, 64, 65), (19456, 65, 33), (19521, 80, 30),
                                   (29185, 96, 64), (40000, 100, 130), (40033, 112, 7),
                                   (50001, 113, 128), (4099, 127, 1024), (70001, 128, 65),
                                   (4500, 3, 20000)])
def test_against_64_bits(pg, n, d, c):
  _check(pg, *_data(n, d, c, seed=n + d))


def test_scaled_features(pg):
  """Scales of 2^-50 .. 2^50 per feature, states scaled back; a zero column."""
  X, y, q = _data(5000, 40, 70, seed=1)
  k = torch.linspace(-50, 50, 40, device='cuda').round()
  X, q = X * 2.0 ** k, q * 2.0 ** -k
  X[:, 7] = 0.0
  _check(pg, X, y, q)


@pytest.mark.parametrize('case', ['wide', 'outlier', 'tiny', 'huge', 'labels'])
def test_kept_on_the_cuda_cores(pg, case):
  X, y, q = _data(5100, 20, 50, seed=3)
  if case == 'wide':
    X[:, 4] = torch.exp(6.0 * X[:, 4])
    q[:, 4] /= X[:, 4].max()
  elif case == 'outlier':
    X[5, 4] = 2.0 ** 40
    q[:, 4] = 2.0 ** -42
  elif case == 'tiny':
    X[:, 4] *= 2.0 ** -70
  elif case == 'huge':
    X[:, 4] *= 2.0 ** 70
    q[:, 4] *= 2.0 ** -70
  else:
    y = 5.0 * y - 1.0
  _check(pg, X, y, q)


def test_one_nonfinite_state_leaves_the_others_alone(pg):
  X, y, q = _data(6000, 30, 140, seed=4)
  t = pg.LogisticRegression(X, y)
  lp0, g0 = t.log_prob_and_grad(q)
  q[17, 3] = float('inf')
  q[130, 0] = float('nan')
  lp, g = t.log_prob_and_grad(q)
  bad = torch.zeros(140, dtype=torch.bool, device='cuda')
  bad[17] = bad[130] = True
  assert not torch.isfinite(lp[bad]).any()
  assert torch.equal(lp[~bad], lp0[~bad]) and torch.equal(g[~bad], g0[~bad])
