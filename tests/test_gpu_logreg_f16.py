"""The FP32 logistic-regression target on the tensor cores (exact leading
products of FP16 slices, csrc/logreg_f16.cu) against 64-bit arithmetic, at the
edges of its tiles (64 rows, 128 chains, 16 and 64 features), of its row limit
(65,536) and of its scaling, and the columns that go to the FP32 kernel
instead.

Bounds.  A residual is off by at most 2^-22 (ex2.approx 2^-22 relative on a
term below 1, times a slope of 1/4, and rcp.approx one ulp of a number below
1), z by 2^-23 of sum_d |x q| (an FP32 rounding of the two accumulators and
the slices' 2^-24), which moves a residual by at most a quarter of that, and
the FP32 sums over splits add 2^-22 of the sum of magnitudes."""
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
  z = x @ b.T
  mag = x.abs() @ b.abs().T
  lp64 = (t * z - torch.nn.functional.softplus(z, threshold=1e9)).sum(0) - 0.5 * (b * b).sum(1) \
      - 0.5 * X.shape[1] * np.log(2 * np.pi)
  g64 = (t - torch.sigmoid(z)).T @ x - b
  dr = 2.0 ** -22 + 2.0 ** -25 * mag                    # [N, C]
  bound_g = dr.T @ x.abs() + 2.0 ** -22 * (x.abs().sum(0) + b.abs())
  terms = torch.nn.functional.softplus(z.abs()) + 0.5 * z.abs()
  bound_l = (2.0 ** -22 * (terms + mag)).sum(0) + 2.0 ** -40 * lp64.abs() + 1e-6
  assert torch.isfinite(lp).all() and torch.isfinite(g).all()
  assert ((lp - lp64).abs() <= bound_l).all()
  assert ((g - g64).abs() <= bound_g).all()


def _data(n, d, c, seed):
  g = torch.Generator('cuda').manual_seed(seed)
  X = torch.randn(n, d, generator=g, device='cuda')
  X[:, 0] = 1.0
  y = (torch.rand(n, generator=g, device='cuda') < 0.4).float()
  return X, y, torch.randn(c, d, generator=g, device='cuda') / d ** 0.5


@pytest.mark.parametrize('n,d,c', [(65535, 30, 9), (65536, 1, 1), (65599, 15, 127),
                                   (65537, 16, 128), (65600, 17, 129), (65664, 48, 5),
                                   (70001, 63, 40), (65537, 64, 300), (66000, 65, 33),
                                   (65601, 100, 130), (65599, 112, 7), (65663, 113, 128),
                                   (131073, 128, 65)])
def test_against_64_bits(pg, n, d, c):
  _check(pg, *_data(n, d, c, seed=n + d))


def test_scaled_features_and_states(pg):
  """Scales of 2^-50 .. 2^50 per feature, states scaled back; one coefficient
  far above the rest, zero columns and states."""
  X, y, q = _data(66000, 40, 70, seed=1)
  k = torch.linspace(-50, 50, 40, device='cuda').round()
  X, q = X * 2.0 ** k, q * 2.0 ** -k
  X[:, 7] = 0.0
  q[3] = 0.0
  _check(pg, X, y, q)
  X, y, q = _data(66000, 40, 70, seed=2)
  q[:, 0] = 300.0
  X[:, 0] = 0.01
  _check(pg, X, y, q)


@pytest.mark.parametrize('case', ['wide', 'outlier', 'tiny', 'huge'])
def test_columns_outside_the_splits(pg, case):
  X, y, q = _data(65900, 20, 50, seed=3)
  if case == 'wide':
    X[:, 4] = torch.exp(6.0 * X[:, 4])
    q[:, 4] /= X[:, 4].max()
  elif case == 'outlier':
    X[5, 4] = 2.0 ** 40
    q[:, 4] = 2.0 ** -42
  elif case == 'tiny':
    X[:, 4] *= 2.0 ** -70
  else:
    X[:, 4] *= 2.0 ** 70
    q[:, 4] *= 2.0 ** -70
  _check(pg, X, y, q)


def test_one_nonfinite_state_leaves_the_others_alone(pg):
  X, y, q = _data(65800, 30, 140, seed=4)
  t = pg.LogisticRegression(X, y)
  lp0, g0 = t.log_prob_and_grad(q)
  q[17, 3] = float('inf')
  q[130, 0] = float('nan')
  lp, g = t.log_prob_and_grad(q)
  bad = torch.zeros(140, dtype=torch.bool, device='cuda')
  bad[17] = bad[130] = True
  assert not torch.isfinite(lp[bad]).any()
  assert torch.equal(lp[~bad], lp0[~bad]) and torch.equal(g[~bad], g0[~bad])
