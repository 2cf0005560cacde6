"""Which columns the FP32 logistic regressions hold as FP16 pairs
(csrc/f16_rows.cuh).  A column whose entries the pairs cannot carry leaves the
target on the CUDA cores (up to 128 features: csrc/logreg_f32.cu; 129 to 256:
csrc/logreg_simt.cu; above: the FP32 GEMMs).

Which of the two ran is seen from the gradient's bits: a last row of zeros adds
nothing to a gradient, but its label, 3, does not fit the pairs either and keeps the
target on the CUDA cores; with the label 0 X alone decides.  Equal bits: the same
kernels ran.

Bounds.  ex2.approx and rcp.approx move a residual by 2^-22, z's d FMAs by a quarter
of d 2^-24 of sum_d |x q|, neither where |z| > 100 (there a residual is exact);
products, their truncated sums and the FP32 sums over tiles and splits lose less than
2^-20 of the sum of magnitudes."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


@pytest.fixture(scope='module')
def pg():
  if not torch.cuda.is_available():
    pytest.skip('no CUDA device')
  import probability_gb300 as pg
  return pg


def _data(n, d, c, seed):
  """n - 1 rows and a last one of zeros."""
  g = torch.Generator('cuda').manual_seed(seed)
  X = torch.randn(n, d, generator=g, device='cuda')
  X[:, 0] = 1.0
  X[-1] = 0.0
  y = (torch.rand(n, generator=g, device='cuda') < 0.4).float()
  y[-1] = 0.0
  return X, y, 0.3 * torch.randn(c, d, generator=g, device='cuda') / d ** 0.5, g


def _grad_error(X, y, q, grad):
  """Error of a gradient over its bound."""
  x, t, b = X.double(), y.double()[:, None], q.double()
  z = x @ b.T
  r = t - torch.sigmoid(z)
  dr = 2.0 ** -22 + X.shape[1] * 2.0 ** -26 * (x.abs() @ b.abs().T)
  dr = torch.where(z.abs() > 100, torch.zeros_like(dr), dr)
  bound = dr.T @ x.abs() + 2.0 ** -20 * (r.abs().T @ x.abs() + b.abs())
  return ((grad.double() - (r.T @ x - b)).abs() / bound).max()


def _fits(pg, X, y, q):
  """(whether the pairs were used, gradient)"""
  grad = pg.LogisticRegression(X, y).log_prob_and_grad(q)[1]
  kept = y.clone()
  kept[-1] = 3.0
  other = pg.LogisticRegression(X, kept).log_prob_and_grad(q)[1]
  return not torch.equal(grad, other), grad


SHAPES = [(5100, 20, 50), (8192, 100, 9), (3000, 150, 50), (5100, 300, 40)]


@pytest.mark.parametrize('n,d,c', SHAPES)
@pytest.mark.parametrize('top', [2.0 ** 24, 1e9, 2.0 ** 34, 2.0 ** 40, 2.0 ** 50])
def test_saturated_outlier(pg, n, d, c, top):
  """One entry far above its column's others, its row fitted exactly (residual 0):
  the column's gradient is the others'."""
  X, y, q, _ = _data(n, d, c, seed=n + d)
  X[5, 4] = top
  y[5] = 1.0
  q[:, 4] = 2e3 / top          # z of row 5 is 2000
  fits, grad = _fits(pg, X, y, q)
  assert _grad_error(X, y, q, grad) <= 1.0
  assert not fits


@pytest.mark.parametrize('n,d,c', SHAPES)
@pytest.mark.parametrize('case', ['lognormal', 'two scales', 'sparse'])
def test_wide_columns(pg, n, d, c, case):
  X, y, q, g = _data(n, d, c, seed=n + d + 1)
  if case == 'lognormal':
    X[:-1, 4] = torch.exp(6.0 * X[:-1, 4])
  elif case == 'two scales':   # one row in ten is what matters
    X[:, 4] *= torch.where(torch.rand(n, generator=g, device='cuda') < 0.1, 1.0, 1e8)
  else:                        # a handful of entries, one of them large
    X[9:, 4] = 0.0
    X[3, 4] = 1e9
  q[:, 4] = 1.0 / X[:, 4].abs().max()
  fits, grad = _fits(pg, X, y, q)
  assert _grad_error(X, y, q, grad) <= 1.0
  assert not fits


@pytest.mark.parametrize('n,d,c', SHAPES)
@pytest.mark.parametrize('case', ['normal', 'constant', 'dummy', 'uniform', 'lognormal', 'sparse',
                                  'scaled', 'one tiny entry', 'moderate outlier', 'zero'])
def test_ordinary_columns_are_held(pg, n, d, c, case):
  X, y, q, g = _data(n, d, c, seed=n + d + 2)
  col = X[:-1, 4]
  if case == 'constant':
    col.fill_(0.1)
  elif case == 'dummy':
    col.copy_((col > 1.0).float())
  elif case == 'uniform':
    col.copy_(torch.rand(n - 1, generator=g, device='cuda'))
  elif case == 'lognormal':
    col.exp_()
  elif case == 'sparse':
    col[torch.rand(n - 1, generator=g, device='cuda') < 0.98] = 0.0
  elif case == 'scaled':
    col *= 2.0 ** -45
  elif case == 'one tiny entry':
    col[11] = 1e-30
  elif case == 'moderate outlier':
    col[11] = 500.0
  elif case == 'zero':
    col.zero_()
  if case == 'moderate outlier':
    q[:, 4] *= 0.01
  fits, grad = _fits(pg, X, y, q)
  assert _grad_error(X, y, q, grad) <= 1.0
  assert fits
