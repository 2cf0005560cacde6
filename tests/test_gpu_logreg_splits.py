"""Row splits of a logistic-regression evaluation and their reduction
(csrc/split_reduce.cuh): up to 32 splits one thread adds them, above that four
groups do, each path at row counts around the change (64- and 128-row tiles)
and at feature counts around a group's 128 threads.  Bounds: each residual within 2^-21
and the sums within 2^-20 of the sum of magnitudes (float32 sums of up to 152
splits)."""
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


def _reference(X, y, q):
  x, t, b = X.double(), y.double()[:, None], q.double()
  z = x @ b.T
  lp = (t * z - torch.nn.functional.softplus(z)).sum(0) - 0.5 * (b * b).sum(1) \
      - 0.5 * X.shape[1] * np.log(2 * np.pi)
  return lp, (t - torch.sigmoid(z)).T @ x - b


@pytest.mark.parametrize('n', [2048, 2049, 2113, 4096, 4097, 9729, 30000])
@pytest.mark.parametrize('d', [3, 128, 129, 256])
def test_splits(pg, n, d):
  g = torch.Generator('cuda').manual_seed(n + d)
  X = torch.randn(n, d, generator=g, device='cuda') / d ** 0.5
  y = (torch.rand(n, generator=g, device='cuda') < 0.4).float()
  for c in (1, 6, 65):
    q = torch.randn(c, d, generator=g, device='cuda')
    lp, grad = pg.LogisticRegression(X, y).log_prob_and_grad(q)
    lp64, g64 = _reference(X, y, q)
    bound = 2.0 ** -20 * (X.double().abs().sum(0) + q.double().abs())
    assert ((grad - g64).abs() <= bound).all()
    np.testing.assert_allclose(lp.cpu().numpy(), lp64.cpu().numpy(), rtol=2e-6)


@pytest.mark.parametrize('c', [2047, 2048, 2051])
@pytest.mark.parametrize('d', [1, 31, 32, 33, 63, 64, 65])
@pytest.mark.parametrize('precision', ['fp32', 'mixed'])
def test_many_chains(pg, c, d, precision):
  """From 2048 chains on a block reduces four chains of up to 32 features or two of up
  to 64."""
  g = torch.Generator('cuda').manual_seed(c + d)
  X = (torch.randn(900, d, generator=g, device='cuda') / d ** 0.5).bfloat16()
  y = (torch.rand(900, generator=g, device='cuda') < 0.4).float()
  q = torch.randn(c, d, generator=g, device='cuda')
  if precision == 'fp32':
    X = X.float()
  lp, grad = pg.LogisticRegression(X, y, precision=precision).log_prob_and_grad(q)
  X = X.float()
  lp64, g64 = _reference(X, y, q)
  # Mixed: the residual as BF16 hi + lo (2^-16), z from BF16 pairs of the state (2^-16
  # of the sum of magnitudes, and a quarter of that in the residual).
  unit = 2.0 ** -20 if precision == 'fp32' else 2.0 ** -12
  bound = unit * (X.double().abs().sum(0) + q.double().abs())
  assert ((grad - g64).abs() <= bound).all()
  np.testing.assert_allclose(lp.cpu().numpy(), lp64.cpu().numpy(), atol=1e-2,
                             rtol=2e-6 if precision == 'fp32' else 1e-5)
