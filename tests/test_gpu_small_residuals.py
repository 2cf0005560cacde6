"""FP32 logistic regression of 129 to 256 features where every row is all but
fitted: labels 0, an intercept far below zero and a wide prior, so that the gradient
is the sum of residuals of e^z each (csrc/logreg_wide.cu keeps their bits by scaling,
csrc/logreg_simt.cu in FP32).

Bound.  A residual is e^z / (1 + e^z): its relative error is z's absolute one, d + 1
roundings of 2^-24 of sum_d |x q|, and a few of 2^-22 for exp and the division; the
products and their sums lose less than 2^-20 of the sum of magnitudes."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


@pytest.mark.parametrize('n,d,c', [(1, 129, 3), (200, 130, 65), (3000, 150, 40), (4161, 256, 130)])
@pytest.mark.parametrize('level', [-12.0, -18.0, -25.0, -40.0, -60.0, -78.0])
def test_gradient_of_fitted_rows(n, d, c, level):
  if not torch.cuda.is_available():
    pytest.skip('no CUDA device')
  import probability_gb300 as pg
  g = torch.Generator('cuda').manual_seed(n + d)
  X = torch.randn(n, d, generator=g, device='cuda')
  X[:, 0] = 1.0
  y = torch.zeros(n, device='cuda')
  q = 0.3 * torch.randn(c, d, generator=g, device='cuda') / d ** 0.5
  q[:, 0] = level + torch.linspace(-2.0, 2.0, c, device='cuda')
  grad = pg.LogisticRegression(X, y, prior_scale=1e18).log_prob_and_grad(q)[1]
  x, b = X.double(), q.double()
  r = -torch.sigmoid(x @ b.T)                      # [N, C]
  g64 = r.T @ x - b * 1e-36
  dz = (d + 1) * 2.0 ** -24 * (x.abs() @ b.abs().T) + 2.0 ** -20
  bound = (r.abs() * dz).T @ x.abs() + 2.0 ** -20 * (r.abs().T @ x.abs() + b.abs() * 1e-36)
  assert ((grad.double() - g64).abs() <= bound).all()
