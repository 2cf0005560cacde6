"""The mixed-precision kernels of 129 to 256 and of 257 to 512 features (there a
pair of CTAs shares a tile of 64 chains: csrc/logreg_tc.cu) at the edges of their
rows, features and chains.

A chain's result does not depend on its place in the tile: with the chains in
another order (other halves, other warps, the other CTA) the outputs are the same
to the bit.  Against 64-bit arithmetic on the same BF16 data: the residuals of the
gradient are BF16 (2^-9 relative, on values up to 1) and their tanh.approx is off by
2^-10, the states' BF16 pairs and truncated sums move z by 2^-14 of sum |x q|, a
quarter of which reaches a residual."""
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


@pytest.mark.parametrize('n,d,c', [
    (1, 129, 1), (127, 130, 15), (128, 143, 16), (129, 144, 17), (256, 192, 33), (257, 193, 48),
    (385, 255, 64), (9729, 256, 65), (19457, 200, 129), (40000, 160, 700),
    (1, 257, 1), (127, 258, 7), (128, 272, 8), (129, 273, 31), (255, 383, 32), (256, 384, 33),
    (257, 385, 40), (1000, 400, 56), (9728, 511, 63), (9729, 512, 64), (19457, 300, 65),
    (4000, 448, 129), (3000, 512, 700)])
def test_chains_anywhere_in_a_tile(pg, n, d, c):
  g = torch.Generator('cuda').manual_seed(n + d + c)
  X = (torch.randn(n, d, generator=g, device='cuda') / d ** 0.5).bfloat16()
  y = (torch.rand(n, generator=g, device='cuda') < 0.4).float()
  q = torch.randn(c, d, generator=g, device='cuda')
  t = pg.LogisticRegression(X, y, precision='mixed')
  lp, grad = t.log_prob_and_grad(q)
  x, b = X.double(), q.double()
  z = x @ b.T
  mag = x.abs() @ b.abs().T
  lp64 = (y.double()[:, None] * z - torch.nn.functional.softplus(z)).sum(0) \
      - 0.5 * (b * b).sum(1) - 0.5 * d * np.log(2 * np.pi)
  g64 = (y.double()[:, None] - torch.sigmoid(z)).T @ x - b
  dr = 2.0 ** -9 + 2.0 ** -10 + 2.0 ** -16 * mag
  assert ((grad - g64).abs() <= dr.T @ x.abs() + 2.0 ** -20 * b.abs()).all()
  terms = torch.nn.functional.softplus(z.abs()) + z.abs()
  assert ((lp - lp64).abs() <= (2.0 ** -14 * mag + 2.0 ** -20 * terms).sum(0) + 1e-5).all()
  perm = torch.randperm(c, generator=g, device='cuda')
  lp2, grad2 = t.log_prob_and_grad(q[perm].contiguous())
  assert torch.equal(lp2, lp[perm]) and torch.equal(grad2, grad[perm])
