"""FP32 logistic regression above 128 features: the products kernel of up to 256
(csrc/logreg_wide.cu) and the gradient from FP16 pairs that it shares with the
GEMM path above that (csrc/grad_tc.cuh), against 64-bit arithmetic at the edges of
their tiles (32, 64 and 128 rows, 64 and 128 chains, 16, 64 and 256 features), and
the columns and labels that stay with the older kernels.  Bounds: those of
test_gpu_logreg_f32_tc.py."""
import pytest

from tests.test_gpu_logreg_f32_tc import _check, _data, pg  # noqa: F401

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


@pytest.mark.parametrize('n,d,c', [
    (1, 129, 1), (31, 256, 3), (32, 144, 64), (33, 145, 65), (63, 160, 63), (64, 129, 128),
    (65, 255, 129), (127, 200, 5), (128, 192, 16), (129, 193, 257), (9727, 240, 64),
    (9729, 241, 33), (19457, 256, 130), (30011, 237, 192), (70001, 129, 7), (2000, 250, 20000),
    (1, 257, 1), (40, 257, 9), (64, 272, 128), (65, 273, 129), (1000, 512, 64), (1001, 513, 65),
    (9729, 768, 3), (12289, 601, 99), (20001, 769, 130), (2100, 1025, 257), (500, 2050, 20)])
def test_against_64_bits(pg, n, d, c):
  _check(pg, *_data(n, d, c, seed=n + d))


@pytest.mark.parametrize('d', [150, 300])
@pytest.mark.parametrize('case', ['wide', 'outlier', 'huge', 'labels', 'zero'])
def test_other_columns(pg, d, case):
  X, y, q = _data(3100, d, 50, seed=3)
  if case == 'wide':
    X[:, 4] = torch.exp(6.0 * X[:, 4])
    q[:, 4] /= X[:, 4].max()
  elif case == 'outlier':
    X[5, 4] = 2.0 ** 40
    q[:, 4] = 2.0 ** -42
  elif case == 'huge':
    X[:, 4] *= 2.0 ** 70
    q[:, 4] *= 2.0 ** -70
  elif case == 'labels':
    y = 5.0 * y - 1.0
  else:
    X[:, 7] = 0.0
  _check(pg, X, y, q)


@pytest.mark.parametrize('d', [150, 300])
def test_one_nonfinite_state_leaves_the_others_alone(pg, d):
  X, y, q = _data(3000, d, 140, seed=4)
  t = pg.LogisticRegression(X, y)
  lp0, g0 = t.log_prob_and_grad(q)
  q[17, 3] = float('inf')
  q[130, 0] = float('nan')
  lp, g = t.log_prob_and_grad(q)
  bad = torch.zeros(140, dtype=torch.bool, device='cuda')
  bad[17] = bad[130] = True
  assert not torch.isfinite(lp[bad]).any()
  assert torch.equal(lp[~bad], lp0[~bad]) and torch.equal(g[~bad], g0[~bad])
