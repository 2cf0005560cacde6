"""FP32 logistic regression above 256 features from 4096 rows on, where X^T R comes from
FP16 pairs with the residuals lying along rows (csrc/grad_tc.cuh, K-major): rows that
are no multiple of 8 or 64, chains around a tile of 128, features around blocks of 16,
64 and 256, nonfinite states, a zero column and labels that keep the target on the
GEMMs.  Bounds: those of test_gpu_logreg_f32_tc.py."""
import pytest

from tests.test_gpu_logreg_f32_tc import _check, _data, pg  # noqa: F401

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


@pytest.mark.parametrize('n,d,c', [
    (4096, 257, 63), (4097, 257, 64), (4103, 272, 127), (4104, 273, 128), (4159, 300, 129),
    (4160, 319, 1), (4161, 320, 65), (4223, 321, 2), (5003, 512, 64), (5004, 513, 127),
    (6001, 513, 128), (8191, 527, 129), (9733, 1024, 63), (9737, 1025, 200)])
def test_against_64_bits(pg, n, d, c):
  _check(pg, *_data(n, d, c, seed=n + d))


@pytest.mark.parametrize('case', ['zero', 'labels', 'huge'])
def test_other_columns(pg, case):
  X, y, q = _data(4999, 300, 70, seed=5)
  if case == 'zero':
    X[:, 7] = 0.0
  elif case == 'labels':
    y = 5.0 * y - 1.0
  else:
    X[:, 4] *= 2.0 ** 70
    q[:, 4] *= 2.0 ** -70
  _check(pg, X, y, q)


def test_one_nonfinite_state_leaves_the_others_alone(pg):
  X, y, q = _data(5007, 300, 140, seed=4)
  t = pg.LogisticRegression(X, y)
  lp0, g0 = t.log_prob_and_grad(q)
  q[17, 3] = float('inf')
  q[130, 0] = float('nan')
  lp, g = t.log_prob_and_grad(q)
  bad = torch.zeros(140, dtype=torch.bool, device='cuda')
  bad[17] = bad[130] = True
  assert not torch.isfinite(lp[bad]).any()
  assert torch.equal(lp[~bad], lp0[~bad]) and torch.equal(g[~bad], g0[~bad])
