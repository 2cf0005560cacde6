"""Multivariate normals at the edges of their tiles (32 and 64 chains, 64
outputs, chunks of 16 and 32 and four stretches of k; csrc/mvn_tile.cuh), alone
and as members of a ragged batch, against 64-bit arithmetic.

Bounds.  u_o is a chain of o FMAs on rounded differences: off by (o + 2) 2^-24 of
the sum of magnitudes.  grad carries that through L^-T and adds as much of its
own; the log-density, summed in 64 bits, carries it once.  A batch gives the
single target's bits whatever its tiles."""
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


def _normal(pg, d, c):
  rng = np.random.default_rng([d, c])
  L = np.tril(rng.normal(size=(d, d)) / np.sqrt(d)) + np.diag(1.0 + rng.random(d))
  t = pg.MultivariateNormalTriL(rng.normal(size=d), L)
  x = torch.from_numpy(rng.normal(size=(c, d)).astype(np.float32)).cuda()
  return t, x


def _check(t, x, lp, g):
  # Parameters as the target holds them (float32).
  m, mu = t._linv_t.double().cuda(), t._loc_t.double().cuda()
  r = x.double() - mu
  u = r @ m.T
  eps = (torch.arange(x.shape[1], device='cuda') + 2) * 2.0 ** -24
  du = eps * (r.abs() @ m.abs().T)
  lp64 = -0.5 * (u * u).sum(1) + t._log_norm
  bound_l = (u.abs() * du + du * du).sum(1) + 2.0 ** -45 * (u * u).sum(1) + 1e-9
  bound_g = du @ m.abs() + (x.shape[1] + 2) * 2.0 ** -24 * (u.abs() @ m.abs())
  assert ((lp - lp64).abs() <= bound_l).all()
  assert ((g - -(u @ m)).abs() <= bound_g).all()


SIZES = [(1, 1), (2, 33), (15, 64), (16, 65), (17, 31), (31, 32), (32, 5), (33, 63), (63, 130),
         (64, 32), (65, 64), (127, 33), (128, 96), (129, 7), (192, 65), (255, 40), (257, 129),
         (640, 3), (1025, 70)]


@pytest.mark.parametrize('d,c', SIZES)
def test_single(pg, d, c):
  t, x = _normal(pg, d, c)
  _check(t, x, *t.log_prob_and_grad(x))


@pytest.mark.parametrize('d,c', [(1, 40000), (8, 38848), (20, 70003), (32, 39001), (33, 38848),
                                 (40, 38847), (64, 45001), (65, 19456), (130, 13001), (300, 8001)])
def test_many_chains(pg, d, c):
  """Past the number of chains from which tiles are 64 x 64; bits as in a small call."""
  t, x = _normal(pg, d, c)
  lp, g = t.log_prob_and_grad(x)
  _check(t, x, lp, g)
  few = torch.arange(c - 100, c, device='cuda')
  lp1, g1 = t.log_prob_and_grad(x[few])
  assert torch.equal(lp[few], lp1) and torch.equal(g[few], g1)


def test_batch_gives_the_same_bits(pg):
  rng = np.random.default_rng(5)
  made = [_normal(pg, d, c) for d, c in SIZES]
  members, states = [], []
  for i, (t, x) in enumerate(made):
    members.append((t, x.shape[0]))
    states.append(x)
    if i % 4 == 0:
      h = pg.NonCentredHierarchicalNormal(rng.normal(size=i + 1), rng.uniform(1, 3, i + 1))
      members.append((h, 3 + i))
      states.append(torch.from_numpy(rng.normal(size=(3 + i, i + 3)).astype(np.float32)).cuda())
  batch = pg.TargetBatch(members)
  lp, g = batch.log_prob_and_grad(batch.pack(states))
  parts, c0 = batch.unpack(g), 0
  for (t, c), x, part in zip(members, states, parts):
    lp1, g1 = t.log_prob_and_grad(x)
    if isinstance(t, pg.MultivariateNormalTriL):
      assert torch.equal(lp[c0:c0 + c], lp1) and torch.equal(part, g1)
    c0 += c
