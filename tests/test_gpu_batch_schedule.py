"""The tile lists of a ragged batch (csrc/batch.cu) where a member has very many chains:
every chain is evaluated once, as by the member's own target, and making the list of
one member's tiles takes no longer than that of as many tiles in many members."""
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


def _hier(pg, groups):
  rng = np.random.default_rng(groups)
  return pg.NonCentredHierarchicalNormal(rng.normal(size=groups) * 5, rng.uniform(5, 20, groups))


def _states(chains, dim, seed):
  g = torch.Generator('cuda').manual_seed(seed)
  return 0.5 * torch.randn(chains, dim, generator=g, device='cuda')


@pytest.mark.parametrize('chains', [4095, 4096, 4097, 32768 + 3, 70001, 300007])
def test_members_of_many_chains(pg, chains):
  rng = np.random.default_rng(3)
  A = rng.standard_normal((9, 11))
  members = [(_hier(pg, 3), chains), (pg.MultivariateNormalTriL(rng.normal(size=9),
                                      np.linalg.cholesky(A @ A.T)), chains // 7 + 1),
             (_hier(pg, 20), 33), (_hier(pg, 1), 1)]
  batch = pg.TargetBatch(members)
  states = [_states(c, t.event_dim, i) for i, (t, c) in enumerate(members)]
  lp, grad = batch.log_prob_and_grad(batch.pack(states))
  lps = torch.split(lp, [c for _, c in members])
  for (t, c), s, l, g in zip(members, states, lps, batch.unpack(grad)):
    l1, g1 = t.log_prob_and_grad(s)
    np.testing.assert_allclose(l.cpu().numpy(), l1.cpu().numpy(), rtol=1e-12, atol=1e-9)
    np.testing.assert_allclose(g.cpu().numpy(), g1.cpu().numpy(), rtol=2e-6, atol=2e-6)


def _time(batch, q):
  times = []
  for _ in range(9):
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    for _ in range(4):
      batch.log_prob_and_grad(q)
    b.record()
    torch.cuda.synchronize()
    times.append(a.elapsed_time(b))
  return sorted(times)[4]


def test_one_member_costs_what_many_do(pg):
  t = _hier(pg, 2)
  q = _states(1 << 20, 4, 5).reshape(-1)
  one = _time(pg.TargetBatch([(t, 1 << 20)]), q)
  many = _time(pg.TargetBatch([(t, 1 << 14)] * 64), q)
  assert one <= 2.0 * many
