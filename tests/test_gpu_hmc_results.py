"""HMC results whose accepted part carries a seed (a proposal's results passed on as
the accepted ones): two chains, as many as a seed has words, several state parts."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


@pytest.mark.parametrize('parts', [1, 2])
@pytest.mark.parametrize('chains', [2, 3])
def test_results_with_a_seed(parts, chains):
  if not torch.cuda.is_available():
    pytest.skip('no CUDA device')
  import probability_gb300 as pg
  g = torch.Generator('cuda').manual_seed(1)
  X = torch.randn(50, 4, generator=g, device='cuda')
  y = (torch.rand(50, generator=g, device='cuda') < 0.5).float()
  q = torch.randn(chains, 4, generator=g, device='cuda')
  state = q if parts == 1 else [q[:, :1].contiguous(), q[:, 1:].contiguous()]
  k = pg.mcmc.HamiltonianMonteCarlo(pg.LogisticRegression(X, y), step_size=0.1,
                                    num_leapfrog_steps=3)
  kr = k.bootstrap_results(state)
  seeded = kr._replace(accepted_results=kr.accepted_results._replace(
      seed=torch.tensor([4, 9], dtype=torch.int64)))
  s1, kr1 = k.one_step(state, kr, seed=(2, 3))
  s2, kr2 = k.one_step(state, seeded, seed=(2, 3))
  assert kr1.accepted_results.seed == [] and kr2.accepted_results.seed == []
  for a, b in zip([s1] if parts == 1 else s1, [s2] if parts == 1 else s2):
    assert torch.equal(a, b)
  assert torch.equal(kr1.accepted_results.target_log_prob, kr2.accepted_results.target_log_prob)
