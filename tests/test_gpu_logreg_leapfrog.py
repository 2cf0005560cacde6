"""Whole HMC trajectories of small FP32 regressions (csrc/logreg_leapfrog.cuh):
row counts around a tile and where the splits outnumber one thread's additions,
clusters of one to eight CTAs, several chains a cluster, and sizes past them that
keep a launch per step.

The proposal's gradient must be the single evaluation's to the bit and its
log-density to float64 rounding (the same terms in another float64 order: 2^-44 of
the sum of magnitudes is ample); the trajectory, replayed with single evaluations
and float64 updates, within 2^-20 of its largest state for each step (a float32
update rounds at 2^-24, and the steps are stable)."""
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


@pytest.mark.parametrize('n,d,c,steps', [
    (1, 1, 1, 1), (63, 2, 3, 5), (64, 25, 64, 2), (65, 24, 16, 4), (130, 128, 20, 3),
    (500, 3, 16, 7), (1000, 25, 64, 10), (1000, 60, 128, 4), (1999, 60, 33, 3), (2000, 33, 130, 3),
    (2000, 100, 64, 3), (2049, 128, 7, 2), (4095, 25, 64, 3), (4095, 128, 5, 2), (4095, 100, 300, 2),
    (300, 10, 700, 3), (300, 10, 2500, 2), (5000, 10, 16, 2)])
@pytest.mark.parametrize('per_chain', [False, True])
def test_trajectory(pg, n, d, c, steps, per_chain):
  g = torch.Generator('cuda').manual_seed(n + d + c)
  X = torch.randn(n, d, generator=g, device='cuda')
  y = (torch.rand(n, generator=g, device='cuda') < 0.4).float()
  q = 0.3 * torch.randn(c, d, generator=g, device='cuda') / d ** 0.5
  t = pg.LogisticRegression(X, y)
  eps = 0.1 / n ** 0.5
  e = eps * (1.0 + torch.arange(c, device='cuda').float() / c) if per_chain else eps
  k = pg.mcmc.UncalibratedHamiltonianMonteCarlo(t, step_size=e, num_leapfrog_steps=steps)
  kr0 = k.bootstrap_results(q)
  state, kr = k.one_step(q, kr0, seed=(5, 6))
  lp, grad = t.log_prob_and_grad(state)
  assert torch.equal(kr.grads_target_log_prob, grad)
  z = X.double() @ state.double().T
  size = torch.nn.functional.softplus(z.abs()).sum(0) + (state.double() ** 2).sum(1) + d + 1
  size = size + (X.double().T @ (y.double() - 0.5)).abs() @ state.double().abs().T
  assert ((kr.target_log_prob - lp).abs() <= 2.0 ** -44 * size).all()
  # Replay.
  e64 = (e if per_chain else torch.full((c,), eps, device='cuda')).float().double()[:, None]
  x, p = q.double(), kr.initial_momentum.double()
  p = p + 0.5 * e64 * kr0.grads_target_log_prob.double()
  for i in range(steps):
    x = (x + e64 * p).float().double()
    gr = t.log_prob_and_grad(x.float())[1].double()
    p = (p + (e64 if i + 1 < steps else 0.5 * e64) * gr).float().double()
  bound = steps * 2.0 ** -20
  assert ((state - x).abs() <= bound * x.abs().max()).all()
  assert ((kr.final_momentum - p).abs() <= bound * p.abs().max()).all()
