"""Whole NUTS trajectories of a hierarchical-normal chain in one warp
(csrc/nuts_chain.cu) against the batched kernels, which a sampler with
profiling on still uses: the same draws give the same trees (mcmc/nuts.py:
321-1010), state bits included.  Only the float64 log-density differs, by
rounding of its prior term: each side rounds a sum of a few terms below
~1e4, a few ulps of 2^-40, so 1e-11 absolute."""
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


def _target(pg, groups, seed):
  rng = np.random.default_rng(seed)
  sigma = rng.uniform(5, 20, groups)
  return pg.NonCentredHierarchicalNormal(4 + 6 * rng.normal(size=groups), sigma)


def _batched(pg, kernel, on):
  pg._native.check(pg._native.lib().gbm_nuts_set_profiling(kernel._handle, int(on)))


def _same(a, b):
  for x, y in zip(a, b):
    if x.dtype == torch.float64:
      np.testing.assert_allclose(x.cpu().numpy(), y.cpu().numpy(), rtol=0, atol=1e-11)
    else:
      assert torch.equal(x, y)


def _results(q, kr):
  return [q, kr.grads_target_log_prob, kr.target_log_prob, kr.energy, kr.leapfrogs_taken,
          kr.is_accepted, kr.reach_max_depth, kr.has_divergence]


# 32 elements and fewer live in registers, 1024 is the longest vector held.
@pytest.mark.parametrize('groups', [1, 3, 8, 30, 31, 62, 63, 510, 1022, 1023])
@pytest.mark.parametrize('mass', [False, True])
def test_transition_matches_batched(pg, groups, mass):
  t = _target(pg, groups, groups)
  C, D = 67, groups + 2
  g = torch.Generator('cuda').manual_seed(groups)
  q = torch.randn(C, D, generator=g, device='cuda') * 0.7
  k = pg.mcmc.NoUTurnSampler(t, step_size=0.15, max_tree_depth=6)
  kr = k.bootstrap_results(q)
  k._ensure(C)
  im = torch.rand(D, generator=g, device='cuda') + 0.5
  if mass:
    pg._native.check(pg._native.lib().gbm_nuts_set_inverse_mass(
        k._handle, pg._native.ptr(im), 0))
  out = []
  for batched in (False, True):
    _batched(pg, k, batched)
    q1, kr1 = k.one_step(q, kr, seed=(3, groups))
    out.append(_results(q1, kr1) + [torch.tensor(k.last_leaf_iterations)])
    run = k.run_free(q, kr, 3, (5, groups))
    out[-1] += [run.all_states, run.transitions_done] + [run.trace[x] for x in sorted(run.trace)]
  _same(*out)


def test_mixed_batch_and_budget_match_batched(pg):
  """Hierarchical members run whole, the normals leaf by leaf, beside them."""
  rng = np.random.default_rng(2)
  members = []
  for d, c in ((5, 9), (40, 6)):
    A = rng.standard_normal((d, d + 2)) / np.sqrt(d)
    members.append((pg.MultivariateNormalTriL(rng.normal(size=d), np.linalg.cholesky(A @ A.T)), c))
  members += [(_target(pg, 8, 1), 12), (_target(pg, 100, 2), 5), (_target(pg, 1100, 3), 2)]
  batch = pg.TargetBatch(members)
  q = batch.pack([torch.from_numpy((0.5 * rng.normal(size=(c, t.event_dim))).astype(np.float32))
                  for t, c in members]).cuda()
  k = pg.BatchedNoUTurnSampler(batch, step_size=[0.3, 0.1, 0.2, 0.15, 0.1], max_tree_depth=7)
  kr = k.bootstrap_results(q)
  out = []
  for batched in (False, True):
    _batched(pg, k, batched)
    q1, kr1 = k.one_step(q, kr, seed=(8, 8))
    out.append(_results(q1, kr1) + [torch.tensor(k.last_leaf_iterations)])
    for budget in (1 << 40, 21):
      run = k.run_free(q, kr, 4, (6, 2), max_leaf_iterations=budget)
      done = run.transitions_done
      keep = torch.arange(4, device='cuda')[:, None] < done[None, :]
      out[-1] += [done, torch.tensor(run.leaf_iterations)]
      out[-1] += [torch.where(keep, run.trace[x], 0) for x in ('leapfrogs_taken', 'is_accepted')]
      if budget > 21:
        out[-1].append(run.all_states)
  _same(*out)
