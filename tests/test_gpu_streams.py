"""Samplers called from another stream than their target's: the transition waits for
what the caller has queued (arguments, and what the call itself makes of them, a
scalar step size among it) and the caller's stream for the results.  Every result
equals the call from the target's own stream, while first the caller's and then the
target's stream is held up for a while."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

_HOLD = 100_000_000   # clocks, about 50 ms


@pytest.fixture(scope='module')
def pg():
  if not torch.cuda.is_available():
    pytest.skip('no CUDA device')
  import probability_gb300 as pg
  return pg


def _problem(n=700, d=6, c=40):
  g = torch.Generator('cuda').manual_seed(11)
  X = torch.randn(n, d, generator=g, device='cuda')
  y = (torch.rand(n, generator=g, device='cuda') < 0.4).float()
  return X, y, 0.3 * torch.randn(c, d, generator=g, device='cuda')


def _tensors(x):
  if isinstance(x, torch.Tensor):
    return [x]
  if isinstance(x, dict):
    return [t for k in sorted(x) for t in _tensors(x[k])]
  if isinstance(x, (list, tuple)):
    return [t for v in x for t in _tensors(v)]
  return []


def _calls(pg, kind, target):
  """call(q as the caller has it) -> results."""
  if kind.startswith('hmc'):
    cls = (pg.mcmc.UncalibratedHamiltonianMonteCarlo if 'uncalibrated' in kind
           else pg.mcmc.HamiltonianMonteCarlo)
    step = [0.02] if 'list' in kind else 0.02
    k = cls(target, step_size=step, num_leapfrog_steps=4)
  elif kind == 'hierarchical':
    t = pg.NonCentredHierarchicalNormal([3., 8., -1., 2.], [10., 12., 9., 11.])
    k = pg.mcmc.NoUTurnSampler(t, step_size=0.2, max_tree_depth=5)
  else:
    k = pg.mcmc.NoUTurnSampler(target, step_size=0.02, max_tree_depth=4)

  def one_step(q):
    kr = k.bootstrap_results(q)
    q1, kr1 = k.one_step(q, kr, seed=(3, 4))
    return k.one_step(q1, kr1, seed=(5, 6))

  if kind == 'run_chain':
    k = pg.mcmc.HamiltonianMonteCarlo(target, step_size=0.02, num_leapfrog_steps=3)
    return lambda q: tuple(pg.mcmc.run_chain(k, 3, q, seed=(1, 2)))
  if kind == 'run_free':
    return lambda q: tuple(k.run_free(q, k.bootstrap_results(q), 3, (7, 8)))
  return one_step


@pytest.mark.parametrize('kind', ['hmc', 'hmc list', 'hmc uncalibrated', 'nuts', 'hierarchical',
                                  'run_chain', 'run_free'])
def test_called_from_another_stream(pg, kind):
  X, y, q = _problem()
  call = _calls(pg, kind, pg.LogisticRegression(X, y))
  want = [t.clone() for t in _tensors(call(q))]
  torch.cuda.synchronize()
  own, other = torch.cuda.current_stream(), torch.cuda.Stream()
  for held in (other, own):
    # Freed memory that the allocator hands out again: a step size read before it
    # is written is not the last call's.
    junk = torch.full((1 << 16,), float('nan'), device='cuda')
    with torch.cuda.stream(other):
      junk2 = torch.full((1 << 16,), float('nan'), device='cuda')
    torch.cuda.synchronize()
    del junk, junk2
    with torch.cuda.stream(held):
      torch.cuda._sleep(_HOLD)
    with torch.cuda.stream(other):
      mine = q + 0.0                       # an argument that the caller has just queued
      got = [t.clone() for t in _tensors(call(mine))]
    other.synchronize()
    assert len(got) == len(want)
    for a, b in zip(got, want):
      assert torch.equal(a, b)
    torch.cuda.synchronize()
