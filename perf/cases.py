"""The calls whose speed is measured: gradient-MCMC work as users run it.

A case is a dict of plain values.  `listed()` names them, `draw(rng)` makes
one more of the same ranges, `prepare` builds what a program holds before the
call (targets, kernels, states, kernel results), `run` is one pass through
the public entry points, `work` is what that pass cannot do without, and
`exact` is what it returns in 64-bit arithmetic, by plain torch.
"""
import math

import numpy as np
import torch

import probability_gb300 as pg


def listed():
  return [
      # One HMC transition of the smallest regression in use (1000 x 25, 64
      # chains, 10 leapfrog steps): launches and latency.
      dict(name='hmc_1000x25_c64', kind='hmc', n=1000, d=25, chains=64, step=0.03, leapfrogs=10),
      # One NUTS transition of the eight-schools model on a few hundred
      # chains: a whole tree per call, small vectors, latency again.
      dict(name='nuts_schools_c256', kind='nuts', groups=8, chains=256, step=0.25),
      # Free-running NUTS over a ragged batch of hierarchical posteriors (the
      # sampler's own kernels: half of a many-posterior batch).
      dict(name='free_hier_16', kind='free', members=16, groups_max=512, chains_max=512, step=0.2,
           transitions=4),
      # FP32 log-density + gradient of the plain NUTS workload (1e5 x 100,
      # 1024 chains): where that sampler's time goes.
      dict(name='fp32_1e5x100_c1024', kind='logreg', data='f32', precision='fp32', n=100000, d=100,
           chains=1024),
      # FP32 regressions with more features, odd sizes: the fused kernel's
      # upper range and the range above it.
      dict(name='fp32_30011x237_c192', kind='logreg', data='f32', precision='fp32', n=30011, d=237,
           chains=192),
      dict(name='fp32_12289x601_c99', kind='logreg', data='f32', precision='fp32', n=12289, d=601,
           chains=99),
      # Mixed precision on FP32 data, the same workload as the FP32 one.
      dict(name='mixed_1e5x100_c1024', kind='logreg', data='f32', precision='mixed', n=100000,
           d=100, chains=1024),
      # Mixed precision on BF16 data: the tall workload, all its chains.
      dict(name='bf16_1e6x512_c4096', kind='logreg', data='bf16', precision='mixed', n=1000000,
           d=512, chains=4096),
      # Two requests of a serving stream (rows 1e3..2e5, features 10..1000,
      # 16..256 chains): a middling one and a wide one.
      dict(name='bf16_12007x173_c77', kind='logreg', data='bf16', precision='mixed', n=12007, d=173,
           chains=77),
      dict(name='bf16_65371x929_c240', kind='logreg', data='bf16', precision='mixed', n=65371,
           d=929, chains=240),
      # One multivariate normal, odd dimension.
      dict(name='mvn_777_c350', kind='mvn', d=777, chains=350),
      # Log-density + gradient of a ragged batch: normals of dimension 8..2048
      # and hierarchical models of 8..512 groups, 32..512 chains each.
      dict(name='batch_24', kind='batch', members=24, d_max=2048, groups_max=512, chains_max=512),
  ]


def _log_int(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  k = rng.choice(['hmc', 'nuts', 'free', 'fp32', 'fp32_wide', 'mixed', 'serve', 'tall', 'mvn',
                  'batch'])
  if k == 'hmc':
    return dict(kind='hmc', n=_log_int(rng, 500, 2000), d=rng.randint(3, 60),
                chains=_log_int(rng, 16, 128), step=0.03, leapfrogs=rng.randint(5, 15))
  if k == 'nuts':
    return dict(kind='nuts', groups=_log_int(rng, 4, 128), chains=_log_int(rng, 32, 2048),
                step=0.25)
  if k == 'free':
    return dict(kind='free', members=rng.randint(4, 24), groups_max=_log_int(rng, 32, 512),
                chains_max=_log_int(rng, 64, 512), step=0.2, transitions=rng.randint(2, 5))
  if k == 'fp32':
    return dict(kind='logreg', data='f32', precision='fp32', n=_log_int(rng, 1000, 200000),
                d=_log_int(rng, 4, 128), chains=_log_int(rng, 16, 2048))
  if k == 'fp32_wide':
    return dict(kind='logreg', data='f32', precision='fp32', n=_log_int(rng, 2000, 60000),
                d=_log_int(rng, 129, 1000), chains=_log_int(rng, 16, 256))
  if k == 'mixed':
    return dict(kind='logreg', data='f32', precision='mixed', n=_log_int(rng, 1000, 200000),
                d=_log_int(rng, 10, 128), chains=_log_int(rng, 16, 2048))
  if k == 'serve':
    return dict(kind='logreg', data='bf16', precision='mixed', n=_log_int(rng, 1000, 200000),
                d=_log_int(rng, 10, 1000), chains=_log_int(rng, 16, 256))
  if k == 'tall':
    return dict(kind='logreg', data='bf16', precision='mixed', n=_log_int(rng, 100000, 1000000),
                d=rng.randint(257, 512), chains=_log_int(rng, 256, 4096))
  if k == 'mvn':
    return dict(kind='mvn', d=_log_int(rng, 8, 2048), chains=_log_int(rng, 32, 512))
  return dict(kind='batch', members=rng.randint(4, 32), d_max=_log_int(rng, 64, 2048),
              groups_max=_log_int(rng, 32, 512), chains_max=_log_int(rng, 64, 512))


# ---- inputs ----------------------------------------------------------------
def _regression(case, seed):
  """X [N, D] with an intercept column and entries N(0, 1/D), labels from a
  true beta ~ N(0, 1), states near it, as a running sampler holds them."""
  g = torch.Generator('cuda').manual_seed(seed)
  n, d = case['n'], case['d']
  dt = torch.bfloat16 if case.get('data') == 'bf16' else torch.float32
  X = torch.empty(n, d, dtype=dt, device='cuda')
  scale = 1.0 if case['kind'] == 'hmc' else d ** -0.5
  beta = torch.randn(d, generator=g, device='cuda')
  y = torch.empty(n, device='cuda')
  for r in range(0, n, 1 << 18):
    m = min(1 << 18, n - r)
    block = torch.randn(m, d, generator=g, device='cuda') * scale
    block[:, 0] = 1.0
    X[r:r + m] = block.to(dt)
    p = torch.sigmoid(X[r:r + m].float() @ beta)
    y[r:r + m] = (torch.rand(m, generator=g, device='cuda') < p).float()
  noise = torch.randn(case['chains'], d, generator=g, device='cuda')
  q = 0.1 * noise if case['kind'] == 'hmc' else beta + 0.1 * noise
  return X, y, q.contiguous()


def _normal(d, seed):
  """loc and the Cholesky factor of a Wishart(d + 2, I/d) covariance (its
  Bartlett factor)."""
  rng = np.random.default_rng([seed, d])
  L = np.tril(rng.standard_normal((d, d)), -1)
  L[np.diag_indices(d)] = np.sqrt(rng.chisquare(d + 2 - np.arange(d)))
  return rng.standard_normal(d), L / math.sqrt(d)


def _normal_states(loc, L, chains, seed):
  g = torch.Generator('cuda').manual_seed(seed)
  z = torch.randn(chains, len(loc), generator=g, device='cuda', dtype=torch.float64)
  x = torch.as_tensor(loc, device='cuda') + z @ torch.as_tensor(L, device='cuda').T
  return x.float().contiguous()


def _groups(j, seed):
  rng = np.random.default_rng([seed, j])
  sigma = rng.uniform(5, 20, j).astype(np.float32)
  theta = 4.0 + 5.0 * rng.standard_normal(j)
  return (theta + sigma * rng.standard_normal(j)).astype(np.float32), sigma


def _group_states(j, chains, seed):
  g = torch.Generator('cuda').manual_seed(seed)
  q = torch.randn(chains, j + 2, generator=g, device='cuda')
  q[:, 0] = 4.0 + 3.0 * q[:, 0]
  q[:, 1] = 1.0 + 0.5 * q[:, 1]
  return q.contiguous()


def _members(case, seed):
  """[(family, dim or groups, chains)]: the shapes are the case's, whatever the seed."""
  rng = np.random.default_rng([case['members'], case['groups_max'], case['chains_max']])
  out = []
  for i in range(case['members']):
    chains = int(rng.integers(32, case['chains_max'] + 1))
    groups = int(rng.integers(8, case['groups_max'] + 1))
    if case['kind'] == 'batch' and i % 2 == 0:
      top = math.log(case['d_max'])
      d = case['d_max'] if i == 0 else int(round(math.exp(rng.uniform(math.log(8), top))))
      out.append(('mvn', d, chains))
    else:
      out.append(('hier', groups, chains))
  return out


def prepare(case, seed):
  kind = case['kind']
  if kind in ('logreg', 'hmc'):
    X, y, q = _regression(case, seed)
    target = pg.LogisticRegression(X, y, precision=case.get('precision', 'fp32'))
    if kind == 'logreg':
      return dict(kind=kind, target=target, q=q)
    kernel = pg.mcmc.HamiltonianMonteCarlo(target, step_size=case['step'],
                                           num_leapfrog_steps=case['leapfrogs'])
    return dict(kind=kind, kernel=kernel, q=q, kr=kernel.bootstrap_results(q), seed=(seed, 17))
  if kind == 'mvn':
    loc, L = _normal(case['d'], seed)
    return dict(kind=kind, target=pg.MultivariateNormalTriL(loc, L),
                q=_normal_states(loc, L, case['chains'], seed))
  if kind == 'nuts':
    target = pg.NonCentredHierarchicalNormal(*_groups(case['groups'], seed))
    kernel = pg.mcmc.NoUTurnSampler(target, step_size=case['step'], max_tree_depth=10)
    q = _group_states(case['groups'], case['chains'], seed)
    return dict(kind=kind, kernel=kernel, q=q, kr=kernel.bootstrap_results(q), seed=(seed, 29))
  members, states = [], []
  for i, (family, d, chains) in enumerate(_members(case, seed)):
    if family == 'mvn':
      loc, L = _normal(d, seed + i)
      members.append((pg.MultivariateNormalTriL(loc, L), chains))
      states.append(_normal_states(loc, L, chains, seed + i))
    else:
      members.append((pg.NonCentredHierarchicalNormal(*_groups(d, seed + i)), chains))
      states.append(_group_states(d, chains, seed + i))
  batch = pg.TargetBatch(members)
  q = batch.pack(states)
  if kind == 'batch':
    return dict(kind=kind, target=batch, q=q)
  kernel = pg.BatchedNoUTurnSampler(batch, step_size=[case['step']] * len(members),
                                    max_tree_depth=10)
  return dict(kind=kind, kernel=kernel, q=q, kr=kernel.bootstrap_results(q), seed=(seed, 43),
              transitions=case['transitions'])


def run(state):
  kind = state['kind']
  if kind in ('logreg', 'mvn', 'batch'):
    log_prob, grad = state['target'].log_prob_and_grad(state['q'])
    return [log_prob, grad]
  if kind == 'hmc':
    q, kr = state['kernel'].one_step(state['q'], state['kr'], seed=state['seed'])
    a, p = kr.accepted_results, kr.proposed_results
    return [q, a.target_log_prob, a.grads_target_log_prob, kr.proposed_state, p.target_log_prob,
            p.grads_target_log_prob, p.initial_momentum, p.final_momentum, kr.log_accept_ratio,
            kr.is_accepted]
  if kind == 'nuts':
    q, kr = state['kernel'].one_step(state['q'], state['kr'], seed=state['seed'])
    return [q, kr.target_log_prob, kr.grads_target_log_prob, kr.log_accept_ratio,
            kr.leapfrogs_taken, kr.is_accepted, kr.reach_max_depth, kr.has_divergence, kr.energy]
  r = state['kernel'].run_free(state['q'], state['kr'], state['transitions'], state['seed'])
  t = r.trace
  return [r.all_states, t['target_log_prob'], t['log_accept_ratio'], t['leapfrogs_taken'],
          t['is_accepted'], t['has_divergence'], r.transitions_done]


# ---- what a pass cannot do without ---------------------------------------------
# Leapfrog steps of a NUTS trajectory at the step sizes above (2^depth - 1
# with the usual depth); the trees themselves are drawn.
_NUTS_LEAVES = 15


def work(case):
  kind = case['kind']
  if kind in ('logreg', 'hmc'):
    n, d, c = case['n'], case['d'], case['chains']
    el = 2 if case.get('data') == 'bf16' else 4
    steps = case.get('leapfrogs', 1)
    flops = 4.0 * n * d * c * steps
    if kind == 'logreg':
      return dict(bytes=el * n * d + 4 * n + 8 * c * d + 8 * c, flops=flops)
    return dict(bytes=el * n * d + 4 * n + 4 * c * d * 8 + 50 * c, flops=flops)
  if kind == 'mvn':
    d, c = case['d'], case['chains']
    return dict(bytes=2.0 * d * (d + 1) + 4 * d + 8 * c * d + 8 * c, flops=2.0 * d * (d + 1) * c)
  if kind == 'nuts':
    j, c = case['groups'], case['chains']
    return dict(bytes=8 * j + 16 * c * (j + 2) + 60 * c, flops=16.0 * j * c * _NUTS_LEAVES)
  b = f = 0.0
  for family, d, c in _members(case, 0):
    if family == 'mvn':
      b += 2.0 * d * (d + 1) + 4 * d + 8 * c * d + 8 * c
      f += 2.0 * d * (d + 1) * c
    elif kind == 'batch':
      b += 8 * d + 8 * c * (d + 2) + 8 * c
      f += 10.0 * d * c
    else:
      k = case['transitions']
      b += 8 * d + 4 * c * (d + 2) * (2 + k) + 30 * c * k
      f += 16.0 * d * c * _NUTS_LEAVES * k
  return dict(bytes=b, flops=f)


# ---- the same in 64 bits -----------------------------------------------------------
def _logreg64(X, y, q):
  """log-density and gradient with a Normal(0, 1) prior; X in row blocks."""
  d = X.shape[1]
  lp = -0.5 * (q * q).sum(1) - 0.5 * d * math.log(2 * math.pi)
  grad = -q
  block = max(1024, (1 << 27) // max(q.shape[0], d))
  for r in range(0, X.shape[0], block):
    x, t = X[r:r + block].double(), y[r:r + block].double()
    z = x @ q.T
    lp = lp + t @ z - torch.nn.functional.softplus(z, threshold=1e9).sum(0)
    grad = grad + (t[:, None] - torch.sigmoid(z)).T @ x
  return lp, grad


def _mvn64(loc, L, q):
  loc, L = torch.as_tensor(loc, device='cuda'), torch.as_tensor(L, device='cuda')
  u = torch.linalg.solve_triangular(L, (q.double() - loc).T, upper=False)
  grad = -torch.linalg.solve_triangular(L.T, u, upper=True).T
  lp = -0.5 * (u * u).sum(0) - L.diagonal().log().sum() - 0.5 * len(loc) * math.log(2 * math.pi)
  return lp, grad


def _hier64(y, sigma, q):
  y, s = torch.as_tensor(y).cuda().double(), torch.as_tensor(sigma).cuda().double()
  q = q.double()
  mu, eta, z = q[:, 0], q[:, 1], q[:, 2:]
  tau = eta.exp()
  t2 = (tau / 5.0) ** 2
  res = (y - mu[:, None] - tau[:, None] * z) / s
  norm = 0.5 * math.log(2 * math.pi)
  lp = ((-0.5 * z * z - 0.5 * res * res - 2 * norm - s.log()).sum(1) - 0.5 * (mu / 5.0) ** 2
        - math.log(5.0) - norm + math.log(2 / math.pi) - math.log(5.0) - torch.log1p(t2) + eta)
  r = res / s
  g = torch.cat([(-mu / 25.0 + r.sum(1))[:, None],
                 (1 - 2 * t2 / (1 + t2) + tau * (r * z).sum(1))[:, None],
                 -z + tau[:, None] * r], 1)
  return lp, g


def _philox(key, elem, site):
  """Philox4x32-10 (Salmon et al. 2011), first two words; counter (elem, site, 0, 0)."""
  m, mask = np.uint64, np.uint64(0xFFFFFFFF)
  c = [elem.astype(np.uint64), np.full(elem.shape, site, np.uint64),
       np.zeros(elem.shape, np.uint64), np.zeros(elem.shape, np.uint64)]
  k0, k1 = m(key[0]), m(key[1])
  for _ in range(10):
    p0, p1 = m(0xD2511F53) * c[0], m(0xCD9E8D57) * c[2]
    c = [(p1 >> m(32)) ^ c[1] ^ k0, p1 & mask, (p0 >> m(32)) ^ c[3] ^ k1, p0 & mask]
    k0, k1 = (k0 + m(0x9E3779B9)) & mask, (k1 + m(0xBB67AE85)) & mask
  return c[0], c[1]


def _hmc64(case, seed):
  X, y, q32 = _regression(case, seed)
  c, d, key = case['chains'], case['d'], (seed & 0xFFFFFFFF, 17)
  a, b = _philox(key, np.arange(c * d), 1 << 24)                       # momentum draws
  u1 = ((a >> np.uint64(8)).astype(np.float64) + 1) * 2.0 ** -24
  u2 = (b >> np.uint64(8)).astype(np.float64) * 2.0 ** -24
  p0 = np.sqrt(-2 * np.log(u1)) * np.cos(2 * np.pi * u2)
  p0 = torch.as_tensor(p0.reshape(c, d)).cuda()
  u, _ = _philox(key, np.arange(c), 5 << 24)                           # accept uniforms
  u = torch.as_tensor((u >> np.uint64(8)).astype(np.float64) * 2.0 ** -24).cuda()
  eps = float(np.float32(case['step']))
  q0 = q32.double()
  l0, g0 = _logreg64(X, y, q0)
  q, p, g = q0, p0, g0
  for _ in range(case['leapfrogs']):
    p = p + 0.5 * eps * g
    q = q + eps * p
    l, g = _logreg64(X, y, q)
    p = p + 0.5 * eps * g
  lar = l - l0 + 0.5 * ((p0 * p0).sum(1) - (p * p).sum(1))
  acc = u.log() < lar
  m = acc[:, None]
  return [torch.where(m, q, q0), torch.where(acc, l, l0), torch.where(m, g, g0), q, l, g, p0, p,
          lar, None]


def exact(case, seed):
  kind = case['kind']
  if kind == 'logreg':
    X, y, q = _regression(case, seed)
    return list(_logreg64(X, y, q.double()))
  if kind == 'hmc':
    return _hmc64(case, seed)
  if kind == 'mvn':
    loc, L = _normal(case['d'], seed)
    return list(_mvn64(loc, L, _normal_states(loc, L, case['chains'], seed)))
  if kind == 'batch':
    lps, gs = [], []
    for i, (family, d, chains) in enumerate(_members(case, seed)):
      if family == 'mvn':
        loc, L = _normal(d, seed + i)
        lp, g = _mvn64(loc, L, _normal_states(loc, L, chains, seed + i))
      else:
        lp, g = _hier64(*_groups(d, seed + i), _group_states(d, chains, seed + i))
      lps.append(lp)
      gs.append(g.reshape(-1))
    return [torch.cat(lps), torch.cat(gs)]
  return None   # NUTS: the trees are decided by comparisons, leaf after leaf
