"""What the job server reckons a job takes (its admission control, its refusals and
the reported device_bytes) against what the job takes: the high-water mark of the
stream-ordered pool that all of a job's memory comes from.

The estimate must cover it, and by no more than a few buffers that are not all alive
at once (half of the truth again and 24 MB)."""
import ctypes

import numpy as np
import pytest

from tests import _problems

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

_USED_HIGH = 8    # CU_MEMPOOL_ATTR_USED_MEM_HIGH


class _Pool:
  """The device's default memory pool."""

  def __init__(self):
    self.cu = ctypes.CDLL('libcuda.so.1')
    self.pool = ctypes.c_void_p()
    assert self.cu.cuDeviceGetDefaultMemPool(ctypes.byref(self.pool),
                                             torch.cuda.current_device()) == 0

  def reset(self):
    zero = ctypes.c_uint64(0)
    assert self.cu.cuMemPoolSetAttribute(self.pool, _USED_HIGH, ctypes.byref(zero)) == 0

  def high(self):
    out = ctypes.c_uint64()
    assert self.cu.cuMemPoolGetAttribute(self.pool, _USED_HIGH, ctypes.byref(out)) == 0
    return out.value


@pytest.fixture(scope='module')
def pg():
  if not torch.cuda.is_available():
    pytest.skip('no CUDA device')
  import probability_gb300 as pg
  return pg


def _logreg(srv, n, d, chains, precision, dtype):
  X, y, _ = _problems.logreg_data(n, d, seed=d, scale=1.0 / np.sqrt(d))
  X = torch.from_numpy(X).cuda().to(dtype)
  return srv.submit_logistic_regression(X, y, _problems.init_state(chains, d, seed=1), 3,
                                        precision=precision, step_size=0.01, max_tree_depth=2,
                                        seed=(1, 1))


def _mvn(srv, d, chains):
  return srv.submit_mvn(np.zeros(d), np.eye(d), np.zeros((chains, d), np.float32), 3,
                        step_size=0.1, max_tree_depth=2, seed=(2, 2))


def _hier(srv, groups, chains):
  return srv.submit_hierarchical_normal(np.zeros(groups), np.full(groups, 10.0),
                                        np.zeros((chains, groups + 2), np.float32), 3,
                                        step_size=0.1, max_tree_depth=2, seed=(3, 3))


F32, BF16 = torch.float32, torch.bfloat16
JOBS = [('logreg', n, d, c, p, t) for n, d, c, p, t in [
    (200000, 20, 64, 'fp32', F32), (200000, 100, 64, 'fp32', F32), (3000, 128, 500, 'fp32', F32),
    (60000, 200, 100, 'fp32', F32), (3000, 256, 300, 'fp32', F32), (20000, 300, 64, 'fp32', F32),
    (20000, 1000, 100, 'fp32', F32), (2000, 700, 64, 'fp32', F32), (200000, 20, 64, 'mixed', F32),
    (200000, 100, 64, 'mixed', BF16), (100000, 200, 64, 'mixed', F32),
    (100000, 260, 64, 'mixed', BF16), (20000, 600, 64, 'mixed', F32),
    (20000, 1000, 64, 'mixed', BF16)]]
JOBS += [('mvn', d, c) for d, c in [(65, 64), (200, 500), (1000, 32), (2048, 16)]]
JOBS += [('hier', g, c) for g, c in [(8, 5000), (512, 700), (5000, 60)]]


@pytest.mark.parametrize('job', JOBS, ids=lambda j: '-'.join(str(v).split('.')[-1] for v in j))
def test_estimate_covers_the_job(pg, job):
  from probability_gb300.serving import Server, DONE
  submit = dict(logreg=_logreg, mvn=_mvn, hier=_hier)[job[0]]
  srv = Server(workers=1, memory_budget_bytes=32 * 2**30)
  torch.cuda.synchronize()
  pool = _Pool()
  pool.reset()
  info = submit(srv, *job[1:]).wait()
  used = pool.high()
  srv.close()
  assert info['status'] == DONE and used > 0
  assert used <= info['device_bytes'] <= 1.5 * used + 24 * 2**20


def test_regression_that_fits_without_its_pairs_is_admitted(pg):
  """A budget for X but not for X and its FP16 pairs: the job runs, without them."""
  from probability_gb300.serving import Server, DONE
  n, d, c = 400000, 100, 16
  srv = Server(workers=1, memory_budget_bytes=32 * 2**30)
  full = _logreg(srv, n, d, c, 'fp32', F32).wait()['device_bytes']
  srv.close()
  srv = Server(workers=1, memory_budget_bytes=int(0.75 * full))
  pool = _Pool()
  pool.reset()
  info = _logreg(srv, n, d, c, 'fp32', F32).wait()
  used = pool.high()
  srv.close()
  assert info['status'] == DONE and used <= info['device_bytes'] <= 0.75 * full
