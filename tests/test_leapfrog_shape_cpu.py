"""The shape of an HMC trajectory's launch (csrc/logreg_leapfrog.cuh), on the host:
what it accepts must fit an SM's shared memory, whatever the number of rows."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r'''
#include <cstdio>
#include "logreg_leapfrog.cuh"
// Reads "rows features chains" lines; prints K G S rowpad smax bytes, or 0.
int main() {
  long long n;
  int d, c;
  while (scanf("%lld %d %d", &n, &d, &c) == 3) {
    gbm::LeapShape h;
    if (gbm::leap_shape(n, d, c, 152, 128, &h))
      printf("%d %d %d %d %d %lld\n", h.K, h.G, h.S, h.rowpad, h.smax, (long long)h.bytes());
    else
      printf("0\n");
  }
}
'''


@pytest.fixture(scope='module')
def shapes(tmp_path_factory):
  from probability_gb300 import build
  try:
    cc = build.nvcc()
  except RuntimeError as e:
    pytest.skip(str(e))
  d = tmp_path_factory.mktemp('leap_shape')
  src, exe = str(d / 'shape.cu'), str(d / 'shape')
  open(src, 'w').write(PROGRAM)
  subprocess.run([cc, src, '-o', exe] + build._flags(), check=True, capture_output=True)

  def run(cases):
    text = ''.join('%d %d %d\n' % c for c in cases)
    out = subprocess.run([exe], input=text, check=True, capture_output=True, text=True).stdout
    return [[int(v) for v in line.split()] for line in out.splitlines()]
  return run


def _bytes(n, d, K, G, S, rowpad, smax):
  threads = 512
  floats = d * rowpad + rowpad + G * rowpad + G * rowpad // 4 + 2 * smax * G * d + 2 * G * d
  return 4 * ((floats + 1) // 2 * 2 + 2 * G * (1 + threads // 32))


def test_accepted_shapes_fit(shapes):
  # Rows from one to past 2^32 elements, some of which wrap a 32-bit product.
  cases = [(40517394, 100, 64)]
  for d in (1, 3, 16, 25, 100, 128):
    for n in (1, 64, 1000, 4095, 5000, 20000, 33554432 // d, 1 << 24, (1 << 31) // d + 1,
              (1 << 32) // d + 12345):
      for c in (1, 64, 700, 20000):
        if n < (1 << 31) - 256:
          cases.append((n, d, c))
  # The rows whose d * stride is a multiple of 2^32 but for a few kilobytes.
  for k in (1, 2, 3):
    for off in range(-40, 400, 17):
      cases.append((max(1, ((1 << 32) * k // 100 + off) // 64 * 64), 100, 64))
  accepted = 0
  for (n, d, c), h in zip(cases, shapes(cases)):
    if h == [0]:
      continue
    accepted += 1
    assert h[5] == _bytes(n, d, *h[:5]) and h[5] <= 227 * 1024, (n, d, c, h)
    assert h[0] * h[3] >= n, (n, d, c, h)     # the cluster holds every row
  assert accepted >= 20
