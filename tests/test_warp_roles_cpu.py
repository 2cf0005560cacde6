"""Roles of one lane in the tensor-core kernels, checked in their source: a warp
whose single lane loads or issues goes on to barriers and TMEM instructions that
want it converged (.aligned), so such a branch ends with __syncwarp()."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    'probability_gb300', 'csrc')
FILES = ['grad_tc.cuh', 'logreg_f32.cu', 'logreg_tc.cu']
# A role's branch: first in `if (warp ...) {`, after at most a comment line.
ROLE = re.compile(r'^  (?:\} else )?if \(warp [^\n]*\{\n(?:    //[^\n]*\n)?'
                  r'    if \((?:lane == 0|tc::elect_one\(\))\) \{\n', re.M)


@pytest.mark.parametrize('name', FILES)
def test_single_lane_roles_reconverge(name):
  src = open(os.path.join(CSRC, name)).read()
  roles = list(ROLE.finditer(src))
  assert len(roles) >= {'grad_tc.cuh': 2, 'logreg_f32.cu': 1, 'logreg_tc.cu': 6}[name]
  for m in roles:
    end = src.index('\n    }\n', m.end())
    after = src[end + len('\n    }\n'):].lstrip(' ')
    line = src.count('\n', 0, m.start()) + 1
    assert after.startswith('__syncwarp();'), '%s:%d' % (name, line)
