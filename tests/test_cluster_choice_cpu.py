"""The choice of a cluster size on the host: sizes that cannot be had."""
import os
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "cluster_choice.h"
// batch, smallest size that holds a sample, largest one with work, then the
// clusters of 1, 2, 4 and 8 CTAs that run at once (0: not at all, or an error)
int main(int, char** v) {
  const int need = atoi(v[2]), top = atoi(v[3]);
  auto at_once = [&](int c) { return atoi(v[c == 1 ? 4 : c == 2 ? 5 : c == 4 ? 6 : 7]); };
  printf("%d", qsx::choose_cluster(atoi(v[1]), 8, [&](int c) { return c >= need; },
                                   [&](int c) { return 2 * c <= top; }, at_once));
}
"""


@pytest.fixture(scope='module')
def choose(tmp_path_factory):
    d = tmp_path_factory.mktemp('cluster_choice')
    (d / 'main.cpp').write_text(PROGRAM)
    subprocess.run(['g++', '-std=c++17', '-I', os.path.join(ROOT, 'qspectra_gb300', 'csrc'),
                    str(d / 'main.cpp'), '-o', str(d / 'main')], check=True)
    return lambda *a: int(subprocess.run([str(d / 'main')] + [str(x) for x in a], check=True,
                                         capture_output=True, text=True).stdout)


@pytest.mark.parametrize('args,size', [
    ((1, 1, 8, 152, 70, 34, 16), 8),       # one sample: every CTA there is work for
    ((64, 4, 8, 152, 70, 34, 16), 4),      # the samples would not all run at once
    ((30, 1, 8, 152, 70, 34, 16), 4),
    ((1, 1, 2, 152, 70, 34, 16), 2),
    ((1, 1, 8, 152, 70, 0, 16), 2),        # the larger one fails: the last good one
    ((300, 1, 8, 152, 70, 34, 16), 1),
    ((1, 4, 8, 152, 70, 0, 16), 0),        # the first one fails: another form
    ((1, 16, 16, 152, 70, 34, 16), 0),     # no cluster holds a sample
])
def test_sizes_that_cannot_be_had(choose, args, size):
    assert choose(*args) == size
