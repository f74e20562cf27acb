"""Host tables against their definitions, element by element."""
import itertools

import numpy as np
import pytest

from qspectra_gb300.dynamics.liouville_space import liouville_subspace_index
from qspectra_gb300.operator_tools import (SubspaceError, n_excitations, transition_operator,
                                            transition_sum)


@pytest.mark.parametrize('n', [1, 2, 5])
@pytest.mark.parametrize('transitions', ['-+', '-', '+', ''])
@pytest.mark.parametrize('subspace', ['g', 'e', 'f', 'ge', 'eg', 'gf', 'ef', 'gef', 'feg'])
def test_transition_sum(n, transitions, subspace):
    rng = np.random.RandomState(n)
    for weights in (rng.randn(n), rng.randn(n) + 1j * rng.randn(n), np.arange(n)):
        ref = sum(weights[i] * transition_operator(i, n, subspace, transitions) for i in range(n))
        out = transition_sum(weights, n, subspace, transitions)
        assert out.dtype == ref.dtype and np.array_equal(out, ref)


@pytest.mark.parametrize('n,vib', [(1, 1), (3, 1), (4, 2)])
def test_liouville_subspace_index(n, vib):
    for full in ('g', 'e', 'ge', 'ef', 'gef'):
        sizes = [int(s) for c, s in zip('gef', n_excitations(n, vib)) if c in full]
        letter = np.repeat(list(full), sizes)
        blocks = [a + b for a, b in itertools.product(full, repeat=2)]
        for k in (1, 2, 3):
            for pick in itertools.product(blocks, repeat=k):
                ref = [a + len(letter) * b for b in range(len(letter)) for a in range(len(letter))
                       if letter[a] + letter[b] in pick]
                out = liouville_subspace_index(','.join(pick), full, n, vib)
                assert out.dtype == np.int64 and np.array_equal(out, ref)
                if k == 3 and len(full) == 3:
                    break
    with pytest.raises(SubspaceError):
        liouville_subspace_index('ef', 'ge', n, vib)
