"""The choice of the real blocked loop's K between time and rounding (CPU)."""
import pytest

from qspectra_gb300 import _native
from qspectra_gb300.simulate import ensemble as ens


@pytest.mark.parametrize('m,nsel', [(9, 3), (25, 5), (25, 25), (49, 7), (64, 8)])
def test_the_tensor_core_build_ends_at_nine_steps(m, nsel, monkeypatch):
    for K in range(2, 65):
        supported = _native.rk4_block_matrix_real_tc_supported(m, K, nsel)
        assert ens._tensor_core_build(m, K, nsel) == (supported and K <= 9)
        monkeypatch.setattr(ens, '_PINNED_K_REAL', K)
        assert ens._tensor_core_build(m, K, nsel) == supported
        monkeypatch.setattr(ens, '_PINNED_K_REAL', None)
    # what the tuner times: K past 9 at the CUDA-core build's cost alone
    tc = lambda k: ens._tensor_core_build(m, k, nsel)  # noqa: E731
    for K in ens.block_k_real_candidates(999, m, nsel, tc):
        assert K <= 9 or not tc(K)


@pytest.mark.parametrize('times,choice', [
    ({5: 0.262, 6: 0.283}, 6), ({5: 0.389, 6: 0.461}, 5), ({5: 0.5, 6: 0.4}, 6),
    ({4: 0.3, 5: 0.2}, 5), ({6: 0.3, 7: 0.2}, 7), ({8: 0.19, 9: 0.2, 10: 0.2, 12: 0.21}, 10)])
def test_a_small_gain_does_not_buy_rounding(times, choice):
    tensor_core = lambda K: K in (2, 3, 4, 5, 8, 9)  # noqa: E731
    assert ens._measured_choice(times, tensor_core) == choice
    assert ens._measured_choice(times, None) == min(times, key=times.get)
