"""The clusters that a recurrence of constant width is dealt over (csrc/lstm_rec.cu): widths around those where the columns of the fullest
cluster change, so that the last cluster has as many columns as the others or one alone, against the oracle's node chain."""
import pytest

from test_gpu_lstm_rec import _release, g, test_recurrence_matches_oracle as matches_oracle   # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,N", [(60, 2), (60, 75), (256, 14), (256, 15), (256, 16), (256, 17), (256, 31), (256, 33), (300, 12), (300, 13), (300, 29), (300, 31), (300, 45)])
def test_widths_around_the_cluster_counts(oracle, g, H, N):   # noqa: F811
    matches_oracle(oracle, g, 24, H, N, 8, None)
