"""The clusters that the columns of a recurrence are dealt over (csrc/lstm_rec.cu): widths around those where the columns of the fullest
cluster change, so that the last cluster has as many columns as the others or one alone, against the oracle's node chain; and ragged batches,
one block of columns per cluster and more, against the oracle sentence by sentence."""
import pytest

from test_gpu_lstm_rec import _release, g, test_recurrence_matches_oracle as matches_oracle   # noqa: F401  (fixtures)
from test_gpu_tagger import test_tagger_driver_matches_per_sentence_oracle as tagger_matches_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,N", [(60, 2), (60, 75), (256, 14), (256, 15), (256, 16), (256, 17), (256, 31), (256, 33), (300, 12), (300, 13), (300, 29), (300, 31), (300, 45)])
def test_widths_around_the_cluster_counts(oracle, g, H, N):   # noqa: F811
    matches_oracle(oracle, g, 24, H, N, 8, None)


@pytest.mark.parametrize("H,S,lo,hi", [(256, 2, 1, 30), (256, 13, 3, 30), (256, 16, 9, 30), (256, 17, 3, 30), (256, 29, 1, 30), (300, 11, 3, 20), (300, 60, 1, 20)])
def test_ragged_batches(oracle, H, S, lo, hi):
    tagger_matches_oracle(oracle, (60, 20, H, 6, 5), S, lo, hi)
