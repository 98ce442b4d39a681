"""The tensor-pipe recurrence (csrc/lstm_rec_tc.cu) at widths in whole 64 units, which have instances of their own, and at one beside them: the last group of columns
full, with one column, empty.  All steps against the oracle."""
import pytest

import test_gpu_lstm_rec as rec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("I,H,B,T,mask", [(24, 64, 1040, 8, "full"), (16, 128, 497, 9, None), (24, 192, 305, 8, "one"), (16, 256, 497, 8, "full"), (20, 256, 528, 8, None),
                                          (20, 224, 305, 8, "full")])
def test_widths_in_whole_64_units(oracle, I, H, B, T, mask):
    import gpu_util as g
    g.ctx()
    try:
        rec.test_recurrence_matches_oracle(oracle, g, I, H, B, T, mask)
    finally:
        g.release()
