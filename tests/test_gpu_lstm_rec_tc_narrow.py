"""The tensor-pipe recurrence (csrc/lstm_rec_tc.cu) at fewer than 64 units, whose forward kernel keeps a step's inputs in registers: units that fill no CTA, the last
group of columns full, with one column, empty.  All steps against the oracle."""
import pytest

import test_gpu_lstm_rec as rec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("I,H,B,T,mask", [(12, 1, 1200, 8, None), (12, 31, 1217, 8, "full"), (16, 32, 1216, 9, None), (16, 33, 625, 9, "one"), (20, 48, 640, 8, "full"),
                                          (24, 63, 609, 8, None)])
def test_fewer_than_64_units(oracle, I, H, B, T, mask):
    import gpu_util as g
    g.ctx()
    try:
        rec.test_recurrence_matches_oracle(oracle, g, I, H, B, T, mask)
    finally:
        g.release()
