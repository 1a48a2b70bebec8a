"""Which steps a scan goes through 32 tokens at a time, and which token by token: the sides of the rule's lines that were measured
(whole steps of two widths, one kernel alone), on the CPU."""
import pytest

from nanohybrid_vlm_b200.kernels import ops

NARROW, WIDE = 64, 128          # (head, 16 columns) of a request at widths 1,024 and 2,048
SMS = 148


@pytest.mark.parametrize("lengths,blocks,gated,mlstm", [
    ([128], WIDE, False, False), ([512], NARROW, False, False), ([512], WIDE, False, False),      # the host is what a step waits for
    ([768], NARROW, True, True), ([4096], WIDE, True, True),
    ([512] * 2, NARROW, False, False), ([512] * 2, WIDE, True, True),
    ([400] * 4, NARROW, False, False), ([400] * 4, WIDE, False, True),                            # every SM is full by tokens too
    ([512] * 8, WIDE, False, True), ([333, 625, 917, 1209, 1501], WIDE, True, True),
    ([1001] + [1] * 23, WIDE, False, True), ([32] * 48, WIDE, False, True), ([16] * 256, WIDE, False, False), ([1] * 64, WIDE, False, False)])
def test_rule(lengths, blocks, gated, mlstm):
    step = sum(lengths), len(lengths), max(lengths), blocks, SMS
    assert ops._by_chunks(*step, normed=False) == gated
    assert ops._by_chunks(*step, normed=True) == mlstm
