"""Which packed chunks the outer recurrence cuts into parallel segments."""

from __future__ import annotations

import pytest

from mini_inference_engine_b200.engine.kernels.recurrence import TILE, segment_tokens


@pytest.mark.parametrize("longest,lanes,per_sm,cut", [
    (2869, 80, 1081.0, True), (2000, 80, 1081.0, False), (4433, 96, 1946.0, True), (3000, 96, 1946.0, False),
    (256, 400, 1.0, False), (5000, 75, 0.0, False)])
def test_requests_that_nearly_fill_the_gpu(longest, lanes, per_sm, cut):
    length = segment_tokens(longest, lanes, per_sm=per_sm)
    assert (length > 0) == cut
    assert length % TILE == 0 and (not cut or 256 <= length < longest)
