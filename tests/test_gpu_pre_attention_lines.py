"""qk_norm_rope_store around the sizes where whole-token passes take over (2368 warps: 4.5 full passes each, eight that are three
quarters full) and where a warp's units end unevenly, one full pass per token (6 / 1 and 4 / 2 heads) among them: bit for bit against the
oracle, slots that are skipped included."""
import pytest

from test_gpu_pre_attention_large import test_large_batches_are_bit_exact as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,h,kvh", [(1775, 32, 8), (1776, 32, 8), (1065, 64, 8), (1066, 64, 8), (2132, 28, 4), (6314, 14, 2),
                                     (6315, 14, 2), (6317, 12, 4), (8191, 9, 8), (8190, 18, 2), (8190, 10, 2),
                                     (8191, 6, 1), (8191, 5, 1), (10655, 6, 1), (10656, 6, 1), (10656, 4, 2), (16384, 6, 1),
                                     (16384, 4, 2)])
def test_lines_and_ragged_units(t, h, kvh):
    check(t, h, kvh)
