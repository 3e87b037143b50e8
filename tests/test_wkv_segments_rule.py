"""CPU: where segments of the matrix-state recurrence go side by side.  They work on whole tiles of 64 x 64, so heads that leave much of a
tile empty are served only while they do not fill the GPU; both sides of the lines were measured."""
import pytest

SLOWER = [(256, 128, 16), (1024, 300, 16), (1024, 444, 16), (256, 260, 8), (256, 444, 4), (256, 96, 32), (1024, 300, 40), (256, 160, 48), (1024, 370, 48),
          (256, 28, 72), (256, 48, 72), (1024, 48, 80), (4096, 128, 88), (256, 20, 96), (1024, 222, 96), (256, 40, 104), (300, 40, 104)]
FASTER = [(256, 1, 64), (256, 32, 64), (256, 444, 64), (4096, 32, 64), (4096, 128, 64), (256, 296, 56), (1024, 370, 60), (256, 16, 128), (256, 222, 128), (512, 40, 104),
          (1024, 222, 100), (256, 74, 16), (256, 74, 32), (4096, 64, 40), (256, 74, 48), (256, 9, 72), (300, 18, 72), (256, 18, 96), (4096, 12, 64)]


@pytest.mark.parametrize("T,H,D", SLOWER)
def test_shapes_that_are_slower_in_segments_go_token_after_token(T, H, D):
    from cold_compress_b200 import _lib
    assert _lib.load_seq().cc_seq_wkv_segments_workspace(T, H, D) == 0


@pytest.mark.parametrize("T,H,D", FASTER)
def test_shapes_that_are_faster_in_segments_go_in_segments(T, H, D):
    from cold_compress_b200 import _lib
    assert _lib.load_seq().cc_seq_wkv_segments_workspace(T, H, D) > 0


def _segments(T, H, D):
    """How many, from the floats that each takes in the workspace."""
    from cold_compress_b200 import _lib
    floats = _lib.load_seq().cc_seq_wkv_segments_workspace(T, H, D) // 4 - (T * H * D + 3) // 4 * 4
    assert floats % (H * D * (D + 1)) == 0
    return floats // (H * D * (D + 1))


@pytest.mark.parametrize("T,H,D,n", [(3699, 32, 64, 27), (3700, 32, 64, 37), (4096, 32, 64, 37), (899, 128, 64, 6), (900, 128, 64, 9), (7299, 16, 64, 55), (7400, 16, 64, 74),
                                     (399, 128, 128, 3), (400, 128, 128, 4), (1399, 40, 100, 11), (1400, 40, 100, 14), (256, 460, 64, 2), (256, 592, 64, 2), (256, 290, 128, 2)])
def test_eight_segments_an_sm_while_they_keep_a_hundred_tokens_and_six_otherwise(T, H, D, n):
    assert _segments(T, H, D) == n


@pytest.mark.parametrize("T,H,D", [(4096, 593, 64), (4096, 297, 128), (256, 290, 100), (300, 290, 104)])
def test_more_heads_than_leave_two_segments_go_token_after_token(T, H, D):
    from cold_compress_b200 import _lib
    assert _lib.load_seq().cc_seq_wkv_segments_workspace(T, H, D) == 0
