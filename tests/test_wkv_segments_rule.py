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
