"""What a step's shape decides on the host (no GPU): which kernel takes 32-bit portions."""
import pytest


# both sides of the line where they were measured (16 and 32 heads of 64 on 8, 8 of 128 on 2, 4 of 64 on 4): portions of one or several
# requests after thousands of positions, or from position 0
@pytest.mark.parametrize("nh,nkv,rows,requests,from_start,tiles", [
    (16, 8, 8, 1, False, False), (16, 8, 64, 1, False, False), (16, 8, 256, 1, False, True), (32, 8, 64, 1, False, False), (32, 8, 256, 1, False, True),
    (8, 2, 256, 1, False, False), (8, 2, 512, 1, False, True), (4, 4, 256, 1, False, False), (4, 4, 512, 1, False, True),
    (16, 8, 256, 32, False, False), (32, 8, 256, 32, False, False), (16, 8, 400, 4, False, True), (16, 8, 80, 16, False, False),
    (16, 8, 16, 1, True, False), (16, 8, 128, 1, True, True), (32, 8, 64, 1, True, True), (16, 8, 1000, 3, True, True), (8, 2, 128, 1, True, False),
    (18, 2, 8, 1, False, True)])
def test_where_32_bit_portions_go_to_the_tiles(nh, nkv, rows, requests, from_start, tiles):
    from imparo_b200.kernels import ops
    assert ops.attention_f32_tiles_pay(rows, requests, nh, nkv, from_start) is tiles
