"""The number of KV ranges that the KV-centric operator takes where none is given."""
import pytest

from sparse_attention_b200_b200.kv_centric import default_segments


@pytest.mark.parametrize("kv_blocks,topk,items,rows,want", [
    (10, 10, 32, 8192, 4),           # us with 1, 2 and 4 ranges: 25.9, 20.6, 20.1
    (11, 9, 29, 7296, 4),            # 24.0, 22.0, 19.7
    (7, 6, 8, 1792, 4),              # 18.6, 17.6, 15.5
    (12, 12, 38, 9600, 2),           # 29.2, 23.3, 26.6
    (62, 31, 160, 40960, 2),         # 112.8, 103.8, 107.4
    (252, 4, 16, 3072, 1),           # 15.4, 16.6, 16.6
    (1024, 64, 4 * 8 * 1024, 64 * 131072, 1),
    (2, 1, 2, 768, 1),               # one block: nothing to divide
])
def test_default_ranges_of_measured_problems(kv_blocks, topk, items, rows, want):
    assert default_segments(kv_blocks, topk, items, rows) == want


def test_default_ranges_without_sizes():
    """Known only by blocks and list length (fp32 partials): four, or as many as there are."""
    assert [default_segments(nb, k) for nb, k in ((64, 16), (3, 16), (64, 2), (1, 1))] == [4, 3, 2, 1]
