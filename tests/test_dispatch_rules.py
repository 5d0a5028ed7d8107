"""Which kernel a size goes to, where the host decides: the lines, on both sides."""
import pytest


@pytest.mark.parametrize("batch,heads,kv,hd,max_len,want", [
    (1, 12, 4, 64, 4096, 64), (8, 12, 4, 64, 4096, 16), (16, 12, 4, 64, 4096, 8),            # fit as they are
    (32, 12, 4, 64, 564, 4), (32, 12, 4, 64, 4352, 4), (32, 12, 4, 64, 4353, 8),             # a full last round: short and long caches
    (48, 12, 4, 64, 1152, 2), (48, 12, 4, 64, 1153, 8), (96, 12, 4, 64, 2064, 8), (48, 16, 4, 128, 577, 8),      # an empty one: short caches alone
    (32, 8, 8, 64, 640, 2), (32, 8, 8, 64, 641, 8), (48, 8, 8, 64, 4096, 8), (96, 8, 8, 64, 288, 1), (96, 8, 8, 64, 289, 8),      # no groups
    (64, 8, 8, 128, 320, 1), (64, 8, 8, 128, 321, 8), (32, 16, 8, 64, 2176, 2), (32, 16, 8, 64, 2177, 8),
    (96, 16, 8, 64, 576, 1), (96, 16, 8, 64, 577, 8),
    (16, 8, 1, 64, 100000, 16), (32, 8, 1, 64, 100000, 8), (64, 8, 1, 64, 4096, 4), (64, 8, 1, 64, 8192, 8)])
def test_pieces_of_a_sequence_in_token_attention(batch, heads, kv, hd, max_len, want):
    from ghassan_b200.inference.engine import attention_splits
    assert attention_splits(batch, heads, kv, hd, max_len) == want
