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


@pytest.mark.parametrize("blocks,seen,dkp,want", [
    (4, 16, 64, 1), (4, 64, 64, 4), (4, 512, 64, 8), (4, 513, 64, 33), (4, 1032, 64, 64), (80, 512, 64, 4), (80, 513, 64, 7), (128, 4096, 64, 4), (600, 4096, 64, 1),
    (5, 256, 128, 8), (5, 257, 128, 17), (160, 256, 128, 2), (160, 1024, 128, 3), (4, 128, 256, 8), (4, 144, 256, 9), (192, 64, 256, 3)])
def test_pieces_of_a_layer_list_token(blocks, seen, dkp, want):
    from ghassan_b200.models.layer_model import attention_splits
    assert attention_splits(blocks, seen, dkp) == want


@pytest.mark.parametrize("N,top,ne,ne1,E,d,want", [
    (3, 2, 8, 9, 768, 768, False), (4, 2, 8, 9, 768, 768, True), (128, 2, 8, 9, 768, 768, True), (129, 2, 8, 9, 768, 768, False),      # most experts are visited
    (128, 4, 8, 9, 1280, 768, True), (128, 2, 16, 16, 1024, 1024, True), (64, 2, 16, 16, 1088, 1024, True), (65, 2, 16, 16, 1088, 1024, False),
    (64, 2, 4, 5, 4096, 1024, True), (96, 2, 4, 5, 4096, 1024, False), (4, 4, 16, 16, 2048, 1024, False), (8, 4, 16, 16, 2048, 1024, True),
    (32, 4, 16, 16, 2048, 1024, True), (33, 4, 16, 16, 2048, 1024, False), (64, 1, 64, 64, 1024, 1024, False), (32, 8, 64, 64, 576, 1024, False),
    (32, 2, 65, 65, 64, 768, False), (32, 9, 16, 16, 64, 768, False), (32, 2, 8, 8, 96, 768, False), (32, 2, 8, 8, 64, 20488, False)])
def test_when_all_rows_go_through_all_experts(N, top, ne, ne1, E, d, want):
    from ghassan_b200.models.cuda_model import few_through_all
    assert few_through_all(N, top, ne, ne1, E, d) is want


@pytest.mark.parametrize("M,N,K,want", [
    (1280, 2048, 1024, True), (1280, 2048, 1023, False), (1536, 2560, 768, True),            # one round of pairs for two of the one-CTA kernel; 60 tiles for any K
    (300, 4616, 2048, False), (300, 6144, 2048, False), (128, 15104, 2048, False), (500, 4864, 2048, True),      # 111, 144 and 118 tiles of 128 x 128, 152
    (128, 9728, 2048, True), (128, 9408, 2048, False), (128, 15360, 2048, True)])            # 152 tiles of 128 x 64, 147; 60 of 256 x 256
def test_products_that_the_pairs_take(M, N, K, want):
    from ghassan_b200.ops import gemm as G
    assert G.pair_fits(M, N, K=K, block_n=G.pick_block_n(M, N)) is want


def test_pair_lines_from_the_environment():
    """One variable moves both lines, as it did when there was one; the second has a variable of its own."""
    import os
    import subprocess
    import sys
    code = "from ghassan_b200.ops import gemm as G; print(G.PAIR_MIN_TILES, G.PAIR_MIN_TILES_ONE)"
    for env, want in (({}, "60 38"), ({"GB200_GEMM_PAIR_MIN_TILES": "70"}, "70 70"), ({"GB200_GEMM_PAIR_MIN_TILES_ONE": "50"}, "60 50")):
        clean = {k: v for k, v in os.environ.items() if not k.startswith("GB200_GEMM_PAIR")}
        out = subprocess.run([sys.executable, "-c", code], env=dict(clean, **env), capture_output=True, text=True, check=True).stdout
        assert out.split("\n")[-2] == want
