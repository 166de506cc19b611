"""Decisions that the kernels' Python face takes on the host (no GPU needed)."""
from inferloop_b200.csrc.ops import tc_row_blocks

SMS = 148


def ctas(tokens, heads, kv_heads, blocks):
    per = blocks * (128 // (heads // kv_heads))
    return -(-tokens // per) * kv_heads


def test_row_blocks_of_the_prefill_attention_kernel():
    # prompts from their start: two blocks once there is a CTA pair for every SM
    assert tc_row_blocks(ctas(1024, 32, 8, 1), ctas(1024, 32, 8, 2), SMS, False) == 1
    assert tc_row_blocks(ctas(2048, 32, 8, 1), ctas(2048, 32, 8, 2), SMS, False) == 2
    # portions behind a long cached prefix run in rounds: 512 tokens of 40 / 8 heads are 168 CTAs
    # (two rounds) or 88 pairs (one round of dearer tiles); 512 tokens of 32 / 8 heads fit one round
    assert tc_row_blocks(ctas(512, 40, 8, 1), ctas(512, 40, 8, 2), SMS, True) == 2
    assert tc_row_blocks(ctas(512, 32, 8, 1), ctas(512, 32, 8, 2), SMS, True) == 1
    assert tc_row_blocks(ctas(384, 40, 8, 1), ctas(384, 40, 8, 2), SMS, True) == 1
    # three rounds of one block against two of pairs: one block
    assert tc_row_blocks(ctas(1536, 32, 8, 1), ctas(1536, 32, 8, 2), SMS, True) == 1


def test_tiles_of_an_exact_product_of_many_tokens():
    """The faster tile of each pair that was measured (K = 4,096; 32 bits: 0, bfloat16: 1)."""
    from inferloop_b200.csrc.build import load_module
    tile = load_module("gemm_simt").ilb_gemm_simt_tile
    for M, N in ((512, 4096), (2048, 1000), (1024, 2048), (2048, 1024), (1024, 24576), (2048, 24576)):
        assert tile(M, N, 1) == 128
    for M, N in ((17, 8), (64, 4096), (200, 6144), (512, 6144), (1024, 4096), (2048, 4096), (1024, 6144), (200, 24576), (512, 24576)):
        assert tile(M, N, 1) == 64
    assert tile(2048, 24576, 0) == 128
    for M, N in ((41, 8), (200, 4096), (512, 4096), (512, 6144), (1024, 4096), (2048, 4096), (2048, 6144), (512, 24576), (1024, 24576)):
        assert tile(M, N, 0) == 64
