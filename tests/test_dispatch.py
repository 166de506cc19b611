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


# ------------------------------------------------------------------ products of few tokens (gemm_few.cuh)
FEW_KEYS = ("served", "rows", "ranges", "stages", "cluster", "fetched", "in_memory", "tiles", "ring", "shares", "smem")
FEW_TOKENS = (1, 2, 7, 8, 9, 16, 17, 24, 33, 40, 48, 64, 65, 72, 96, 104, 128)


B200 = (SMS, 74, 33, 15, 148, 71, 33)


def few_plan(T, N, K, adds=False, in_memory=True, gated=False, device=B200):
    """The plan on a device of 148 SMs that holds 74, 33 and 15 clusters of 2, 4 and 8 CTAs with one CTA to an SM and 148, 71 and 33
    with two."""
    import ctypes

    from inferloop_b200.csrc.build import load_module
    lib = load_module("gemm_tcgen05")
    lib.ilb_gemm_tc_sums_in_memory(1 if in_memory else 0)
    try:
        out = (ctypes.c_int * len(FEW_KEYS))()
        assert lib.ilb_gemm_few_plan(T, N, K, 2 if gated else 1 if adds else 0, (ctypes.c_int * 7)(*device), out) == 0
        return dict(zip(FEW_KEYS, out))
    finally:
        lib.ilb_gemm_tc_sums_in_memory(1)


def test_ranges_whose_order_is_kept_belong_to_the_weight():
    """A row's sum is cut alike whatever it is computed beside: as many equal K ranges as tiles of 128 rows allow (two CTAs to an SM,
    clusters that fit the device at once), for every token count, and for adding products too once sums in memory are off."""
    for (N, K), ranges in {(6144, 4096): 4, (4096, 4096): 8, (24576, 4096): 1, (4096, 12288): 8, (7168, 5120): 4, (5120, 5120): 4,
                           (34816, 5120): 1, (5120, 17408): 4, (10240, 5120): 2, (5120, 25600): 4, (4096, 2048): 8, (2048, 6144): 8,
                           (4224, 4096): 8, (4352, 4096): 4, (9472, 1024): 4, (9600, 1024): 2, (18944, 512): 2, (19072, 512): 1,
                           (37888, 320): 1, (768, 256): 4, (512, 384): 4, (256, 64): 1, (256, 72): 2, (72, 8): 1}.items():
        for T in FEW_TOKENS:
            for adds in (False, True):
                plan = few_plan(T, N, K, adds, in_memory=False)
                assert plan["served"] and plan["ranges"] == ranges and not plan["in_memory"], (T, N, K, plan)
                assert plan["cluster"] == ranges, (T, N, K, plan)
            assert few_plan(T, N, K)["ranges"] == ranges                       # a product that adds nothing never asks
            if 8 < T <= 64:
                assert few_plan(T, N, K, adds=True)["ranges"] == ranges        # and between 9 and 64 tokens nor does one that does


def test_ranges_that_meet_in_memory():
    """Up to 8 tokens with a weight of 2,048 x 2,048 or more, or 65 to 128 with a wide output; never when switched off."""
    for T in FEW_TOKENS:
        for (N, K), few, many in (((4096, 4096), True, True), ((2048, 2048), True, False), ((2047, 4096), False, False), ((4096, 512), False, True),
                                  ((4096, 448), False, False), ((3072, 1024), False, False), ((3328, 1024), False, True), ((18944, 2048), True, True),
                                  ((19200, 2048), False, False)):
            may = (T <= 8 and few) or (T > 64 and many)
            plan = few_plan(T, N, K, adds=True)
            assert not plan["in_memory"] or may, (T, N, K, plan)
            assert not may or plan["in_memory"] or plan["ranges"] == 1, (T, N, K, plan)
    assert few_plan(1, 4096, 4096, adds=True)["in_memory"] and few_plan(128, 4096, 4096, adds=True)["in_memory"]


def test_weights_of_more_tiles_than_ctas():
    """They keep the form that shares tiles out block by block, unless the rows they read differ from run to run as it is."""
    for T in FEW_TOKENS:
        free = T <= 8 or T > 64
        plan = few_plan(T, 51200, 5120)
        assert plan["served"] == free and (not free or plan["ranges"] == 1), (T, plan)
        assert not few_plan(T, 51200, 5120, in_memory=False)["served"]
        assert few_plan(T, 50000, 1024)["served"] == 0                         # rows of 1,024 never meet in memory
        assert few_plan(T, 151936, 4096)["served"] == 0
    assert few_plan(129, 4096, 4096)["served"] == 0


def test_shared_memory_of_a_plan_holds_what_the_kernel_lays_out():
    """1,024 bytes of alignment, the ring, the area for shares, barriers and flags; what the MMA reads beyond the tokens, the tile on its
    way out and the shares of a cluster, sent or parked, all inside."""
    forms = set()
    for N in (1, 16, 72, 515, 768, 1000, 2048, 3072, 4096, 5120, 6144, 7168, 9472, 10240, 12288, 18944, 24576, 34816, 37888, 51200, 75776):
        for K in (8, 64, 72, 320, 512, 1024, 4096, 12288, 25600):
            for T in FEW_TOKENS:
                for adds in (False, True):
                    p = few_plan(T, N, K, adds)
                    if not p["served"]:
                        continue
                    what = (T, N, K, adds, p)
                    padded, chunks, blocks = -(-T // 8) * 8, p["rows"] // 16, -(-K // 64)
                    stage = (padded + p["rows"]) * 128
                    assert p["rows"] % 16 == 0 and 16 <= p["rows"] <= 256 and (p["tiles"] - 1) * p["rows"] < N <= p["tiles"] * p["rows"], what
                    assert 1 <= p["ranges"] <= blocks and 1 <= p["stages"] <= 12, what
                    deep = T > 64 and p["in_memory"] and p["tiles"] * p["ranges"] <= SMS
                    assert 1023 + p["ring"] + p["shares"] + (2 * 12 + 4) * 8 <= p["smem"] <= (224 if deep else 112) * 1024, what
                    assert p["ring"] >= max(p["stages"] * stage, (p["stages"] - 1) * stage + (64 if T <= 64 else 128) * 128), what
                    if p["cluster"] == 1:
                        assert p["ring"] >= T * (p["rows"] + 4) * 4 and p["shares"] == 0 and not p["fetched"], what
                    else:
                        assert p["cluster"] == p["ranges"] and p["ranges"] in (2, 4, 8) and not p["in_memory"], what
                        if p["fetched"]:
                            assert p["ring"] >= chunks * padded * 64 and p["shares"] == 0, what
                        else:
                            assert p["shares"] >= p["ranges"] * -(-chunks // p["ranges"]) * padded * 64, what
                    forms.add((p["cluster"] > 1, p["fetched"], p["in_memory"]))
    assert forms == {(False, 0, 0), (False, 0, 1), (True, 0, 0), (True, 1, 0)}


def test_plans_of_products_that_had_become_slower():
    """Products that the kernel of few tokens took longer over than the kernels before it (4,096 x 512 adding at 64 tokens 7.9 -> 9.5 us,
    5,120 x 17,408 adding at 128 38.1 -> 40.9, 6,144 x 1,024 gated at 24 6.65 -> 7.05, 3,072 x 4,096 at 1 token 8.0 -> 8.6): more
    of the SMs' slots, a deeper ring, gated tiles that are fetched in whole blocks."""
    for T in (57, 64):
        plan = few_plan(T, 4096, 512, adds=True)
        assert plan["tiles"] * plan["ranges"] >= 220, plan
    for T in (72, 80, 96, 112, 128):
        for N, K in ((4096, 12288), (5120, 5120), (5120, 8192), (5120, 17408), (5120, 25600)):
            plan = few_plan(T, N, K, adds=True)
            assert plan["in_memory"] and plan["stages"] >= 5 and plan["tiles"] * plan["ranges"] <= SMS, (T, N, K, plan)
    for T in (19, 24, 32):
        assert few_plan(T, 6144, 1024, gated=True)["rows"] % 64 == 0, T
    for T in (1, 2, 4, 8):
        assert few_plan(T, 3072, 4096)["rows"] <= 144, T


def test_no_third_cta_of_a_product_of_few_tokens_fits_an_sm():
    """Each holds up to 256 of the 512 columns of tensor memory while it waits for its cluster: three on an SM could wait for one
    another without end.  An SM has 228 KB of shared memory, 1 KB of it kept for every CTA."""
    for N, K in ((4096, 512), (6144, 256), (24576, 192), (72, 8), (768, 256), (2048, 2048), (1, 64), (1024, 1024), (4096, 4096)):
        for T in FEW_TOKENS:
            for adds in (False, True):
                plan = few_plan(T, N, K, adds)
                assert plan["rows"] <= 256 and 3 * (plan["smem"] + 1024) > 228 * 1024, (T, N, K, plan)


def test_a_wait_that_runs_out_leaves_no_thread_of_a_product_of_few_tokens_behind():
    """Read in the kernel's source: no barrier, and no load that a whole warp has to issue, stands under a condition that threads could see
    differently once a wait has run out; nothing returns early; and what was requested from memory is awaited at the end."""
    import os
    import re

    import inferloop_b200.csrc as csrc
    text = open(os.path.join(csrc.__path__[0], "gemm_few.cuh")).read()
    body = text[text.index("gemm_few_kernel("):text.index("// ------------------------------------------------------------------ host side")]
    body = re.sub(r'"[^"\n]*bar\.sync[^"\n]*"', "BARRIER", re.sub(r"//[^\n]*", "", body))
    body = re.sub(r'"[^"\n]*"', "", re.sub(r"for \([^{]*?;[^{]*?;[^{]*?\)", "for ()", body))
    together = re.compile(r"BARRIER|__syncthreads\(|__syncwarp\(|cluster_sync_all\(|tmem_load_16\(")
    private = re.compile(r"\b(failed|bad|ok|arrived|mbar_wait)\b")
    around, statement, found = [], "", 0
    for piece in re.split(r"([{};])", body):
        if piece == "{":
            around.append(statement)
            statement = ""
        elif piece == "}":
            around.pop()
            statement = ""
        elif piece == ";":
            if together.search(statement):
                found += 1
                for condition in around + [statement]:
                    assert not private.search(condition), (statement.strip(), condition.strip())
            statement = ""
        else:
            statement += piece
    assert found >= 12 and not around and not re.search(r"\breturn\b", body)
    end = body[body.rindex("__syncthreads("):]
    assert re.search(r"\*failed\)\s*for \(\)\s*mbar_wait\(full0", end), "requested blocks have to land before the block ends"


def test_a_plan_belongs_to_the_device_it_was_made_for():
    """Plans are kept by all that they depend on: one made for a device of half the size is not handed to a whole one."""
    half = (74, 37, 16, 7, 74, 35, 16)
    for T, N, K in ((8, 34816, 5120), (3, 24576, 5120)):                     # one range on either, so that the sizes alone don't tell them apart
        whole, small = few_plan(T, N, K, gated=True), few_plan(T, N, K, gated=True, device=half)
        assert whole["ranges"] == small["ranges"] == 1 and small["tiles"] <= 2 * 74 < whole["tiles"] <= 2 * SMS, (T, N, K, small, whole)
        assert few_plan(T, N, K, gated=True) == whole, (T, N, K)
