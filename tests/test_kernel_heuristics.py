"""Launch-shape rules of the GPU operators (pure Python: which kernel, how many splits)."""

import math

from mfq_b200.ops import kernels as K


def test_decode_attention_splits_fill_one_wave():
    # a batch that fills the GPU by itself is not split; small batches split until one wave (592 CTAs at D <= 128) is full
    assert K.attn_splits_for(64, 8, 4096, 128, rows=4) == 1
    assert K.attn_splits_for(128, 8, 4096, 128, rows=4) == 1
    for batch, heads, ctx, d in ((1, 8, 4096, 128), (8, 8, 4096, 128), (64, 2, 4096, 128), (32, 2, 16384, 128), (64, 2, 4096, 256)):
        s = K.attn_splits_for(batch, heads, ctx, d, rows=4)
        slots = 148 * (4 if d <= 128 else 2)
        assert 1 <= s <= 32 and batch * heads * s <= slots and ctx // s >= 256
        more = s + 1
        assert batch * heads * more > slots or ctx // more < 256 or more > 32  # and it is the largest such count
    # windows wider than 8 (row, head) pairs run the 16-row kernel, which keeps its own rule
    assert K.attn_splits_for(64, 8, 4096, 128, rows=16) == 3
    assert K.attn_splits_for(1, 8, 512, 128, rows=4) == 2


def test_split_k_choice():
    for m in (1, 16, 64):
        for n, k in ((6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336), (128256, 4096), (1536, 4096), (3584, 4096), (4096, 512)):
            s = K.pick_splits(m, n, k)
            tiles, kb = math.ceil(n / 128), k // 128
            assert 1 <= s <= 8, "decode tiles never leave the cluster path"
            assert s == 1 or math.ceil(kb / s) >= 2
            ctas = tiles * math.ceil(kb / math.ceil(kb / s))
            assert s == 1 or not 128 < ctas <= 148 or (tiles, kb) in K._MEASURED_SPLITS, (m, n, k, s, ctas)
    assert K.pick_splits(64, 28672, 4096) == 1 and K.pick_splits(64, 128256, 4096) == 1  # enough tiles already
    assert K.pick_splits(64, 6144, 4096) == 4  # measured override of the wave model's 3
    assert K.pick_splits(64, 1536, 4096) == 8  # 11 would leave the cluster path
    assert K.pick_splits(4096, 4096, 4096) == 1


def test_kernel_choice_by_rows():
    assert K.use_gemv(1, 28672, 4096) and K.use_gemv(8, 128256, 4096)
    assert K.use_gemv(16, 4096, 4096) and not K.use_gemv(16, 28672, 4096) and not K.use_gemv(12, 4096, 14336)
    assert K.use_gemv(64, 768, 4096) and not K.use_gemv(64, 3072, 4096)
    assert not K.use_gemv(4, 100, 4096)  # rows of 16 only
    assert K.act_gemv_ok(4, 4096, 4096) and not K.act_gemv_ok(5, 4096, 4096) and not K.act_gemv_ok(1, 4096, 32768)
    assert not K.act_gemv_pays(1, 4096, 4096)  # measured slower: off unless asked for


def test_pair_kernels_are_chosen_only_where_they_run():
    from mfq_b200.ops import dense
    from mfq_b200.ops import kernels as K
    for m in (1, 8, 64, 65, 100, 129, 357, 1000, 4097):
        for n, k in ((256, 128), (4096, 4096), (6144, 4096), (28672, 4096), (4096, 14336), (128256, 4096), (384, 512)):
            t = K.pair_tile(m, n, k)
            assert t in (0, 128, 256) and (t == 0 or (m >= K.PAIR_MIN_ROWS and n % 256 == 0))
            tile, splits = dense.plan(m, n, k, pairs=True)
            assert splits >= 1 or (splits == dense.PAIR and tile in (128, 256) and m > 128)
            assert dense.plan(m, n, k)[1] >= 1
    assert K.pair_tile(4096, 28672, 4096) and K.pair_tile(357, 4096, 14336)
    assert not K.pair_tile(128, 4096, 14336)  # few tiles over a long K range: the one-SM kernel splits it


def test_pair_kernel_leaves_split_ranges_of_few_tiles_alone():
    """One pair walks the K range that the one-SM kernel splits over many CTAs: measured on B200, 6.2 against 20.0 us in the first shape,
    11.6 against 19.1 in the last."""
    for m, n, k in ((65, 256, 2048), (100, 1024, 2048), (500, 256, 4096), (128, 2048, 1024), (129, 1536, 4096), (72, 5120, 768), (128, 4096, 4096)):
        assert K.pair_tile(m, n, k) == 0, (m, n, k)
    for m, n, k in ((357, 4096, 14336), (700, 4096, 4096), (1000, 6144, 4096), (500, 2048, 1024), (100, 6144, 2048), (1000, 2560, 14336)):
        assert K.pair_tile(m, n, k), (m, n, k)  # 39.5 against 83 us, 29 against 50, ...


def test_the_choice_for_a_shape_is_worked_out_once():
    """A prompt asks for the same few shapes in every layer, and the wave models cost about as much host time as a launch."""
    K.pair_tile(777, 4096, 4096), K.split_blocks(777, 4096, 4096)
    before = K.pick_splits.cache_info().misses, K.split_blocks.cache_info().misses
    for _ in range(8):
        K.pair_tile(777, 4096, 4096), K.split_blocks(777, 4096, 4096), K.pick_splits(777, 4096, 4096)
    assert (K.pick_splits.cache_info().misses, K.split_blocks.cache_info().misses) == before


def test_splits_fit_the_scratch():
    """The split-K kernels refuse partial sums beyond the workspace's scratch: no rule may ask for them."""
    import inspect

    from mfq_b200.ops.lib import Workspace
    assert inspect.signature(Workspace.__init__).parameters["splitk_bytes"].default == K.SPLIT_SCRATCH_BYTES
    unsplit = 0
    for rows in (1, 3, 5, 7, 13, 15, 33, 65, 129, 257, 513):
        for k in (512, 2048, 4096, 14336, 28672):
            for m in (1, 64, 65, 129, 700, 1500, 3000, 4096, 8192):
                s, tile, blocks = K.pick_splits(m, rows * 128, k), K._token_tile(m), k // 128
                partials = math.ceil(blocks / math.ceil(blocks / s)) * rows * math.ceil(m / tile) * tile * 128 * 4
                assert s == 1 or partials <= K.SPLIT_SCRATCH_BYTES, (m, rows * 128, k, s)
                unsplit += s == 1 and K._best_splits(m, rows * 128, k, 148) > 1
    assert unsplit and K.pick_splits(8192, 640, 14336) == 1


def test_sums_of_a_dense_pair_product_fit_its_accumulators():
    from mfq_b200.ops import dense
    seen = set()
    for m in (129, 160, 200, 257, 357, 500, 1000, 2048):
        for n in (256, 1040, 2560, 3072, 4096, 6144, 11008, 28672):
            for k in (512, 1536, 2048, 4096, 5632, 14336):
                tile, splits = dense.plan(m, n, k, pairs=True)
                if splits == dense.PAIR:
                    sums = dense.pair_sums(m, n, k)
                    assert 1 <= sums <= 512 // tile and sums == dense.plan(m, n, k)[1]
                    seen.add(sums)
    assert seen > {1}


def test_half_of_the_pairs_leave_long_weights_of_few_tokens_to_all_sms():
    # 100 x 9216 x 14336: 31.5 us on all SMs, 34.7 on 36 pairs; more pairs, more tokens or shorter rows are as they were
    for m in (65, 100, 128):
        assert K.pair_tile(m, 9216, 14336) == 0 and K.pair_tile(m, 9216, 8192) == 128 and K.pair_tile(m, 9728, 14336) == 128
    assert K.pair_tile(129, 9216, 14336) == 128 and K.pair_tile(300, 3072, 14336) == 128
