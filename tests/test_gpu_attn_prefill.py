"""tcgen05 prefill attention against the fp32 reference."""

import math

import pytest
import torch

from mfq_b200 import ops
from mfq_b200.ops import reference as ref
from gpu_common import assert_close, check_status, require_gpu_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,hq,hk", [(128, 4, 2), (300, 8, 2), (1024, 4, 4), (1, 4, 1), (129, 2, 1)])
def test_prefill_attention_matches_reference(t, hq, hk):
    require_gpu_lib()
    g = torch.Generator(device="cuda").manual_seed(t)
    q = torch.randn((t, hq, 128), generator=g, device="cuda").to(torch.bfloat16)
    k = torch.randn((t, hk, 128), generator=g, device="cuda").to(torch.bfloat16)
    v = torch.randn((t, hk, 128), generator=g, device="cuda").to(torch.bfloat16)
    scale = 1 / math.sqrt(128)
    got = ops.kernels.attn_prefill_bf16(q, k, v, scale)
    check_status()
    want = ref.attention(q, k, v, scale, causal_offset=0)
    assert_close(got, want, rel=2e-2, what=f"prefill attention T={t}")


@pytest.mark.parametrize("t,past,hq,hk", [(128, 0, 4, 2), (300, 0, 8, 1), (1024, 0, 2, 2), (1, 0, 4, 1), (200, 77, 8, 2),
                                           (64, 1000, 4, 1), (2048, 0, 2, 1)])
def test_prefill_attention_head_dim_256(t, past, hq, hk):
    """The 256-wide kernel keeps O in TMEM and rescales it lazily; large-magnitude late keys force rescales."""
    require_gpu_lib()
    g = torch.Generator(device="cuda").manual_seed(7 * t + past)
    q = torch.randn((t, hq, 256), generator=g, device="cuda").to(torch.bfloat16)
    k = torch.randn((past + t, hk, 256), generator=g, device="cuda")
    # growing key magnitude: the running maximum keeps rising, so the rescale path runs many times
    k = (k * torch.linspace(0.5, 3.0, past + t, device="cuda")[:, None, None]).to(torch.bfloat16)
    v = torch.randn((past + t, hk, 256), generator=g, device="cuda").to(torch.bfloat16)
    scale = 1 / math.sqrt(256)
    got = ops.kernels.attn_prefill_bf16(q, k, v, scale)
    check_status()
    want = ref.attention(q, k, v, scale, causal_offset=past)
    assert_close(got, want, rel=2e-2, what=f"prefill attention D=256 T={t} past={past}")


def test_packed_sequences_do_not_mix():
    require_gpu_lib()
    q = torch.randn((200, 4, 128), device="cuda").to(torch.bfloat16)
    k = torch.randn((200, 2, 128), device="cuda").to(torch.bfloat16)
    v = torch.randn((200, 2, 128), device="cuda").to(torch.bfloat16)
    got = ops.attn_prefill(q, k, v, [0, 70, 200], 0.09)
    want = torch.cat([ref.attention(q[:70], k[:70], v[:70], 0.09, 0), ref.attention(q[70:], k[70:], v[70:], 0.09, 0)])
    assert_close(got, want, rel=2e-2)
    check_status()


@pytest.mark.parametrize("tq,past", [(128, 128), (200, 77), (64, 1000), (300, 1)])
def test_prefill_attention_with_past_keys(tq, past):
    """Queries of a later chunk attend to the cached past + the chunk (causal with an offset)."""
    import torch
    from mfq_b200.ops import kernels as K
    from mfq_b200.ops import reference as ref
    from gpu_common import assert_close, check_status, require_gpu_lib
    require_gpu_lib()
    g = torch.Generator(device="cuda").manual_seed(tq + past)
    hq, hk, d = 8, 2, 128
    q = torch.randn((tq, hq, d), generator=g, device="cuda").to(torch.bfloat16)
    k = torch.randn((past + tq, hk, d), generator=g, device="cuda").to(torch.bfloat16)
    v = torch.randn((past + tq, hk, d), generator=g, device="cuda").to(torch.bfloat16)
    got = K.attn_prefill_bf16(q, k, v, 0.088)
    check_status()
    want = ref.attention(q, k, v, 0.088, causal_offset=past)
    assert_close(got.float(), want.float(), rel=2e-2, what="prefill attention with past")


def test_kv_gather_dequant_and_chunked_engine_prefill():
    import torch
    from mfq_b200.engine.llm_engine import LLMEngine
    from mfq_b200.models.llama import LlamaConfig, LlamaModel, LlamaWeights
    from mfq_b200.ops import kernels as K
    from mfq_b200.ops import reference as ref
    from gpu_common import assert_close, check_status, require_gpu_lib
    require_gpu_lib()
    cfg = LlamaConfig.tiny()
    w = LlamaWeights.random_init(cfg, "cuda", seed=2, std=0.05)
    prompt = torch.randint(0, cfg.vocab_size, (300,), generator=torch.Generator().manual_seed(3))
    whole = LLMEngine(LlamaModel(cfg, w), max_batch=2, max_seq_len=512)
    parts = LLMEngine(LlamaModel(cfg, w), max_batch=2, max_seq_len=512, prefill_chunk=128)
    a = whole.generate([prompt], 8).tokens[0].tolist()
    b = parts.generate([prompt], 8).tokens[0].tolist()
    check_status()
    n = 0
    while n < 8 and a[n] == b[n]:
        n += 1
    assert n >= 6, (a, b)  # chunk boundaries change the summation order of the attention slightly
    # the gather kernel returns exactly what the pages hold
    kv = parts.cache.layer(0)
    row = parts.cache.block_table[0]
    kd, vd = K.kv_gather_dequant(kv, row, 200)
    t = torch.arange(200, device="cuda")
    kr, vr = ref.gather_slots(kv, row[(t // 16).long()] * 16 + t % 16)
    assert_close(kd.float(), kr.float(), rel=1e-2, what="gathered K")
    assert_close(vd.float(), vr.float(), rel=1e-2, what="gathered V")


def test_prefix_cache_restores_pages_on_gpu(tmp_path):
    import torch
    from mfq_b200 import native
    from mfq_b200.engine.llm_engine import LLMEngine
    from mfq_b200.models.llama import LlamaConfig, LlamaModel, LlamaWeights
    from gpu_common import check_status, require_gpu_lib
    require_gpu_lib()
    cfg = LlamaConfig.tiny()
    w = LlamaWeights.random_init(cfg, "cuda", seed=2, std=0.05)
    g = torch.Generator().manual_seed(0)
    shared = torch.randint(0, cfg.vocab_size, (300,), generator=g)
    p1 = torch.cat([shared, torch.randint(0, cfg.vocab_size, (20,), generator=g)])
    pc = native.PrefixCache(tmp_path / "kv", ram_budget=256 << 20, disk_budget=0, block_tokens=256)
    eng = LLMEngine(LlamaModel(cfg, w), max_batch=2, max_seq_len=512, prefix_cache=pc, prefix_salt="tiny")
    first = eng.generate([p1], 6).tokens[0].tolist()
    assert eng.prefix_stats["blocks_stored"] == 1
    eng.release(0)
    again = eng.generate([p1], 6).tokens[0].tolist()  # 256 tokens restored, 64 recomputed against them
    check_status()
    assert eng.prefix_stats["blocks_hit"] == 1
    n = 0
    while n < 6 and first[n] == again[n]:
        n += 1
    assert n >= 5, (first, again)
    pc.close()


@pytest.mark.parametrize("t,past,hq,hk,scale", [(1, 0, 2, 1, 0.09), (127, 1, 6, 2, 0.09), (129, 0, 3, 3, 0.09), (257, 126, 3, 1, 0.09), (385, 0, 8, 2, 0.09),
                                                (256, 130, 4, 1, 0.0), (128, 0, 148, 74, 0.09), (128, 1, 150, 75, 0.09), (257, 126, 51, 17, 0.09),
                                                (257, 126, 50, 25, 0.0), (385, 0, 45, 15, 0.09), (130, 1000, 2, 1, 0.09)])
def test_prefill_attention_over_tiles_and_heads(t, past, hq, hk, scale):
    """One key block up to nine, so that both S buffers and stages come around; odd counts of heads and blocks, more tiles than SMs; keys
    that grow, so that O is rescaled in every block; a scale of zero."""
    require_gpu_lib()
    g = torch.Generator(device="cuda").manual_seed(t + past)
    q = torch.randn((t, hq, 128), generator=g, device="cuda").to(torch.bfloat16)
    k = torch.randn((past + t, hk, 128), generator=g, device="cuda")
    k = (k * torch.linspace(0.25, 4.0, past + t, device="cuda")[:, None, None]).to(torch.bfloat16)
    v = torch.randn((past + t, hk, 128), generator=g, device="cuda").to(torch.bfloat16)
    got = ops.kernels.attn_prefill_bf16(q, k, v, scale)
    check_status()
    # probabilities and the result are rounded to bf16 (2^-9 each, relative): well inside 2 % of (|ref| + rms / 4)
    assert_close(got, ref.attention(q, k, v, scale, causal_offset=past), rel=2e-2, what=f"T={t} past={past}")


@pytest.mark.parametrize("t,past,hq,hk", [(257, 0, 84, 21), (385, 126, 64, 16), (1000, 130, 32, 8), (100, 1000, 256, 64)])
def test_grids_that_fill_two_ctas_per_sm(t, past, hq, hk):
    """All heads in one call, and a few at a time, which leave SMs free and take the other form: the same bits, with keys that grow."""
    require_gpu_lib()
    g = torch.Generator(device="cuda").manual_seed(t)
    q = torch.randn((t, hq, 128), generator=g, device="cuda").to(torch.bfloat16)
    k = (torch.randn((past + t, hk, 128), generator=g, device="cuda") * torch.linspace(0.25, 4.0, past + t, device="cuda")[:, None, None]).to(torch.bfloat16)
    v = torch.randn((past + t, hk, 128), generator=g, device="cuda").to(torch.bfloat16)
    blocks, per = -(-t // 128), hq // hk
    assert blocks * hq >= 250 > blocks * per
    got = ops.kernels.attn_prefill_bf16(q, k, v, 0.09)
    for h in range(hk):
        want = ops.kernels.attn_prefill_bf16(q[:, h * per : (h + 1) * per].contiguous(), k[:, h : h + 1].contiguous(), v[:, h : h + 1].contiguous(), 0.09)
        assert torch.equal(got[:, h * per : (h + 1) * per], want), h
    check_status()


def _form(t, past, hq):
    return ops.kernels.lib().mfq_attn_prefill_form(t, past + t, hq)


@pytest.mark.parametrize("t,past,hq,hk", [(513, 0, 84, 21), (1300, 0, 32, 8), (385, 126, 128, 32), (3100, 0, 16, 4), (200, 8000, 128, 16)])
def test_two_ctas_per_sm_give_the_bits_of_one(t, past, hq, hk):
    """Grids that take the pair form, and a few heads of them, which take the other: the same bits."""
    require_gpu_lib()
    g = torch.Generator(device="cuda").manual_seed(t)
    q = torch.randn((t, hq, 128), generator=g, device="cuda").to(torch.bfloat16)
    k = (torch.randn((past + t, hk, 128), generator=g, device="cuda") * torch.linspace(0.25, 4.0, past + t, device="cuda")[:, None, None]).to(torch.bfloat16)
    v = torch.randn((past + t, hk, 128), generator=g, device="cuda").to(torch.bfloat16)
    per = hq // hk
    assert _form(t, past, hq) and not _form(t, past, per)
    got = ops.kernels.attn_prefill_bf16(q, k, v, 0.09)
    for h in range(0, hk, 3):
        want = ops.kernels.attn_prefill_bf16(q[:, h * per : (h + 1) * per].contiguous(), k[:, h : h + 1].contiguous(), v[:, h : h + 1].contiguous(), 0.09)
        assert torch.equal(got[:, h * per : (h + 1) * per], want), h
    check_status()


def test_grids_whose_longest_tiles_would_stand_alone_keep_one_cta_per_sm():
    """Measured on either side: few tiles a head, tiles of many lengths with too few of them for all SMs, and three full rounds of tiles alike."""
    require_gpu_lib()
    for t, past, hq, pair in ((2028, 0, 16, 0), (2540, 0, 16, 0), (4076, 0, 16, 1), (1004, 0, 32, 0), (1516, 0, 32, 1), (2028, 0, 32, 1),
                              (1004, 1000, 32, 0), (1004, 8000, 32, 1), (1516, 8000, 32, 0), (2028, 8000, 32, 1), (120, 0, 32, 0)):
        assert _form(t, past, hq) == pair, (t, past, hq)


@pytest.mark.parametrize("t,past,hq,hk", [(513, 0, 84, 21), (385, 126, 128, 32)])
def test_infinite_values_by_either_form(t, past, hq, hk):
    """Keys, queries and values that are infinite or NaN, behind the diagonal and ahead of it: where either form gives NaN, the other does, and the
    rest are the same bits."""
    require_gpu_lib()
    g = torch.Generator(device="cuda").manual_seed(t)
    q, k, v = (torch.randn((n, h, 128), generator=g, device="cuda").to(torch.bfloat16) for n, h in ((t, hq), (past + t, hk), (past + t, hk)))
    q[5, 0, 3], k[past + 200, 1, 7], k[130, 2, 0], k[past + t - 1, 3, 9] = float("inf"), -float("inf"), float("inf"), float("nan")
    v[past + 3, 4, 5], v[past + 250, 5, 6], v[140, 6, 0] = float("inf"), -float("inf"), float("nan")
    per = hq // hk
    assert _form(t, past, hq) and not _form(t, past, per)
    got = ops.kernels.attn_prefill_bf16(q, k, v, 0.09)
    for h in range(8):
        want = ops.kernels.attn_prefill_bf16(q[:, h * per : (h + 1) * per].contiguous(), k[:, h : h + 1].contiguous(), v[:, h : h + 1].contiguous(), 0.09)
        own = got[:, h * per : (h + 1) * per]
        assert torch.equal(own.isnan(), want.isnan()) and torch.equal(own[~want.isnan()], want[~want.isnan()]), h
    check_status()
