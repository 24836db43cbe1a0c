"""Kernels that wide batches and prompts take: products on pairs of SMs, row quantization in one pass, several heads of a token per
warp, router logits through the dense product -- at the edges of their tiles and of the rules that choose them."""

import dataclasses
import math

import pytest
import torch

from mfq_b200 import ops
from mfq_b200.engine.kv_cache import PagedKVCache, PlainPagedKVCache
from mfq_b200.ops import dense, moe, w4, window_attn
from mfq_b200.ops import kernels as K
from mfq_b200.ops.dense import DenseLinear
from gpu_common import check_status, require_gpu_lib

pytestmark = pytest.mark.gpu
FP8 = torch.float8_e4m3fn


def _normal(seed, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * std).to(dtype)


def _fp8(seed, m, n, k):
    xq = _normal(seed, m, k, std=60, dtype=torch.float32).clamp(-448, 448).to(FP8)
    wq = _normal(seed + 1, n, k, std=60, dtype=torch.float32).clamp(-448, 448).to(FP8)
    g = torch.Generator(device="cuda").manual_seed(seed + 2)
    return xq, torch.rand(m, generator=g, device="cuda") + 0.1, wq, torch.rand((math.ceil(n / 128), k // 128), generator=g, device="cuda") + 0.1


@pytest.mark.parametrize("m,n,k", [(65, 256, 128), (129, 512, 640), (257, 256, 2048), (400, 4096, 256), (1300, 256, 1152), (130, 256, 33 * 1024),
                                   (2100, 4608, 640)])
def test_fp8_pair_kernel_gives_the_bits_of_the_one_sm_kernel(m, n, k):
    """Both fold K block after K block into fp32 registers and round the same way, residual included; 33 * 1024 is a K range whose
    multipliers do not fit the shared-memory copy; in the last shape a pair walks several tiles of either width, of five K blocks each
    (a number that the stages and the accumulators do not divide), the last ones ragged."""
    require_gpu_lib()
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    assert m != 2100 or math.ceil(m / 256) * (n // 256) > 2 * pairs
    args = _fp8(m + k, m, n, k)
    res = _normal(m, m, n)
    want = ops.fp8_gemm(*args, residual=res, splits=1, token_tile=128)
    for tile in (128, 256):
        h = res.clone()
        assert torch.equal(ops.fp8_gemm(*args, residual=h, out=h, pair=tile), want)
        assert torch.equal(ops.fp8_gemm(*args, pair=tile), ops.fp8_gemm(*args, splits=1, token_tile=128))
    check_status()


@pytest.mark.parametrize("m,n,k", [(300, 256, 4096), (130, 512, 1408), (700, 4096, 4096), (65, 4352, 1024), (130, 2816, 768)])
def test_fp8_product_of_a_wide_batch_keeps_the_sums_of_the_split_form(m, n, k, monkeypatch):
    """Chosen by itself (the last three), the two-SM kernel adds up the partial sums that the one-SM kernel's K splits would, 16 of them in
    the first shape."""
    require_gpu_lib()
    args = _fp8(m, m, n, k)
    res = _normal(m, m, n)
    assert K.split_blocks(m, n, k)
    if m == 300 or k == 1408:
        monkeypatch.setattr(K, "pair_tile", lambda *_: 128)
    assert K.pair_tile(m, n, k) == 128
    got, want = ops.fp8_gemm(*args, residual=res), ops.fp8_gemm(*args, residual=res, pair=0)
    check_status()
    assert torch.equal(got, want)


@pytest.mark.parametrize("m,n,k,tile", [(128, 1536, 1024, 0), (96, 5120, 768, 0), (1300, 2048, 2048, 0), (300, 4608, 1024, 128), (300, 4608, 1024, 256)])
def test_fp8_pair_kernel_passes_its_output_places_on(m, n, k, tile, monkeypatch):
    """The output places in shared memory hold, in turn, split sums (tile 0: several of them), the residual and the results, of a token
    range that ends inside a place; output and residual off a 16-byte boundary go round them."""
    require_gpu_lib()
    args = _fp8(m, m, n, k)
    res = _normal(m, m, n)
    off = torch.empty(m * n + 1, device="cuda", dtype=torch.bfloat16)[1:].view(m, n)
    assert off.data_ptr() % 16 and (tile or K.split_blocks(m, n, k))
    monkeypatch.setattr(K, "pair_tile", lambda *_: tile or 128)
    one = dict(splits=1, token_tile=128) if tile else dict(pair=0)
    for r in (None, res) * 3:
        want = ops.fp8_gemm(*args, residual=r, **one)
        assert torch.equal(ops.fp8_gemm(*args, residual=r, pair=tile or None), want)
        assert torch.equal(ops.fp8_gemm(*args, residual=r, out=off, pair=tile or None), want)
    h = off.copy_(res)
    assert torch.equal(ops.fp8_gemm(*args, residual=h, out=h, pair=tile or None), want)
    check_status()


def test_fp8_product_whose_partial_sums_exceed_the_scratch():
    """Rows that are not whole pairs of blocks stay on the one-SM kernel, whose wave model asks for 80 MB of partial sums here."""
    require_gpu_lib()
    args = _fp8(1, 8192, 640, 14336)
    assert K._best_splits(8192, 640, 14336, 148) > 1
    assert torch.equal(ops.fp8_gemm(*args), ops.fp8_gemm(*args, splits=1, token_tile=128))
    check_status()


@pytest.mark.parametrize("tile", [128, 256])
@pytest.mark.parametrize("m,n,k", [(1, 16, 8), (129, 272, 72), (257, 512, 4096), (300, 48, 200), (1400, 1040, 64), (4100, 2832, 72)])
def test_dense_pair_kernel_on_every_output_stage(m, n, k, tile):
    """Ragged rows, tokens and K against 64 bits; in the last shape a pair walks more tiles than it has accumulators, so that they are
    handed back and used again."""
    require_gpu_lib()
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    assert m != 4100 or math.ceil(m / tile) * math.ceil(n / 256) > 512 // tile * pairs
    w, x, bias = _normal(n, n, k, std=k ** -0.5), _normal(m, m, k), _normal(k, n, dtype=torch.float32)
    table, ids = _normal(3, 50, n), torch.arange(m, device="cuda", dtype=torch.int32) % 50
    y = x.double() @ w.double().T
    slack = (x.double().abs() @ w.double().abs().T) * (k + 8) * 2.0 ** -24

    def check(got, want, factor=1.0):
        # bf16 results: half a step; factor: how much the output stage can enlarge an error of the sum (plus its own fp32 steps)
        bound = want.abs() * (2.0 ** -8 if got.dtype == torch.bfloat16 else 2.0 ** -20) + factor * slack.amax() + 1e-5
        assert bool(((got.double() - want).abs() <= bound).all())

    how = dict(tile=tile, splits=dense.PAIR)
    check(DenseLinear(w, bias)(x, **how), y + bias.double())
    check(DenseLinear(w)(x, fp32=True, **how), y)
    check(DenseLinear(w)(x, softcap=3.0, **how), 3 * torch.tanh(y / 3))
    check(DenseLinear(w, act="relu2")(x, **how), y.clamp_min(0).square(), 2 * float(y.abs().max()))
    check(DenseLinear(w)(x, table=table, ids=ids, **how), torch.nn.functional.gelu(y, approximate="tanh") * table[ids.long()].double(), 6.0)
    stream = _normal(5, m, n, dtype=torch.float32)
    want = stream.double() + 0.5 * y
    check(DenseLinear(w)(x, add_to=stream, scale=0.5, **how), want)
    if n % 16 == 0:
        gate, up = (y.view(m, n // 16, 2, 8)[:, :, i].reshape(m, n // 2) for i in (0, 1))
        check(DenseLinear(w, glu="silu")(x, **how), torch.nn.functional.silu(gate) * up, 2 * float(y.abs().max()) + 2)
    check_status()


@pytest.mark.parametrize("m,n,k,tile,sums", [(200, 6144, 4096, 128, 2), (129, 2560, 1536, 128, 3), (300, 1040, 1104, 128, 4), (1300, 2832, 1096, 128, 3),
                                             (1500, 4112, 520, 256, 2)])
def test_dense_pair_kernel_keeps_the_sums_of_the_split_form(m, n, k, tile, sums):
    """The first two are taken by themselves; in the last two a pair walks several tiles of several accumulators each, over a K range that
    the parts do not divide."""
    require_gpu_lib()
    x, w = _normal(m, m, k), _normal(n, n, k, std=k ** -0.5)
    want = DenseLinear(w)(x, fp32=True, tile=tile, splits=sums)
    assert torch.equal(DenseLinear(w)(x, fp32=True, tile=tile, splits=-1 - sums), want)
    if k in (4096, 1536):
        assert dense.plan(m, n, k, pairs=True) == (tile, dense.PAIR) and dense.pair_sums(m, n, k) == sums
        assert torch.equal(DenseLinear(w)(x, fp32=True), want)
    check_status()


@pytest.mark.parametrize("m", [3, 511, 512, 1025])
@pytest.mark.parametrize("k", [8, 520, 4096, 14336, 16384, 16392])
def test_row_quantization_in_one_pass(m, k):
    """Rows that are and are not held in registers between the maximum and the encoding: the codes of plain fp32 arithmetic."""
    require_gpu_lib()
    x = _normal(m + k, m, 2 * k)
    x[0] = 0
    y = x[:, :k].float()
    q, s = ops.quant_rows(x[:, :k])
    # quotients through 64 bits: rounded once to fp32, as the kernel's divisions are (torch multiplies by the reciprocal of a scalar)
    scale = (y.abs().amax(1).clamp_min(1e-12).double() / 448).float()
    inverse = (1 / scale.double()).float()
    assert torch.equal(s, scale)
    assert torch.equal(q.view(torch.uint8), (y * inverse[:, None]).clamp(-448, 448).to(FP8).view(torch.uint8))
    q, s = ops.silu_mul_quant(x)
    q1, s1 = ops.silu_mul_quant(x[-1:])  # a single row: another split of the same row
    assert torch.equal(q[-1:].view(torch.uint8), q1.view(torch.uint8)) and torch.equal(s[-1:], s1)
    check_status()


@pytest.mark.parametrize("m", [255, 256, 4999, 5001])
@pytest.mark.parametrize("k", [8, 248, 264, 512, 520, 1024])
def test_quantization_of_short_rows(m, k):
    """A warp or a block per row: the codes of plain fp32 arithmetic, and of a single row."""
    test_row_quantization_in_one_pass(m, k)


@pytest.mark.parametrize("rot", [None, 64])
@pytest.mark.parametrize("d", [64, 128, 256])
def test_rotation_of_many_tokens_gives_the_bits_of_few(d, rot):
    """Enough tokens that a warp takes several heads, with a count of heads that does not divide: the same pages and queries as from
    calls that are too small for that."""
    require_gpu_lib()
    t, hq, hk = 5003, 11, 2
    rows = _normal(d, t, (hq + 2 * hk) * d)
    pos = torch.randint(0, 9000, (t,), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda", dtype=torch.int32)
    got = []
    for step in (t, 1000):
        cache = PagedKVCache(layers=1, kv_heads=hk, head_dim=d, num_pages=t // 16 + 2, max_seqs=1, max_pages_per_seq=t // 16 + 1, device="cuda")
        cache.assign(0, 0, t)
        slots = cache.slots(0, 0, t).to("cuda")
        slots[5] = -1
        kd, vd = torch.zeros((t, hk, d), device="cuda", dtype=torch.bfloat16), torch.zeros((t, hk, d), device="cuda", dtype=torch.bfloat16)
        q = torch.cat([ops.rope_kv_write(rows[a : a + step], pos[a : a + step], slots[a : a + step], cache.layer(0), n_q=hq, n_kv=hk, head_dim=d,
                                         theta=1e4, rot=rot, kd_out=kd[a : a + step], vd_out=vd[a : a + step]) for a in range(0, t, step)])
        got.append([q, cache.k.view(torch.uint8), cache.v.view(torch.uint8), cache.k_scale, cache.v_scale, kd, vd])
    check_status()
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("d", [128, 256])
def test_rotation_into_rows_off_a_vector(d):
    """Outputs that begin 2 bytes past a vector, as views of a larger buffer may: the same values as in aligned ones."""
    require_gpu_lib()
    t, hq, hk = 3003, 12, 2
    rows, pos = _normal(d, t, (hq + 2 * hk) * d), torch.arange(t, device="cuda", dtype=torch.int32)
    got = []
    for shift in (0, 1):
        cache = PagedKVCache(layers=1, kv_heads=hk, head_dim=d, num_pages=t // 16 + 2, max_seqs=1, max_pages_per_seq=t // 16 + 1, device="cuda")
        cache.assign(0, 0, t)
        q, kd, vd = (torch.zeros(t * h * d + 8, device="cuda", dtype=torch.bfloat16)[shift : shift + t * h * d].view(t, h, d) for h in (hq, hk, hk))
        assert q.data_ptr() % 8 == 2 * shift
        ops.rope_kv_write(rows, pos, cache.slots(0, 0, t).to("cuda"), cache.layer(0), n_q=hq, n_kv=hk, head_dim=d, theta=1e4, q_out=q, kd_out=kd,
                          vd_out=vd)
        got.append([q, kd, vd, cache.k.view(torch.uint8)])
    check_status()
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("t,e", [(65, 16), (200, 512), (700, 48)])
def test_router_logits_of_a_prompt(t, e):
    require_gpu_lib()
    x, w, h = _normal(t, t, 256), _normal(e, e, 256, std=0.1), 256
    ids, weights, scores = moe.router_topk(x, w, 4, want_scores=True)
    check_status()
    want = torch.softmax(x.double() @ w.double().T, -1)
    # fp32 sums of 256 terms before an exponential: a relative error of their absolute error, and that of exp itself
    slack = ((x.double().abs() @ w.double().abs().T) * (h + 8) * 2.0 ** -24).amax() * 2 + 2.0 ** -20
    assert bool(((scores.double() - want).abs() <= want * slack).all())
    picked = want.gather(1, ids.long())
    assert bool((picked >= want.topk(4, -1).values * (1 - 2 * slack)).all())
    assert bool(((weights.double() - picked / picked.sum(1, keepdim=True)).abs() <= 4 * slack).all())


@pytest.mark.parametrize("m,i", [(1, 8), (6, 2056), (295, 264), (296, 264), (3, 0)])
def test_gated_rows_over_one_and_several_blocks(m, i):
    """The last sizes before and after the rule's line, rows that end in the middle of a block, a batch of rows set apart by padding, rows
    of no width."""
    require_gpu_lib()
    rows = _normal(m, m, 2 * i + 8)[:, :2 * i]
    a, b = rows[:, :i].double(), rows[:, i:].double()
    want = a * torch.sigmoid(a) * b
    # rounded to bf16 once (2^-8); fp32 exponential and divide are far below that
    assert ((K.silu_mul(rows).double() - want).abs() <= 2.0 ** -7.9 * want.abs() + 1e-30).all()


@pytest.mark.parametrize("m", [1, 16, 17])
def test_w4_rows_off_a_vector_are_refused(m):
    """By the host, on either route of the rule on rows."""
    require_gpu_lib()
    w = w4.quantize_torch(_normal(1, 128, 256, dtype=torch.float32))
    x = torch.zeros(m * 256 + 8, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        w4.w4_gemm(x[1:1 + m * 256].view(m, 256), w)


@pytest.mark.parametrize("dtype,ulp", [(torch.float32, 2.0 ** -23), (torch.bfloat16, 2.0 ** -7)])
@pytest.mark.parametrize("d,rot,v_rot", [(128, 128, 0), (128, 64, 0), (16, 16, 16), (256, 256, 128), (80, 48, 0), (96, 0, 32)])
def test_heads_rotated_by_vectors_agree_with_the_general_form(d, rot, v_rot, dtype, ulp):
    """A table 8 bytes past a 16-byte boundary takes the general form.  Both evaluate a cos + b sin, a and b at most the row's largest
    value: each rounds at most twice, so they differ by 4 * 2 * 2^-24 of it, and by one place more where that is rounded to the type."""
    require_gpu_lib()
    t, h, g = 149, 6, 2  # the fewest tokens of the rule
    rows = _normal(1, t, (h + 2 * g) * d, dtype=dtype)
    pos = torch.randint(0, 900, (t,), device="cuda", dtype=torch.int32)
    slots = (torch.randperm(160, device="cuda")[:t] + 16).int()
    slots[5] = -1

    def finish(shift):
        def table(r):
            if not r:
                return None
            whole = torch.zeros(1000 * r + 4, device="cuda")
            assert whole.data_ptr() % 16 == 0
            part = whole[shift:shift + 1000 * r].view(1000, r // 2, 2)
            return part.copy_(window_attn.rope_table(3e4, r, 1000, "cuda"))
        cache = PlainPagedKVCache([(g, d, d)], dtype, num_pages=11, max_seqs=1, max_pages_per_seq=11, device="cuda")
        turn = window_attn.ValueTurn(table(v_rot), v_rot) if v_rot else None
        norm = _normal(2, d, dtype=torch.float32)
        q = window_attn.qkv_finish(rows, cache.layer(0), pos, slots, heads=h, kv_heads=g, dim=d, q_norm=norm, k_norm=norm, rope=table(rot),
                                   rot=rot, eps=1e-5, turn=turn)
        return q, cache.layer(0).k.clone(), cache.layer(0).v.clone()

    for got, want in zip(finish(0), finish(2)):
        got, want = got.double(), want.double()
        assert ((got - want).abs() <= (2.0 ** -21 + ulp) * want.abs().amax(-1, keepdim=True)).all()


@pytest.mark.parametrize("m", [148, 149, 296, 297, 592, 593, 1036, 1037])
@pytest.mark.parametrize("w", [8, 512, 520, 1024, 1032, 2048, 2056, 4096, 4104])
def test_stream_rows_by_vectors_per_thread(m, w):
    """Widths around one and two vectors per thread, rows around the lines of the rule."""
    require_gpu_lib()
    y, f, x = _normal(m, m, w), _normal(1, w, dtype=torch.float32), _normal(2, m, w, dtype=torch.float32)
    want, act = x.double() + y.double() * torch.rsqrt(y.double().square().mean(1, keepdim=True) + 1e-5) * f.double(), torch.empty_like(y)
    size = x.double().abs() + (want - x.double()).abs()
    dense.norm_add(y, f, x, act, w, 1e-5)
    # a tree of w squares, its root and three more roundings: below 32 of 2^-24, of the size of the two terms
    assert ((x.double() - want).abs() <= 2.0 ** -19 * size).all() and torch.equal(act, x.bfloat16())


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("how", ["pages", "offset", "mixed", "none first"])
def test_values_that_go_to_whole_pages_together(d, how):
    """Slots in one piece from a page's start or from inside one, in pieces that change places, and slots that take nothing: the pages and rows
    that calls too small for whole pages write, and what reading the pages back gives."""
    require_gpu_lib()
    t, hq, hk, first = 1100, 12, 4, 5 if how == "offset" else 0
    rows = _normal(d, t, (hq + 2 * hk) * d)
    pos = torch.arange(t, device="cuda", dtype=torch.int32)
    slots = torch.arange(first, first + t, dtype=torch.int32) + 16
    if how == "mixed":
        slots = torch.cat([slots[40:300], slots[:40], slots[300:301], slots[302:], slots[301:302]])
    if how == "none first":
        slots[0], slots[500:520] = -1, -1
    slots = slots.cuda()
    got = []
    for step in (t, 300):
        cache = PagedKVCache(layers=1, kv_heads=hk, head_dim=d, num_pages=90, max_seqs=1, max_pages_per_seq=80, device="cuda")
        kd, vd = torch.zeros((t, hk, d), device="cuda", dtype=torch.bfloat16), torch.zeros((t, hk, d), device="cuda", dtype=torch.bfloat16)
        assert (step * (hq + 2 * hk) >= 18000) == (step == t)
        q = torch.cat([ops.rope_kv_write(rows[a : a + step], pos[a : a + step], slots[a : a + step], cache.layer(0), n_q=hq, n_kv=hk, head_dim=d, theta=1e4,
                                         kd_out=kd[a : a + step], vd_out=vd[a : a + step]) for a in range(0, t, step)])
        got.append([q, cache.k.view(torch.uint8), cache.v.view(torch.uint8), cache.k_scale, cache.v_scale, kd, vd])
    for a, b in zip(*got):
        assert torch.equal(a, b)
    table = torch.arange(1, 80, device="cuda", dtype=torch.int32)
    for n in (1, 15, 16, 17, 333, 1100):
        kr, vr = K.kv_gather_dequant(cache.layer(0), table, n)
        for i, s in enumerate(slots.tolist()):
            if 0 <= s - 16 < n and i % 7 == 0:
                assert torch.equal(kr[s - 16], kd[i]) and torch.equal(vr[s - 16], vd[i])
    check_status()


@pytest.mark.parametrize("d,t,hq,hk", [(128, 1200, 12, 2), (128, 400, 32, 8), (256, 1200, 12, 2), (256, 500, 28, 9), (64, 4000, 6, 1), (64, 6000, 6, 1),
                                       (64, 8000, 6, 1), (64, 10000, 6, 1)])
def test_rotation_of_prompts_packed_one_after_the_other(d, t, hq, hk):
    """Pieces of 1 to 90 tokens, each from the start of a page or from inside one, so that whole pages begin at any token of the batch, a page
    whose tokens are interrupted by another's, and the last page cut short: the pages and rows of calls too small for whole pages."""
    require_gpu_lib()
    g, slots, page = torch.Generator().manual_seed(t), [], 1
    while len(slots) < t:
        n, inside = (int(torch.randint(a, b, (1,), generator=g)) for a, b in ((1, 90), (0, 5)))
        slots += range(page * 16 + 3 * inside, page * 16 + 3 * inside + n)
        page = slots[-1] // 16 + 1
    slots[100:108], slots[300] = reversed(slots[100:108]), -1
    slots = torch.tensor(slots[:t], dtype=torch.int32, device="cuda")
    rows, pos = _normal(d, t, (hq + 2 * hk) * d), torch.arange(t, device="cuda", dtype=torch.int32)
    got = []
    for step in (t, 160):
        cache = PagedKVCache(layers=1, kv_heads=hk, head_dim=d, num_pages=page + 1, max_seqs=1, max_pages_per_seq=page, device="cuda")
        kd, vd = torch.zeros((t, hk, d), device="cuda", dtype=torch.bfloat16), torch.zeros((t, hk, d), device="cuda", dtype=torch.bfloat16)
        q = torch.cat([ops.rope_kv_write(rows[a : a + step], pos[a : a + step], slots[a : a + step], cache.layer(0), n_q=hq, n_kv=hk, head_dim=d, theta=1e4,
                                         kd_out=kd[a : a + step], vd_out=vd[a : a + step]) for a in range(0, t, step)])
        got.append([q, cache.k.view(torch.uint8), cache.v.view(torch.uint8), cache.k_scale, cache.v_scale, kd, vd])
    check_status()
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("beside", ["one", "another", "bounds", "any"])
def test_pairs_of_gates_have_the_bits_of_the_division(beside):
    """The fp32 quotients themselves: every bf16 gate in either lane of a pair, next to gates of either side of the bounds from which a pair
    divides (64 and 1e-30), and any bits at all."""
    require_gpu_lib()
    gates = torch.arange(1 << 16, device="cuda").to(torch.int32).to(torch.int16).view(torch.bfloat16).float()
    if beside == "any":
        g = torch.Generator(device="cuda").manual_seed(0)
        pairs = [torch.randint(-(1 << 31), 1 << 31, (1 << 22,), generator=g, device="cuda").to(torch.int32).view(torch.float32).view(-1, 2)]
    elif beside == "bounds":
        edge = torch.tensor([64.0, 1e-30], device="cuda").view(torch.int32)
        edge = torch.cat([edge + i for i in range(-2, 3)]).view(torch.float32)
        edge = torch.cat([edge, -edge])
        pairs = [torch.stack([gates, e.expand_as(gates)], 1) for e in edge] + [torch.cartesian_prod(edge, edge)]
    else:
        other = torch.ones_like(gates) if beside == "one" else gates.roll(12345)
        pairs = [torch.stack([gates, other], 1)]
    x = torch.cat(pairs + [p.flip(1) for p in pairs]).contiguous()
    paired, divided = torch.empty_like(x), torch.empty_like(x)
    K.check(K.lib().mfq_silu_check(K.ptr(x), K.ptr(paired), K.ptr(divided), x.shape[0], K.stream_ptr()), "silu_check")
    assert torch.equal(paired.isnan(), divided.isnan())
    assert torch.equal(paired.view(torch.int32)[~divided.isnan()], divided.view(torch.int32)[~divided.isnan()])


@pytest.mark.parametrize("few,many,h", [(296, 297, 4104), (296, 297, 8192), (200, 1000, 16384), (1600, 1601, 2560), (1600, 1601, 4096), (1025, 2000, 2056)])
@pytest.mark.parametrize("residual", [False, True])
def test_norms_of_few_rows_give_the_bits_of_many(few, many, h, residual):
    """Either side of the lines from which residual and multipliers are requested ahead."""
    require_gpu_lib()
    x, w = _normal(h, many, h), 1 + _normal(1, h, std=0.1)
    got = []
    for m in (few, many):
        r = _normal(h + 1, many, h)[:m] if residual else None
        got.append([t[:few] for t in K.rmsnorm_quant(x[:m], w, 1e-5, residual=r, want_y=True) if t is not None])
    check_status()
    assert len(got[0]) == 3 + residual and all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(*got))


@pytest.mark.parametrize("d", [64, 128, 256])
def test_past_rows_off_a_vector(d):
    """Pages that begin at an odd byte, rows 2 bytes past a vector: the rows that aligned ones give, and nothing beside them."""
    require_gpu_lib()
    t, hk = 77, 3
    cache = PagedKVCache(layers=1, kv_heads=hk, head_dim=d, num_pages=7, max_seqs=1, max_pages_per_seq=6, device="cuda")
    table = torch.tensor([3, 1, 6, 2, 5], device="cuda", dtype=torch.int32)
    ops.rope_kv_write(_normal(d, 96, 3 * hk * d), torch.arange(96, device="cuda", dtype=torch.int32), torch.arange(16, 112, device="cuda", dtype=torch.int32),
                      cache.layer(0), n_q=hk, n_kv=hk, head_dim=d, theta=1e4)
    kv = cache.layer(0)
    want = K.kv_gather_dequant(kv, table, t)

    def shifted(x, by):
        flat = torch.zeros(x.numel() + 16, device="cuda", dtype=x.dtype)[by : by + x.numel()]
        flat.view(torch.uint8).copy_(x.reshape(-1).view(torch.uint8))
        return flat.view(x.shape)

    rows = [torch.full((t * hk * d + 16,), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    for pages, row in ((0, 1), (3, 0), (1, 1)):
        odd = dataclasses.replace(kv, k=shifted(kv.k, pages), v=shifted(kv.v, pages))
        for r in rows:
            r.fill_(7.0)
        got = K.kv_gather_dequant(odd, table, t, *(r[row : row + t * hk * d].view(t, hk, d) for r in rows))
        assert all(torch.equal(a, b) for a, b in zip(want, got))
        assert all((r[:row] == 7).all() and (r[row + t * hk * d :] == 7).all() for r in rows)
    check_status()


@pytest.mark.parametrize("m,k", [(16, 4096), (600, 4096), (300, 14336), (200, 14336), (5200, 512)])
def test_gates_of_every_value_round_as_the_division_does(m, k):
    """All bf16 values as gates, zeros of either sign, subnormal, infinite and NaN among them, through every kernel that quantizes gated rows:
    the codes of the rows that the plain product of gate and value gives."""
    require_gpu_lib()
    g = torch.arange(m * k, device="cuda") % 65521  # a prime: another gate in every place of a row
    gate = g.to(torch.int32).to(torch.int16).view(torch.bfloat16).view(m, k)
    gate = torch.where(gate.isfinite() | (torch.arange(m, device="cuda") % 5 == 0)[:, None], gate, torch.ones_like(gate))
    x = torch.cat([gate, _normal(m, m, k)], 1)
    q, s = ops.silu_mul_quant(x)
    want, ws = ops.quant_rows(K.silu_mul(x))
    assert torch.equal(s.view(torch.int32), ws.view(torch.int32)) and torch.equal(q.view(torch.uint8), want.view(torch.uint8))
    check_status()
