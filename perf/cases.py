"""The work a serving process has this framework do, as cases that can be timed and compared.

Four paths, each through the entry points a program calls:

* ``fp8``: the dense Llama decoder in block-scaled FP8 over FP8 pages (``LlamaModel.forward``), the geometry of ``LlamaConfig.llama_8b``;
* ``w4``: the same decoder with its block projections in 4-bit codes (``W4Linear``);
* ``bf16``: the Tepetar decoder of equal geometry, unquantized, in ragged batches (``TepetarModel.forward``);
* ``experts``: the routed experts of one layer of the 512-expert hybrid (``ops.moe``).

Decoders keep their full width, heads and vocabulary; their depth is cut to :data:`LAYERS` so that a state fits the card several times.
A decode step runs as a CUDA graph that is captured once, as the engine does; a prompt runs eagerly, as the engine does.
"""

from __future__ import annotations

import math
import zlib

import torch

from mfq_b200 import ops
from mfq_b200.engine.kv_cache import PagedKVCache
from mfq_b200.models.llama import Fp8Linear, LlamaConfig, LlamaLayer, LlamaModel, LlamaWeights, StepBuffers, W4Linear
from mfq_b200.models.tepetar import TepetarConfig, TepetarModel, TepetarWeights
from mfq_b200.ops import moe
from mfq_b200.ops.kernels import attn_splits_for

LAYERS = 8
WIDTH, FF, HEADS, KV_HEADS, DIM, VOCAB = 4096, 14336, 32, 8, 128, 128256
THETA, EPS = 5e5, 1e-5
EXPERTS, TOP_K, MOE_WIDTH, MOE_FF = 512, 10, 2048, 512
WINDOW, SIDE, CAP, LIMIT, SIDE_EPS = 1024, 256, 50.0, 7.0, 1e-6
GROUP = 32  # inputs per 4-bit group
PAGE = 16
E4M3_MAX = 448.0


# ---- cases ------------------------------------------------------------------------------------------------------------

def _decode(path, rows, context, ragged=False):
    return {"path": path, "rows": rows, "context": context, "ragged": ragged, "portion": 0, "past": 0}


def _prompt(path, portion, past=0, rows=0, context=0):
    return {"path": path, "rows": rows, "context": context, "ragged": False, "portion": portion, "past": past}


def listed():
    return [
        {"name": "fp8 decode 1", **_decode("fp8", 1, 600)},  # one user's stream: latency of every launch counts
        {"name": "fp8 decode 64", **_decode("fp8", 64, 4096)},  # a full batch over long contexts: the benchmark's step
        {"name": "fp8 decode 21 ragged", **_decode("fp8", 21, 2900, True)},  # a serving batch: any count of rows, any lengths
        {"name": "fp8 prompt 4096", **_prompt("fp8", 4096)},  # a long prompt in one pass
        {"name": "fp8 prompt 357", **_prompt("fp8", 357)},  # a chat turn: not a multiple of any tile
        {"name": "fp8 prompt 1000 past 3001", **_prompt("fp8", 1000, 3001)},  # the next turn of a conversation kept in the pages
        {"name": "w4 decode 6", **_decode("w4", 6, 1024)},  # a small deployment of a 4-bit checkpoint
        {"name": "experts 32", "path": "experts", "tokens": 32},  # routed experts of a decode batch
        {"name": "experts 3000", "path": "experts", "tokens": 3000},  # ... and of a prompt
        {"name": "bf16 decode 16", **_decode("bf16", 16, 2000)},  # an unquantized model, a batch of streams
        {"name": "bf16 prompt 1500 beside 8", **_prompt("bf16", 1500, 0, 8, 900)},  # continuous batching: a prompt beside eight streams
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["fp8 decode", "fp8 decode", "fp8 prompt", "fp8 prompt", "w4", "experts", "bf16 decode", "bf16 prompt"])
    if kind == "experts":
        return {"path": "experts", "tokens": size(1, 4096)}
    if kind.endswith("decode"):
        return _decode(kind.split()[0], size(1, 64), size(17, 4096), rng.random() < 0.5)
    if kind == "w4":
        return _decode("w4", size(1, 64), size(17, 2048), rng.random() < 0.5) if rng.random() < 0.6 else _prompt("w4", size(17, 1500))
    if kind == "fp8 prompt":
        portion = size(17, 3500)
        return _prompt("fp8", portion, size(16, 4096) if portion < 2000 and rng.random() < 0.4 else 0)
    rows = size(1, 16) if rng.random() < 0.5 else 0
    return _prompt("bf16", size(17, 2048), 0, rows, size(17, 2048) if rows else 0)


def _sequences(case):
    """``(tokens in the pages, new tokens)`` of every sequence, single tokens first."""
    n, c = case["rows"], case["context"]
    if case["ragged"] and n > 1:
        low = max(1, c // 20)
        seqs = [(low + (c - low) * ((7 * i) % n) // (n - 1) - 1, 1) for i in range(n)]
    else:
        seqs = [(c - 1, 1)] * n
    return seqs + ([(case["past"], case["portion"])] if case["portion"] else [])


# ---- seeded data: every tensor from the seed and its own name -------------------------------------------------------------

def _generator(seed, name):
    return torch.Generator(device="cuda").manual_seed(zlib.crc32(f"{seed}/{name}".encode()))


def _normal(seed, name, shape, std=1.0, dtype=torch.bfloat16):
    return torch.randn(shape, generator=_generator(seed, name), device="cuda", dtype=torch.float32).mul_(std).to(dtype)


def _ids(case, seed):
    count = sum(m for _, m in _sequences(case))
    return torch.randint(0, VOCAB, (count,), generator=_generator(seed, "ids"), device="cuda", dtype=torch.int32)


def _fp8_matrix(seed, name, n, k, std=0.02, stack=1):
    """E4M3 codes and 128 x 128 multipliers of a N(0, std) matrix: a block's largest value (about 4 std) sits at 448."""
    q = torch.empty((stack * n, k), dtype=torch.float8_e4m3fn, device="cuda")
    gen, step = _generator(seed, name), max(1, (1 << 28) // k)
    for a in range(0, stack * n, step):
        part = torch.randn((min(step, stack * n - a), k), generator=gen, device="cuda").mul_(112.0).clamp_(-E4M3_MAX, E4M3_MAX)
        q[a : a + step] = part.to(torch.float8_e4m3fn)
    s = torch.rand((stack * math.ceil(n / 128), k // 128), generator=gen, device="cuda").mul_(0.5).add_(0.75).mul_(std / 112.0)
    return (q, s) if stack == 1 else (q.view(stack, n, k), s.view(stack, -1, k // 128))


# The two projections that write into the stream are drawn smaller: a layer then adds a few hundredths of the stream, as in trained
# models, and the rounding of 8-bit activations does not pile up from layer to layer.
STD = {"o": 0.00025, "down": 0.00025}
MATRICES = {"qkv": ((HEADS + 2 * KV_HEADS) * DIM, WIDTH), "o": (WIDTH, HEADS * DIM), "gate_up": (2 * FF, WIDTH), "down": (WIDTH, FF)}


def _llama_norms(seed, name):
    return 1 + _normal(seed, name, (WIDTH,), 0.1)


def _past_rows(seed, layer, seqs):
    """What the q | k | v projection gave for the tokens that are in the pages already (one query head: it is not used)."""
    return _normal(seed, f"past{layer}", (sum(p for p, _ in seqs), (1 + 2 * KV_HEADS) * DIM), 1.28)


class _TepetarTensors:
    """Checkpoint tensors of the Tepetar under its canonical names."""

    def __init__(self, seed):
        self.seed = seed

    def shape(self, name):
        leaf = name.removeprefix("model.").split(".", 2)[2] if name.startswith("model.block.") else name
        return {
            "model.token_embedding.weight": (VOCAB, WIDTH), "model.output.weight": (VOCAB, WIDTH), "model.output_norm.weight": (WIDTH,),
            "model.token_side.embedding.weight": (VOCAB, LAYERS * SIDE), "attention.query.weight": (HEADS * DIM, WIDTH),
            "attention.query.bias": (HEADS * DIM,), "attention.key.weight": (KV_HEADS * DIM, WIDTH), "attention.key.bias": (KV_HEADS * DIM,),
            "attention.value.weight": (KV_HEADS * DIM, WIDTH), "attention.value.bias": (KV_HEADS * DIM,), "attention.output.weight": (WIDTH, HEADS * DIM),
            "attention.output.bias": (WIDTH,), "attention.query_norm.weight": (DIM,), "attention.key_norm.weight": (DIM,),
            "attention.post_norm.weight": (WIDTH,), "mlp.gate.weight": (FF, WIDTH), "mlp.up.weight": (FF, WIDTH), "mlp.down.weight": (WIDTH, FF),
            "mlp.post_norm.weight": (WIDTH,), "token_side.gate.weight": (SIDE, WIDTH), "token_side.projection.weight": (WIDTH, SIDE),
            "token_side.norm.weight": (WIDTH,)}[leaf]

    def __getitem__(self, name):
        if name.endswith("value_mix"):
            return torch.tensor(0.3)
        near_one = name.endswith(("query_norm.weight", "key_norm.weight", "token_side.norm.weight"))
        t = _normal(self.seed, name, self.shape(name), 0.1 if near_one else 0.02)
        return 1 + t if near_one else t


# ---- states -----------------------------------------------------------------------------------------------------------------

class _State:
    """Model, pages and the step of one case; ``graph`` replays a decode step, a batch with a prompt runs eagerly."""

    graph = None


def _llama(case, seed):
    weights = []
    for i in range(LAYERS):
        lin = {}
        for name, (n, k) in MATRICES.items():
            if case["path"] == "w4":
                lin[name] = W4Linear.from_float(_normal(seed, f"{name}{i}", (n, k), STD.get(name, 0.02)), GROUP)
            else:
                lin[name] = Fp8Linear(*_fp8_matrix(seed, f"{name}{i}", n, k, STD.get(name, 0.02)))
        weights.append(LlamaLayer(_llama_norms(seed, f"attn_norm{i}"), lin["qkv"], lin["o"], _llama_norms(seed, f"mlp_norm{i}"), lin["gate_up"], lin["down"]))
    cfg = LlamaConfig(vocab_size=VOCAB, hidden_size=WIDTH, intermediate_size=FF, num_layers=LAYERS, num_heads=HEADS, num_kv_heads=KV_HEADS,
                      head_dim=DIM, rope_theta=THETA, rms_eps=EPS)
    embed = _normal(seed, "embed", (VOCAB, WIDTH))  # a stream of unit size, as trained models have it
    return LlamaModel(cfg, LlamaWeights(embed, weights, _llama_norms(seed, "final_norm"), Fp8Linear(*_fp8_matrix(seed, "head", VOCAB, WIDTH))))


def _tepetar(seed):
    cfg = TepetarConfig.uniform(vocab_size=VOCAB, hidden_size=WIDTH, num_layers=LAYERS, heads=HEADS, kv_heads=KV_HEADS, dim=DIM, vdim=DIM,
                                window=WINDOW, ff=FF, side_dim=SIDE, rot_base=THETA, softcap=CAP, limit=LIMIT, norm_eps=SIDE_EPS)
    return TepetarModel(cfg, TepetarWeights(cfg, _TepetarTensors(seed), "cuda"))


def _i32(values):
    return torch.tensor(values, dtype=torch.int32).to("cuda")


def prepare(case, seed):
    s = _State()
    s.case = case
    if case["path"] == "experts":
        s.x = _normal(seed, "x", (case["tokens"], MOE_WIDTH))
        s.router = _normal(seed, "router", (EXPERTS, MOE_WIDTH), 0.02)
        s.gate_up = _fp8_matrix(seed, "experts.gate_up", 2 * MOE_FF, MOE_WIDTH, stack=EXPERTS)
        s.down = _fp8_matrix(seed, "experts.down", MOE_WIDTH, MOE_FF, stack=EXPERTS)
        return s
    seqs = _sequences(case)
    lens = [p + m for p, m in seqs]
    s.model = _tepetar(seed) if case["path"] == "bf16" else _llama(case, seed)
    pool = dict(num_pages=1 + sum(-(-n // PAGE) for n in lens), max_seqs=len(seqs), max_pages_per_seq=-(-max(lens) // PAGE), device="cuda")
    if case["path"] == "bf16":
        s.cache = s.model.make_cache(**pool)
        for i, l in enumerate(s.cache.pools):
            l.k.copy_(_normal(seed, f"keys{i}", l.k.shape))
            l.v.copy_(_normal(seed, f"values{i}", l.v.shape, 1.28))
        s.pages = [t for l in s.cache.pools for t in (l.k, l.v)]
    else:
        s.cache = PagedKVCache(layers=LAYERS, kv_heads=KV_HEADS, head_dim=DIM, **pool)
        s.pages = [s.cache.k, s.cache.v, s.cache.k_scale, s.cache.v_scale]
    for i, n in enumerate(lens):
        s.cache.assign(i, i, n)
    if case["path"] != "bf16" and any(p for p, _ in seqs):
        slots = torch.cat([s.cache.slots(i, 0, p) for i, (p, _) in enumerate(seqs)]).to("cuda")
        at = torch.cat([torch.arange(p, dtype=torch.int32) for p, _ in seqs]).to("cuda")
        for i in range(LAYERS):
            ops.rope_kv_write(_past_rows(seed, i, seqs), at, slots, s.cache.layer(i), n_q=1, n_kv=KV_HEADS, head_dim=DIM, theta=THETA)
    starts = [0]
    for _, m in seqs:
        starts.append(starts[-1] + m)
    s.ids = _ids(case, seed)
    s.positions = torch.cat([torch.arange(p, p + m, dtype=torch.int32) for p, m in seqs]).to("cuda")
    s.slots = torch.cat([s.cache.slots(i, p, m) for i, (p, m) in enumerate(seqs)]).to("cuda")
    s.seqs, s.starts, s.q_starts, s.seq_lens = seqs, starts, _i32(starts), _i32(lens)
    s.tok_seq = _i32([i for i, (_, m) in enumerate(seqs) for _ in range(m)])
    s.last_rows = _i32([e - 1 for e in starts[1:]])
    if case["path"] == "bf16":
        s.model.attn_splits = s.model.decode_splits(max(1, case["rows"]), max(lens))
    elif not case["portion"]:
        s.model.attn_splits = attn_splits_for(len(seqs), KV_HEADS, max(lens), DIM, HEADS // KV_HEADS)
    if not case["portion"]:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                _decode_forward(s)
        torch.cuda.current_stream().wait_stream(side)
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph):
            s.logits = _decode_forward(s)
    return s


def _decode_forward(s):
    step = StepBuffers(input_ids=s.ids, positions=s.positions, slots=s.slots, block_table=s.cache.block_table, seq_lens=s.seq_lens)
    return s.model.forward(step, s.cache, prefill=False)


def run(state):
    s = state
    if s.case["path"] == "experts":
        ids, weights = moe.router_topk(s.x, s.router, TOP_K)
        out = moe.moe_ffn_fp8(*ops.quant_rows(s.x), ids, weights, *s.gate_up, *s.down, base=s.x)
        return {"ids": ids, "weights": weights, "out": out}
    if s.graph is not None:
        s.graph.replay()
        return {"logits": s.logits, "pages": s.pages}
    if s.model.ragged:
        step = StepBuffers(input_ids=s.ids, positions=s.positions, slots=s.slots, block_table=s.cache.block_table, seq_lens=s.seq_lens,
                           cu_seqlens=s.starts, q_starts=s.q_starts, tok_seq=s.tok_seq, max_q=s.case["portion"], num_decode=s.case["rows"],
                           portions=s.seqs)
    else:
        past = s.case["past"]
        step = StepBuffers(input_ids=s.ids, positions=s.positions, slots=s.slots, cu_seqlens=s.starts, past_len=past,
                           block_table=s.cache.block_table if past else None)
    return {"logits": s.model.forward(step, s.cache, prefill=True, logits_rows=s.last_rows), "pages": s.pages}


# ---- what a pass cannot do without --------------------------------------------------------------------------------------------

def work(case):
    if case["path"] == "experts":
        t, one = case["tokens"], 3 * MOE_WIDTH * MOE_FF
        touched = EXPERTS * (1 - (1 - TOP_K / EXPERTS) ** t)  # experts that some token takes
        return {"bytes": touched * one * (1 + 4 / 128 ** 2) + 2 * EXPERTS * MOE_WIDTH + 4 * t * MOE_WIDTH + 8 * t * TOP_K,
                "flops": 2.0 * t * (TOP_K * one + EXPERTS * MOE_WIDTH)}
    seqs, bf16 = _sequences(case), case["path"] == "bf16"
    t, rows = sum(m for _, m in seqs), len(seqs)
    block = LAYERS * sum(n * k for n, k in MATRICES.values())
    per = {"fp8": 1 + 4 / 128 ** 2, "w4": 0.5 + 4 / GROUP, "bf16": 2.0}[case["path"]]
    side = 2 * LAYERS * SIDE * WIDTH if bf16 else 0
    token = 2 * KV_HEADS * DIM * (2 if bf16 else 1) + (0 if bf16 else 8 * KV_HEADS)  # page bytes of a token in a layer
    seen = [min(p, WINDOW) if bf16 else p for p, _ in seqs]
    reads = block * per + 2 * side + VOCAB * WIDTH * (2 if bf16 else 1) + LAYERS * token * sum(seen) + t * (2 * WIDTH + (2 * LAYERS * SIDE if bf16 else 0))
    writes = LAYERS * token * t + 2 * rows * VOCAB
    pairs = 0
    for p, m in seqs:
        full = p * m + m * (m + 1) // 2  # (query, key) pairs of a causal mask
        if bf16:
            full = sum(min(p + i + 1, WINDOW) for i in range(m))
        pairs += full
    return {"bytes": reads + writes, "flops": 2.0 * t * (block + side) + 2.0 * rows * VOCAB * WIDTH + 4.0 * LAYERS * HEADS * DIM * pairs}


def tolerance(case):
    """Bounds for another order of the sums.  ``fp8``, ``w4``: any difference moves some values across a step of the 8-bit rows (one
    step is 6 to 12 % of a value), and after a few layers the logits differ by 0.016 to 0.023 (largest single value 0.2) whatever
    the first difference was: measured between two roundings of the residual sum.  ``bf16`` logits are 0.009 off the exact ones,
    expert outputs 0.002; router scores tie within 32-bit sums about once in ten thousand places."""
    if case["path"] == "experts":
        return {"rel": 0.008, "max": 0.5, "differ": 0.002}
    if case["path"] == "bf16":
        return {"rel": 0.02, "max": 0.3}
    return {"rel": 0.03, "max": 0.6}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------------------

def _e4m3(x):
    """``x`` as E4M3 codes with one multiplier per row (last axis), the form activations and cached rows have."""
    s = x.abs().amax(-1, keepdim=True).clamp_min(1e-12) / E4M3_MAX
    return (x / s).clamp(-E4M3_MAX, E4M3_MAX).float().to(torch.float8_e4m3fn).double() * s


def _blocks(q, s):
    return q.double() * s.double().repeat_interleave(128, 0)[: q.shape[0]].repeat_interleave(128, 1)


def _four_bits(w):
    """The reconstruction of a matrix from 4-bit codes with a bf16 step and offset per group."""
    g = w.double().view(w.shape[0], -1, GROUP)
    lo = g.amin(-1, keepdim=True)
    step = (g.amax(-1, keepdim=True) - lo) / 15
    codes = ((g - lo) / step).round().clamp(0, 15)
    return (codes * step.bfloat16().double() + lo.bfloat16().double()).bfloat16().double().view(w.shape)


def _rms(x, w, eps):
    return x / (x.square().mean(-1, keepdim=True) + eps).sqrt() * w.double()


def _turn(x, at):
    """``x [T, heads, DIM]`` turned by position, channel i with i + DIM / 2."""
    f = THETA ** (-2 * torch.arange(DIM // 2, device=x.device, dtype=torch.float64) / DIM)
    a = at.double()[:, None, None] * f
    u, v = x[..., : DIM // 2], x[..., DIM // 2 :]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def _attend(q, k, v, past, window=None, cap=0.0):
    m, n, g = q.shape[0], k.shape[0], HEADS // KV_HEADS
    first = max(0, past + 1 - window) if window else 0  # keys before it are out of every query's sight
    k, v = k[first:], v[first:]
    back = (past + torch.arange(m, device=q.device))[:, None] - torch.arange(first, n, device=q.device)
    hidden = (back < 0) | (back >= window) if window else back < 0
    out = torch.empty_like(q)
    for h in range(HEADS):
        s = (q[:, h] @ k[:, h // g].T) / math.sqrt(DIM)
        s = cap * torch.tanh(s / cap) if cap else s
        out[:, h] = torch.softmax(s.masked_fill_(hidden, -math.inf), -1) @ v[:, h // g]
    return out


def _exact_llama(case, seed):
    seqs = _sequences(case)
    w4 = case["path"] == "w4"

    def product(x, name, i=""):
        n, k = MATRICES.get(name, (VOCAB, WIDTH))
        if w4 and name != "head":
            return x @ _four_bits(_normal(seed, f"{name}{i}", (n, k), STD.get(name, 0.02))).T
        return _e4m3(x) @ _blocks(*_fp8_matrix(seed, f"{name}{i}", n, k, STD.get(name, 0.02))).T

    x = _normal(seed, "embed", (VOCAB, WIDTH))[_ids(case, seed).long()].double()
    at = torch.cat([torch.arange(p, p + m) for p, m in seqs]).to("cuda")
    for i in range(LAYERS):
        qkv = product(_rms(x, _llama_norms(seed, f"attn_norm{i}"), EPS), "qkv", i).view(len(x), -1, DIM)
        q, k, v = qkv.split([HEADS, KV_HEADS, KV_HEADS], 1)
        q, k, v = _turn(q, at), _e4m3(_turn(k, at)), _e4m3(v)
        past, o, row, done = _past_rows(seed, i, seqs).view(-1, 1 + 2 * KV_HEADS, DIM), torch.empty_like(q), 0, 0
        for p, m in seqs:
            old = past[done : done + p].double()
            kk = torch.cat([_e4m3(_turn(old[:, 1 : 1 + KV_HEADS], torch.arange(p, device="cuda"))), k[row : row + m]])
            vv = torch.cat([_e4m3(old[:, 1 + KV_HEADS :]), v[row : row + m]])
            o[row : row + m] = _attend(q[row : row + m], kk, vv, p)
            row, done = row + m, done + p
        x = x + product(o.reshape(len(x), -1), "o", i)
        gate, up = product(_rms(x, _llama_norms(seed, f"mlp_norm{i}"), EPS), "gate_up", i).chunk(2, 1)
        x = x + product(torch.nn.functional.silu(gate) * up, "down", i)
    ends = torch.tensor([m for _, m in seqs]).cumsum(0).sub(1).to("cuda")
    logits = product(_rms(x[ends], _llama_norms(seed, "final_norm"), EPS), "head")
    return {"logits": logits, "pages": [None] * 4}  # pages hold 8-bit codes


def _exact_tepetar(case, seed):
    seqs, w = _sequences(case), _TepetarTensors(seed)
    get = lambda name: w[name].to("cuda").double()  # noqa: E731
    ids = _ids(case, seed).long()
    x = w["model.token_embedding.weight"][ids].double()
    table = w["model.token_side.embedding.weight"][ids].double()
    at = torch.cat([torch.arange(p, p + m) for p, m in seqs]).to("cuda")
    counts = [-(-(p + m) // PAGE) for p, m in seqs]
    page_shape = (1 + sum(counts), KV_HEADS, PAGE, DIM)
    first, pages = None, []

    def add(x, y, name):
        return x + _rms(y, 1 + get(name), SIDE_EPS)

    for i in range(LAYERS):
        p = f"model.block.{i}."
        q, k, v = (x @ get(p + f"attention.{n}.weight").T + get(p + f"attention.{n}.bias") for n in ("query", "key", "value"))
        q, k, v = q.view(len(x), HEADS, DIM), k.view(len(x), KV_HEADS, DIM), v.view(len(x), KV_HEADS, DIM)
        q, k = (_turn(_rms(t, get(p + f"attention.{n}_norm.weight"), SIDE_EPS), at) for t, n in ((q, "query"), (k, "key")))
        first = v if i == 0 else first
        v = v if i == 0 else 0.7 * v + 0.3 * first
        pk, pv = _normal(seed, f"keys{i}", page_shape).double(), _normal(seed, f"values{i}", page_shape, 1.28).double()
        o, row, page = torch.empty_like(q), 0, 1  # pages are handed out in order, from the second on
        for (n, m), c in zip(seqs, counts):
            for pool, new in ((pk, k), (pv, v)):
                rows = pool[page : page + c].transpose(1, 2).reshape(c * PAGE, KV_HEADS, DIM)
                rows[n : n + m] = new[row : row + m]
                pool[page : page + c] = rows.view(c, PAGE, KV_HEADS, DIM).transpose(1, 2)
                kk, vv = (rows[: n + m], None) if pool is pk else (kk, rows[: n + m])
            o[row : row + m] = _attend(q[row : row + m], kk, vv, n, WINDOW, CAP)
            row, page = row + m, page + c
        pages += [pk, pv]
        x = add(x, o.reshape(len(x), -1) @ get(p + "attention.output.weight").T + get(p + "attention.output.bias"), p + "attention.post_norm.weight")
        g = (x @ get(p + "mlp.gate.weight").T).clamp_max(LIMIT)
        u = (x @ get(p + "mlp.up.weight").T).clamp(-LIMIT, LIMIT)
        x = add(x, (g * torch.sigmoid(1.702 * g) * (u + 1)) @ get(p + "mlp.down.weight").T, p + "mlp.post_norm.weight")
        y = torch.nn.functional.gelu(x @ get(p + "token_side.gate.weight").T, approximate="tanh") * table[:, i * SIDE : (i + 1) * SIDE]
        x = x + _rms(y @ get(p + "token_side.projection.weight").T, get(p + "token_side.norm.weight"), SIDE_EPS)
    ends = torch.tensor([m for _, m in seqs]).cumsum(0).sub(1).to("cuda")
    logits = _rms(x[ends], 1 + get("model.output_norm.weight"), SIDE_EPS) @ get("model.output.weight").T
    return {"logits": logits, "pages": pages}


def _exact_experts(case, seed):
    x = _normal(seed, "x", (case["tokens"], MOE_WIDTH)).double()
    scores = torch.softmax(x @ _normal(seed, "router", (EXPERTS, MOE_WIDTH), 0.02).double().T, -1)
    weights, ids = scores.topk(TOP_K, -1)
    weights = weights / weights.sum(-1, keepdim=True)
    gq, gs = _fp8_matrix(seed, "experts.gate_up", 2 * MOE_FF, MOE_WIDTH, stack=EXPERTS)
    dq, ds = _fp8_matrix(seed, "experts.down", MOE_WIDTH, MOE_FF, stack=EXPERTS)
    out, xq = x.clone(), _e4m3(x)
    for e in range(EXPERTS):
        tok, place = (ids == e).nonzero(as_tuple=True)
        if tok.numel():
            gate, up = (xq[tok] @ _blocks(gq[e], gs[e]).T).chunk(2, 1)
            y = _e4m3(torch.nn.functional.silu(gate) * up) @ _blocks(dq[e], ds[e]).T
            out.index_add_(0, tok, y * weights[tok, place][:, None])
    return {"ids": ids.int(), "weights": weights, "out": out}


def exact(case, seed):
    return {"experts": _exact_experts, "bf16": _exact_tepetar}.get(case["path"], _exact_llama)(case, seed)
