"""The work whose speed is measured: steps of the engine, from one decoded token to a full prompt batch.

A pass is what the engine does for one step of ``LLM.generate``: the packed step buffer (block tables, positions, token ids) goes
from pinned host memory to the GPU, the model runs over the paged cache, and the logits of every sequence's last token come out.
Decode steps are padded to the engine's batch buckets and replayed from a CUDA graph, prompt steps run eagerly, as in
``engine/worker.py``.  Logits are returned instead of sampled tokens, because a token says nothing about how close a result is,
and beside them what the step has written for the first few sequences: the newest keys and values, latents and states.

A case says which model, how many layers of it, how many sequences (``seqs``), and the range that their lengths are spread over
(``lo`` to ``hi``).  The layers of a model are alike, and the roundings of bf16 add up over them: a stack of 12 (4 with block-scaled
fp8 weights, whose activations are rounded to e4m3 as well) is deep enough for a step's real proportions and shallow enough that
results of two correct implementations can be told from wrong ones.
For ``decode`` a length is the number of cached tokens with the new one; for ``prefill`` it is the length of the prompt, to
which ``prefix`` cached tokens shared by all sequences (a hit of the prefix cache) come on top.
"""
import math
import random

import numpy as np
import torch
import torch.nn.functional as F

from tinyllmforge_b200 import Config, preset
from tinyllmforge_b200.engine.request import Request
from tinyllmforge_b200.engine.step_batch import build_decode, build_prefill
from tinyllmforge_b200.engine.worker import DeviceBatch, Worker, graph_buckets
from tinyllmforge_b200.models.goselix_config import GoselixConfig, example_dict
from tinyllmforge_b200.ops.quant import Fp8BlockWeight
from tinyllmforge_b200.parallel.comm import TPGroup

BLOCK = 256                     # the engine's default cache block
MAX_LEN = 4096 + 512            # longest sequence of any case
GOSELIX_WIDTH = 2048
LAYERS, LAYERS_FP8 = 12, 4
SHOWN = 8                       # sequences whose newest memory is returned


def listed():
    small, large, hybrid = "qwen3-0.6b", "qwen3-8b", "goselix"
    return [
        # one user of the small model, early in an answer: the smallest call, all latency
        {"name": "small decode 1", "model": small, "layers": LAYERS, "kind": "decode", "seqs": 1, "lo": 300, "hi": 300, "prefix": 0, "fp8": False},
        # a batch that has thinned out, or a modest server load
        {"name": "small decode 61", "model": small, "layers": LAYERS, "kind": "decode", "seqs": 61, "lo": 200, "hi": 2000, "prefix": 0, "fp8": False},
        # steady state of the 256-request benchmark workload
        {"name": "small decode 256", "model": small, "layers": LAYERS, "kind": "decode", "seqs": 256, "lo": 100, "hi": 1500, "prefix": 0, "fp8": False},
        # first token of one short question: latency of a prompt step
        {"name": "small prefill 1", "model": small, "layers": LAYERS, "kind": "prefill", "seqs": 1, "lo": 107, "hi": 107, "prefix": 0, "fp8": False},
        # a full token budget of ragged prompts, as the benchmark workload admits them
        {"name": "small prefill 28", "model": small, "layers": LAYERS, "kind": "prefill", "seqs": 28, "lo": 100, "hi": 1024, "prefix": 0, "fp8": False},
        # one user of the large model, some way into a conversation
        {"name": "large decode 1", "model": large, "layers": LAYERS, "kind": "decode", "seqs": 1, "lo": 3001, "hi": 3001, "prefix": 0, "fp8": False},
        # the large model under load
        {"name": "large decode 64", "model": large, "layers": LAYERS, "kind": "decode", "seqs": 64, "lo": 300, "hi": 2000, "prefix": 0, "fp8": False},
        # one long document
        {"name": "large prefill 1", "model": large, "layers": LAYERS, "kind": "prefill", "seqs": 1, "lo": 3777, "hi": 3777, "prefix": 0, "fp8": False},
        # requests that share a system prompt of 4096 tokens: only their suffixes are computed
        {"name": "large prefix 8", "model": large, "layers": LAYERS, "kind": "prefill", "seqs": 8, "lo": 256, "hi": 256, "prefix": 4096, "fp8": False},
        # block-scaled e4m3 weights, a few users
        {"name": "large fp8 decode 13", "model": large, "layers": LAYERS_FP8, "kind": "decode", "seqs": 13, "lo": 200, "hi": 2000, "prefix": 0, "fp8": True},
        # latent attention and retention: prompts and decode
        {"name": "goselix prefill 8", "model": hybrid, "layers": 4, "kind": "prefill", "seqs": 8, "lo": 500, "hi": 1024, "prefix": 0, "fp8": False},
        {"name": "goselix decode 64", "model": hybrid, "layers": 4, "kind": "decode", "seqs": 64, "lo": 500, "hi": 1500, "prefix": 0, "fp8": False},
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    model = rng.choice(["qwen3-0.6b", "qwen3-0.6b", "qwen3-8b", "qwen3-8b", "goselix"])
    kind = rng.choice(["decode", "prefill"])
    fp8 = model == "qwen3-8b" and kind == "decode" and rng.random() < 0.3
    case = {"model": model, "layers": 4 if model == "goselix" else LAYERS_FP8 if fp8 else LAYERS, "kind": kind, "prefix": 0, "fp8": fp8}
    if kind == "decode":
        top = {"qwen3-0.6b": 256, "qwen3-8b": 64, "goselix": 64}[model]
        case["seqs"] = _log_uniform(rng, 1, top)
        lo = _log_uniform(rng, 100, 1000)
        case.update(lo=lo, hi=rng.randint(lo, 2000 if case["seqs"] <= 64 else 1500))
        return case
    if model == "qwen3-8b" and rng.random() < 0.5:
        case["prefix"] = BLOCK * rng.randint(1, 16)
    budget = {"qwen3-0.6b": 16000, "qwen3-8b": 2048 if case["prefix"] else 3700, "goselix": 6000}[model]
    hi = _log_uniform(rng, 17, min(budget, 4000 if not case["prefix"] else 400))
    case.update(lo=rng.randint(max(1, hi // 3), hi), hi=hi)
    case["seqs"] = min(64, rng.randint(1, max(1, budget // hi)))
    return case


# ------------------------------------------------------------------------------------------------ shapes of a case
def _lengths(case):
    """Lengths of the sequences: part of the case, not of the seed (the work must not depend on the seed)."""
    r = random.Random(f"{case['seqs']} {case['lo']} {case['hi']}")
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["seqs"])]


def _config(case):
    if case["model"] == "goselix":
        # dense feed-forwards in every layer: with routed ones a near-tie sends a token to another expert, and no tolerance tells that from an error
        d = example_dict(GOSELIX_WIDTH, case["layers"])
        for layer in d["layers"]:
            layer["mlp"] = d["layers"][0]["mlp"]
        return GoselixConfig.from_dict(d)
    return preset(case["model"], num_hidden_layers=case["layers"])


def _requests(case, vocab, seed):
    """Requests with their tokens, blocks in shuffled order (a pool that has been in use), and one state slot each."""
    rng = np.random.default_rng(seed)
    lengths = _lengths(case)
    shared = case["prefix"] // BLOCK
    need = [-(-n // BLOCK) for n in lengths]
    blocks = rng.permutation(shared + sum(need)).tolist()
    head, at = blocks[:shared], shared
    prefix = rng.integers(0, vocab, case["prefix"]).tolist()
    reqs = []
    for i, (n, k) in enumerate(zip(lengths, need)):
        r = Request(prefix + rng.integers(0, vocab, n).tolist())
        r.block_table = head + blocks[at:at + k]
        r.num_cached_tokens = case["prefix"]
        r.state_slot = i
        at += k
        reqs.append(r)
    return reqs, shared + sum(need)


# ------------------------------------------------------------------------------------------------ a pass
class State:
    pass


def _fill_memory(model, seed):
    """What earlier steps have left behind: keys of unit size after their norm, values of a projection's size that have a direction
    in common (as the values of one text do), latents of unit size, retention states."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    if hasattr(model, "kv_cache"):
        size = 0.7 * 0.02 * model.cfg.hidden_size ** 0.5
        for layer in model.kv_cache:
            layer.normal_(generator=gen)
            common = torch.randn(1, layer.shape[2], 1, layer.shape[4], device="cuda", generator=gen)
            layer[1].mul_(size).add_((size * common).to(layer.dtype))
        return
    for m in model.memory:
        m.normal_(0.0, 0.5 if m.dtype == torch.float32 else 1.0, generator=gen)


@torch.inference_mode()
def prepare(case, seed):
    cfg = _config(case)
    reqs, blocks = _requests(case, cfg.vocab_size, seed)
    config = Config("perf", hf_config=cfg, load_format="dummy", seed=seed, max_model_len=MAX_LEN, max_num_batched_tokens=16384, enforce_eager=True,
                    num_kvcache_blocks=blocks, max_num_seqs=max(1, len(reqs)), quantization="fp8_block" if case["fp8"] else None)
    s = State()
    s.worker = worker = Worker(config, 0, TPGroup())
    s.model = worker.model
    s.graph = None
    if case["kind"] == "decode":
        bucket = next(b for b in graph_buckets(512) if b >= len(reqs))
        s.step = build_decode(reqs, BLOCK, pad_to=bucket, table_width=worker.table_width)
    else:
        s.step = build_prefill(reqs, BLOCK)
    s.host = torch.from_numpy(s.step.buf[:s.step.num_words].copy()).pin_memory()
    s.words = s.host.cuda()
    s.batch = DeviceBatch(s.step, s.words)
    if case["kind"] == "decode":
        _forward(s)                                 # ahead of the capture, as the engine does
        torch.cuda.synchronize()
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph):
            s.logits = _forward(s)
    _fill_memory(s.model, seed)
    s.newest = _newest(s, reqs[:SHOWN])
    torch.cuda.synchronize()
    return s


def _newest(s, reqs):
    """Views of what a step writes last for these requests."""
    at = [(r.block_table[(len(r) - 1) // BLOCK], (len(r) - 1) % BLOCK) for r in reqs]
    if hasattr(s.model, "kv_cache"):
        return [s.model.kv_cache[:, :, b, :, o] for b, o in at]
    return [m[:len(reqs)] if layer.mix.recurrent else [m[b, o] for b, o in at] for layer, m in zip(s.model.layers, s.model.memory)]


def _forward(s):
    return s.model.compute_logits(s.model.forward(s.batch), s.batch)


@torch.inference_mode()
def run(s):
    s.words.copy_(s.host, non_blocking=True)
    if s.graph is None:
        s.logits = _forward(s)
    else:
        s.graph.replay()
    return {"logits": s.logits[:s.step.num_seqs], "newest": s.newest}


# ------------------------------------------------------------------------------------------------ work and tolerance
def _queries_and_keys(case):
    """[(queries, keys seen by the last one)] per sequence."""
    return [(1, n) if case["kind"] == "decode" else (n, case["prefix"] + n) for n in _lengths(case)]


def work(case):
    cfg = _config(case)
    seqs = _queries_and_keys(case)
    T, rows = sum(q for q, _ in seqs), len(seqs)
    keys = sum(k for _, k in seqs) - (len(seqs) - 1) * case["prefix"]             # a shared prefix is read once
    pairs = sum(q * k - q * (q - 1) // 2 for q, k in seqs)
    W, V = cfg.hidden_size, cfg.vocab_size
    nbytes, flops = 2.0 * (V * W + T * W + rows * V), 2.0 * V * W * rows          # head, embedding rows, logits
    if case["model"] != "goselix":
        d, H, G, I, L = cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.intermediate_size, cfg.num_hidden_layers
        params = W * (H + 2 * G) * d + H * d * W + 3 * W * I
        nbytes += L * (params * (1 if case["fp8"] else 2) + 4 * G * d * (keys + (0 if case["kind"] == "prefill" and not case["prefix"] else T)))
        flops += L * (2.0 * params * T + 4.0 * H * d * pairs)
        return {"bytes": nbytes, "flops": flops}
    for i in range(len(cfg.layers)):
        m, ff = cfg.layers[i].mixer, cfg.layers[i].mlp
        if cfg.layers[i].type == "latent_attention":
            params = (m.q_rank + m.kv_rank + m.rot_dim) * W + m.heads * ((m.dim + m.rot_dim) * m.q_rank + (m.dim + m.vdim) * m.kv_rank + m.vdim * W)
            nbytes += 2 * (m.kv_rank + m.rot_dim) * (keys + T)
            flops += 2.0 * m.heads * pairs * ((2 * m.kv_rank + m.rot_dim) if case["kind"] == "decode" else (m.dim + m.rot_dim + m.vdim))
        else:
            params = m.heads * (2 * m.dim + 3 * m.vdim) * W
            nbytes += 4 * rows * m.heads * m.dim * m.vdim * (2 if case["kind"] == "decode" else 1)
            flops += 4.0 * T * m.heads * m.dim * m.vdim
        nbytes += 2 * params
        flops += 2.0 * params * T
        nbytes += 2 * 3 * W * ff.ff
        flops += 2.0 * T * 3 * W * ff.ff
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """bf16 operands and a bf16 residual stream (Qwen3): a rounding of 2^-9 at each addition of the stream and at each operand.  With
    the attention's sums in another order, logits of 12 layers were 0.002 to 0.016 apart (largest single value 0.08); 0.006 to 0.023 from 64 bits."""
    return {"rel": 0.03, "max": 0.2}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _norm(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, positions, base):
    """x [tokens, heads, d]: entry i together with entry i + d / 2."""
    half = x.shape[-1] // 2
    angle = positions[:, None].double() * base ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    return torch.cat([x[..., :half] * c - x[..., half:] * s, x[..., half:] * c + x[..., :half] * s], dim=-1)


def _attend(q, k, v, scale, first):
    """Causal attention; q [n, H, d] at positions first.., k and v [m, G, .] from position 0."""
    share = q.shape[1] // k.shape[1]
    hidden = torch.arange(k.shape[0], device=q.device)[None] > first + torch.arange(q.shape[0], device=q.device)[:, None]
    out = []
    for h in range(q.shape[1]):
        scores = (q[:, h] @ k[:, h // share].T * scale).masked_fill_(hidden, float("-inf"))
        out.append(torch.softmax(scores, -1) @ v[:, h // share])
    return torch.stack(out, 1)


def _weight(w):
    if not isinstance(w, Fp8BlockWeight):
        return w.double()
    n, k = w.shape
    return w.q.double() * w.scale.double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)


def _linear(x, w, quantized):
    """x @ w.T; with block-scaled e4m3 weights, steps of up to 128 tokens round their activations to e4m3 too, per token and 128 features."""
    if quantized and x.shape[0] <= 128:
        b = x.view(x.shape[0], -1, 128)
        scale = b.abs().amax(-1, keepdim=True) / 448.0
        x = ((b / scale).float().to(torch.float8_e4m3fn).double() * scale).view(x.shape)
    return x @ _weight(w).T


def _slots(table, n):
    """(blocks, offsets) of tokens 0..n-1."""
    at = torch.arange(n, device="cuda")
    return table[at // BLOCK], at % BLOCK


def _exact_qwen3(case, s, cfg):
    model, fp8 = s.model, case["fp8"]
    seqs = _queries_and_keys(case)
    tokens = sum(q for q, _ in seqs)
    ids = torch.from_numpy(s.step.input_ids[:tokens].copy()).cuda().long()
    positions = torch.from_numpy(s.step.positions[:tokens].copy()).cuda()
    tables = torch.from_numpy(s.step.block_tables.copy()).cuda().long()
    H, G, d = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim
    x = model.embed_tokens.weight[ids].double()
    last = torch.tensor([q for q, _ in seqs], device="cuda").cumsum(0) - 1
    newest = []
    for layer, cache in zip(model.layers, model.kv_cache):
        qkv = _linear(_norm(x, cfg.rms_norm_eps), layer.qkv_proj.weight, fp8).view(tokens, H + 2 * G, d)
        q = _rotate(_norm(qkv[:, :H], cfg.rms_norm_eps), positions, cfg.rope_theta)
        k = _rotate(_norm(qkv[:, H:H + G], cfg.rms_norm_eps), positions, cfg.rope_theta)
        newest.append(torch.stack([k[last[:SHOWN]], qkv[last[:SHOWN], H + G:]], 1))
        out, at = [], 0
        for i, (n, m) in enumerate(seqs):
            b, o = _slots(tables[i], m - n)
            past = cache[:, b, :, o].double()                                    # [m - n, 2, G, d]: indexed dimensions come first
            keys, values = (torch.cat([past[:, j], new[at:at + n]]) for j, new in ((0, k), (1, qkv[:, H + G:])))
            out.append(_attend(q[at:at + n], keys, values, d ** -0.5, m - n))
            at += n
        x = x + _linear(torch.cat(out).reshape(tokens, H * d), layer.o_proj.weight, fp8)
        gate, up = _linear(_norm(x, cfg.rms_norm_eps), layer.gate_up_proj.weight, fp8).chunk(2, dim=-1)
        x = x + _linear(F.silu(gate) * up, layer.down_proj.weight, fp8)
    logits = _norm(x[last], cfg.rms_norm_eps) @ model.lm_head.weight.double().T
    return {"logits": logits, "newest": list(torch.stack(newest, 1))}


def _exact_latent(h, mix, m, cache, seqs, positions, tables, eps):
    T = h.shape[0]
    both = h @ mix.a_proj.double().T
    q = (_norm(both[:, :m.q_rank], eps) @ mix.uq.double().T).view(T, m.heads, m.dim + m.rot_dim)
    q = torch.cat([q[..., :m.dim], _rotate(q[..., m.dim:], positions, m.rot.base)], -1)
    c = torch.cat([_norm(both[:, m.q_rank:m.q_rank + m.kv_rank], eps), _rotate(both[:, None, m.q_rank + m.kv_rank:], positions, m.rot.base)[:, 0]], -1)
    out, at = [], 0
    for i, (n, total) in enumerate(seqs):
        b, o = _slots(tables[i], total - n)
        rows = torch.cat([cache[b, o].double(), c[at:at + n]])
        kv = (rows[:, :m.kv_rank] @ mix.ukv.double().T).split([m.heads * m.dim, m.heads * m.vdim], -1)
        k = torch.cat([kv[0].view(total, m.heads, m.dim), rows[:, None, m.kv_rank:].expand(-1, m.heads, -1)], -1)
        out.append(_attend(q[at:at + n], k, kv[1].view(total, m.heads, m.vdim), m.scale, total - n))
        at += n
    last = torch.tensor([q for q, _ in seqs], device="cuda").cumsum(0) - 1
    return torch.cat(out).reshape(T, -1) @ mix.o.double().T, list(c[last[:SHOWN]])


def _exact_retention(h, mix, m, state, seqs, positions, decode, eps):
    """o_i = sum over j <= i of decay^(i - j) (q_i k_j) v_j, plus decay^(i + 1) times the state before the step (decode)."""
    T = h.shape[0]
    q, k, v, g = (h @ mix.qkvg.double().T).split([m.heads * m.dim, m.heads * m.dim, m.heads * m.vdim, m.heads * m.vdim], -1)
    q = _rotate(q.reshape(T, m.heads, m.dim), positions, m.rot.base)
    k = _rotate(k.reshape(T, m.heads, m.dim), positions, m.rot.base) * m.dim ** -0.5
    v = v.reshape(T, m.heads, m.vdim)
    decay = mix.decay.double()
    out, states, at = [], [], 0
    for i, (n, _) in enumerate(seqs):
        steps = torch.arange(n, device="cuda", dtype=torch.float64)
        back = steps[:, None] - steps[None]
        qi, ki, vi = (t[at:at + n].transpose(0, 1) for t in (q, k, v))
        weights = decay[:, None, None] ** back.clamp(min=0) * (back >= 0)
        o = (qi @ ki.transpose(1, 2) * weights) @ vi
        after = (ki * weights[:, -1, :, None]).transpose(1, 2) @ vi
        if decode:
            o = o + (decay[:, None] ** (steps + 1))[..., None] * (qi @ state[i].double())
            after = after + decay[:, None, None] ** n * state[i].double()
        if i < SHOWN:
            states.append(after)
        out.append(o.transpose(0, 1))
        at += n
    y = _norm(torch.cat(out), eps).reshape(T, -1) * F.silu(g)
    return y @ mix.o.double().T, torch.stack(states)


def _gated(h, gate_up, down):
    gate, up = (h @ gate_up.double().T).chunk(2, -1)
    return (F.silu(gate) * up) @ down.double().T


def _exact_goselix(case, s, cfg):
    model, eps, decode = s.model, cfg.rms_norm_eps, case["kind"] == "decode"
    seqs = _queries_and_keys(case)
    tokens = sum(q for q, _ in seqs)
    positions = torch.from_numpy(s.step.positions[:tokens].copy()).cuda()
    tables = torch.from_numpy(s.step.block_tables.copy()).cuda().long()
    x = model.embed.weight[torch.from_numpy(s.step.input_ids[:tokens].copy()).cuda().long()].double()
    newest = []
    for layer, memory in zip(model.layers, model.memory):
        h, m = _norm(x, eps), layer.mix.spec
        if layer.mix.recurrent:
            y, new = _exact_retention(h, layer.mix, m, memory, seqs, positions, decode, eps)
        else:
            y, new = _exact_latent(h, layer.mix, m, memory, seqs, positions, tables, eps)
        newest.append(new)
        x = x + y + _gated(h, layer.mlp.gate_up, layer.mlp.down)
    last = torch.tensor([q for q, _ in seqs], device="cuda").cumsum(0) - 1
    return {"logits": _norm(x[last], eps) @ model.head.weight.double().T, "newest": newest}


@torch.inference_mode()
def exact(case, seed):
    s = prepare(case, seed)
    return (_exact_goselix if case["model"] == "goselix" else _exact_qwen3)(case, s, _config(case))
