"""The work that users have this framework do, as cases of known size: model sessions and the serving engine.

A case is a dict of plain values.  ``listed()`` gives the fixed ones, ``draw(rng)`` one more of the same ranges,
``prepare`` what a program holds before the call (a session or an engine with its weights, and the inputs),
``run`` one pass through the public entry points, ``exact`` what a session's pass gives in 64 bits, ``work`` the bytes
and operations a pass cannot do without.

Models are the ones the package builds itself, with random weights.  Two scales differ from the builders' defaults,
both in the serving cases: token embeddings are as large as in a trained decoder (standard deviation 0.14 for GPT-2,
2 for BitNet) and BitNet's residual projections carry the 1 / sqrt(2 layers) that GPT-2's have.  With the default
scales next-token scores are nearly level and two correct implementations choose different tokens; with these the
winner leads clearly, as it does after training, and every shape, layer and kernel is the same.
"""
from __future__ import annotations

import functools
import math

import torch
import torch.nn.functional as F

from ronn_b200 import Model, SessionOptions
from ronn_b200.models.bitnet_llama import BitNetConfig, build_bitnet_llama
from ronn_b200.models.distilbert import DistilBertConfig, build_distilbert
from ronn_b200.models.gpt2 import GPT2Config, build_gpt2
from ronn_b200.models.mlp784 import build_mlp784
from ronn_b200.models.resnet18 import build_resnet18
from ronn_b200.serving import EngineConfig, LLMEngine, SamplingParams

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
_BLOCK = 16                                    # tokens of a KV-cache block


# ---------------------------------------------------------------------------------------------------- the cases
def _mlp(name, batch, dtype="bf16"):
    return dict(name=name, model="mlp784", batch=batch, dtype=dtype)


def _resnet(name, batch, image, dtype, graph):
    return dict(name=name, model="resnet18", batch=batch, image=image, dtype=dtype, graph=graph)


def _encoder(name, batch, seq, dtype, graph, padded):
    return dict(name=name, model="distilbert", batch=batch, seq=seq, dtype=dtype, graph=graph, padded=padded)


def _scores(name, batch, seq, dtype, graph):
    return dict(name=name, model="gpt2-scores", batch=batch, seq=seq, dtype=dtype, graph=graph)


def _serve(name, size, requests, lo, hi, new, dtype="bf16", chunk=0, sample=False):
    return dict(name=name, model="gpt2-serve", size=size, requests=requests, lo=lo, hi=hi, new=new, dtype=dtype, chunk=chunk,
                sample=sample)


def _bitnet(name, requests, lo, hi, new):
    return dict(name=name, model="bitnet-serve", requests=requests, lo=lo, hi=hi, new=new, dtype="bf16")


def listed():
    return [
        # one classification of a digit-sized vector, handed over from the host: the smallest call of a session
        _mlp("mlp784_b1", 1),
        # image classification: one picture as it arrives, the batch of the headline latency figure, a large offline batch
        # of an odd size in the other data type and without graph replay
        _resnet("resnet18_b1", 1, 224, "fp16", True),
        _resnet("resnet18_b32", 32, 224, "fp16", True),
        _resnet("resnet18_b117", 117, 224, "bf16", False),
        # sentence encoder: a single query of odd length run node by node, and the batch of the headline figure with
        # sentences of different lengths padded to one
        _encoder("distilbert_1x23", 1, 23, "fp16", False, False),
        _encoder("distilbert_64x128", 64, 128, "bf16", True, True),
        # scores of every position of whole documents (perplexity, reranking): the decoder as a plain graph session
        _scores("gpt2_scores_6x777", 6, 777, "bf16", False),
        # serving: one conversation (latency of a decode step), the headline workload with many requests at once (a
        # quarter of its 256 new tokens), long prompts read in chunks, a small model with every sampling option in fp16
        _serve("gpt2_chat_1", "medium", 1, 50, 50, 48),
        _serve("gpt2_serve_256", "medium", 256, 64, 512, 64),
        _serve("gpt2_prompts_24", "medium", 24, 500, 1000, 3, chunk=512),
        _serve("gpt2_sampled_37", "small", 37, 5, 300, 24, dtype="fp16", sample=True),
        # ternary weights: the batch of the headline figure
        _bitnet("bitnet_128", 128, 40, 88, 24),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    model = rng.choice(["mlp784", "resnet18", "distilbert", "gpt2-scores", "gpt2-serve", "gpt2-serve", "bitnet-serve"])
    dtype = rng.choice(["bf16", "fp16"])
    graph = rng.random() < 0.5
    if model == "mlp784":
        case = _mlp("", _log_int(rng, 1, 4096), dtype)
    elif model == "resnet18":
        case = _resnet("", _log_int(rng, 1, 128), rng.randrange(160, 257, 2), dtype, graph)
    elif model == "distilbert":
        seq = _log_int(rng, 8, 512)
        case = _encoder("", _log_int(rng, 1, max(1, 16384 // seq)), seq, dtype, graph, rng.random() < 0.5)
    elif model == "gpt2-scores":
        seq = _log_int(rng, 16, 1024)
        case = _scores("", _log_int(rng, 1, max(1, 6000 // seq)), seq, dtype, graph)
    elif model == "gpt2-serve":
        lo = _log_int(rng, 4, 512)
        case = _serve("", rng.choice(["small", "medium"]), _log_int(rng, 1, 224), lo, rng.randint(lo, min(2 * lo + 64, 960)),
                      _log_int(rng, 2, 48), dtype, rng.choice([0, 0, 256, 512]), rng.random() < 0.3)
    else:
        lo = _log_int(rng, 4, 128)
        case = _bitnet("", _log_int(rng, 1, 128), lo, 2 * lo, _log_int(rng, 2, 24))
    del case["name"]
    return case


# ---------------------------------------------------------------------------------------------------- models and sessions
@functools.lru_cache(maxsize=None)
def _gpt2_config(size):
    return GPT2Config.medium() if size == "medium" else GPT2Config.small()


@functools.lru_cache(maxsize=None)
def _session(model, image, dtype, graph):
    """A session, kept as a program keeps it: it is built once and then fed many inputs."""
    t = _DTYPES[dtype]
    if model == "mlp784":
        g = build_mlp784(seed=1)
    elif model == "resnet18":
        g = build_resnet18(dtype=t, seed=1, image=image)
    elif model == "distilbert":
        g = build_distilbert(DistilBertConfig.base(), dtype=t, seed=1)
    else:
        g = build_gpt2(GPT2Config.small(), dtype=t, seed=1)
    return Model.from_graph(g).create_session(SessionOptions().with_provider("gpu").with_optimization_level("O3")
                                              .with_dtype(dtype).with_cuda_graph(graph))


@functools.lru_cache(maxsize=2)
def _gpt2_model(size, dtype):
    g = build_gpt2(_gpt2_config(size), dtype=_DTYPES[dtype], seed=1, with_lm_head=False)
    g.initializers["wte"] = g.initializers["wte"] * 7.0
    return _on_device(g)


@functools.lru_cache(maxsize=1)
def _bitnet_model():
    """The builder's graph for one layer, and the weights of all 24 made on the device (packing 1.9 billion ternary
    values on the host takes most of a minute); the engine reads weights and metadata."""
    cfg = BitNetConfig.b158_2b()
    g = build_bitnet_llama(BitNetConfig(n_layer=1), dtype=torch.bfloat16, seed=1, with_lm_head=False)
    init = g.initializers
    init["embed"] = init["embed"] * 100.0
    gen = torch.Generator(device="cuda").manual_seed(1)
    for i in range(cfg.n_layer):
        for n in ("attn_norm", "ffn_norm"):
            init[f"layers.{i}.{n}.weight"] = init[f"layers.0.{n}.weight"]
        for n in ("qkv", "o", "gate_up", "down"):
            rows, quads = init[f"layers.0.{n}.weight"].shape
            packed = torch.zeros(rows, quads, dtype=torch.uint8, device="cuda")
            for shift in (0, 2, 4, 6):                                        # codes 0, 1, 2 stand for -1, 0, +1
                packed += torch.randint(0, 3, (rows, quads), generator=gen, device="cuda", dtype=torch.uint8) << shift
            residual = 1.0 / math.sqrt(2 * cfg.n_layer) if n in ("o", "down") else 1.0
            init[f"layers.{i}.{n}.scale"] = torch.tensor(residual / math.sqrt(quads * 4 * 2.0 / 3.0))
            init[f"layers.{i}.{n}.weight"] = packed
    g.metadata["ronn.n_layer"] = str(cfg.n_layer)
    return _on_device(g)


def _on_device(g):
    """Engines are built more than once here: their weights come from the device instead of the host."""
    for k, v in g.initializers.items():
        if v.is_floating_point() and v.dim() > 0:
            g.initializers[k] = v.cuda()
    return Model.from_graph(g)


def _lengths(case):
    """Prompt lengths spread over [lo, hi] in a scattered order, the same for every seed."""
    lo, span, n = case["lo"], case["hi"] - case["lo"], case["requests"]
    return [lo + int(span * ((i * 0.6180339887498949) % 1.0) + 0.5) for i in range(n)]


def _params(case, seed):
    if not case.get("sample"):
        return SamplingParams(max_new_tokens=case["new"])
    return SamplingParams(max_new_tokens=case["new"], temperature=0.8, top_k=50, top_p=0.95, repeat_penalty=1.1, seed=seed)


def _prepare_serving(case, seed):
    if case["model"] == "bitnet-serve":
        model, vocab = _bitnet_model(), BitNetConfig.b158_2b().vocab_size
    else:
        model, vocab = _gpt2_model(case["size"], case["dtype"]), _gpt2_config(case["size"]).vocab_size
    lens = _lengths(case)
    blocks = sum(-(-(n + case["new"]) // _BLOCK) + 1 for n in lens) + 8
    engine = LLMEngine(model, EngineConfig(max_num_seqs=case["requests"], max_model_len=1024, num_blocks=blocks,
                                           dtype=case["dtype"], prefill_chunk=case.get("chunk", 0)))
    gen = torch.Generator().manual_seed(seed)
    ids = torch.randint(0, vocab, (sum(lens),), generator=gen).tolist()
    ends = torch.tensor(lens).cumsum(0).tolist()
    prompts = [ids[e - n:e] for n, e in zip(lens, ends)]
    # a server warms up before it takes requests: step graphs are captured here
    engine.generate([[7] * n for n in lens], _params(case, 0))
    return dict(case=case, engine=engine, prompts=prompts, params=_params(case, seed))


def prepare(case, seed):
    model = case["model"]
    if model.endswith("-serve"):
        return _prepare_serving(case, seed)
    session = _session(model, case.get("image", 0), case["dtype"], case.get("graph", False))
    feed = _feed(case, seed)
    session.run(feed)                            # kernels loaded, and with graph replay the graph of this shape captured
    return dict(case=case, session=session, feed=feed)


def _feed(case, seed):
    model = case["model"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if model == "mlp784":
        feed = {"input": torch.rand(case["batch"], 784, generator=torch.Generator().manual_seed(seed))}
    elif model == "resnet18":
        shape = (case["batch"], 3, case["image"], case["image"])
        feed = {"input": torch.randn(shape, generator=gen, device="cuda", dtype=_DTYPES[case["dtype"]])}
    else:
        vocab = DistilBertConfig.base().vocab_size if model == "distilbert" else GPT2Config.small().vocab_size
        shape = (case["batch"], case["seq"])
        feed = {"input_ids": torch.randint(0, vocab, shape, generator=gen, device="cuda")}
        if model == "distilbert":
            lens = torch.full((case["batch"], 1), case["seq"], device="cuda")
            if case["padded"]:
                lens = torch.randint(max(1, case["seq"] // 4), case["seq"] + 1, lens.shape, generator=gen, device="cuda")
            feed["attention_mask"] = (torch.arange(case["seq"], device="cuda")[None, :] < lens).to(torch.int64)
    return feed


def run(state):
    if "session" in state:
        return state["session"].run(state["feed"])
    engine = state["engine"]
    tokens = engine.generate(state["prompts"], state["params"])
    # the tokens, and the keys and values that the engine holds after the pass
    return dict(tokens=torch.tensor(tokens, dtype=torch.int32), keys=engine.runner.kcache, values=engine.runner.vcache)


# ---------------------------------------------------------------------------------------------------- the same in 64 bits
@functools.lru_cache(maxsize=2)
def _weights64(model, image, dtype):
    """The weights a session starts from, in 64 bits on the device."""
    t = _DTYPES[dtype]
    if model == "mlp784":
        g = build_mlp784(seed=1)
    elif model == "resnet18":
        g = build_resnet18(dtype=t, seed=1, image=image)
    elif model == "distilbert":
        g = build_distilbert(DistilBertConfig.base(), dtype=t, seed=1)
    else:
        g = build_gpt2(GPT2Config.small(), dtype=t, seed=1)
    return {k: v.cuda().double() for k, v in g.initializers.items() if v.is_floating_point()}


def _resnet64(w, x):
    def conv(x, n, stride, pad, eps=1e-5):
        y = F.conv2d(x, w[n + ".weight"], stride=stride, padding=pad)
        return F.batch_norm(y, w[n + ".bn.running_mean"], w[n + ".bn.running_var"], w[n + ".bn.weight"], w[n + ".bn.bias"], eps=eps)

    x = F.max_pool2d(conv(x, "stem", 2, 3).relu(), 3, 2, 1)
    for stage in range(4):
        for blk in range(2):
            n, stride = f"layer{stage + 1}.{blk}", 2 if stage > 0 and blk == 0 else 1
            y = conv(conv(x, n + ".a", stride, 1).relu(), n + ".b", 1, 1)
            skip = conv(x, n + ".down", stride, 0) if n + ".down.weight" in w else x
            x = (y + skip).relu()
    return x.mean((2, 3)) @ w["fc.weight"].t() + w["fc.bias"]


def _attend64(q, k, v, heads, mask):
    b, s, h = q.shape
    q, k, v = (t.view(b, s, heads, h // heads).transpose(1, 2) for t in (q, k, v))
    p = (q @ k.transpose(-1, -2) / math.sqrt(h // heads)).masked_fill(~mask, float("-inf")).softmax(-1)
    return (p @ v).transpose(1, 2).reshape(b, s, h)


def _distilbert64(w, c, ids, mask):
    def lin(x, n):
        return x @ w[n + ".weight"] + w[n + ".bias"]

    def norm(x, n):
        return F.layer_norm(x, (c.dim,), w[n + ".weight"], w[n + ".bias"], c.eps)

    x = w["embeddings.word_embeddings.weight"][ids] + w["embeddings.position_embeddings.weight"][:ids.shape[1]]
    x = norm(x, "embeddings.LayerNorm")
    for i in range(c.n_layers):
        p = f"transformer.layer.{i}"
        q, k, v = (lin(x, f"{p}.attention.{n}_lin") for n in "qkv")
        x = norm(lin(_attend64(q, k, v, c.n_heads, mask[:, None, None, :] > 0), p + ".attention.out_lin") + x, p + ".sa_layer_norm")
        f = lin(F.gelu(lin(x, p + ".ffn.lin1"), approximate="tanh"), p + ".ffn.lin2")
        x = norm(f + x, p + ".output_layer_norm")
    return x


def _gpt2_64(w, c, ids):
    def lin(x, n):
        return x @ w[n + ".weight"] + w[n + ".bias"]

    def norm(x, n):
        return F.layer_norm(x, (c.n_embd,), w[n + ".weight"], w[n + ".bias"], c.layer_norm_epsilon)

    s = ids.shape[1]
    seen = torch.ones(s, s, dtype=torch.bool, device=ids.device).tril()
    x = w["wte"][ids] + w["wpe"][:s]
    for i in range(c.n_layer):
        p = f"h.{i}"
        q, k, v = lin(norm(x, p + ".ln_1"), p + ".attn.c_attn").chunk(3, -1)
        x = x + lin(_attend64(q, k, v, c.n_head, seen), p + ".attn.c_proj")
        x = x + lin(F.gelu(lin(norm(x, p + ".ln_2"), p + ".mlp.c_fc"), approximate="tanh"), p + ".mlp.c_proj")
    return norm(x, "ln_f")


def exact(case, seed):
    """Sessions in 64 bits, with the weights they start from.  An engine chooses tokens and then reads its own choices:
    its pass has no such value."""
    model = case["model"]
    if model.endswith("-serve"):
        return None
    feed = _feed(case, seed)
    w = _weights64(model, case.get("image", 0), case["dtype"])
    with torch.no_grad():
        if model == "mlp784":
            x = feed["input"].cuda().double()
            x = (x @ w["fc1.weight"] + w["fc1.bias"]).relu()
            return {"probs": (x @ w["fc2.weight"] + w["fc2.bias"]).softmax(-1)}
        if model == "resnet18":
            return {"logits": torch.cat([_resnet64(w, x.double()) for x in feed["input"].split(8)])}
        if model == "distilbert":
            c, mask = DistilBertConfig.base(), feed["attention_mask"]
            parts = [_distilbert64(w, c, i, m) for i, m in zip(feed["input_ids"].split(16), mask.split(16))]
            return {"last_hidden_state": torch.cat(parts)}
        hidden = torch.cat([_gpt2_64(w, GPT2Config.small(), i) for i in feed["input_ids"].split(4)])
        return {"last_hidden_state": hidden, "logits": hidden @ w["wte"].t()}


# ---------------------------------------------------------------------------------------------------- what a pass needs
def _decoder_work(layer_params, layer_weight_bytes, n_layer, width, vocab, lens, new, rows_scored):
    """Operations and bytes of reading prompts and generating ``new`` tokens for each: every token passes every layer once
    (the last token drawn passes none), attends to the tokens before it, and ``rows_scored`` rows meet the vocabulary."""
    flops = bytes_ = 0.0
    steps = max(new - 1, 0)
    tokens = sum(lens) + len(lens) * steps
    flops += 2.0 * tokens * n_layer * layer_params
    for n in lens:
        # prompt token i looks at i + 1 keys; decode step j of a request at n + 1 + j
        seen = n * (n + 1) / 2 + sum(n + 1 + j for j in range(steps))
        flops += 4.0 * seen * width * n_layer
        bytes_ += 4.0 * n_layer * width * sum(n + 1 + j for j in range(steps))        # keys and values of decode, 2 bytes
        bytes_ += 4.0 * n_layer * width * (n + steps)                                 # written once each
    flops += 2.0 * rows_scored * width * vocab
    bytes_ += (1 + steps) * (n_layer * layer_weight_bytes + 2.0 * width * vocab)      # weights: prompts once, each step once
    return flops, bytes_


def work(case):
    model = case["model"]
    if model == "mlp784":
        b, params = case["batch"], 784 * 128 + 128 * 10
        return {"flops": 2.0 * b * params, "bytes": 4.0 * b * 784 + 2.0 * params + 2.0 * b * 10}
    if model == "resnet18":
        b, im = case["batch"], case["image"]
        half = lambda v, k, s, p: (v + 2 * p - k) // s + 1
        h = half(im, 7, 2, 3)
        macs, params = h * h * 64 * 147, 64 * 147
        h, cin = half(h, 3, 2, 1), 64
        for stage, cout in enumerate((64, 128, 256, 512)):
            for blk in range(2):
                first = stage > 0 and blk == 0
                if first:
                    h = half(h, 3, 2, 1)
                    macs, params = macs + h * h * cin * cout, params + cin * cout
                w = 9 * cout * (cin + cout)
                macs, params, cin = macs + h * h * w, params + w, cout
        macs, params = macs + 512000, params + 512000
        return {"flops": 2.0 * b * macs, "bytes": 2.0 * (b * 3 * im * im + params + b * 1000)}
    if model == "distilbert":
        c, tokens = DistilBertConfig.base(), case["batch"] * case["seq"]
        per_layer = 4 * c.dim * c.dim + 2 * c.dim * c.hidden_dim
        return {"flops": c.n_layers * (2.0 * tokens * per_layer + 4.0 * tokens * case["seq"] * c.dim),
                "bytes": 2.0 * c.n_layers * per_layer + 16.0 * tokens + 4.0 * tokens * c.dim}
    if model == "gpt2-scores":
        c, tokens = GPT2Config.small(), case["batch"] * case["seq"]
        per_layer = 12 * c.n_embd * c.n_embd
        return {"flops": c.n_layer * (2.0 * tokens * per_layer + 2.0 * tokens * (case["seq"] + 1) * c.n_embd)
                + 2.0 * tokens * c.n_embd * c.vocab_size,
                "bytes": 2.0 * (c.n_layer * per_layer + c.vocab_size * c.n_embd + tokens * (c.vocab_size + 2 * c.n_embd))}
    lens = _lengths(case)
    rows = case["requests"] * case["new"]
    if model == "gpt2-serve":
        c = _gpt2_config(case["size"])
        per_layer = 12 * c.n_embd * c.n_embd
        f, b = _decoder_work(per_layer, 2.0 * per_layer, c.n_layer, c.n_embd, c.vocab_size, lens, case["new"], rows)
    else:
        c = BitNetConfig.b158_2b()
        per_layer = 4 * c.hidden * c.hidden + 3 * c.hidden * c.ffn
        f, b = _decoder_work(per_layer, per_layer / 4.0, c.n_layer, c.hidden, c.vocab_size, lens, case["new"], rows)
    return {"flops": f, "bytes": b}


def tolerance(case):
    """About four times the largest difference seen, over the listed cases, against the same graph or engine on library
    calls at the same precision and in fp32 (relative 2-norm of the worst output / largest difference):
    mlp784 bf16 0.0015 / 0.002; resnet18 fp16 0.0004 / 0.0015, bf16 0.003 / 0.012; distilbert fp16 0.0013 / 0.0054,
    bf16 0.0087 / 0.062; gpt2 bf16 0.0138 / 0.098, fp16 0.0013 / 0.0076; bitnet 0.018 / 0.12 (int8 activations: a
    rounding that falls the other way moves a value by 1/127 of its row's largest).  Tokens were the same in all; one
    that differs would change everything its request writes after it."""
    half = case["dtype"] == "fp16"
    rel, most = {
        "mlp784": (0.0015, 0.006) if half else (0.006, 0.02),
        "resnet18": (0.0016, 0.006) if half else (0.012, 0.05),
        "distilbert": (0.005, 0.03) if half else (0.03, 0.25),
        "gpt2-scores": (0.005, 0.03) if half else (0.03, 0.3),
        "gpt2-serve": (0.005, 0.03) if half else (0.03, 0.4),
        "bitnet-serve": (0.03, 0.4),
    }[case["model"]]
    return {"rel": rel, "max": most, "differ": 0.002}
