"""The work that programs written on this framework have it do, as cases that can be timed and compared.

Every case is one decoder graph that a program compiles once (`Compiler.compile("cuda", ...)`), fills with its weights and
caches, and then runs once per step or prompt (`Executor.run()`).  `kind` says how the program wrote its graph:

  operators  a prompt in the plain operators of an exported model (MatMul, Transpose, Where, Softmax, ...), fp32
  attention  a prompt or a step in the language-model operators (RmsNormalization, MatMul, RotaryPositionEmbedding,
             Attention with a cache that lives in the graph), any of the three floating types
  step       one generated token for one sequence, the whole step as one node
  steps      one generated token for 2 to 4 sequences in the fused operators
  batch      one generated token for 2 to 48 sequences, contiguous or paged cache, greedy or top-k sampling
  prompt     a prompt of 1 to 4 sequences in the fused prefill operators
"""
import math

import numpy as np
import torch

from refactorgraph_b200.config import LlamaConfig
from refactorgraph_b200.graph_builder import BF16, F32, FP16, I64, GraphBuilder
from refactorgraph_b200.llama import (decode_step_graph, decode_step_graph_batched, decode_step_graph_single_kernel, prefill_graph,
                                      prefill_graph_reference_ops, weight_inputs)

DTYPES = {"fp32": (F32, torch.float32), "fp16": (FP16, torch.float16), "bf16": (BF16, torch.bfloat16)}
PAGE = 16  # tokens of one block of a paged cache

# Widths of the decoders that the configurations, tests and benchmark of this repository use.
WIDTHS = {
    "tiny": dict(hidden=256, heads=4, kv_heads=4, head_dim=64, ffn=688, vocab=1000),
    "small": dict(hidden=1024, heads=8, kv_heads=8, head_dim=128, ffn=2752, vocab=32000),
    "small64": dict(hidden=1024, heads=16, kv_heads=16, head_dim=64, ffn=2752, vocab=32000),
    "7b": dict(hidden=4096, heads=32, kv_heads=32, head_dim=128, ffn=11008, vocab=32000),
    "7b-gqa": dict(hidden=4096, heads=32, kv_heads=8, head_dim=128, ffn=11008, vocab=32000),
    "70b": dict(hidden=8192, heads=64, kv_heads=8, head_dim=128, ffn=28672, vocab=32000),
}


def listed():
    return [
        # A tiny fp32 model exported operator by operator: many launches of almost no work each.
        dict(name="operators_tiny", kind="operators", width="tiny", dtype="fp32", layers=2, seq=32),
        # The same kind of export of a model of useful size, an odd prompt length.
        dict(name="operators_small", kind="operators", width="small64", dtype="fp32", layers=4, seq=509),
        # An fp16 model in the language-model operators, weights [in, out] as exporters store them: a prompt into an empty cache ...
        dict(name="attention_prompt", kind="attention", width="7b", dtype="fp16", layers=2, batch=1, seq=300, past=0, trans_b=False),
        # ... and the generation step of a small batch with a thousand tokens in the cache, weights [out, in].
        dict(name="attention_step", kind="attention", width="7b", dtype="fp16", layers=2, batch=4, seq=1, past=1037, trans_b=True),
        # Generation for one user: a small model with a short cache (the shortest step there is), and the 7B shape at 2048 tokens
        # (31 of its 32 layers: every layer's caches are among the outputs, of which 64 can be looked at).
        dict(name="step_small", kind="step", width="small", dtype="fp16", layers=8, past=300),
        dict(name="step_7b", kind="step", width="7b", dtype="fp16", layers=31, past=2048),
        # A few users whose sequences have different lengths.
        dict(name="batch_3", kind="batch", width="7b", dtype="fp16", layers=8, batch=3, shortest=200, longest=1500, paged=False, top_k=1),
        # A serving batch in bf16, contiguous caches.
        dict(name="batch_8", kind="batch", width="7b", dtype="bf16", layers=8, batch=8, shortest=300, longest=1200, paged=False, top_k=1),
        # Grouped-query attention at the 70B widths, ten layers (one GPU's share of memory), 4096 tokens in every cache.
        dict(name="batch_16_70b", kind="batch", width="70b", dtype="fp16", layers=10, batch=16, shortest=4096, longest=4096, paged=False, top_k=1),
        # A paged cache with lengths all over the place and top-50 sampling.
        dict(name="batch_32_paged", kind="batch", width="7b", dtype="fp16", layers=8, batch=32, shortest=512, longest=4096, paged=True, top_k=50),
        # One user's short prompt of odd length, and a full prefill batch.
        dict(name="prompt_333", kind="prompt", width="7b", dtype="fp16", layers=8, batch=1, seq=333),
        dict(name="prompt_4x2048", kind="prompt", width="7b", dtype="bf16", layers=8, batch=4, seq=2048),
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(["operators", "attention", "step", "steps", "batch", "prompt"])
    if kind == "operators":
        return dict(kind=kind, width=rng.choice(["tiny", "small", "small64"]), dtype="fp32", layers=rng.randint(1, 4), seq=_log_int(rng, 2, 509))
    if kind == "attention":
        c = dict(kind=kind, width=rng.choice(["small", "small64", "7b", "7b-gqa"]), dtype=rng.choice(["fp32", "fp16", "fp16", "bf16"]),
                 layers=rng.randint(1, 2), trans_b=rng.random() < 0.5)
        if rng.random() < 0.5:  # a step
            return dict(c, batch=rng.randint(1, 8), seq=1, past=_log_int(rng, 1, 2000))
        batch = rng.randint(1, 3)
        return dict(c, batch=batch, seq=_log_int(rng, 2, 300 // batch), past=rng.choice([0, 0, rng.randint(1, 600)]))
    if kind == "step":
        return dict(kind=kind, width=rng.choice(["tiny", "small", "small64", "7b", "7b-gqa"]), dtype=rng.choice(["fp16", "bf16"]),
                    layers=_log_int(rng, 2, 31), past=_log_int(rng, 1, 4000))
    longest = _log_int(rng, 64, 4096)
    lengths = dict(shortest=rng.randint(1, longest), longest=longest)
    if kind == "steps":
        return dict(kind=kind, width=rng.choice(["small", "small64"]), dtype=rng.choice(["fp16", "bf16"]), layers=rng.randint(2, 8),
                    batch=rng.randint(2, 4), **lengths)
    if kind == "batch":
        return dict(kind=kind, width=rng.choice(["small", "7b", "7b-gqa", "70b"]), dtype=rng.choice(["fp16", "bf16"]), layers=rng.randint(2, 6),
                    batch=_log_int(rng, 2, 48), paged=rng.random() < 0.5, top_k=rng.choice([1, 50]), **lengths)
    return dict(kind=kind, width=rng.choice(["small", "7b", "7b-gqa", "70b"]), dtype=rng.choice(["fp16", "bf16"]), layers=rng.randint(1, 2),
                batch=rng.randint(1, 4), seq=_log_int(rng, 16, 1536))


def _tokens(case):
    """(sequences, new tokens of each) of one pass."""
    return case.get("batch", 1), case.get("seq", 1)


def _config(case):
    batch, seq = _tokens(case)
    longest = case.get("longest", case.get("past", 0)) + seq
    return LlamaConfig(layers=case["layers"], batch=batch, max_seq=-(-longest // 128) * 128, dtype=DTYPES[case["dtype"]][0], **WIDTHS[case["width"]])


def _attention_graph(cfg, case):
    """The decoder in the language-model operators: the caches are edges of the graph, in which they stay from run to run."""
    g = GraphBuilder()
    n, s = _tokens(case)
    hidden, heads, kv, dim, ffn, t = cfg.hidden, cfg.heads, cfg.kv_heads, cfg.head_dim, cfg.ffn, n * s
    trans = case["trans_b"]
    ids, positions, past, last = g.input("ids", I64, (t,)), g.input("positions", I64, (t,)), g.input("past", I64, (1,)), g.input("last", I64, (n,))
    g.input("embed", cfg.dtype, (cfg.vocab, hidden))

    def linear(x, name, rows, cols):
        g.input(name, cfg.dtype, (rows, cols) if trans else (cols, rows))
        return g.op("llm::MatMul", [x, name], transB=int(trans))

    def norm(x, name):
        g.input(name, cfg.dtype, (hidden,))
        return g.op("llm::RmsNormalization", [x, name], epsilon=cfg.eps)

    def by_head(x, count, rope):
        x = g.op("onnx::Reshape", [x], shape=[t, count, dim])
        if rope:
            x = g.op("llm::RotaryPositionEmbedding", [x, positions], theta=cfg.theta)
        return g.op("onnx::Transpose", [g.op("onnx::Reshape", [x], shape=[n, s, count, dim])], perm=[0, 2, 1, 3])

    caches = []
    x = g.op("onnx::Gather", ["embed", ids], axis=0)
    for i in range(cfg.layers):
        y = norm(x, f"l{i}.norm1")
        q, k, v = (by_head(linear(y, f"l{i}.w{m}", count * dim, hidden), count, m != "v") for m, count in (("q", heads), ("k", kv), ("v", kv)))
        a, k_cache, v_cache = g.op("llm::Attention", [q, k, v, past], n_out=3, max_seq_len=cfg.max_seq)
        caches += [g.output(k_cache), g.output(v_cache)]
        a = g.op("onnx::Reshape", [g.op("onnx::Transpose", [a], perm=[0, 2, 1, 3])], shape=[t, heads * dim])
        x = g.op("onnx::Add", [x, linear(a, f"l{i}.wo", hidden, heads * dim)])
        y = norm(x, f"l{i}.norm2")
        gate, up = linear(y, f"l{i}.wg", ffn, hidden), linear(y, f"l{i}.wu", ffn, hidden)
        gate = g.op("onnx::Mul", [g.op("onnx::Mul", [gate, g.op("onnx::Sigmoid", [gate])]), up])
        x = g.op("onnx::Add", [x, linear(gate, f"l{i}.wd", hidden, ffn)])
    logits = linear(norm(g.op("onnx::Gather", [x, last], axis=0), "norm_f"), "lm_head", cfg.vocab, hidden)
    probs, best = g.op("llm::TopK", [logits], n_out=2, k=1, softmax=1)
    index = {"logits": g.output(logits), "probs": g.output(probs), "next": g.output(best), "caches": caches}
    index.update({name: i for i, name in enumerate(g.inputs)})
    return g, index


class _Memory:
    """Device memory of an executor, in the form that torch takes over without a copy (and that keeps the executor alive)."""

    def __init__(self, executor, address, shape, typestr):
        self.executor = executor
        self.__cuda_array_interface__ = {"data": (address, False), "shape": tuple(shape), "typestr": typestr, "strides": None, "version": 3}


def _view(executor, address, shape, dtype):
    typestr = {torch.float32: "<f4", torch.float16: "<f2", torch.bfloat16: "<i2", torch.int64: "<i8"}[dtype]
    t = torch.as_tensor(_Memory(executor, address, shape, typestr), device="cuda")
    return t.view(torch.bfloat16) if dtype == torch.bfloat16 else t


def _normal(gen, shape, dtype, std=0.02):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=gen)


def _weights(gen, shapes, dtype):
    """(name, values) of every weight, drawn as the benchmark draws them.  The output head is tied to the embedding, whose
    values outweigh what the layers add: the next token is then as decided as a trained model's and not a tie of noise."""
    embed = None
    for name, shape in shapes:
        if name == "embed":
            w = embed = _normal(gen, shape, dtype, 4.0)
        elif name == "lm_head":
            w = (embed if tuple(embed.shape) == tuple(shape) else embed.t().contiguous()) * (0.02 / 4.0)
        else:
            w = _normal(gen, shape, dtype)
            if "norm" in name:
                w += 1.0
        yield name, w


def prepare(case, seed):
    cfg = _config(case)
    kind, (batch, seq) = case["kind"], _tokens(case)
    code, dtype = DTYPES[case["dtype"]]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    host = np.random.default_rng(seed)
    past = host.integers(case["shortest"], case["longest"] + 1, batch) if "shortest" in case else np.full(batch, case.get("past", 0))
    past = past.astype(np.int64)
    ids = host.integers(0, cfg.vocab, batch * seq).astype(np.int64)
    feeds, passes = {}, []
    cache_shape = (batch, cfg.kv_heads, cfg.max_seq, cfg.head_dim)
    if kind == "operators":
        weights = {name: w.cpu().numpy() for name, w in _weights(gen, weight_inputs(cfg), dtype)}
        g, index = prefill_graph_reference_ops(cfg, weights, seq)
        index["ids"] = 0
        feeds["ids"] = ids
    elif kind == "attention":
        g, index = _attention_graph(cfg, case)
        feeds.update(ids=ids, positions=(past[:, None] + np.arange(seq)).ravel(), past=past[:1], last=(np.arange(batch) + 1) * seq - 1)
    elif kind == "prompt":
        g, index = prefill_graph(cfg, seq)
        feeds.update(ids=ids, positions=np.tile(np.arange(seq), batch), last=(np.arange(batch) + 1) * seq - 1)
    elif kind == "step":
        g, index = decode_step_graph_single_kernel(cfg)
        feeds.update(token=ids, pos=past)
    elif kind == "steps":
        g, index = decode_step_graph(cfg)
        feeds.update(token=ids, pos=past, lens=past + 1)
    else:
        blocks = cfg.max_seq // PAGE
        sample = dict(top_k=case["top_k"], sample=case["top_k"] > 1, temperature=1.0, seed=0)
        g, index = decode_step_graph_batched(cfg, paged=case["paged"], page=PAGE, max_blocks=blocks, n_blocks=batch * blocks, **sample)
        passes = ["fuse"] if batch > 4 else []  # the fused forms for 2 to 4 tokens take narrower layers than the 7B shape's
        feeds.update(token=ids, pos=past, lens=past + 1)
        if case["top_k"] > 1:
            feeds["step"] = np.zeros(1, np.int64)
        if case["paged"]:
            cache_shape = (batch * blocks, cfg.kv_heads, PAGE, cfg.head_dim)
    ex = g.compiler().compile("cuda", "flat", passes)
    if kind == "attention":
        for name, w in _weights(gen, [(n, tuple(g.edges[n].shape)) for n in g.inputs if n in g.edges and n not in feeds], dtype):
            ex.set_input_blob(index[name], w.data_ptr(), w.numel() * w.element_size())
    elif kind != "operators":
        for name, w in _weights(gen, weight_inputs(cfg), dtype):
            ex.set_input_blob(index[name], w.data_ptr(), w.numel() * w.element_size())
    if kind == "batch" and case["paged"]:
        ex.set_input(index["block_table"], host.permutation(cache_shape[0]).astype(np.int32).reshape(batch, -1))
    # the tokens before this step lie in the caches; a prompt finds them empty
    out = {}
    for i in range(cfg.layers if kind != "operators" else 0):
        for m, name in enumerate(("k_cache", "v_cache")):
            address = ex.output_address(index["caches"][2 * i + m]) if kind == "attention" else ex.input_address(index[f"l{i}.{name}"])
            out[f"l{i}.{name}"] = _view(ex, address, cache_shape, dtype)
            if past.any():
                out[f"l{i}.{name}"].normal_(0.0, 1.0, generator=gen)
    rows = seq if kind == "operators" else batch
    out["logits"] = _view(ex, ex.output_address(index["logits"]), (rows, cfg.vocab), dtype)
    if kind == "operators":
        out["top"] = _view(ex, ex.output_address(index["topk_idx"]), (rows, 5), torch.int64)
        out["top_logits"] = _view(ex, ex.output_address(index["topk_val"]), (rows, 5), dtype)
    else:
        out["next"] = _view(ex, ex.output_address(index["next"]), (rows,), torch.int64)
    # what the program sends with every step lies in pinned memory
    feeds = [(index[name], torch.from_numpy(np.ascontiguousarray(a, dtype=np.int64)).pin_memory()) for name, a in feeds.items()]
    return {"executor": ex, "feeds": feeds, "outputs": out, "stream": torch.cuda.ExternalStream(ex.cuda_stream()),
            "inputs_free": torch.cuda.Event(), "outputs_ready": torch.cuda.Event()}


def run(state):
    """One step or prompt: the host's tokens and positions in, one run, the outputs ready for the caller's stream."""
    ex, stream, caller = state["executor"], state["stream"], torch.cuda.current_stream()
    state["inputs_free"].record(caller)
    stream.wait_event(state["inputs_free"])
    for i, a in state["feeds"]:
        ex.set_input_async(i, a.data_ptr(), a.nbytes)
    ex.run()
    state["outputs_ready"].record(stream)
    caller.wait_event(state["outputs_ready"])
    return state["outputs"]


def work(case):
    cfg = _config(case)
    batch, seq = _tokens(case)
    tokens, size = batch * seq, 4 if case["dtype"] == "fp32" else 2
    heads, kv, dim = cfg.heads, cfg.kv_heads, cfg.head_dim
    layer = (heads + 2 * kv) * dim * cfg.hidden + cfg.hidden * heads * dim + 3 * cfg.ffn * cfg.hidden
    head_rows = tokens if case["kind"] == "operators" else batch
    past = (case["shortest"] + case["longest"]) / 2 if "shortest" in case else case.get("past", 0)
    seen = tokens * (past + (seq + 1) / 2)  # (query, key) pairs under the causal mask
    row = 2 * kv * dim * size  # K and V of one token in one layer
    cached = 0 if case["kind"] == "operators" else cfg.layers * row * (batch * past + tokens)
    moved = size * (cfg.layers * (layer + 2 * cfg.hidden) + cfg.hidden * cfg.vocab + cfg.hidden + tokens * cfg.hidden + head_rows * cfg.vocab) + cached
    return {"bytes": moved, "flops": 2 * tokens * cfg.layers * layer + 2 * head_rows * cfg.hidden * cfg.vocab + cfg.layers * 4 * seen * heads * dim}


def tolerance(case):
    """About four times what the logits are off from the same decoder evaluated without rounding between its operators
    (2-norm 6e-7 in fp32; over the ranges above 6e-4 and 5e-3 times the root of the layer count in fp16 and bf16)."""
    if case["dtype"] == "fp32":
        return {"rel": 3e-6, "max": 3e-5, "differ": 4e-3}
    rel = min(0.03, (2.4e-3 if case["dtype"] == "fp16" else 1.5e-2) * math.sqrt(case["layers"]))
    return {"rel": rel, "max": 10 * rel}
