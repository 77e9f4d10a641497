"""The work this framework is used for, as measurable cases: student training steps and teacher collection batches,
each one call of the public per-batch entry points (``DistillEngine.train_step``, ``TeacherCollector.submit`` /
``fetch``) from host batch to result.

A case names a model preset with its overrides, the batch (``batch`` conversations of up to ``seq`` tokens), the stored
teacher distribution (``topk`` entries per row) and the options in force:

    kind      train | collect
    rows      "all": every position carries a target (the benchmark's synthetic batches); "content": conversations of
              uneven length whose turn markers are left out, as the dataset reader produces them
    precision bf16, or 4bit / 8bit (frozen NF4 / int8 decoder matrices, the shipped default)
    accum     micro-batches per optimizer step
    chunk     > 0: prefill in chunks of that many positions against a key / value cache
    full      collection stores the whole distribution instead of the top-K entries
"""
import math

import numpy as np
import torch

from llm_distillery_b200.collect.collector import TeacherCollector
from llm_distillery_b200.data.convo import ConvoTokenized
from llm_distillery_b200.engine.trainer import DistillEngine, HostBatch
from llm_distillery_b200.models import llama

_TRAIN = dict(kind="train", layers=0, window=0, batch=1, seq=256, topk=200, loss="kl", temperature=1.0, rows="content",
              precision="bf16", optimizer="adamw", accum=1, checkpoint=False)
_COLLECT = dict(kind="collect", layers=0, window=0, batch=1, seq=256, topk=200, rows="content", chunk=0, full=False)


def listed():
    return [
        # the plumbing configuration's student: a step that is all launches and host work
        dict(_TRAIN, name="train_plumbing", model="plumbing-student", batch=2, seq=256, rows="all"),
        # one short conversation of a small student with a 150 k vocabulary, the reference's loss
        dict(_TRAIN, name="train_one_conversation", model="qwen2.5-0.5b", batch=1, seq=777, loss="reference"),
        # the headline benchmark
        dict(_TRAIN, name="train_tinyllama", model="tinyllama-1.1b", batch=8, seq=2048, temperature=2.0, rows="all"),
        # config.json as shipped: 4-bit base weights, 8-bit AdamW, batches of 4 accumulated 4 times, top-400, reference loss
        dict(_TRAIN, name="train_shipped_config", model="tinyllama-1.1b", batch=4, seq=1893, topk=400, loss="reference",
             precision="4bit", optimizer="adamw8bit", accum=4),
        # a 1 B student with tied 128 k embeddings on long sequences, JSD
        dict(_TRAIN, name="train_llama_1b", model="llama-3.2-1b", batch=4, seq=4096, loss="jsd", rows="all"),
        # layers of the 7 - 8 B students (heads of 128), recomputed in the backward, reverse KL; four of them, so that
        # the optimizer state of a step fits several times
        dict(_TRAIN, name="train_wide_layers", model="mistral-7b", layers=4, batch=2, seq=4000, topk=128, loss="rkl",
             checkpoint=True),
        # a single short conversation through a teacher: latency
        dict(_COLLECT, name="collect_short", model="tinyllama-1.1b", batch=1, seq=93),
        # the benchmark's collection batch
        dict(_COLLECT, name="collect_tinyllama", model="tinyllama-1.1b", batch=8, seq=2048, rows="all"),
        # an 8 B teacher over a long context, chunked prefill
        dict(_COLLECT, name="collect_8b_chunked", model="llama-3-8b", batch=1, seq=8192, topk=128, rows="all", chunk=2048),
        # a conversation longer than the teacher's attention window
        dict(_COLLECT, name="collect_beyond_window", model="mistral-7b", window=4096, batch=1, seq=6001),
        # layers of a sparse mixture-of-experts teacher; six of them, since with random weights the router's near ties
        # turn the last bits of one layer into other experts in the next
        dict(_COLLECT, name="collect_experts", model="tinymixtral-8x1b", layers=6, batch=4, seq=1531),
    ]


def draw(rng):
    """One more case of the same ranges: sizes log-uniform, odd ones included, at most the work of the largest listed."""
    most = max(work(c)["flops"] for c in listed())

    def log_int(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    while True:
        kind = rng.choice(["train", "train", "train", "collect", "collect"])
        if kind == "collect":
            model = rng.choice(["tinyllama-1.1b", "llama-3.2-1b", "llama-3-8b", "mistral-7b", "qwen2.5-7b", "tinymixtral-8x1b"])
            c = dict(_COLLECT, model=model, layers=6 if model == "tinymixtral-8x1b" else 0,
                     window=4096 if model == "mistral-7b" else 0, topk=rng.choice([50, 100, 128, 200, 400]),
                     rows=rng.choice(["all", "content"]), full=rng.random() < 0.15)
            c["seq"] = log_int(32, min(8192, llama.preset(model).max_position_embeddings))
            c["chunk"] = 128 * rng.randint(1, c["seq"] // 128) if c["seq"] > 256 and rng.random() < 0.25 else 0
        else:
            model = rng.choice(["plumbing-student", "qwen2.5-0.5b", "qwen2.5-1.5b", "tinyllama-1.1b", "tinyllama-1.1b",
                                "llama-3.2-1b", "mistral-7b"])
            c = dict(_TRAIN, model=model, layers=4 if model == "mistral-7b" else 0,
                     topk=rng.choice([50, 100, 128, 200, 400]), loss=rng.choice(["reference", "reference", "kl", "rkl", "jsd"]),
                     temperature=rng.choice([1.0, 1.0, 2.0]), rows=rng.choice(["all", "content"]),
                     precision=rng.choice(["bf16", "bf16", "4bit", "8bit"]) if model == "tinyllama-1.1b" else "bf16")
            c["seq"] = log_int(64, min(4096, llama.preset(model).max_position_embeddings))
            c.update(optimizer=rng.choice(["adamw", "adamw8bit"]), accum=rng.choice([1, 1, 2, 4]),
                     checkpoint=rng.random() < 0.2)
        c["batch"] = log_int(1, max(1, min(16, 16384 // c["seq"])))
        if work(c)["flops"] <= most:
            return c


# ------------------------------------------------------------------------------------------------ inputs
def _config(case):
    over = {}
    if case["layers"]:
        over["num_hidden_layers"] = case["layers"]
    if case["window"]:
        over["sliding_window"] = case["window"]
    return llama.preset(case["model"], **over)


def _tokens(cfg, batch, seq, rnd):
    """Token ids with the skew of text: frequent ids repeat."""
    return (cfg.vocab_size * rnd.random((batch, seq)) ** 2).astype(np.int64)


def _conversations(case, cfg, rnd):
    """[batch, seq] padded tokens and one ``ConvoTokenized`` per row. Datasets are sorted by length, so the members of a
    batch are of similar length; the first is the longest. Turns of 30 - 300 tokens behind 5 marker tokens each; where
    they lie belongs to the case, what they say to the seed."""
    B, L = case["batch"], case["seq"]
    tokens = _tokens(cfg, B, L, rnd)
    shape = np.random.default_rng(B * 10007 + L)
    convos = []
    for b in range(B):
        n = L if b == 0 or case["rows"] == "all" else int(shape.integers(max(1, (9 * L) // 10), L + 1))
        if case["rows"] == "all":
            ranges = [(0, n)]
        else:
            ranges, at = [], 0
            while at + 6 < n:
                end = min(n - 1, at + 5 + int(shape.integers(30, 300)))
                ranges.append((at + 5, end))
                at = end
        tokens[b, n:] = 0
        convos.append(ConvoTokenized(tokens[b], ranges, L - n, False, b))
    return tokens, convos


def _teacher_rows(rows, vocab, k, gen):
    """Top-``k`` ids (ascending, as the store's reader hands them over) and log-probs of a teacher whose logits are
    N(0, 3): a few likely tokens and a long tail."""
    ids = torch.empty((rows, k), dtype=torch.int32, device="cuda")
    logp = torch.empty((rows, k), dtype=torch.float32, device="cuda")
    step = max(1, (128 << 20) // vocab)
    for r in range(0, rows, step):
        z = torch.randn((min(step, rows - r), vocab), generator=gen, device="cuda") * 3.0
        v, i = z.topk(k, dim=-1)
        i, order = i.sort(dim=-1)
        ids[r:r + step] = i
        logp[r:r + step] = v.gather(1, order) - z.logsumexp(-1, keepdim=True)
    return ids, logp


def _host_batch(case, cfg, rnd, gen):
    tokens, convos = _conversations(case, cfg, rnd)
    B, L = tokens.shape
    rows, seg, labels, avoid = [], [], [], []
    for b, c in enumerate(convos):
        ci = c.content_indices()
        ce, av = c.ce_indices(L)
        lab = np.full(len(ci), -1, dtype=np.int64)
        n = min(len(ci), len(ce))
        inside = ce[:n] < L
        lab[:n][inside] = c.tokenized[ce[:n][inside]]
        out = np.zeros(len(ci), dtype=bool)
        out[av[av < len(ci)]] = True
        rows.append(ci + b * L)
        seg.append(np.full(len(ci), b, dtype=np.int64))
        labels.append(lab)
        avoid.append(out)
    M = sum(map(len, rows))
    ids, logp = _teacher_rows(M, cfg.vocab_size, case["topk"], gen)
    host = lambda parts: torch.from_numpy(np.concatenate(parts))  # noqa: E731
    reference = case["loss"] == "reference"
    return HostBatch(input_ids=torch.from_numpy(tokens), ids=ids.cpu(), logp=logp.to(torch.float16).float().cpu(), seg=host(seg),
                     n_seg=B, rows=None if case["rows"] == "all" else host(rows), labels=host(labels) if reference else None,
                     avoid=host(avoid) if reference else None, n_tokens=B * L).pin()


def prepare(case, seed):
    """The model with its weights, the engine or collector a program keeps, and the batches of one call in pinned (or,
    for collection, ordinary) host memory."""
    cfg = _config(case)
    rnd = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    model = llama.build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=seed)
    if case["kind"] == "collect":
        for p in model.parameters():
            p.requires_grad_(False)
        model.lm_head.mul_(3.0)                     # a trained head is peaked: logits of about N(0, 3)
        tokens, convos = _conversations(case, cfg, rnd)
        collector = TeacherCollector(model, topk=case["topk"], crop_to_size=cfg.vocab_size, enable_topk=not case["full"],
                                     prefill_chunk_len=case["chunk"])
        return {"kind": "collect", "model": model, "collector": collector, "tokens": tokens, "convos": convos,
                "vocab": cfg.vocab_size}
    model.grad_checkpointing = bool(case["checkpoint"])
    if case["precision"] != "bf16":
        model.quantize_frozen_linears({"4bit": "nf4", "8bit": "int8"}[case["precision"]])
    engine = DistillEngine(model, loss=case["loss"], temperature=case["temperature"], alpha=2.0, crop_to_size=cfg.vocab_size,
                           optimizer=case["optimizer"], lr=1e-4, grad_accum=case["accum"])
    batches = [_host_batch(case, cfg, rnd, gen) for _ in range(case["accum"])]
    return {"kind": case["kind"], "model": model, "engine": engine, "batches": batches}


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    """train: loss and updated weights (fp32 master and bf16) of one optimizer step. collect: the log-probs in pinned host
    memory and, as one flag per vocabulary entry, which entries each row keeps (rows rank nearly equal entries in an
    order that the last bit decides; the set and the ranked values do not depend on it)."""
    # a program holds one model with frozen low-bit weights; here several are alive, so say whose layers are expanded
    quant = state["model"].quant
    llama.LAYER_WEIGHTS_PRE[0] = quant.before_layer if quant is not None else None
    if state["kind"] == "train":
        engine = state["engine"]
        loss = engine.train_step(state["batches"])
        return {"loss": loss, "master": engine.flat.master, "weights": engine.flat.model}
    collector = state["collector"]
    logp, ids, _ = collector.fetch(collector.submit(state["tokens"], state["convos"]))
    if ids is None:
        return {"logp": logp}
    kept = torch.zeros((ids.shape[0], state["vocab"]), dtype=torch.uint8, device="cuda")
    kept.scatter_(1, ids.to("cuda", non_blocking=True).long(), 1)
    return {"logp": logp, "kept": kept}


# ------------------------------------------------------------------------------------------------ what a pass needs
def work(case):
    cfg = _config(case)
    B, L, h, V = case["batch"], case["seq"], cfg.hidden_size, cfg.vocab_size
    d, H, q, kv = cfg.head_dim, cfg.num_attention_heads, cfg.q_size, cfg.kv_size
    n_exp = max(1, cfg.num_local_experts)
    used = cfg.num_experts_per_tok if cfg.num_local_experts else 1
    attn_w, ffn_w = h * (q + 2 * kv) + q * h, 3 * h * cfg.intermediate_size
    layers = cfg.num_hidden_layers
    decoder = layers * (attn_w + n_exp * ffn_w)                       # stored matrix elements
    active = layers * (attn_w + used * ffn_w)                         # elements that multiply each token
    tokens, rows = B * L, B * L if case["rows"] == "all" else int(B * L * 0.93)
    W = min(L, case["window"] or L)
    pairs = B * (W * (W + 1) // 2 + (L - W) * W)                      # visible (query, key) pairs
    attn = layers * 4.0 * pairs * H * d
    head_entries = V * h
    embed = 0 if cfg.tie_word_embeddings else V * h
    if case["kind"] == "collect":
        stored = rows * (V * 2 if case["full"] else case["topk"] * 6)
        return {"flops": 2.0 * active * tokens + attn + 2.0 * head_entries * rows,
                "bytes": 2.0 * (decoder + head_entries) + 2.0 * min(tokens, V) * h + 8.0 * tokens + stored}
    frozen = case["precision"] != "bf16"
    batch_bytes = 8.0 * tokens + rows * case["topk"] * 8.0
    dec_bytes = decoder * ({"bf16": 2.0, "4bit": 0.52, "8bit": 1.0}[case["precision"]])
    forward = 2.0 * active * tokens + attn + 2.0 * head_entries * rows
    backward = (2.0 if frozen else 4.0) * active * tokens + 2.5 * attn + 4.0 * head_entries * rows
    trained = head_entries + embed + (0 if frozen else decoder)
    state = {"adamw": 8.0, "adamw8bit": 2.0}[case["optimizer"]]
    # per trained element: weight read and written (bf16), fp32 gradient written, fp32 master and state read and written
    update = trained * (2 + 2 + 4 + 2 * (4 + state))
    return {"flops": case["accum"] * (forward + backward),
            "bytes": update + (dec_bytes if frozen else 0) + case["accum"] * batch_bytes}


def tolerance(case):
    """Measured against the same models with library GEMMs (fp32 accumulation in another order) and library attention:
    after one AdamW step the weights differ by 0.0001 - 0.0011 of their norm (elements whose gradient is within rounding
    of zero move the other way: single ones by 0.012 of the rms), two steps nearly double that; a step that is left
    out shows as 0.002 - 0.005. Collected log-probs differ by 0.005 - 0.013 (single ones by 0.05 - 0.13, behind a router
    0.4), and 3 - 7 % of the entries at the edge of a row's top-K are others (behind a router 9 %)."""
    if case["kind"] == "train":
        return {"rel": 0.003, "max": 0.05}
    router = case["model"].startswith("tinymixtral")
    swapped = 0.35 if router else 0.2                   # of a row's K entries; each shows twice in the V flags
    vocab = _config(case).vocab_size
    return {"rel": 0.03, "max": 0.9 if router else 0.5, "differ": min(0.01, 2 * swapped * case["topk"] / vocab)}
