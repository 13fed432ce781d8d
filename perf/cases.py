"""Performance cases of the verify path: what a host program has it do, through the public entry points.

A serving process loads one model, keeps sessions (KV pool, recurrent state) and calls verify steps, prompt
passes and speculative generation on them; a host with its own runtime calls the quantized GEMM and the
acceptance stage directly. `listed()` names one case per regime, `draw()` gives more of the same ranges:

  step      Session.verify: chains and trees, greedy and rejection sampling, 1..32 sequences, any KV format
  prompt    Session.forward: the prompt of a new request, or more tokens behind a context (plain decode, next turn)
  generate  spec_generate_device: a whole request with prompt-lookup drafts
  gemm      gemm_quant: one quantized matrix product on tile-ordered weights
  accept    accept_tree: the acceptance stage over logits that are already on the device

Models are the repository's own shapes with seeded random weights. The head is made to favour one successor of
every token, as a trained model does, so that greedy tokens and acceptance decisions are decisive: they do not
hang on the last bits of a sum, drafts are accepted at a realistic rate on every pass, and greedy text repeats
itself after 32 tokens, which is what prompt lookup lives on.
"""
import math

import numpy as np
import torch

from yuuka_b200 import cuda, synth

KV = {"f16": (cuda.KV_F16, 2.0), "f32": (cuda.KV_F32, 4.0), "q8_0": (cuda.KV_Q8_0, 34.0 / 32.0)}
GEMM_DTYPE = {"q4_k": synth.Q4_K, "q5_k": synth.Q5_K, "q6_k": synth.Q6_K, "q8_0": synth.Q8_0}
ACCEPT_RATE = 0.7   # share of draft tokens that are the model's own next token
GROWTH = 256        # tokens a sequence may grow by before the next request takes its place
WIDE_ROWS = 48      # rows from which a launch multiplies fp16-rounded weights and activations


# --------------------------------------------------------------------------- cases

def listed():
    return [
        # the smallest step there is: a draft model's or a test's; launches and host work are all of it
        {"name": "tiny step 5", "kind": "step", "model": "tiny", "batch": 1, "nodes": 5, "tree": False, "mode": "greedy",
         "context": 64, "context_max": 64, "kv": "f16"},
        # one token of plain decode behind a conversation, logits to the host for the host's own sampler
        {"name": "decode 1", "kind": "prompt", "model": "dense4b", "tokens": 1, "context": 700, "kv": "f16"},
        # the interactive verify step: one sequence, eight drafts, a context of a few pages
        {"name": "chain 9", "kind": "step", "model": "dense4b", "batch": 1, "nodes": 9, "tree": False, "mode": "greedy",
         "context": 1500, "context_max": 1500, "kv": "f16"},
        # a handful of users at once, contexts of different lengths
        {"name": "chain 4x9", "kind": "step", "model": "dense4b", "batch": 4, "nodes": 9, "tree": False, "mode": "greedy",
         "context": 256, "context_max": 1900, "kv": "f16"},
        # a full server: one GPU's share of 256 sequences, 16-node draft trees, sampling
        {"name": "tree 32x17", "kind": "step", "model": "dense4b", "batch": 32, "nodes": 17, "tree": True, "mode": "rejection",
         "context": 256, "context_max": 3072, "kv": "f16"},
        # mixture of experts, a full server
        {"name": "moe 32x5", "kind": "step", "model": "moe", "batch": 32, "nodes": 5, "tree": False, "mode": "greedy",
         "context": 1024, "context_max": 1024, "kv": "f16"},
        # a new request with a long prompt of no round length
        {"name": "prompt 1837", "kind": "prompt", "model": "dense4b", "tokens": 1837, "context": 0, "kv": "f16"},
        # a whole request: prompt, then bursts of device-drafted steps
        {"name": "generate 96+128", "kind": "generate", "model": "dense4b", "prompt": 96, "max_tokens": 128, "max_draft": 8},
        # direct GEMM calls: a small matrix for two rows, the LM head for a verify step, a projection for a full batch
        {"name": "gemm 2560x2560 2", "kind": "gemm", "dtype": "q4_k", "n_out": 2560, "n_in": 2560, "rows": 2, "x": "bf16"},
        {"name": "gemm 248320x2560 9", "kind": "gemm", "dtype": "q6_k", "n_out": 248320, "n_in": 2560, "rows": 9, "x": "bf16"},
        {"name": "gemm 9216x2560 576", "kind": "gemm", "dtype": "q4_k", "n_out": 9216, "n_in": 2560, "rows": 576, "x": "bf16"},
        # the acceptance stage alone, over a full server's logits
        {"name": "accept 64x9", "kind": "accept", "batch": 64, "nodes": 9, "vocab": 248320, "mode": "rejection"},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "prompt", "prompt", "gemm", "gemm", "gemm", "accept", "generate"])
    if kind == "step":
        model = rng.choice(["dense4b", "dense4b", "dense4b", "dense4b", "moe", "tiny"])
        batch, nodes = _log(rng, 1, 32), rng.randint(1, 17)
        mode = rng.choice(["greedy", "greedy", "rejection"])
        lo, hi = sorted((_log(rng, 32, 400 if model == "tiny" else 3000), _log(rng, 32, 400 if model == "tiny" else 3000)))
        if model == "moe":
            hi = min(hi, 1024)
            lo = min(lo, hi)
        if model == "tiny":
            hi = min(hi, 512 - 17 - 16)
            lo = min(lo, hi)
        return {"kind": "step", "model": model, "batch": batch, "nodes": nodes, "tree": nodes > 4 and rng.random() < 0.4,
                "mode": mode, "context": lo, "context_max": hi, "kv": rng.choice(["f16", "f16", "f32", "q8_0"])}
    if kind == "prompt":
        model = rng.choice(["dense4b", "dense4b", "dense4b", "moe", "tiny"])
        n = _log(rng, 1, {"dense4b": 1837, "moe": 1024, "tiny": 200}[model])
        context = rng.choice([0, _log(rng, 16, 1500 if model != "tiny" else 200)])
        return {"kind": "prompt", "model": model, "tokens": n, "context": context, "kv": rng.choice(["f16", "f16", "f32", "q8_0"])}
    if kind == "generate":
        return {"kind": "generate", "model": rng.choice(["dense4b", "tiny"]), "prompt": _log(rng, 8, 200),
                "max_tokens": _log(rng, 16, 128), "max_draft": rng.randint(2, 12)}
    if kind == "gemm":
        dtype = rng.choice(list(GEMM_DTYPE))
        n_in = 256 * _log(rng, 2, 36)
        n_out = _log(rng, 256, 32768)
        return {"kind": "gemm", "dtype": dtype, "n_out": n_out, "n_in": n_in, "rows": _log(rng, 1, 576), "x": rng.choice(["bf16", "f32"])}
    return {"kind": "accept", "batch": _log(rng, 1, 64), "nodes": rng.randint(2, 9), "vocab": _log(rng, 4096, 248320),
            "mode": rng.choice(["greedy", "rejection"])}


# --------------------------------------------------------------------------- models

CONFIGS = {
    "tiny": lambda: synth.tiny_config(),
    "dense4b": lambda: synth.dense4b_config(),
    "moe": lambda: synth.moe_config(layers=8),
}
SCHEME = {"tiny": "q8_0", "dense4b": "q4_k_m", "moe": "q4_k_m"}
# embedding scale (against the residual additions of the layers) and the logit of a token's favoured successor
HEAD = {"tiny": (1.0, 14.0), "dense4b": (20.0, 22.0), "moe": (4.0, 20.0)}

_device, _stream, _models = None, None, {}


def device():
    global _device, _stream
    if _device is None:
        _device = cuda.Device(0)
        _stream = _device.stream()
    return _device


def successor(tokens):
    """The favoured next token: the vocabulary in cycles of 32."""
    t = np.asarray(tokens)
    return (t & ~31) | ((t + 1) & 31)


def _matrix(values, dtype):
    rows, cols = values.shape
    out = np.empty(rows * synth.row_bytes(dtype, cols), np.uint8)
    rb, step = synth.row_bytes(dtype, cols), 16384
    for r in range(0, rows, step):
        out[r * rb:(r + step) * rb] = synth.quantize(values[r:r + step].cpu().numpy(), dtype)
    return out


def _tensors(name):
    """One recurrent and one attention layer from the package's generator, repeated over the depth of the model, and
    an embedding and a head of which token t's successor answers to t's embedding."""
    cfg = CONFIGS[name]()
    V, H, every = cfg["vocab"], cfg["hidden"], cfg["full_attention_interval"]
    kinds = {}
    for recurrent, interval in ((True, 4), (False, 1)):
        one = dict(cfg, block_count=1, vocab=32, full_attention_interval=interval)
        kinds[recurrent] = synth.make_model(one, SCHEME[name], seed=11 + interval, unit_norms=False)
    t = {"output_norm.weight": kinds[True]["output_norm.weight"]}
    for i in range(cfg["block_count"]):
        for key, value in kinds[(i + 1) % every != 0].items():
            if key.startswith("blk.0."):
                t[f"blk.{i}." + key[6:]] = value
    pick = synth.quant_plan(SCHEME[name])
    g = torch.Generator(device="cuda").manual_seed(5)
    scale, favoured = HEAD[name]
    e = torch.randn(V, H, generator=g, device="cuda")
    t["token_embd.weight"] = (pick("token_embd"), _matrix(e * scale, pick("token_embd")), V, H)
    head = torch.randn(V, H, generator=g, device="cuda") * 0.02
    head[torch.from_numpy(successor(np.arange(V))).cuda()] += e * (favoured / H)
    t["output.weight"] = (pick("output"), _matrix(head, pick("output")), V, H)
    del e, head
    torch.cuda.empty_cache()
    return cfg, t


def model(name):
    """Loaded once per process, as a server does."""
    if name not in _models:
        dev = device()
        cfg, tensors = _tensors(name)
        _models[name] = cuda.Model(dev, cfg, tensors)
    return _models[name]


# --------------------------------------------------------------------------- inputs

class DeviceBuffer(cuda.Buffer):
    """Device memory of the library that is given back with the last thing that refers to it."""

    def __del__(self):
        torch.cuda.synchronize()
        self.free()


class View:
    """A device buffer as torch sees it; a tensor made from it keeps it alive."""

    def __init__(self, buffer, shape, typestr):
        self.buffer = buffer
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "version": 3,
                                         "data": (cuda.lib().yuuka_buffer_ptr(buffer.h), False)}


def view(buffer, shape, typestr="<f4"):
    return torch.as_tensor(View(buffer, shape, typestr), device="cuda")


class State:
    """What a program keeps between calls; its session is closed with it."""

    def __init__(self, case):
        self.case, self.session = case, None

    def __del__(self):
        if self.session is not None:
            torch.cuda.synchronize()
            self.session.close()


def _drafts(rng, pending, parent, vocab):
    """Tokens of one sequence's rows: of every row's children one is the model's own next token at ACCEPT_RATE."""
    n = parent.size
    tokens = rng.integers(0, vocab, n).astype(np.int32)
    tokens[0] = pending
    for row in range(n):
        children = np.flatnonzero(parent == row)
        if children.size and rng.random() < ACCEPT_RATE:
            tokens[rng.choice(children)] = successor(tokens[row])
    return tokens


def _fill_draft_probs(probs, tokens, g):
    """probs [rows, vocab]: a perturbed softmax with a good part of its mass on the drafted token."""
    vocab = probs.shape[-1]
    for r in range(probs.shape[0]):
        probs[r] = torch.softmax(3.0 * torch.randn(vocab, generator=g, device="cuda"), -1)
    share = 0.2 + 0.6 * torch.rand(probs.shape[0], 1, generator=g, device="cuda")
    probs *= 1.0 - share
    probs.scatter_add_(1, torch.from_numpy(tokens.reshape(-1, 1).astype(np.int64)).cuda(), share)


def prepare(case, seed):
    s = State(case)
    rng = np.random.default_rng(seed)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    {"step": _prepare_step, "prompt": _prepare_prompt, "generate": _prepare_generate, "gemm": _prepare_gemm,
     "accept": _prepare_accept}[case["kind"]](s, case, rng, g)
    torch.cuda.synchronize()
    return s


def _prepare_step(s, case, rng, g):
    m = model(case["model"])
    vocab, limit = m.vocab, m.cfg["context_length"]
    batch, nodes = case["batch"], case["nodes"]
    s.capacity = min(limit, (case["context_max"] + GROWTH + nodes + 15) // 16 * 16)
    s.session = cuda.Session(m, max_batch=batch, max_nodes=nodes, capacity=s.capacity, kv_format=KV[case["kv"]][0])
    blocks = s.capacity // 16
    order = rng.permutation(batch * blocks).astype(np.int32)
    s.lengths = rng.integers(case["context"], case["context_max"] + 1, batch)
    s.positions = s.lengths.copy()
    s.parent = synth.tree_16()[:nodes] if case["tree"] else np.arange(-1, nodes - 1, dtype=np.int32)
    s.tokens = np.empty((batch, nodes), np.int32)
    for b in range(batch):
        s.session.set_block_table(b, order[b * blocks:(b + 1) * blocks])
        prompt = rng.integers(0, vocab, int(s.lengths[b])).astype(np.int32)
        s.session.forward(prompt, seq=b, want_logits=False)
        s.tokens[b] = _drafts(rng, int(successor(prompt[-1])), s.parent, vocab)
    s.args = {"parent": s.parent if case["tree"] else None, "mode": cuda.ACCEPT_GREEDY}
    if case["mode"] == "rejection":
        s.probs = DeviceBuffer(device(), batch * nodes * vocab * 4)
        _fill_draft_probs(view(s.probs, (batch * nodes, vocab)), s.tokens, g)
        s.args.update(mode=cuda.ACCEPT_REJECTION, temperature=0.8, draft_probs=s.probs,
                      uniforms=rng.random((batch, nodes, 2), dtype=np.float32) * np.float32(0.999))


def _prepare_prompt(s, case, rng, g):
    m = model(case["model"])
    room = case["tokens"] if case["context"] == 0 else case["tokens"] + max(GROWTH, case["tokens"])
    s.base = min(case["context"], m.cfg["context_length"] - room)
    s.session = cuda.Session(m, max_batch=1, max_nodes=9, capacity=s.base + room, kv_format=KV[case["kv"]][0])
    s.tokens = rng.integers(0, m.vocab, case["tokens"]).astype(np.int32)
    if s.base:
        s.session.forward(rng.integers(0, m.vocab, s.base).astype(np.int32), want_logits=False)
    s.position = s.base


def _prepare_generate(s, case, rng, g):
    m = model(case["model"])
    capacity = case["prompt"] + case["max_tokens"] + 8 * (case["max_draft"] + 1)
    s.session = cuda.Session(m, max_batch=1, max_nodes=case["max_draft"] + 1, capacity=min(capacity, m.cfg["context_length"]))
    s.tokens = rng.integers(0, m.vocab, case["prompt"]).astype(np.int32)


def _prepare_gemm(s, case, rng, g):
    dev, dtype = device(), GEMM_DTYPE[case["dtype"]]
    n_out, n_in, rows = case["n_out"], case["n_in"], case["rows"]
    base = min(n_out, 4096)  # a large matrix repeats its first rows: the values of a row do not matter to the others
    packed = synth.normal_quant(base, n_in, dtype, 0.02, int(rng.integers(1 << 40)))
    packed = np.tile(packed, -(-n_out // base))[:n_out * synth.row_bytes(dtype, n_in)]
    raw = dev.upload(packed)
    s.weights = DeviceBuffer(device(), cuda.tiled_bytes(dtype, n_out, n_in) + 256)
    cuda.tile_weights(_stream, s.weights, raw, dtype, n_out, n_in)
    _stream.synchronize()
    raw.free()
    x = torch.randn(rows, n_in, generator=g, device="cuda")
    bf16 = case["x"] == "bf16"
    s.x = DeviceBuffer(device(), rows * n_in * (2 if bf16 else 4))
    if bf16:
        view(s.x, (rows, n_in), "<i2").copy_(x.to(torch.bfloat16).view(torch.int16))
    else:
        view(s.x, (rows, n_in)).copy_(x)
    s.out = DeviceBuffer(device(), rows * n_out * 4)
    s.product = view(s.out, (rows, n_out))
    s.dtype, s.x_dtype = dtype, cuda.BF16 if bf16 else cuda.F32


def _prepare_accept(s, case, rng, g):
    batch, nodes, vocab = case["batch"], case["nodes"], case["vocab"]
    rows = batch * nodes
    temperature = 0.7
    s.logits = DeviceBuffer(device(), rows * vocab * 4)
    logits = view(s.logits, (rows, vocab))
    logits.normal_(0.0, 3.0, generator=g)
    s.tokens = rng.integers(0, vocab, (batch, nodes)).astype(np.int32)
    s.args = {"mode": cuda.ACCEPT_GREEDY}
    if case["mode"] == "greedy":
        best = logits.argmax(-1).cpu().numpy().reshape(batch, nodes)
        keep = rng.random((batch, nodes - 1)) < ACCEPT_RATE
        s.tokens[:, 1:][keep] = best[:, :-1][keep]
        return
    # row c's draft distribution perturbs the target distribution of the row before it; the draft is drawn from it
    s.probs = DeviceBuffer(device(), rows * vocab * 4)
    probs = view(s.probs, (rows, vocab))
    for r in range(rows):
        if r % nodes == 0:
            probs[r] = 0.0
            continue
        probs[r] = torch.softmax(logits[r - 1] / temperature + torch.randn(vocab, generator=g, device="cuda"), -1)
        at = torch.searchsorted(probs[r].double().cumsum(0), torch.rand(1, generator=g, device="cuda").double())
        s.tokens[r // nodes, r % nodes] = min(int(at), vocab - 1)
    s.args.update(mode=cuda.ACCEPT_REJECTION, temperature=temperature, draft_probs=s.probs,
                  uniforms=rng.random((batch, nodes, 2), dtype=np.float32) * np.float32(0.999))


# --------------------------------------------------------------------------- passes

def run(s):
    return {"step": _run_step, "prompt": _run_prompt, "generate": _run_generate, "gemm": _run_gemm,
            "accept": _run_accept}[s.case["kind"]](s)


def _run_step(s):
    r = s.session.verify(s.tokens, **s.args)
    s.positions += r.accepted + 1
    for b in np.flatnonzero(s.positions + s.tokens.shape[1] > s.capacity):
        s.session.set_position(int(b), int(s.lengths[b]))  # the sequence is full: the slot goes back to its prompt
        s.positions[b] = s.lengths[b]
    return r.accepted, r.emitted, r.path


def _run_prompt(s):
    if s.base == 0:
        s.session.reset(0)  # a new request
    elif s.position + s.tokens.size > s.session.capacity:
        s.session.set_position(0, s.base)  # the context is full: back to where the conversation began
        s.position = s.base
    s.position += s.tokens.size
    return s.session.forward(s.tokens)


def _run_generate(s):
    c = s.case
    tokens, r = cuda.spec_generate_device(s.session, s.tokens, c["max_tokens"], max_draft=c["max_draft"])
    return np.array(tokens, np.int32), r.steps, r.draft_tokens, r.accepted_draft


def _run_gemm(s):
    c = s.case
    cuda.gemm_quant(_stream, s.out, s.x, s.weights, c["n_in"], c["n_out"], c["rows"], s.dtype, s.x_dtype, flags=cuda.GEMM_TILED)
    return s.product


def _run_accept(s):
    return cuda.accept_tree(_stream, s.logits, s.tokens, s.case["vocab"], **s.args)


# --------------------------------------------------------------------------- work

def _model_work(name, rows):
    """(weight bytes, multiply-adds per row, recurrent state bytes of one sequence, attention layers) of a pass over
    `rows` rows; head aside. Of the routed experts the ones that rows of an even router touch are counted."""
    cfg, pick = CONFIGS[name](), synth.quant_plan(SCHEME[name])
    H, S, R, inner = cfg["hidden"], cfg["state_size"], cfg["time_step_rank"], cfg["inner_size"]
    conv = 2 * cfg["group_count"] * S + inner
    q, kv, o = cfg["heads"] * cfg["head_dim"] * 2, cfg["kv_heads"] * cfg["head_dim"], cfg["heads"] * cfg["head_dim"]
    experts, used = cfg["expert_count"], cfg["expert_used"]
    nbytes = macs = state = attention = 0.0
    for i in range(cfg["block_count"]):
        if synth.is_recurrent(cfg, i):
            parts = [("attn_qkv", conv, H), ("attn_gate", inner, H), ("ssm_out", H, inner), ("ssm_beta", 2 * R, H)]
            state += 4.0 * (R * S * S + conv * (cfg["conv_kernel"] - 1))
        else:
            parts = [("attn_q", q, H), ("attn_k", kv, H), ("attn_v", kv, H), ("attn_output", H, o)]
            attention += 1
        if experts:
            ef, sf = cfg["expert_ffn"], cfg["shared_ffn"]
            touched = experts * (1.0 - (1.0 - used / experts) ** rows)
            for role, n, k in (("ffn_gate_exps", 2 * ef, H), ("ffn_down_exps", H, ef)):
                nbytes += touched * n * synth.row_bytes(pick(role), k)
                macs += used * n * k
            nbytes += 4.0 * experts * H
            parts += [("ffn_gate_shexp", 2 * sf, H), ("ffn_down_shexp", H, sf)]
        else:
            parts += [("ffn_gate", 2 * cfg["ffn"], H), ("ffn_down", H, cfg["ffn"])]
        for role, n, k in parts:
            nbytes += n * synth.row_bytes(pick(role), k)
            macs += n * k
    return nbytes, macs, state, attention, cfg


def _pass_work(name, rows, context, batch, logit_rows, kv):
    """A pass of rows per sequence over `batch` sequences with `context` committed positions each on average."""
    total = rows * batch
    nbytes, macs, state, attention, cfg = _model_work(name, total)
    head = cfg["vocab"] * synth.row_bytes(synth.quant_plan(SCHEME[name])("output"), cfg["hidden"])
    kv_row = 2.0 * cfg["kv_heads"] * cfg["head_dim"] * KV[kv][1] * attention
    nbytes += head + batch * (2.0 * state + kv_row * (context + rows))
    keys = context + (rows + 1) / 2.0
    flops = 2.0 * macs * total + 2.0 * logit_rows * cfg["vocab"] * cfg["hidden"] + \
        4.0 * total * keys * cfg["heads"] * cfg["head_dim"] * attention
    return nbytes, flops


def work(case):
    kind = case["kind"]
    if kind == "step":
        context = (case["context"] + case["context_max"]) / 2.0
        nbytes, flops = _pass_work(case["model"], case["nodes"], context, case["batch"], case["batch"] * case["nodes"], case["kv"])
        if case["mode"] == "rejection":  # the draft rows of about three nodes a sequence
            nbytes += case["batch"] * min(3, case["nodes"]) * 4.0 * CONFIGS[case["model"]]()["vocab"]
    elif kind == "prompt":
        nbytes, flops = _pass_work(case["model"], case["tokens"], case["context"], 1, 1, case["kv"])
    elif kind == "generate":
        # the prompt, one row per step through the first cycle of 32 tokens, then whole drafts are accepted
        nbytes, flops = _pass_work(case["model"], case["prompt"], 0, 1, 1, "f16")
        plain = min(case["max_tokens"], 32)
        steps = plain + (case["max_tokens"] - plain) / (case["max_draft"] + 1.0)
        b, f = _pass_work(case["model"], 1, case["prompt"] + case["max_tokens"] / 2.0, 1, 1, "f16")
        nbytes, flops = nbytes + b * steps, flops + f * case["max_tokens"]
    elif kind == "gemm":
        n_out, n_in, rows = case["n_out"], case["n_in"], case["rows"]
        nbytes = n_out * synth.row_bytes(GEMM_DTYPE[case["dtype"]], n_in) + rows * n_in * (2 if case["x"] == "bf16" else 4) + rows * n_out * 4
        flops = 2.0 * rows * n_out * n_in
    else:
        # greedy reads every row; a walk reads logits and draft probabilities of the nodes it visits, about three
        row = 4.0 * case["vocab"]
        seen = case["nodes"] if case["mode"] == "greedy" else min(3, case["nodes"]) * 2
        nbytes = case["batch"] * seen * row
        flops = nbytes / 2.0
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    kind = case["kind"]
    if kind == "prompt":
        # contexts and prompts of 48 tokens and more pass through fp16-rounded products, layer after layer
        return {"rel": 1e-2}
    if kind == "gemm":
        return {"rel": 1e-5} if case["rows"] < WIDE_ROWS else {"rel": 1e-3}
    if kind == "step" and case["mode"] == "rejection":
        # a token drawn from the bulk of the vocabulary changes with the last bits of the logits
        return {"rel": 0.0, "differ": 0.01}
    return "exact"
