"""The workloads whose speed is tracked: what a program that serves a model with this engine has it do.

Every case goes through the public entry points: `Cache.infer` (one reference-style call per token: host ids in, FP16
logits and the next token out), the batched entry points `Cache.batch_prefill` / `Cache.batch_step`, and the
device sampler `llmb_sample_logits`.  The decoded tokens are given (as in scoring or speculative verification), not
the greedy ones, so that the inputs of every step are the same whatever the last bit of the logits before it.

Kinds of case
  request       a prompt of `n_prompt` tokens, then `n_new` - 1 more tokens one call at a time; answers the logits of
                all `n_new` calls.  `n_new` = 1 is the prompt phase alone (time to first token).
  batch         `n_steps` steps of a running batch: `n_seqs` sequences, one token each per step, behind prompts of
                `n_prompt` tokens that were processed before; answers the last step's logits of every sequence.
  batch_prompt  `n_seqs` new prompts of `n_prompt` tokens each, and the batch's first step; answers its logits.
  sample        one temperature / top-k / top-p draw from each of `rows` rows of logits; answers the tokens.

A program loads its weights once and serves many requests, so the model (seeded synthetic weights in the published
shape) is kept per process; prompts, given tokens and logits come from the seed, and each state has a KV cache of
its own.
"""
import weakref

import numpy as np
import torch

from __graft_entry__ import load_package

REQUEST_SEQ = 4224   # cache rows of a request: a 4096-token prompt and 128 tokens
BATCH_SEQ = 1536     # cache rows per sequence of a batch
LOGIT_STD = 1.3      # spread of the logits of a model with these weights


def listed():
    return [
        # the smallest requests: a two-layer model, where launches, synchronisation and host work are all there is
        {"name": "request_tiny_16_32", "kind": "request", "model": "tiny", "n_prompt": 16, "n_new": 32},
        # the headline use: a chat turn at batch 1 (128-token prompt, then token by token)
        {"name": "request_8b_128_64", "kind": "request", "model": "llama3_8b", "n_prompt": 128, "n_new": 64},
        # a long document, then an answer: decode behind thousands of cached rows
        {"name": "request_8b_4096_64", "kind": "request", "model": "llama3_8b", "n_prompt": 4096, "n_new": 64},
        # time to first token: a short question (odd length), an ordinary ragged prompt, a long document
        {"name": "prompt_8b_37", "kind": "request", "model": "llama3_8b", "n_prompt": 37, "n_new": 1},
        {"name": "prompt_8b_517", "kind": "request", "model": "llama3_8b", "n_prompt": 517, "n_new": 1},
        {"name": "prompt_8b_4096", "kind": "request", "model": "llama3_8b", "n_prompt": 4096, "n_new": 1},
        # serving several users at once: a handful (odd number, odd lengths), a full batch, more than one row tile
        {"name": "batch_8b_5x333", "kind": "batch", "model": "llama3_8b", "n_seqs": 5, "n_prompt": 333, "n_steps": 8},
        {"name": "batch_8b_32x1024", "kind": "batch", "model": "llama3_8b", "n_seqs": 32, "n_prompt": 1024, "n_steps": 8},
        {"name": "batch_8b_96x200", "kind": "batch", "model": "llama3_8b", "n_seqs": 96, "n_prompt": 200, "n_steps": 8},
        # the widest layer shape that the engine is configured for (two layers of it)
        {"name": "batch_70b_l2_16x100", "kind": "batch", "model": "llama3_70b_l2", "n_seqs": 16, "n_prompt": 100, "n_steps": 8},
        # new prompts of a batch
        {"name": "batch_prompt_8b_16x150", "kind": "batch_prompt", "model": "llama3_8b", "n_seqs": 16, "n_prompt": 150},
        # the reference's sampler with its own constants, over the 8B vocabulary
        {"name": "sample_128256x8", "kind": "sample", "vocab": 128256, "rows": 8, "temperature": 0.7, "top_k": 50, "top_p": 0.9},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["request", "request", "prompt", "prompt", "batch", "batch", "batch_prompt", "sample"])
    if kind in ("request", "prompt"):
        return {"kind": "request", "model": rng.choice(["tiny", "llama3_8b_prof", "llama3_8b", "llama3_8b"]),
                "n_prompt": _log_int(rng, 1, 4096), "n_new": _log_int(rng, 2, 64) if kind == "request" else 1}
    if kind == "batch":
        n_seqs = _log_int(rng, 1, 128)
        return {"kind": kind, "model": rng.choice(["llama3_8b", "llama3_8b", "llama3_70b_l2"]), "n_seqs": n_seqs,
                "n_prompt": _log_int(rng, 1, min(1024, 32768 // n_seqs)), "n_steps": 8}
    if kind == "batch_prompt":
        n_seqs = _log_int(rng, 1, 64)
        return {"kind": kind, "model": rng.choice(["llama3_8b", "llama3_8b", "llama3_70b_l2"]), "n_seqs": n_seqs,
                "n_prompt": _log_int(rng, 2, min(1024, 8192 // n_seqs))}
    return {"kind": kind, "vocab": rng.choice([4096, 32768, 128256]), "rows": _log_int(rng, 1, 16),
            "temperature": round(rng.uniform(0.5, 1.3), 2), "top_k": _log_int(rng, 1, 200), "top_p": round(rng.uniform(0.5, 0.99), 2)}


_MODELS = {}


def _model(name, max_seq):
    """The loaded model, as a serving process keeps it."""
    if (name, max_seq) not in _MODELS:
        pkg = load_package()
        _MODELS[name, max_seq] = pkg.Model.synthetic(pkg.CONFIGS[name], seed=0, max_seq=max_seq)
    return _MODELS[name, max_seq]


class _Session:
    """A KV cache with what is fed to it; gives its device memory back when the last reference goes."""

    def __init__(self, case, seed):
        pkg = load_package()
        self.case = case
        self.cfg = pkg.CONFIGS[case["model"]]
        self.cache = pkg.Cache(_model(case["model"], REQUEST_SEQ if case["kind"] == "request" else BATCH_SEQ))
        weakref.finalize(self, self.cache.close)
        self.rng = np.random.default_rng(seed)

    def ids(self, *shape):
        return self.rng.integers(0, self.cfg.vocab, shape, dtype=np.int32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sample":
        pkg = load_package()
        gen = torch.Generator(device="cuda").manual_seed(seed)
        logits = (torch.randn(case["rows"], case["vocab"], generator=gen, device="cuda") * LOGIT_STD).half()
        return {"case": case, "seed": seed, "lib": pkg.lib, "logits": logits,
                "scratch": torch.zeros(pkg.lib.llmb_sample_scratch_bytes(case["vocab"]), dtype=torch.uint8, device="cuda"),
                "tokens": torch.zeros(case["rows"], dtype=torch.int32, device="cuda")}
    s = _Session(case, seed)
    if kind == "request":
        s.tokens = s.ids(case["n_prompt"] + case["n_new"] - 1).tolist()
        return s
    s.cache.batch_init(case["n_seqs"])
    s.prompts = s.ids(case["n_seqs"], case["n_prompt"])
    if kind == "batch":
        s.given = s.ids(BATCH_SEQ, case["n_seqs"])
        s.cache.batch_prefill(s.prompts)
        s.rows = case["n_prompt"] - 1
        _batch_steps(s)   # a running batch: its first steps are behind it
    return s


def _batch_steps(s):
    """`n_steps` steps of the batch; when the cache rows are used up, the batch starts over with its prompts."""
    if s.rows + s.case["n_steps"] > BATCH_SEQ:
        s.cache.batch_prefill(s.prompts)
        s.rows = s.case["n_prompt"] - 1
    logits = None
    for i in range(s.case["n_steps"]):
        _, logits = s.cache.batch_step(s.given[s.rows], want_logits=i == s.case["n_steps"] - 1)
        s.rows += 1
    return logits.view(np.float16)


def run(state):
    if isinstance(state, dict):  # sample
        c, lib = state["case"], state["lib"]
        logits, tokens = state["logits"], state["tokens"]
        for r in range(c["rows"]):
            rc = lib.llmb_sample_logits(logits[r].data_ptr(), c["vocab"], c["temperature"], c["top_k"], c["top_p"], state["seed"], r,
                                        state["scratch"].data_ptr(), tokens[r:].data_ptr(), None, None, 0, 0,
                                        torch.cuda.current_stream().cuda_stream)
            if rc != 0:
                raise RuntimeError("llmb_sample_logits: status %d" % rc)
        return tokens
    case, cache = state.case, state.cache
    if case["kind"] == "request":
        n = case["n_prompt"]
        cache.reset()
        seq = state.tokens[:n]
        out = []
        while True:
            cache.infer(seq)
            out.append(cache.logits().view(np.float16))
            if len(out) == case["n_new"]:
                return out
            seq.append(state.tokens[len(seq)])
    if case["kind"] == "batch":
        return _batch_steps(state)
    cache.batch_prefill(state.prompts)
    return cache.batch_step(None, want_logits=True)[1].view(np.float16)


def work(case):
    if case["kind"] == "sample":
        return {"bytes": case["rows"] * (2 * case["vocab"] + 4), "flops": 4 * case["rows"] * case["vocab"]}
    cfg = load_package().CONFIGS[case["model"]]
    mm, head, kv = cfg.matmul_params(), cfg.vocab * cfg.d_model, cfg.kv_bytes_per_position()
    qk_pv = 4 * cfg.n_q_heads * cfg.head_dim * cfg.n_layers     # flops of one query row against one cached row

    def forward(rows, seen, heads):
        """One pass over the weights for `rows` new rows that see `seen` rows in all (summed), `heads` rows of logits."""
        return 2.0 * (mm * rows + head * heads) + qk_pv * seen

    if case["kind"] == "request":
        n, new = case["n_prompt"], case["n_new"]
        bytes_, flops = cfg.weight_bytes_per_token() + kv * n, forward(n, n * (n + 1) / 2, 1)
        for i in range(n, n + new - 1):
            bytes_ += cfg.decode_bytes(i)
            flops += forward(1, i + 1, 1)
        return {"bytes": bytes_ + 2 * cfg.vocab * new, "flops": flops}
    b, n = case["n_seqs"], case["n_prompt"]
    logits = 2 * cfg.vocab * b
    if case["kind"] == "batch_prompt":
        return {"bytes": cfg.weight_bytes_per_token() + kv * n * b + logits, "flops": b * forward(n, n * (n + 1) / 2, 1)}
    bytes_, flops = logits, 0.0
    for i in range(n + case["n_steps"], n + 2 * case["n_steps"]):
        bytes_ += cfg.weight_bytes_per_token() + b * kv * (i + 1)
        flops += b * forward(1, i + 1, 1)
    return {"bytes": bytes_, "flops": flops}


# Four times what two summation orders differ by (prompt as blocks of rows or token by token, whole-step kernel or one
# kernel per operation, batch rows against single sequences), FP16 rounding points the same: measured, over prompts of
# 16 to 4096 tokens, (2-norm, largest) 0.0060, 0.031 at 32 layers, 0.0017, 0.0076 at 4 layers, 0.0007, 0.0030 for the
# tiny model, 0.0012, 0.0059 for two layers of the 70B shape: each layer rounds to FP16 seven times, so it grows with depth.
TOLERANCE = {
    "llama3_8b": {"rel": 0.024, "max": 0.125},
    "llama3_8b_prof": {"rel": 0.0068, "max": 0.03},
    "llama3_70b_l2": {"rel": 0.0048, "max": 0.024},
    "tiny": {"rel": 0.0028, "max": 0.012},
}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"   # the draw is the same token unless u lies within FP32 ulps of a boundary between two entries
    return TOLERANCE[case["model"]]
