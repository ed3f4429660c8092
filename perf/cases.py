"""The calls whose speed this framework is judged by, as a serving program makes them.

Almost every case is one packed step (`Engine.step`) of a model held by an engine, followed by what the caller reads of it and by
the acceptance that lets the next step begin: decode rows, speculative verify blocks, prompt chunks and mixtures of them, over
the two shapes the repository names (the tiny hybrid and the 27B shape, all 64 blocks), over MLX 4-bit and GGUF weights. One case
is a pass over tensors of the caller's own built from the engine's primitives, as a drafter makes it.

An engine, its weights and the pages of its sessions are what a server keeps: they are built once per case and shared by
the states of a process. A state is a set of sessions of that engine: the recurrent state, the tokens and the accepted lengths come
from the seed; KV pages hold pseudo-random codes as the benchmark's do. Weights are seeded synthetic ones.
"""
import json

import numpy as np
import torch

import splosh_b200 as S
from splosh_b200 import synthetic

WEIGHT_SEED = 0x5EED6D17
STATES = 4              # sets of sessions an engine has room for at a time
TURNS = 8               # steps after which a session's positions start over (its recurrent state goes on)
PAGE = 256
GGUF = {"q4_k": "Q4_K", "q5_k": "Q5_K", "q6_k": "Q6_K"}
BLOCK_BYTES = {"mlx4": 0.5625, "q4_k": 144 / 256, "q5_k": 176 / 256, "q6_k": 210 / 256}     # per weight
DRAFT_LAYERS, DRAFT_ATTENTION = 5, 4096


def _step(name, model, weights="mlx4", sessions=0, block=1, context=0, prompt=0, fed=0, read="topk"):
    return {"name": name, "model": model, "weights": weights, "sessions": sessions, "block": block, "context": context, "prompt": prompt, "fed": fed,
            "read": read}


def listed():
    return [
        # The smallest call: one decoding session of the tiny hybrid, its logits read by the host. Launches and latency.
        _step("tiny_decode_1", "tiny", sessions=1, context=1024, read="logits"),
        # The tiny hybrid's packed step: a 512-token prompt chunk and two decoders that verify 4-token drafts.
        _step("tiny_packed_520", "tiny", sessions=2, block=4, context=1536, prompt=512),
        # One user on the 27B shape, no draft: a row a step at 10.7K tokens of context, sampled by the host from the logits.
        _step("decode_1", "27b", sessions=1, context=10700, read="logits"),
        # Continuous batching without drafts: twelve sessions of ordinary chat length, a row each.
        _step("decode_12", "27b", sessions=12, context=3000),
        # A lightly loaded server with drafts: three sessions with verify blocks of 7 rows.
        _step("verify_3x7", "27b", sessions=3, block=7, context=12000),
        # The headline: eight sessions around 39K tokens, each verifying an 8-token draft.
        _step("verify_8x8", "27b", sessions=8, block=8, context=39000),
        # The same decoders with 64 rows of a long prompt riding in the step.
        _step("rider_8x8_64", "27b", sessions=8, block=8, context=39000, prompt=64, fed=10500),
        # Time to first token of an ordinary question: a new session's 301-token prompt in one step.
        _step("prompt_301", "27b", prompt=301, read="logits"),
        # A long prompt's chunk: 2,048 rows over 24K tokens already fed.
        _step("prefill_2048", "27b", prompt=2048, fed=24576, read="logits"),
        # GGUF weights, one session with a very long context and 16-token drafts.
        _step("gguf_verify_16", "27b", weights="q5_k", sessions=1, block=16, context=171000),
        # GGUF weights of the smaller type: a new session's prompt of 200 tokens beside two decoding sessions.
        _step("gguf_prompt_200", "27b", weights="q4_k", sessions=2, context=5000, prompt=200),
        # A draft pass over the caller's own tensors: eight sessions' blocks of eight rows through five layers and the target's head.
        {"name": "own_tensors_64", "model": "27b", "weights": "mlx4", "pass_rows": 64},
    ]


def draw(rng):
    def log(low, high):
        return int(round(low * (high / low) ** rng.random()))
    kind = rng.choice(["tiny", "decode", "verify", "verify", "rider", "prompt", "prefill", "gguf", "gguf_prompt", "own"])
    if kind == "tiny":
        return _draw(_step("", "tiny", sessions=rng.randint(1, 4), block=rng.choice([1, 1, 4, 8]), context=log(200, 4000), prompt=rng.choice([0, log(8, 512)])))
    if kind == "decode":
        sessions = log(1, 16)
        return _draw(_step("", "27b", sessions=sessions, context=log(200, 300000 // sessions // 4), read="logits" if sessions == 1 else "topk"))
    if kind == "verify":
        sessions = log(1, 8)
        return _draw(_step("", "27b", sessions=sessions, block=rng.randint(2, 8), context=log(500, 40000)))
    if kind == "rider":
        return _draw(_step("", "27b", sessions=rng.randint(2, 8), block=rng.randint(1, 8), context=log(500, 38000), prompt=log(8, 128), fed=log(100, 20000)))
    if kind == "prompt":
        return _draw(_step("", "27b", prompt=log(20, 1500), read="logits"))
    if kind == "prefill":
        return _draw(_step("", "27b", prompt=log(200, 2048), fed=log(1000, 24000), read="logits"))
    if kind == "gguf":
        return _draw(_step("", "27b", weights=rng.choice(["q4_k", "q5_k"]), sessions=rng.randint(1, 2), block=rng.choice([1, 5, 8, 16]), context=log(500, 80000)))
    if kind == "gguf_prompt":
        # Short prompts of every type, longer ones of Q4_K alone: steps of more than 32 rows of the byte-wide types were unsafe to run when
        # this was written (the weight ring of their kernel).
        weights = rng.choice(["q4_k", "q5_k", "q6_k"])
        return _draw(_step("", "27b", weights=weights, prompt=log(20, 400) if weights == "q4_k" else rng.randint(5, 32), read="logits"))
    return {"model": "27b", "weights": "mlx4", "pass_rows": rng.randint(8, 128)}


def _draw(case):
    del case["name"]
    return case


# ---- sizes ---------------------------------------------------------------------------------------
def _geometry(case):
    return S.tiny_geometry() if case["model"] == "tiny" else S.b27_geometry(layers=4 if "pass_rows" in case else 64)


def _contexts(case):
    """Tokens in front of each session's first step: around `context`, ragged, with room for the turns' rows in the last page."""
    room = PAGE - TURNS * case["block"] - 20
    out = []
    for s in range(case["sessions"]):
        tokens = int(case["context"] * (0.9 + 0.2 * ((s * 0.618034) % 1.0))) if case["sessions"] > 1 else case["context"]
        out.append(tokens // PAGE * PAGE + min(max(tokens % PAGE, 1), room))
    return out


def _weights(g):
    """(in the blocks, in the head)."""
    H, VD, VH = g.hidden, g.value_dim, g.gdn_value_heads
    AD, KV = g.heads * g.head_dim, g.kv_heads * g.head_dim
    n_full = g.layers // 4
    linear = (g.channels + VD + 2 * VH) * H + H * VD + 3 * H * g.inter
    full = (2 * AD + 2 * KV) * H + H * AD + 3 * H * g.inter
    return (g.layers - n_full) * linear + n_full * full, g.vocab * H


def work(case):
    g = _geometry(case)
    blocks, head = _weights(g)
    if "pass_rows" in case:
        rows = case["pass_rows"]
        own = DRAFT_LAYERS * (2 * DRAFT_ATTENTION * g.hidden + 3 * g.hidden * g.inter)
        return {"bytes": (own + head) * 0.5625 + rows * (g.vocab + g.hidden) * 4, "flops": 2.0 * rows * (own + head)}
    contexts = _contexts(case)
    rows = case["sessions"] * case["block"] + case["prompt"]
    logit_rows = case["sessions"] * case["block"] + (1 if case["prompt"] and (case["read"] == "logits" or not case["fed"]) else 0)
    head_bytes = BLOCK_BYTES["mlx4" if case["weights"] == "mlx4" else "q6_k"]
    n_full = g.layers // 4
    tokens = sum(contexts) + (case["fed"] + case["prompt"] if case["prompt"] else 0)
    attended = sum(case["block"] * (c + case["block"] / 2) for c in contexts) + case["prompt"] * (case["fed"] + case["prompt"] / 2)
    state = (g.layers - n_full) * g.gdn_value_heads * 128 * 128
    holders = case["sessions"] + (1 if case["prompt"] else 0)
    returned = logit_rows * (g.vocab if case["read"] == "logits" else 20) * 4
    return {"bytes": blocks * BLOCK_BYTES[case["weights"]] + head * head_bytes + tokens * n_full * 2 * g.kv_heads * (g.head_dim + 4)
                     + holders * state * 4 * 2 + returned,
            "flops": 2.0 * rows * blocks + 2.0 * logit_rows * head + 4.0 * g.heads * g.head_dim * n_full * attended + 6.0 * rows * state}


def tolerance(case):
    """Every GEMM input is rounded to bf16 (2^-9) and keys and values to 8 bits, at points that move with the order of 32-bit sums, and
    the blocks carry the differences on: the same rows in steps of other widths differ by 1.5e-2 over the 64 blocks' whole logits,
    3e-3 over the largest twenty, a third of that over few blocks."""
    if "pass_rows" in case:
        return {"rel": 5e-3, "max": 0.05}
    if case["read"] == "logits":
        return {"rel": 2e-2, "max": 0.15} if case["model"] == "27b" else {"rel": 1e-2, "max": 0.08}
    return {"rel": 8e-3, "max": 0.05}


# ---- engines and sessions ------------------------------------------------------------------------
class _Server:
    """One engine with its weights and room for STATES sets of the case's sessions, KV pages filled."""

    def __init__(self, case):
        g = _geometry(case)
        self.free = list(range(STATES))
        if "pass_rows" in case:
            self.engine = S.Engine(g, S.EngineConfig(max_slots=1, max_rows=max(64, case["pass_rows"]), kv_pages=4, max_context=1024))
            self.engine.synthesize_q4(WEIGHT_SEED)
            self.own = self._own_tensors(g)
            return
        contexts = _contexts(case)
        ends = contexts + ([case["fed"] + case["prompt"]] if case["prompt"] else [])
        rows = case["sessions"] * case["block"] + case["prompt"]
        pages = sum(-(-(e + TURNS * case["block"]) // PAGE) + 1 for e in ends)
        self.per_state = len(ends)
        self.engine = S.Engine(g, S.EngineConfig(max_slots=STATES * len(ends), max_rows=max(64, rows), kv_pages=STATES * pages,
                                                 max_context=max(ends) + TURNS * case["block"] + PAGE))
        synthetic.load_vectors(self.engine, WEIGHT_SEED)
        if case["weights"] == "mlx4":
            self.engine.synthesize_q4(WEIGHT_SEED)
        else:
            self.engine.synthesize_gguf(WEIGHT_SEED, GGUF[case["weights"]], "Q6_K")
        self.held = contexts + ([case["fed"]] if case["prompt"] else [])      # tokens in front of a state's first step
        for state in range(STATES):
            self.open(state)
            for slot in self.slots(state):
                self.engine.debug_fill_kv(slot)

    def slots(self, state):
        return range(state * self.per_state, (state + 1) * self.per_state)

    def open(self, state):
        """Sessions of a state with their pages and an empty recurrent state (a page goes back to the place it came from)."""
        for slot in reversed(self.slots(state)):
            self.engine.truncate(slot, 0)
        for slot in self.slots(state):
            self.engine.reset_slot(slot)
        rows = [S.EngineRow(slot, 1000, held - 1, False) for slot, held in zip(self.slots(state), self.held) if held]
        if rows:
            self.engine.step(rows)

    def _own_tensors(self, g):
        rng = np.random.default_rng(WEIGHT_SEED)

        def q4(rows, inner):
            packed = rng.integers(0, 1 << 32, (rows, inner // 8), np.uint32)
            scales = synthetic.to_bf16(rng.uniform(0.004, 0.008, (rows, inner // 64)).astype(np.float32))
            biases = synthetic.to_bf16(-7.5 * (scales.astype(np.uint32) << 16).view(np.float32))
            return self.engine.tensor_q4(packed, scales, biases)

        def vector():
            return self.engine.tensor_vector(synthetic.to_bf16((1.0 + 0.02 * rng.standard_normal(g.hidden)).astype(np.float32)))
        layers = [dict(norm=vector(), q=q4(DRAFT_ATTENTION, g.hidden), o=q4(g.hidden, DRAFT_ATTENTION), post=vector(), gate=q4(g.inter, g.hidden),
                       up=q4(g.inter, g.hidden), down=q4(g.hidden, g.inter)) for _ in range(DRAFT_LAYERS)]
        return layers, vector()


class _State:
    def __init__(self, server, index):
        self.server, self.index, self.engine = server, index, server.engine

    def __del__(self):
        self.server.free.append(self.index)
        self.server.free.sort()


_latest = {}


def _server(case):
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    server = _latest.get(key)
    if server is None or not server.free:
        _latest.clear()           # an engine nobody holds is closed before the next is built
        server = None
        server = _latest[key] = _Server(case)
    return server


def prepare(case, seed):
    server = _server(case)
    state = _State(server, server.free.pop(0))
    rng = np.random.default_rng(seed)
    g = _geometry(case)
    if "pass_rows" in case:
        rows = case["pass_rows"]

        def buffer(width):
            return torch.empty((rows, width), device="cuda")
        state.rows, state.g = rows, g
        state.tokens = torch.from_numpy(rng.integers(0, g.vocab, rows).astype(np.uint32)).cuda()
        state.h, state.x, state.a, state.act, state.scratch, state.logits = (buffer(n) for n in (g.hidden, g.hidden, DRAFT_ATTENTION, g.inter, g.inter, g.vocab))
        torch.cuda.synchronize()
        return state
    server.open(state.index)
    slots = list(server.slots(state.index))
    for n, slot in enumerate(slots):
        server.engine.debug_fill_state(slot, (seed * 1000003 + n * 7919 - slot) % (1 << 64))
    # The rows of each turn, and how many of a session's verify rows its acceptance keeps.
    block, verify = case["block"], case["block"] > 1
    position = _contexts(case)
    state.sessions, state.block, state.verify = slots[:case["sessions"]], block, verify
    state.prompt = slots[-1] if case["prompt"] else None
    state.fresh = case["prompt"] > 0 and case["fed"] == 0
    state.read, state.limit = case["read"], min(248077, g.vocab)
    state.turns, state.turn = [], 0
    last = case["prompt"] - 1 if state.fresh or case["read"] == "logits" else -1
    prompt = [S.EngineRow(state.prompt, int(t), case["fed"] + i, i == last) for i, t in enumerate(rng.integers(0, state.limit, case["prompt"]))]
    for _ in range(TURNS):
        rows = [S.EngineRow(slot, int(rng.integers(0, state.limit)), position[s] + i, True, verify) for s, slot in enumerate(state.sessions) for i in range(block)]
        kept = [int(rng.integers(1, block + 1)) for _ in state.sessions]
        position = [p + k for p, k in zip(position, kept)]
        state.turns.append((rows + prompt, [(slot, k, p) for slot, k, p in zip(state.sessions, kept, position)]))
    return state


def run(state):
    if hasattr(state, "tokens"):
        return _run_own(state)
    engine = state.engine
    rows, accepted = state.turns[state.turn]
    state.turn = (state.turn + 1) % TURNS
    if state.fresh:
        engine.reset_slot(state.prompt)          # a new session
    engine.step(rows)
    # What the sampler reads: a single row's logits, or the twenty largest of every row. (The ids of nearly equal logits change places with
    # the order of 32-bit sums; the values are the result.)
    out = engine.logits(0) if state.read == "logits" else engine.topk(20, state.limit)[1]
    if state.verify:
        for slot, kept, tokens in accepted:
            engine.accept_verify(slot, kept, tokens)
    return out


def _run_own(state):
    e, g, n = state.engine, state.g, state.rows
    layers, final = state.server.own
    h, x, a, act, scratch, logits = (t.data_ptr() for t in (state.h, state.x, state.a, state.act, state.scratch, state.logits))
    e.pass_begin()
    e.pass_embed(state.tokens.data_ptr(), n, h)
    for w in layers:
        e.pass_norm(h, w["norm"], n, g.hidden, x)
        e.pass_gemm(w["q"], x, n, a)
        e.pass_gemm(w["o"], a, n, h, h)
        e.pass_norm(h, w["post"], n, g.hidden, x)
        e.pass_mlp_in(w["gate"], w["up"], x, n, act, scratch)
        e.pass_gemm(w["down"], act, n, h, h)
    e.pass_norm(h, final, n, g.hidden, x)
    e.pass_gemm_head(x, n, logits)
    e.pass_wait()
    return {"hidden": state.h, "logits": state.logits}
