"""The work a user of ribn_b200 has it do, as cases that can be timed and compared.

A case is one request shape on one of the models this repository is configured for: the Qwen3-8B architecture with a
Q4_K_M-style checkpoint (with and without the operand cache), Qwen3-0.6B with Q8_0, and the reduced Gemma-4 job.  The
executor with its weights is what a serving process keeps for its whole life, so one executor per model serves every
case; `prepare` admits the sequences of a case (their contexts already cached, their contents seeded) and `run` goes
through the executor's protocol, prepare -> submit -> poll, exactly as the engines in this package do.
"""
import itertools

import numpy as np

import ribn_b200
from ribn_b200 import BatchItem, StepKind

CHUNK = 2048         # prefill chunk of the serving benchmark: tokens of one prompt per step
SLOTS = 224          # concurrent sequences of a serving executor (at most 64 of them in one batch here)
TURN = 256           # output budget of a decoding request; a new request of the same shape takes its place after that
WEIGHT_SEED = 0x5EED

#: Scheduling limits and the KV arena (16-token pages) of each executor.
EXECUTORS = {
    # dense 8B, Q4_K with Q6_K for attn_v, ffn_down and the output head
    "8b": dict(model=ribn_b200.QWEN3_8B, scheme=ribn_b200.SCHEME_Q4_K_M, flags=ribn_b200.FLAG_KEEP_LOGITS, pages=16384),
    # the same model with its matrices also kept as tensor-core operands
    "8b-cache": dict(model=ribn_b200.QWEN3_8B, scheme=ribn_b200.SCHEME_Q4_K_M,
                     flags=ribn_b200.FLAG_KEEP_LOGITS | ribn_b200.FLAG_OPERAND_CACHE, pages=6144),
    # small model, every matrix Q8_0
    "0.6b": dict(model=ribn_b200.QWEN3_0_6B, scheme=ribn_b200.SCHEME_Q8_0, flags=ribn_b200.FLAG_KEEP_LOGITS, pages=12288),
}
CONTEXT = 8192 + TURN + 64
GEMMA = ribn_b200.GEMMA4_REDUCED
GEMMA_PROMPTS = (1.0, 0.43, 0.21, 0.057)    # the job's prompt lengths as shares of the longest: 300, 129, 64, 17

_executors = {}
_ids = itertools.count(1)


def executor(name):
    if name not in _executors:
        e = EXECUTORS[name]
        ex = ribn_b200.QwenB200(e["model"], context_tokens=CONTEXT, max_sequences=SLOTS, max_batch_tokens=CHUNK + 64,
                                kv_pages=e["pages"], flags=e["flags"])
        ex.init_synthetic(WEIGHT_SEED, e["scheme"])
        ex.finalize()
        _executors[name] = ex
    return _executors[name]


def gemma_model():
    if "gemma" not in _executors:
        model = ribn_b200.GemmaB200(GEMMA, max_sequences=4, max_batch_tokens=128)
        model.init_synthetic(WEIGHT_SEED)
        model.finalize()
        _executors["gemma"] = model
    return _executors["gemma"]


# ---- the cases ---------------------------------------------------------------------------------------------------
def listed():
    return [
        # one interactive user: latency of a token
        dict(name="decode 8b x1", kind="decode", model="8b", rows=1, context=1024, spread=0.0, logits=False),
        # two long conversations whose tokens are sampled on the host, which takes the logits of every step
        dict(name="decode 8b x2 long logits", kind="decode", model="8b", rows=2, context=6144, spread=0.5, logits=True),
        # a handful of users at different depths of their answers
        dict(name="decode 8b x5 ragged", kind="decode", model="8b", rows=5, context=700, spread=0.8, logits=False),
        # moderate load on a deployment that spends memory on the operand cache
        dict(name="decode 8b x16 cache", kind="decode", model="8b-cache", rows=16, context=1500, spread=0.6, logits=False),
        # full decode batch: throughput
        dict(name="decode 8b x64", kind="decode", model="8b", rows=64, context=1024, spread=0.0, logits=False),
        # time to first token of a short question, of a full chunk (the logits of its last token are read back)
        dict(name="prefill 8b 47", kind="prefill", model="8b", tokens=47, chunk=CHUNK, logits=True),
        dict(name="prefill 8b 2048", kind="prefill", model="8b", tokens=2048, chunk=CHUNK, logits=True),
        # continuous batching: a new prompt's chunk rides along with the decoding rows
        dict(name="mixed 8b 24+1023", kind="mixed", model="8b", rows=24, context=900, spread=0.7, tokens=1023),
        # the small model: latency, a moderate ragged batch, a prompt
        dict(name="decode 0.6b x1", kind="decode", model="0.6b", rows=1, context=1024, spread=0.0, logits=False),
        dict(name="decode 0.6b x32 ragged", kind="decode", model="0.6b", rows=32, context=1024, spread=0.5, logits=False),
        dict(name="prefill 0.6b 777", kind="prefill", model="0.6b", tokens=777, chunk=CHUNK, logits=True),
        # BF16 decoder: a whole greedy job, four prompts batched
        dict(name="generate gemma x4", kind="generate", model="gemma", rows=4, longest=300, output=32),
    ]


def _log(rng, low, high):
    return int(round(low * (high / low) ** rng.random()))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "decode", "prefill", "prefill", "mixed", "generate"))
    if kind == "decode":
        model = rng.choice(("8b", "8b", "8b-cache", "0.6b"))
        rows = _log(rng, 1, 32 if model == "8b-cache" else 64)
        most = {"8b": 65536, "8b-cache": 24576, "0.6b": 32768}[model]   # cached tokens of one case
        context = min(_log(rng, 96, 8192), most // rows)
        return dict(kind=kind, model=model, rows=rows, context=context, spread=round(rng.random() * 0.9, 2),
                    logits=rows <= 2 and rng.random() < 0.3)
    if kind == "prefill":
        return dict(kind=kind, model=rng.choice(("8b", "0.6b")), tokens=_log(rng, 5, 2048), chunk=rng.choice((512, CHUNK, CHUNK)),
                    logits=True)
    if kind == "mixed":
        return dict(kind=kind, model=rng.choice(("8b", "8b", "0.6b")), rows=_log(rng, 1, 48), context=_log(rng, 96, 1024),
                    spread=round(rng.random() * 0.9, 2), tokens=_log(rng, 32, 1536))
    return dict(kind=kind, model="gemma", rows=rng.randint(1, 4), longest=_log(rng, 24, 440), output=rng.randint(4, 32))


def contexts(case):
    """Cached tokens of each decoding row: spread below `context` as requests at different ages are."""
    return [max(16, round(case["context"] * (1.0 - case["spread"] * ((i * 0.6180339887498949) % 1.0)))) for i in range(case["rows"])]


def gemma_prompts(case):
    return [max(1, round(case["longest"] * share)) for share in GEMMA_PROMPTS[:case["rows"]]]


# ---- states ------------------------------------------------------------------------------------------------------
class Decoding:
    """Admitted sequences of one executor, each with a cached context and its next token pending."""

    def __init__(self, ex, lengths, seed):
        self.ex, self.lengths, self.rng = ex, lengths, np.random.default_rng(seed)
        self.sequences = [next(_ids) for _ in lengths]
        self.positions = [0] * len(lengths)
        self.left = [0] * len(lengths)
        for i in range(len(lengths)):
            self.begin(i)

    def begin(self, i):
        """A request with its context already cached takes place i of the batch."""
        vocab, n, seq = self.ex.cfg.vocab, self.lengths[i], self.sequences[i]
        self.ex.release(seq)
        if not self.ex.admit(seq, seq, self.rng.integers(0, vocab, n, dtype=np.uint32), TURN).ready:
            raise RuntimeError("the executor has no room for the case")
        self.ex.debug_set_context(seq, n, int(self.rng.integers(0, vocab)), seed=int(self.rng.integers(1, 1 << 62)))
        self.positions[i], self.left[i] = n, TURN

    def items(self):
        for i, left in enumerate(self.left):
            if left == 0:
                self.begin(i)
        return [BatchItem(s, StepKind.DECODE, p, 1, 1) for s, p in zip(self.sequences, self.positions)]

    def advance(self, done):
        for i, row in enumerate(done):
            self.positions[i] = row.prefix
            self.left[i] -= 1

    def __del__(self):
        for seq in self.sequences:
            self.ex.release(seq)


def prepare(case, seed):
    if case["kind"] == "generate":
        rng = np.random.default_rng(seed)
        return dict(case=case, model=gemma_model(), prompts=[rng.integers(0, GEMMA["vocab"], n).tolist() for n in gemma_prompts(case)])
    ex = executor(case["model"])
    state = dict(case=case, ex=ex)
    if "tokens" in case:
        state["prompt"] = np.random.default_rng([seed, 1]).integers(0, ex.cfg.vocab, case["tokens"], dtype=np.uint32)
    if "rows" in case:
        state["decoding"] = Decoding(ex, contexts(case), seed)
    return state


# ---- passes ------------------------------------------------------------------------------------------------------
def completions(done):
    """StepCompletion rows as numbers: place in the batch, prefix after the step, tokens given, token."""
    return np.array([[i, row.prefix, len(row.tokens), row.tokens[0] if row.tokens else 0] for i, row in enumerate(done)], dtype=np.int64)


def step(ex, items):
    ex.prepare(items)
    return ex.wait(ex.submit(items))


def run(state):
    return {"decode": run_decode, "prefill": run_prefill, "mixed": run_mixed, "generate": run_generate}[state["case"]["kind"]](state)


def run_decode(state):
    """One decode step of the whole batch."""
    ex, decoding = state["ex"], state["decoding"]
    done = step(ex, decoding.items())
    decoding.advance(done)
    if not state["case"]["logits"]:
        return completions(done)
    return completions(done), np.stack([ex.copy_logits(i) for i in range(len(done))])


def run_prefill(state):
    """A request from admission to its first token, in chunks, and its release."""
    ex, prompt, case = state["ex"], state["prompt"], state["case"]
    seq, n, at = next(_ids), len(state["prompt"]), 0
    if not ex.admit(seq, seq, prompt, TURN).ready:
        raise RuntimeError("the executor has no room for the case")
    while at < n:
        take = min(case["chunk"], n - at)
        done = step(ex, [BatchItem(seq, StepKind.PREFILL, at, take, int(at + take == n))])
        at += take
    logits = ex.copy_logits(0)
    ex.release(seq)
    return completions(done), logits


def run_mixed(state):
    """One step of continuous batching: the decoding rows first, then a new request's prompt as one chunk."""
    ex, decoding, prompt = state["ex"], state["decoding"], state["prompt"]
    seq = next(_ids)
    if not ex.admit(seq, seq, prompt, TURN).ready:
        raise RuntimeError("the executor has no room for the case")
    done = step(ex, decoding.items() + [BatchItem(seq, StepKind.PREFILL, 0, len(prompt), 1)])
    decoding.advance(done[:-1])
    ex.release(seq)
    return completions(done)


def run_generate(state):
    """Greedy generation of a few prompts, batched, from admission to the last token."""
    prompts, output = state["prompts"], state["case"]["output"]
    ex = ribn_b200.GemmaExecutor(state["model"])
    for seq, prompt in enumerate(prompts):
        if not ex.admit(seq, seq, prompt, output).ready:
            raise RuntimeError("the executor has no room for the case")
    tokens, at = [[] for _ in prompts], [0] * len(prompts)
    while any(len(t) < output for t in tokens):
        batch = []
        for seq, prompt in enumerate(prompts):
            if len(tokens[seq]) == output:
                continue
            if at[seq] < len(prompt):
                take = min(128 // len(prompts), len(prompt) - at[seq])
                batch.append(BatchItem(seq, StepKind.PREFILL, at[seq], take, int(at[seq] + take == len(prompt))))
            else:
                batch.append(BatchItem(seq, StepKind.DECODE, at[seq], 1, 1))
        ex.prepare(batch)
        for row in ex.poll(ex.submit(batch)):
            at[row.sequence] = row.prefix
            tokens[row.sequence].extend(row.tokens)
    ex.synchronize()
    return np.array(tokens, dtype=np.int64)


# ---- what a pass cannot do without -------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "generate":
        g = GEMMA
        qd, kd = g["heads"] * g["head_dim"], g["kv_heads"] * g["head_dim"]
        layer = g["hidden"] * (2 * qd + 2 * kd + 3 * g["ffn"] + 2 * g["ple"])
        once = g["layers"] * layer + g["vocab"] * g["hidden"] + g["hidden"] * g["layers"] * g["ple"]
        prompts, output = gemma_prompts(case), case["output"]
        fed = sum(prompts) + len(prompts) * (output - 1)
        pairs = sum((n + output) ** 2 / 2 for n in prompts)
        cached = sum(n + t for n in prompts for t in range(1, output)) + sum(prompts)
        # the prompts in one pass over the weights, then one pass for each further token
        return {"bytes": 2.0 * once * output + 2.0 * 2 * kd * g["layers"] * cached,
                "flops": 2.0 * once * fed + 4.0 * qd * g["layers"] * pairs}
    e = EXECUTORS[case["model"]]
    m = e["model"]
    qd, kd = m["q_heads"] * m["head_dim"], m["kv_heads"] * m["head_dim"]
    base, wide = (34 / 32, 34 / 32) if e["scheme"] == ribn_b200.SCHEME_Q8_0 else (144 / 256, 210 / 256)
    narrow_weights = m["hidden"] * (2 * qd + kd + 2 * m["ffn"])
    wide_weights = m["hidden"] * (kd + m["ffn"])
    head = m["hidden"] * m["vocab"]
    decoding = contexts(case) if "rows" in case else []
    prompt = case.get("tokens", 0)
    passes = -(-prompt // case["chunk"]) if case["kind"] == "prefill" else 1   # every chunk is a step over the weights
    fed, sampled = len(decoding) + prompt, len(decoding) + (1 if prompt else 0)
    cached = sum(decoding) + fed                                               # K / V rows read or written
    pairs = sum(n + 1 for n in decoding) + prompt * (prompt + 1) / 2           # query-key pairs
    bytes_ = passes * m["layers"] * (base * narrow_weights + wide * wide_weights) + wide * head + m["layers"] * cached * 2 * kd * 2
    flops = 2.0 * m["layers"] * (narrow_weights + wide_weights) * fed + 2.0 * head * sampled + m["layers"] * 4.0 * qd * pairs
    return {"bytes": bytes_ + (4.0 * m["vocab"] * sampled if case.get("logits") else 0.0), "flops": flops}


def tolerance(case):
    if case["kind"] == "generate":
        return "exact"      # BF16 rounding after every operation and sums in a fixed order: tokens are reproducible
    # F32 activations and sums over exact block integers; keys and values are stored in F16, so a last-bit difference
    # of a key can move its stored value by one part in 2048.  A token may differ where two logits tie to that accuracy.
    return {"rel": 1e-3, "max": 2e-2, "differ": 0.01}
