"""Tensor parallelism on two GPUs (one process per GPU, NCCL all-reduce after the attention output and the ffn
down projections): a reduced-width dense-Qwen3 model whose ffn splits unevenly (5 blocks: 3 + 2), prefill
through the batched kernels and greedy decode through the GEMV chain (replayed from a captured graph), logits
within max-abs 2e-2 / rel 1e-2 of the CPU oracle on the WHOLE model and the same tokens on both ranks.

On one GPU one rank of the group runs by itself, with a stand-in for NCCL whose all-reduce adds nothing to the rank's own
sums: its results are those of the model that the rank's shard is, which the oracle runs.  That is every kernel and every
step of the tensor-parallel path but the transfer."""
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TP_MODEL = dict(layers=3, hidden=1024, q_heads=8, kv_heads=2, head_dim=128, ffn=1280, vocab=2048, rope_base=1.0e6,
                rms_eps=1.0e-6)


def _rank(rank: int, world: int, group_id: bytes, scheme: str, out):
    sys.path.insert(0, ROOT)
    import ribn_b200
    from ribn_b200 import BatchItem, StepKind
    from tests import helpers as H
    tensors = H.make_model(TP_MODEL, seed=23, scheme=scheme)          # the same whole checkpoint on every rank
    ex = ribn_b200.QwenB200(TP_MODEL, context_tokens=128, max_sequences=2, max_batch_tokens=32, device=rank,
                            flags=ribn_b200.FLAG_KEEP_LOGITS, tp_size=world, tp_rank=rank)
    for name, (kind, rows, cols, data) in tensors.items():
        ex.load_tensor(name, kind, rows, cols, data)                   # whole tensors in; each rank keeps its shard
    kind, rows, cols, shard = ex.read_tensor("blk.1.ffn_down.weight")
    shard_shape = (rows, cols)
    ex.tp_init(group_id)
    ex.finalize()
    rng = np.random.default_rng(9)
    prompt = rng.integers(0, TP_MODEL["vocab"], size=21).tolist()
    assert ex.admit(1, 1, prompt, 12).ready
    item = BatchItem(1, StepKind.PREFILL, 0, len(prompt), 1)
    ex.prepare([item])
    done = ex.wait(ex.submit([item]))
    logits = [ex.copy_logits(0)]
    tokens = [done[0].tokens[0]]
    for step in range(10):
        item = BatchItem(1, StepKind.DECODE, len(prompt) + step, 1, 1)
        ex.prepare([item])
        done = ex.wait(ex.submit([item]))
        logits.append(ex.copy_logits(0))
        tokens.append(done[0].tokens[0])
    _, launches = ex.last_step_stats()
    ex.release(1)
    ex.close()
    out.put((rank, shard_shape, tokens, np.stack(logits), launches))


@pytest.mark.parametrize("scheme", ["q4_k_m", "q8_0"])
def test_two_rank_tensor_parallel_logits_match_the_oracle(built_library, scheme):
    import torch
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    import torch.multiprocessing as mp
    import ribn_b200
    from oracle import binding as orc
    from tests import helpers as H
    group_id = ribn_b200.tp_unique_id()
    ctx = mp.get_context("spawn")
    out = ctx.Queue()
    procs = [ctx.Process(target=_rank, args=(r, 2, group_id, scheme, out)) for r in range(2)]
    for p in procs:
        p.start()
    results = sorted((out.get(timeout=300) for _ in procs), key=lambda r: r[0])
    for p in procs:
        p.join(timeout=60)
        assert p.exitcode == 0
    (_, shape0, tokens0, logits0, launches0), (_, shape1, tokens1, logits1, _) = results
    assert shape0 == (1024, 768) and shape1 == (1024, 512)             # ffn 1280 = 5 blocks: 3 + 2
    assert tokens0 == tokens1
    assert np.array_equal(logits0.view(np.uint32), logits1.view(np.uint32))   # the replicated head sees the same bits
    # the oracle runs the whole model
    tensors = H.make_model(TP_MODEL, seed=23, scheme=scheme)
    orc.set_threads(8)
    oracle = orc.Qwen3Oracle(H.oracle_config(TP_MODEL, 128), tensors)
    seq = oracle.new_sequence()
    rng = np.random.default_rng(9)
    prompt = rng.integers(0, TP_MODEL["vocab"], size=21).tolist()
    for t in prompt[:-1]:
        seq.step(t, want_logits=False)
    want = seq.step(prompt[-1])
    worst = 0.0
    for step, token in enumerate(tokens0):
        err = np.abs(logits0[step] - want)
        worst = max(worst, float(err.max()))
        assert np.all((err < 2e-2) | (err < 1e-2 * np.abs(want))), (step, float(err.max()))
        assert token == orc.argmax(logits0[step])
        want = seq.step(token)                                         # teacher-forced with the device's token
    print(f"tp2 {scheme}: max |logit diff| {worst:.3e}, {launches0} launches per decode step")
    seq.close(); oracle.close()


ALONE = r"""
#include <string.h>
#include <stddef.h>
typedef struct { char bytes[128]; } id_t_;
static int group;
int ncclGetUniqueId(id_t_* id) { memset(id, 0, sizeof *id); return 0; }
int ncclCommInitRank(void** comm, int ranks, id_t_ id, int rank) { (void)ranks; (void)id; (void)rank; *comm = &group; return 0; }
int ncclAllReduce(const void* in, void* out, size_t n, int type, int op, void* comm, void* stream) {
    (void)n; (void)stream;
    return in == out && type == 7 && op == 0 && comm == &group ? 0 : 4;   /* in place, F32, sum: the other ranks add zeros */
}
int ncclCommDestroy(void* comm) { return comm == &group ? 0 : 4; }
const char* ncclGetErrorString(int code) { return code == 0 ? "no error" : "unexpected call"; }
"""
LENGTHS = (150, 21, 9)    # row groups of 64 + 64 + 22, one of 21, one of 9
STEPS = 4                 # then decode batches of three rows: the last replays a captured graph


def _alone(rank: int, flags: int, scheme: str, library: str, out):
    sys.path.insert(0, ROOT)
    import ribn_b200
    from ribn_b200 import BatchItem, StepKind
    from tests import helpers as H
    tensors = H.make_model(TP_MODEL, seed=23, scheme=scheme)
    ex = ribn_b200.QwenB200(TP_MODEL, context_tokens=256, max_sequences=3, max_batch_tokens=192, tp_size=2, tp_rank=rank,
                            flags=ribn_b200.FLAG_KEEP_LOGITS | flags)
    for name, (kind, rows, cols, data) in tensors.items():
        ex.load_tensor(name, kind, rows, cols, data)
    shard = {name: ex.read_tensor(name) for name in ex.tensor_names()}
    ex.tp_init(bytes(128), library)
    ex.finalize()
    rng = np.random.default_rng(9)
    prompts = [rng.integers(0, TP_MODEL["vocab"], size=n).tolist() for n in LENGTHS]
    logits, tokens = [[] for _ in prompts], [[] for _ in prompts]
    for i, prompt in enumerate(prompts):
        assert ex.admit(i + 1, i + 1, prompt, 8).ready
        item = BatchItem(i + 1, StepKind.PREFILL, 0, len(prompt), 1)
        ex.prepare([item])
        tokens[i] += ex.wait(ex.submit([item]))[0].tokens
        logits[i].append(ex.copy_logits(0))
    for step in range(STEPS):
        items = [BatchItem(i + 1, StepKind.DECODE, n + step, 1, 1) for i, n in enumerate(LENGTHS)]
        ex.prepare(items)
        for i, done in enumerate(ex.wait(ex.submit(items))):
            tokens[i] += done.tokens
            logits[i].append(ex.copy_logits(i))
    ex.close()
    out.put((shard, prompts, tokens, np.array(logits)))


@pytest.mark.parametrize("scheme", ["q4_k_m", "q8_0"])
@pytest.mark.parametrize("rank", [0, 1])
def test_one_rank_alone_matches_the_oracle_of_its_shard(built_library, tmp_path, scheme, rank):
    """Prefill in row groups and decode batches of one rank (ffn 1280 = 5 blocks: 3 or 2 of them) against the oracle, and
    with the operand cache (K-quant matrices kept as operands) bit for bit the same; once more with the integer kernels."""
    import torch.multiprocessing as mp
    import ribn_b200
    from oracle import binding as orc
    from tests import helpers as H
    gcc = shutil.which("gcc")
    if gcc is None:
        pytest.skip("no gcc")
    source, library = tmp_path / "alone.c", tmp_path / "libalone.so"
    source.write_text(ALONE)
    subprocess.run([gcc, "-shared", "-fPIC", "-o", str(library), str(source)], check=True)
    ctx = mp.get_context("spawn")
    runs = {}
    for flags in (0, ribn_b200.FLAG_OPERAND_CACHE, ribn_b200.FLAG_NO_TCGEN05):
        out = ctx.Queue()
        child = ctx.Process(target=_alone, args=(rank, flags, scheme, str(library), out))
        child.start()
        runs[flags] = out.get(timeout=240)
        child.join(timeout=60)
        assert child.exitcode == 0
    shard, prompts, _, _ = runs[0]
    model = dict(TP_MODEL, q_heads=4, kv_heads=1, ffn=(3, 2)[rank] * 256)
    orc.set_threads(8)
    oracle = orc.Qwen3Oracle(H.oracle_config(model, 256), shard)
    for flags, (_, _, tokens, logits) in runs.items():
        for i, prompt in enumerate(prompts):
            seq = oracle.new_sequence()
            for t in prompt[:-1]:
                seq.step(t, want_logits=False)
            feed = prompt[-1]
            for got, token in zip(logits[i], tokens[i]):
                want = seq.step(feed)
                err = np.abs(got - want)
                assert np.all((err < 2e-2) | (err < 1e-2 * np.abs(want))), (flags, i, float(err.max()))
                assert token == orc.argmax(got)
                feed = token                                           # teacher-forced with the device's token
            seq.close()
    oracle.close()
    plain, cached = runs[0], runs[ribn_b200.FLAG_OPERAND_CACHE]
    assert plain[2] == cached[2]
    assert np.array_equal(plain[3].view(np.uint32), cached[3].view(np.uint32))
