"""Decode steps whose logits are read back: eager at first, replayed from a captured graph later, through pinned memory up to 4 MiB."""
import numpy as np
import pytest
import torch

from oracle import hybrid as oh
from oracle import model as om

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 3])
def test_replayed_steps_return_the_logits_of_eager_ones(kge, tmp_path, B):
    cfg = om.CONFIGS["tiny-llama"]
    om.save_model_dir(tmp_path, cfg, om.make_weights(cfg, seed=0))
    ids = [np.asarray(p, dtype=np.int32) for p in om.make_prompts(cfg, B, 20, seed=7)]
    bs, per, n = 16, 4, 14

    def tables():
        return 1 + np.arange(B * per, dtype=np.int32).reshape(B, per)

    def step(llm, spans, want):
        tok = np.concatenate([np.resize(t, 64)[a:b] for t, (a, b) in zip(ids, spans)])
        pos = np.concatenate([np.arange(a, b, dtype=np.int32) for a, b in spans])
        slots = np.concatenate([tables()[r, np.arange(a, b) // bs].astype(np.int64) * bs + np.arange(a, b) % bs for r, (a, b) in enumerate(spans)])
        qsl = np.concatenate([[0], np.cumsum([b - a for a, b in spans])]).astype(np.int32)
        return llm.raw_step(tok, pos, qsl, np.asarray([b for _, b in spans], dtype=np.int32), tables(), per, slots, qsl[1:] - 1, want_logits=want)

    def run(always):
        """Logits of n decode steps; always: the first of them eleven times over."""
        llm = kge.LLM(str(tmp_path), max_model_len=64, max_num_seqs=4, max_num_batched_tokens=128, block_size=bs, num_gpu_blocks_override=B * per + 1,
                      enable_prefix_caching=False)
        step(llm, [(0, 20)] * B, False)
        out = []
        for k in range(n):
            turns = 11 if always and k == 0 else 1             # the same step again and again: eager, captured, replayed
            out += [step(llm, [(20 + k, 21 + k)] * B, True) for _ in range(turns)]
        llm.close()
        return out

    once, often = run(False), run(True)
    for tokens, logits in often[:11]:
        assert np.array_equal(tokens, once[0][0]) and np.array_equal(logits, once[0][1])
    for (t0, l0), (t1, l1) in zip(once[1:], often[11:]):       # replayed in one engine from here on, eager in the other up to the eighth
        assert np.array_equal(t0, t1) and np.array_equal(l0, l1)


def decode_llm(kge, path, B, bs=16, per=4):
    """An engine and a function that runs the same decode step of B requests again."""
    llm = kge.LLM(str(path), max_model_len=64, max_num_seqs=4, max_num_batched_tokens=128, block_size=bs, num_gpu_blocks_override=B * per + 1, enable_prefix_caching=False)
    table = 1 + np.arange(B * per, dtype=np.int32).reshape(B, per)
    at = np.arange(B + 1, dtype=np.int32)

    def step(want):
        return llm.raw_step(np.full(B, 5, dtype=np.int32), np.zeros(B, dtype=np.int32), at, np.ones(B, dtype=np.int32), table, per, table[:, 0].astype(np.int64) * bs, at[:B], want_logits=want)
    return llm, step


def test_steps_that_launch_the_same_share_a_graph(kge, tmp_path):
    cfg = om.CONFIGS["tiny-llama"]
    om.save_model_dir(tmp_path, cfg, om.make_weights(cfg, seed=0))
    llm, step = decode_llm(kge, tmp_path, 2)
    eager = step(True)
    for want in [False] * 2 + [True] * 12:
        got = step(want)
        assert llm.decode_graphs <= 1
    assert llm.decode_graphs == 1 and all(np.array_equal(a, b) for a, b in zip(eager, got))
    llm.close()


def test_layer_list_steps_with_logits_have_a_graph_of_their_own(kge, tmp_path):
    cfg = oh.make_config()
    oh.save_model_dir(str(tmp_path), cfg, oh.make_weights(cfg, seed=0))
    llm, step = decode_llm(kge, tmp_path, 2)
    for want, graphs in [(False, 0), (False, 1), (True, 1)] + [(True, 1)] * 7 + [(True, 2)] * 2 + [(False, 2)]:
        step(want)
        assert llm.decode_graphs == graphs
    llm.close()


@pytest.mark.parametrize("name,lengths", [
    ("tiny-opt", [1, 62, 63, 64, 65, 127]),                  # one to three tiles; the last key alone in its tile, at its start and at its end
    ("tiny-opt", [250]),
    ("tiny-llama", [255, 256, 318, 321, 40, 511]),           # two splits merged in a cluster, one of them empty; a last key behind the tiles of the start
    ("tiny-llama", [700, 3]),
    ("tiny-llama", [200 + (i % 17) for i in range(160)]),    # more CTAs than two an SM: three tiles under way
])
def test_keys_before_the_step_read_ahead(kge, tmp_path, name, lengths):
    """A decode step whose attention fetches the keys before each request's last while the projection still runs: eager and replayed against
    the oracle; and a step of two rows of one sequence, where a row's earlier key is written by the other, which must wait for it."""
    cfg = om.CONFIGS[name]
    w = om.make_weights(cfg, seed=0)
    om.save_model_dir(tmp_path, cfg, w)
    lengths = [min(n, 240) for n in lengths] if name == "tiny-opt" else lengths      # (its positions end at 256)
    prompts = [om.make_prompts(cfg, 1, n, seed=11 + i)[0] for i, n in enumerate(lengths)]
    ids, ref = om.OracleModel(cfg, w, torch.bfloat16, max_pos=1024).generate_greedy(prompts, 2, return_logits=True)
    bs, per, B = 16, (max(lengths) + 2 + 15) // 16, len(lengths)
    llm = kge.LLM(str(tmp_path), max_model_len=per * bs, max_num_seqs=B + 1, max_num_batched_tokens=max(256, sum(lengths)), block_size=bs,
                  num_gpu_blocks_override=B * per + 1, enable_prefix_caching=False)
    table = 1 + np.arange(B * per, dtype=np.int32).reshape(B, per)

    def step(rows, want=True):
        """rows: (request, first position, tokens)"""
        tok = np.concatenate([np.asarray(t, dtype=np.int32) for _, _, t in rows])
        pos = np.concatenate([np.arange(a, a + len(t), dtype=np.int32) for _, a, t in rows])
        slots = np.concatenate([table[r, np.arange(a, a + len(t)) // bs].astype(np.int64) * bs + np.arange(a, a + len(t)) % bs for r, a, t in rows])
        qsl = np.concatenate([[0], np.cumsum([len(t) for _, _, t in rows])]).astype(np.int32)
        return llm.raw_step(tok, pos, qsl, np.asarray([a + len(t) for _, a, t in rows], dtype=np.int32), table[[r for r, _, _ in rows]], per, slots, qsl[1:] - 1, want_logits=want)

    def close(got, want, what):
        want = want.numpy() if isinstance(want, torch.Tensor) else want
        err, scale = np.abs(got - want), np.abs(want).max()
        assert (err <= 3e-2 * scale + 1.6e-2 * np.abs(want)).all(), f"{what}: {err.max():.4g} of {scale:.3g}"

    step([(r, 0, p) for r, p in enumerate(prompts)], False)
    turns = [step([(r, len(p), [ids[r][0]]) for r, p in enumerate(prompts)])[1] for _ in range(11)]
    close(turns[0], ref[1], "decode step")
    for t in turns[1:]:                                       # eager, captured, replayed
        assert np.array_equal(t, turns[0])
    long = int(np.argmax(lengths))
    n = lengths[long]
    step([(long, 0, [7] * (n + 1))], False)                   # other keys where the two rows' will be
    step([(long, 0, prompts[long][:n - 1])], False) if n > 1 else None
    both = step([(long, n - 1, prompts[long][n - 1:]), (long, n, [ids[long][0]])])[1]
    close(both, np.stack([ref[0][long], ref[1][long]]), "two rows of one sequence")
    llm.close()


@pytest.mark.parametrize("block_size,graphs", [(16, 2), (32, 1)])
def test_steps_whose_launches_are_alike_share_a_graph(kge, tmp_path, block_size, graphs):
    """Steps of two requests with blocks of their own, and steps in which one row writes a block that the other reads: attention over blocks of
    16 tokens reads ahead in the first kind only, over blocks of 32 in neither."""
    cfg = om.CONFIGS["tiny-llama"]
    om.save_model_dir(tmp_path, cfg, om.make_weights(cfg, seed=0))
    llm = kge.LLM(str(tmp_path), max_model_len=128, max_num_seqs=2, max_num_batched_tokens=128, block_size=block_size, num_gpu_blocks_override=2 * 128 // block_size + 1,
                  enable_prefix_caching=False)
    per = 128 // block_size
    table = 1 + np.arange(2 * per, dtype=np.int32).reshape(2, per)
    for rows in ([(0, 40), (1, 40)], [(0, 40), (0, 41)]):
        for _ in range(12):
            pos = np.asarray([n for _, n in rows], dtype=np.int32)
            slots = np.asarray([table[r, n // block_size] * block_size + n % block_size for r, n in rows], dtype=np.int64)
            llm.raw_step(np.asarray([5, 6], dtype=np.int32), pos, np.arange(3, dtype=np.int32), pos + 1, table[[r for r, _ in rows]], per, slots, np.arange(2, dtype=np.int32))
    assert llm.decode_graphs == graphs
    llm.close()
