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
