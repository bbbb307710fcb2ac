"""Layer-list models (the Safupel design) in the engine against the plain float64 oracle (oracle/hybrid.py): every
mechanism alone, whole prompts against pieces and token-by-token decoding, mixed batches, reused pages and state slots,
chunk edges and far keys with peaked scores, the first tokens, long decoding, odd sizes, and greedy generation through
the scheduler.  float32 engines give the sharp comparison; bfloat16 ones are held to a rounding-sized bound."""
import numpy as np
import pytest
import torch

from oracle import hybrid as oh

pytestmark = pytest.mark.gpu

FULL = dict(layers=("parallel", "rglru", "parallel", "rglru"), mlps=("moe", "dense", "dense", "moe-noshared"))


def make_engine(kge, tmp_path, cfg, W, dtype="float32", tokens=512, bs=16, seqs=4, name="m", batched=0):
    d = str(tmp_path / name)
    oh.save_model_dir(d, cfg, W)
    nb = (tokens + bs - 1) // bs
    return kge.LLM(d, dtype=dtype, block_size=bs, num_gpu_blocks_override=nb + 1, max_model_len=nb * bs + 1, max_num_seqs=seqs,
                   max_num_batched_tokens=batched or nb * bs, enable_prefix_caching=False)


def run_pieces(llm, rid, tokens, pieces):
    """Feed `tokens` in steps of the given sizes, asking for every position's logits."""
    out, at = [], 0
    for n in pieces:
        llm.trace_add(rid, tokens[at:at + n])
        out.append(llm.trace_step([(rid, n, list(range(n)))]))
        at += n
    assert at == len(tokens)
    return np.concatenate(out)


def check(got, want, dtype, what=""):
    want = want.numpy() if isinstance(want, torch.Tensor) else want
    scale = np.sqrt((want ** 2).mean())
    err = np.sqrt(((got - want) ** 2).mean(-1)) / scale
    lim = 2e-4 if dtype == "float32" else 4e-2
    assert err.max() < lim, f"{what}: worst row {err.argmax()} is {err.max():.3g} of the logits' size (limit {lim})"


def prompt(cfg, n, seed=1):
    return torch.randint(0, cfg["vocab"], (n,), generator=torch.Generator().manual_seed(seed)).tolist()


ALONE = {
    "rglru": dict(layers=("rglru",), mlps=(None,)),
    "attention": dict(layers=("parallel",), mlps=(None,), right_scale=0.0, chunk=16),
    "mlstm": dict(layers=("parallel",), mlps=(None,), left_scale=0.0),
    "moe": dict(layers=("parallel",), mlps=("moe",), left_scale=0.0, right_scale=0.0),
    "moe-noshared": dict(layers=("parallel",), mlps=("moe-noshared",), left_scale=0.0, right_scale=0.0, top=3),
    "dense": dict(layers=("parallel",), mlps=("dense",), left_scale=0.0, right_scale=0.0),
}


@pytest.mark.parametrize("mech", sorted(ALONE))
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_mechanism_alone(kge, tmp_path, mech, dtype):
    cfg = oh.make_config(**ALONE[mech])
    W = oh.make_weights(cfg, seed=3)
    toks = prompt(cfg, 45)
    llm = make_engine(kge, tmp_path, cfg, W, dtype)
    got = run_pieces(llm, 0, toks, [45])
    llm.close()
    check(got, oh.forward(cfg, W, toks), dtype, mech)


@pytest.mark.parametrize("experts,m_heads", [(5, 3), (17, 4), (32, 9)])
def test_narrow_projections(kge, tmp_path, experts, m_heads):
    """Gates and routers of up to 8, 16 and 32 columns over rows long enough (width 264) for the kernel that splits K over warps,
    with a K that ends inside a piece; one row, a ragged last row tile, several tiles."""
    cfg = oh.make_config(width=264, layers=("parallel", "rglru"), mlps=("moe", "moe"), experts=experts, m_heads=m_heads, top=experts)
    W = oh.make_weights(cfg, seed=17)
    toks = prompt(cfg, 75)
    want = oh.forward(cfg, W, toks)
    llm = make_engine(kge, tmp_path, cfg, W, "bfloat16")
    for rid, pieces in enumerate([[75], [16, 1, 17, 41]]):
        check(run_pieces(llm, rid, toks, pieces), want, "bfloat16", f"pieces {pieces}")
        llm.trace_end(rid)
    llm.close()


@pytest.mark.parametrize("rows", [4096, 4097])
def test_narrow_projections_of_long_steps(kge, tmp_path, rows):
    """A router of 20 columns over a width of 264: the last row count of the kernel above and the first of the general ones."""
    cfg = oh.make_config(width=264, layers=("rglru",), mlps=("moe",), experts=20, top=20)
    W = oh.make_weights(cfg, seed=29)
    toks = prompt(cfg, rows)
    llm = make_engine(kge, tmp_path, cfg, W, "bfloat16", tokens=rows + 16)
    at = [0, 17, 2048, rows - 2, rows - 1]
    llm.trace_add(0, toks)
    check(llm.trace_step([(0, rows, at)]), oh.forward(cfg, W, toks)[at], "bfloat16", f"{rows} rows")
    llm.close()


@pytest.mark.parametrize("width,taps,pieces", [(1032, 4, [1, 2, 3, 4, 5, 60]), (1024, 2, [75]), (2048, 7, [33, 1, 41]), (72, 4, [1030, 1, 9]), (72, 4, [1024, 16])])
def test_convolution_in_pieces_of_eight_channels(kge, tmp_path, width, taps, pieces):
    """bfloat16 rows by eight channels of four tokens: widths with a last block of one thread, of all, of two blocks, tails carried over
    pieces shorter than the taps; narrow rows with enough tokens for it, and one token too few."""
    cfg = oh.make_config(layers=("rglru",), mlps=(None,), r_width=width, r_blocks=8, r_conv=taps)
    W = oh.make_weights(cfg, seed=31)
    toks = prompt(cfg, sum(pieces))
    llm = make_engine(kge, tmp_path, cfg, W, "bfloat16", tokens=max(sum(pieces), 512) + 16)
    check(run_pieces(llm, 0, toks, pieces), oh.forward(cfg, W, toks), "bfloat16", f"pieces {pieces}")
    llm.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width", [33, 36, 66, 128])
def test_gated_recurrence_by_width(kge, tmp_path, width, dtype):
    """The recurrence of prompt steps in stages of 16 tokens, of 8 where most requests bring one: widths that are copied number by
    number and in fours, a last block of 32 channels with one of them and with all, pieces around a stage's edge, more stages than
    the ring has, one token; then single tokens beside pieces."""
    cfg = oh.make_config(layers=("rglru",), mlps=(None,), r_width=width, r_blocks=3 if width % 3 == 0 else 2)
    W = oh.make_weights(cfg, seed=23)
    toks = prompt(cfg, 340)
    want = oh.forward(cfg, W, toks)
    llm = make_engine(kge, tmp_path, cfg, W, dtype, tokens=1024, seqs=16)
    for rid, pieces in enumerate([[340], [15, 16, 17, 33, 1, 2, 64, 65, 127]]):
        check(run_pieces(llm, rid, toks, pieces), want, dtype, f"pieces {pieces}")
        llm.trace_end(rid)
    n = 12
    for rid in range(n):
        llm.trace_add(rid, toks[:2 + rid])
        llm.trace_step([(rid, 2 + rid, [])])
    for turn, long in enumerate((7, 8, 9, 25)):
        for rid in range(n):
            llm.trace_add(rid, [toks[2 + rid + turn]])
        llm.trace_add(n + turn, toks[:long])
        got = llm.trace_step([(rid, 1, [0]) for rid in range(n)] + [(n + turn, long, list(range(long)))])
        check(got, want[[2 + rid + turn for rid in range(n)] + list(range(long))], dtype, f"beside {long} rows")
    llm.close()


@pytest.mark.parametrize("m_dim,m_vdim", [(16, 8), (64, 40), (128, 256)])
def test_matrix_memory_in_chunks_of_64(kge, tmp_path, m_dim, m_vdim):
    """bfloat16 head sizes that take the tensor-core chunks: pieces that end before, at and behind a chunk's edge, single tokens
    among them, with and without a state from before; then many single-token requests beside a prompt, whose column blocks start
    at different times and must all read the normaliser as it was.  A row whose normaliser cancels amplifies the rounding of the
    bfloat16 projections; it does so alike when the same tokens come one by one (fp32 recurrence), so a row may be off by three
    times what it is there, beside the bound of rows that do not cancel."""
    cfg = oh.make_config(layers=("parallel",), mlps=(None,), left_scale=0.0, m_dim=m_dim, m_vdim=m_vdim)
    W = oh.make_weights(cfg, seed=13)
    toks = prompt(cfg, 150)
    want = oh.forward(cfg, W, toks).numpy()
    llm = make_engine(kge, tmp_path, cfg, W, "bfloat16", tokens=2048, seqs=48)
    size = np.sqrt((want ** 2).mean())

    def off(got, rows):
        return np.sqrt(((got - want[rows]) ** 2).mean(-1)) / size
    singly = off(run_pieces(llm, 99, toks, [1] * 150), slice(None))
    llm.trace_end(99)
    assert np.median(singly) < 1e-2

    def close(got, rows, what):
        assert (off(got, rows) <= 3 * singly[rows] + 2e-2).all(), (what, off(got, rows).max())
    for rid, pieces in enumerate([[150], [63, 64, 23], [64, 65, 1, 20], [1, 2, 127, 20]]):
        close(run_pieces(llm, rid, toks, pieces), slice(None), pieces)
        llm.trace_end(rid)
    n = 40
    for rid in range(n):
        llm.trace_add(rid, toks[:3 + rid % 5])
        llm.trace_step([(rid, 3 + rid % 5, [])])
    for rid in range(n):
        llm.trace_add(rid, [toks[3 + rid % 5]])
    llm.trace_add(n, toks[:70])
    got = llm.trace_step([(rid, 1, [0]) for rid in range(n)] + [(n, 70, [69])])
    close(got, [3 + rid % 5 for rid in range(n)] + [69], "mixed step")
    llm.close()


@pytest.mark.parametrize("dtype,m_vdim,long", [("float32", 256, 70), ("bfloat16", 256, 70), ("bfloat16", 256, 240), ("bfloat16", 264, 70)])
def test_matrix_memory_of_more_requests_than_fit_at_once(kge, tmp_path, dtype, m_vdim, long):
    """A head's value columns are spread over blocks that all read its normaliser, and with 70 requests not all blocks of a launch
    start together: a pure decode step, then a step of single tokens beside a prompt (32 tokens at a time in fp32; 64 on
    tensor cores where the prompt is long: 240), then another decode step on the state that it left."""
    cfg = oh.make_config(layers=("parallel",), mlps=(None,), left_scale=0.0, m_heads=4, m_dim=128, m_vdim=m_vdim)
    W = oh.make_weights(cfg, seed=19)
    toks = prompt(cfg, long + 10)
    want = oh.forward(cfg, W, toks).numpy()
    n = 70
    llm = make_engine(kge, tmp_path, cfg, W, dtype, tokens=2560, seqs=n + 1)
    size = np.sqrt((want ** 2).mean())
    singly = np.sqrt(((run_pieces(llm, 999, toks, [1] * len(toks)) - want) ** 2).mean(-1)) / size
    llm.trace_end(999)

    def close(got, rows, what):
        off = np.sqrt(((got - want[rows]) ** 2).mean(-1)) / size
        # rows whose normaliser cancels are off by what they are when their tokens come one by one, beside the usual bound
        assert (off <= 3 * singly[rows] + (2e-4 if dtype == "float32" else 2e-2)).all(), (what, off.max(), int(off.argmax()))
    have = [3 + rid % 5 for rid in range(n)]
    for rid in range(n):
        llm.trace_add(rid, toks[:have[rid]])
        llm.trace_step([(rid, have[rid], [])])
    for turn in ("decode", "mixed", "decode again"):
        for rid in range(n):
            llm.trace_add(rid, [toks[have[rid]]])
        rows = [(rid, 1, [0]) for rid in range(n)]
        if turn == "mixed":
            llm.trace_add(n, toks[:long])
            rows.append((n, long, [long - 1]))
        close(llm.trace_step(rows), have + ([long - 1] if turn == "mixed" else []), turn)
        have = [h + 1 for h in have]
    llm.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_prefill_decode_and_pieces_agree_with_the_oracle(kge, tmp_path, dtype):
    cfg = oh.make_config(**FULL, chunk=24)
    W = oh.make_weights(cfg, seed=5)
    toks = prompt(cfg, 75)
    want = oh.forward(cfg, W, toks)
    llm = make_engine(kge, tmp_path, cfg, W, dtype)
    for rid, pieces in enumerate([[75], [30] + [1] * 45, [1] * 75, [2, 3, 17, 2, 31, 5, 2, 2, 9, 2], [23, 2, 24, 26], [47, 2, 1, 1, 24]]):
        got = run_pieces(llm, rid, toks, pieces)
        llm.trace_end(rid)
        check(got, want, dtype, f"pieces {pieces[:6]}")
    llm.close()


def test_layer_outputs_match(kge, tmp_path):
    cfg = oh.make_config(**FULL)
    W = oh.make_weights(cfg, seed=6)
    toks = prompt(cfg, 33)
    _, layers = oh.forward(cfg, W, toks, return_layers=True)
    llm = make_engine(kge, tmp_path, cfg, W, "float32")
    buf = np.zeros((4, 33, cfg["width"]), dtype=np.float32)
    llm.set_layer_dump(buf)
    run_pieces(llm, 0, toks, [33])
    llm.set_layer_dump(None)
    llm.close()
    for i, x in enumerate(layers):
        assert np.abs(buf[i] - x.numpy()).max() < 2e-4 * float(x.abs().max()), f"layer {i}"


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_mixed_batches_of_unequal_requests(kge, tmp_path, dtype):
    cfg = oh.make_config(**FULL, chunk=20)
    W = oh.make_weights(cfg, seed=7)
    P = {0: prompt(cfg, 61, 10), 1: prompt(cfg, 9, 11), 2: prompt(cfg, 40, 12), 3: prompt(cfg, 1, 13)}
    want = {r: oh.forward(cfg, W, t).numpy() for r, t in P.items()}
    # each step: (request, number of tokens); prompt pieces beside single tokens, requests pausing and resuming
    steps = [[(0, 19), (1, 1), (3, 1)], [(1, 1), (2, 2), (0, 2)], [(0, 20), (1, 1)], [(2, 18), (1, 1), (0, 1)], [(1, 5), (2, 1)],
             [(0, 1), (2, 1)], [(0, 18), (2, 18)]]
    llm = make_engine(kge, tmp_path, cfg, W, dtype)
    at = {r: 0 for r in P}
    got = {r: [] for r in P}
    for st in steps:
        entries = []
        for r, n in st:
            llm.trace_add(r, P[r][at[r]:at[r] + n])
            entries.append((r, n, list(range(n))))
        lg = llm.trace_step(entries)
        k = 0
        for r, n in st:
            got[r].append(lg[k:k + n])
            k += n
            at[r] += n
    llm.close()
    for r in P:
        assert at[r] == len(P[r])
        check(np.concatenate(got[r]), want[r], dtype, f"request {r}")


def test_pages_and_slots_are_used_again(kge, tmp_path):
    """Two slots and a pool of 96 tokens: five requests pass through, each starting in a slot and in pages that an
    earlier request filled; each must come out as if it had run alone."""
    cfg = oh.make_config(**FULL, chunk=24)
    W = oh.make_weights(cfg, seed=8)
    llm = make_engine(kge, tmp_path, cfg, W, "float32", tokens=96, bs=16, seqs=2)
    P = {r: prompt(cfg, n, 20 + r) for r, n in enumerate([40, 33, 47, 18, 30])}
    want = {r: oh.forward(cfg, W, t).numpy() for r, t in P.items()}
    got = {}
    got[0] = run_pieces(llm, 0, P[0], [40])
    llm.trace_add(1, P[1][:20])
    a = llm.trace_step([(1, 20, list(range(20)))])
    with pytest.raises(kge.KgeError):                     # no third slot
        llm.trace_add(2, P[2])
        llm.trace_step([(2, 5, [])])
    llm.trace_end(2)
    llm.trace_end(0)
    llm.trace_add(2, P[2])
    llm.trace_add(1, P[1][20:])
    b = llm.trace_step([(2, 30, list(range(30))), (1, 13, list(range(13)))])
    got[1] = np.concatenate([a, b[30:]])
    c = llm.trace_step([(2, 17, list(range(17)))])
    got[2] = np.concatenate([b[:30], c])
    llm.trace_end(1)
    got[3] = run_pieces(llm, 3, P[3], [2, 16])
    llm.trace_end(2)
    llm.trace_end(3)
    got[4] = run_pieces(llm, 4, P[4], [29, 1])
    llm.close()
    for r in P:
        check(got[r], want[r], "float32", f"request {r}")


@pytest.mark.parametrize("dims", [(12, 20), (32, 40)])       # the per-row kernel; the tensor-core kernel (bfloat16, key size a multiple of 16)
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_chunk_edges_with_peaked_scores(kge, tmp_path, dtype, dims):
    """Attention alone, scores large enough that single keys carry most of the weight: a key that is wrongly seen or
    missed at a chunk's edge, or a page border that is misread, moves the logits far beyond rounding."""
    cfg = oh.make_config(layers=("parallel",), mlps=(None,), right_scale=0.0, chunk=21, scale=1.6 * (12 / dims[0]) ** 0.5, heads=4, kv_heads=1,
                         dim=dims[0], vdim=dims[1])
    W = oh.make_weights(cfg, seed=9)
    toks = prompt(cfg, 70, 30)
    want = oh.forward(cfg, W, toks)
    ref = want.numpy()
    assert np.abs(ref[21] - oh.forward(dict(cfg, layers=[dict(cfg["layers"][0], mixer=dict(cfg["layers"][0]["mixer"], left=dict(
        cfg["layers"][0]["mixer"]["left"], mask={"size": 22})))]), W, toks).numpy()[21]).max() > 0.05      # the edge matters in this setup
    llm = make_engine(kge, tmp_path, cfg, W, dtype, bs=16)
    check(run_pieces(llm, 0, toks, [70]), want, dtype, "whole")
    check(run_pieces(llm, 1, toks, [19] + [1] * 30 + [21]), want, dtype, "decoding over two edges")
    check(run_pieces(llm, 2, toks, [20, 2, 20, 2, 26]), want, dtype, "pieces that straddle the edges")
    llm.close()


def test_far_keys_tensor_core_kernel(kge, tmp_path):
    """bfloat16, 32-wide keys and 56-wide values, several key tiles per warp and a chunk edge in the middle of the prompt;
    grouped heads."""
    cfg = oh.make_config(layers=("parallel",), mlps=(None,), right_scale=0.0, chunk=200, scale=0.7, heads=6, kv_heads=2, dim=32, vdim=56)
    W = oh.make_weights(cfg, seed=15)
    toks = prompt(cfg, 290, 32)
    want = oh.forward(cfg, W, toks)
    llm = make_engine(kge, tmp_path, cfg, W, "bfloat16", bs=64)
    got = np.concatenate([run_pieces(llm, 0, toks[:150], [150]), run_pieces(llm, 0, toks[150:260], [3, 45, 2, 60]), run_pieces(llm, 0, toks[260:], [1] * 30)])
    llm.close()
    check(got, want, "bfloat16")


def test_far_keys_among_hundreds(kge, tmp_path):
    """One long chunk: the second head's distance penalty is weak, so keys hundreds of positions back keep real weight."""
    cfg = oh.make_config(layers=("parallel",), mlps=(None,), right_scale=0.0, chunk=400, scale=1.2, heads=2, kv_heads=2, dim=8, vdim=8)
    W = oh.make_weights(cfg, seed=10)
    toks = prompt(cfg, 330, 31)
    want = oh.forward(cfg, W, toks)
    llm = make_engine(kge, tmp_path, cfg, W, "float32", bs=64)
    got = np.concatenate([run_pieces(llm, 0, toks[:300], [300]), run_pieces(llm, 0, toks[300:], [1] * 30)])
    llm.close()
    check(got, want, "float32")


def test_experts_with_many_routed_rows(kge, tmp_path):
    """A prompt long enough that the routed rows are made contiguous per expert and run as one tensor-core GEMM pair per
    expert (bfloat16; expert width a multiple of 64); the same prompt fed in short pieces takes the grouped kernel."""
    cfg = oh.make_config(layers=("rglru",), mlps=("moe",), experts=6, top=2, expert_ff=64, shared_ff=64, r_width=64, r_blocks=2)
    W = oh.make_weights(cfg, seed=16)
    toks = prompt(cfg, 300, 33)
    want = oh.forward(cfg, W, toks)
    llm = make_engine(kge, tmp_path, cfg, W, "bfloat16", bs=64)
    check(run_pieces(llm, 0, toks, [300]), want, "bfloat16", "one step")
    llm.trace_end(0)
    check(run_pieces(llm, 1, toks, [280, 7, 13]), want, "bfloat16", "pieces")
    llm.close()


def test_first_tokens(kge, tmp_path):
    cfg = oh.make_config(**FULL)
    W = oh.make_weights(cfg, seed=11)
    llm = make_engine(kge, tmp_path, cfg, W, "float32")
    for rid, n in enumerate([1, 2, 3, 5]):
        toks = prompt(cfg, n, 40 + n)
        got = run_pieces(llm, rid, toks, [n])
        llm.trace_end(rid)
        check(got, oh.forward(cfg, W, toks), "float32", f"{n} tokens")
    llm.close()


def test_long_decoding(kge, tmp_path):
    cfg = oh.make_config(**FULL, chunk=32)
    W = oh.make_weights(cfg, seed=12)
    toks = prompt(cfg, 200, 50)
    llm = make_engine(kge, tmp_path, cfg, W, "float32")
    got = run_pieces(llm, 0, toks, [4] + [1] * 196)
    llm.close()
    check(got, oh.forward(cfg, W, toks), "float32")


@pytest.mark.parametrize("sizes", [
    dict(heads=3, kv_heads=3, dim=16, vdim=16, m_heads=1, m_dim=16, m_vdim=16, r_blocks=1, r_conv=1, experts=2, top=1, chunk=7),
    dict(vocab=53, width=40, heads=6, kv_heads=2, dim=10, vdim=14, m_heads=2, m_dim=6, m_vdim=36, r_width=60, r_blocks=5, r_conv=7,
         ff=50, experts=9, top=4, expert_ff=11, shared_ff=13, chunk=64, left_scale=0.7, right_scale=1.3, gate_cap=4.0, logit_scale=2.0, eps=1e-3),
])
def test_other_sizes(kge, tmp_path, sizes):
    cfg = oh.make_config(**FULL, **sizes)
    W = oh.make_weights(cfg, seed=13)
    toks = prompt(cfg, 50, 60)
    want = oh.forward(cfg, W, toks)
    llm = make_engine(kge, tmp_path, cfg, W, "float32")
    check(run_pieces(llm, 0, toks, [50]), want, "float32", "whole")
    check(run_pieces(llm, 1, toks, [13, 2, 1, 1, 1, 32]), want, "float32", "pieces")
    llm.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_greedy_generation_through_the_scheduler(kge, tmp_path, dtype):
    """LLM.generate: the continuous-batching scheduler cuts the prompts into 16-token steps, admits the third request
    when a slot frees up, and samples greedily."""
    cfg = oh.make_config(**FULL, chunk=24)
    W = oh.make_weights(cfg, seed=14)
    prompts = [prompt(cfg, n, 70 + n) for n in (37, 5, 21)]
    llm = make_engine(kge, tmp_path, cfg, W, dtype, seqs=2, batched=16)
    outs = llm.generate(prompts, kge.SamplingParams(max_tokens=12, temperature=0.0, ignore_eos=True))
    assert llm.kernel_launches > 0
    llm.close()
    for p, o in zip(prompts, outs):
        got = o.outputs[0].token_ids
        assert len(got) == 12
        toks = list(p)
        for k, g in enumerate(got):       # teacher-forced: a different choice must be a near-tie of the oracle
            lg = oh.forward(cfg, W, toks)[-1]
            best = int(torch.argmax(lg))
            if g != best:
                gap = float(lg[best] - lg[g])
                assert gap < (1e-3 if dtype == "float32" else 0.15), f"token {k}: chose {g}, oracle {best} leads by {gap}"
            toks.append(g)


def test_trace_runner_command_line(kge, tmp_path):
    """bin/trace_run end to end: JSON steps on stdin (pieces of two requests side by side, a request that ends and one
    that takes its slot and pages), float32 files out, 'done <step>' lines; and exit code 3 for a family without float32."""
    import json
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    cfg = oh.make_config(layers=("rglru", "parallel", "parallel"), mlps=("dense", "moe", None), chunk=24)
    W = oh.make_weights(cfg, seed=17)
    d = str(tmp_path / "m")
    oh.save_model_dir(d, cfg, W)
    P = {"a": prompt(cfg, 50, 80), "b": prompt(cfg, 31, 81), "c": prompt(cfg, 40, 82)}
    want = {k: oh.forward(cfg, W, v).numpy() for k, v in P.items()}
    steps = [
        {"step": 0, "entries": [{"id": "a", "tokens": P["a"][:30], "want": [0, 29]}, {"id": "b", "tokens": P["b"][:2], "want": []}], "end": []},
        {"step": 1, "entries": [{"id": "b", "tokens": P["b"][2:], "want": [0, 28]}, {"id": "a", "tokens": P["a"][30:31], "want": [0]}], "end": ["b"]},
        {"step": 2, "entries": [{"id": "a", "tokens": P["a"][31:], "want": [18]}, {"id": "c", "tokens": P["c"], "want": [39, 5]}], "end": ["a", "c"]},
    ]
    rows = {0: [("a", 0), ("a", 29)], 1: [("b", 2), ("b", 30), ("a", 30)], 2: [("a", 49), ("c", 39), ("c", 5)]}
    for dtype in ("float32", "bfloat16"):
        out = str(tmp_path / ("out_" + dtype))
        r = subprocess.run([sys.executable, os.path.join(root, "bin", "trace_run"), "--model", d, "--dtype", dtype, "--out", out, "--max-tokens", "128"],
                           input="".join(json.dumps(s) + "\n" for s in steps), capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        assert [l for l in r.stdout.splitlines() if l.startswith("done")] == ["done 0", "done 1", "done 2"]
        for st, rr in rows.items():
            got = np.fromfile(os.path.join(out, f"{st}.f32"), dtype="<f4").reshape(len(rr), cfg["vocab"])
            check(got, np.stack([want[k][i] for k, i in rr]), dtype, f"step {st}")
    from oracle import model as om
    lcfg = om.CONFIGS["tiny-llama"]
    ld = str(tmp_path / "llama")
    om.save_model_dir(ld, lcfg, om.make_weights(lcfg, seed=0))
    r = subprocess.run([sys.executable, os.path.join(root, "bin", "trace_run"), "--model", ld, "--dtype", "float32", "--out", str(tmp_path / "o2"),
                        "--max-tokens", "128"], input="", capture_output=True, text=True, timeout=600)
    assert r.returncode == 3, (r.returncode, r.stderr[-500:])



def last_layer_designs():
    """A last layer of every kind whose rows behind the mixer run for the asked tokens only, with and without a feed-forward, one and
    several residual streams, plain and normed results."""
    from oracle import girolorn as og, kogonex as okg, nosolix as on, zezilix as oz
    out = {f"{mixer}-{mlp}": (oh, oh.make_config(layers=("rglru", mixer), mlps=("dense", mlp))) for mixer in ("rglru", "parallel") for mlp in ("dense", "moe", None)}
    out["attention-moe"] = og, og.make_config(n_layers=2)
    out["delta-moe"] = okg, okg.make_config([okg.latent_layer(), okg.delta_layer()], width=96)
    out["shared-latent"] = okg, okg.make_config([okg.latent_layer(), okg.latent_layer(size=9, kv_from=0, mlp=None)], width=96)
    out["scan-dense"] = on, on.make_config([on.mamba_layer(mlp=on.dense_mlp()), on.mamba_layer(mlp=on.dense_mlp(28))], width=96)
    out["scan-moe"] = on, on.make_config([on.mamba_layer(), on.mamba_layer()], width=96)
    out["wkv-streams"] = oz, oz.make_config([oz.latent_layer(mlp="moe"), oz.wkv_layer(mlp="dense")])
    out["latent-streams"] = oz, oz.make_config([oz.wkv_layer(mlp="dense"), oz.latent_layer(gated=True, mlp="moe")], loop=(0, 2, 2))
    return out


@pytest.mark.parametrize("design", ["rglru-dense", "rglru-moe", "rglru-None", "parallel-dense", "parallel-moe", "parallel-None", "attention-moe", "delta-moe",
                                    "shared-latent", "scan-dense", "scan-moe", "wkv-streams", "latent-streams"])
def test_last_layer_of_the_asked_rows(kge, tmp_path, design):
    """Prompt steps that ask for few of their tokens' logits: none (the next piece stands on its caches and states), the first row, rows
    side by side, more than one turn of the copying kernel, one row for four tokens, and places out of order."""
    o, cfg = last_layer_designs()[design]
    W = o.make_weights(cfg, seed=31)
    toks = prompt(cfg, 150, 32)
    want = o.forward(cfg, W, toks).numpy()
    d = str(tmp_path / "m")
    o.save_model_dir(d, cfg, W)
    llm = kge.LLM(d, dtype="float32", block_size=16, num_gpu_blocks_override=33, max_model_len=513, max_num_seqs=64, max_num_batched_tokens=512, enable_prefix_caching=False)
    at = 0
    for n, places in ((9, []), (21, [20]), (12, [0, 1, 11]), (80, list(range(0, 80, 4))), (20, [7, 3]), (8, [7])):
        llm.trace_add(0, toks[at:at + n])
        got = llm.trace_step([(0, n, places)])
        if places: check(got, want[[at + p for p in places]], "float32", f"{n} tokens, places {places}")
        at += n
    # beside other requests, one of which wants nothing
    llm.trace_add(1, toks[:40]); llm.trace_add(2, toks[:33]); llm.trace_add(3, toks[:1])
    check(llm.trace_step([(3, 1, [0]), (1, 40, []), (2, 33, [5, 32])]), want[[0, 5, 32]], "float32", "three requests")
    llm.close()


@pytest.mark.parametrize("dtype,mlp,width,n,places", [
    ("float32", None, 2048, 511, [0, 510]), ("bfloat16", None, 2048, 512, [0, 511]),      # without a feed-forward: the last step before 2^20 numbers, and the first
    ("bfloat16", "dense", 64, 16, [15]), ("bfloat16", "dense", 64, 17, [0, 16]),          # the first step that is worth the copy
    ("float32", "dense", 640, 409, range(0, 408, 4)), ("bfloat16", "dense", 640, 412, range(1, 412, 4)),      # many rows: from 2^18 numbers on; more than 48 KB of shared memory
    ("float32", "moe", 98, 400, range(3, 400, 4)), ("float32", "moe", 96, 1024, range(0, 1024, 4)),           # rows that are no multiple of 16 bytes; the most rows there are
    ("bfloat16", "moe", 512, 5, [4]), ("bfloat16", "moe", 512, 4, [1])])
def test_last_layer_of_asked_rows_where_it_pays(kge, tmp_path, dtype, mlp, width, n, places):
    """Steps on either side of the lines for the copy of the asked rows, and the copy's own edges."""
    cfg = oh.make_config(width=width, layers=("rglru",), mlps=(mlp,), ff=48, expert_ff=16, shared_ff=16)
    W = oh.make_weights(cfg, seed=37)
    toks = prompt(cfg, n, 38)
    llm = make_engine(kge, tmp_path, cfg, W, dtype, tokens=1024, seqs=2)
    llm.trace_add(0, toks)
    check(llm.trace_step([(0, n, list(places))]), oh.forward(cfg, W, toks)[list(places)], dtype)
    llm.close()
