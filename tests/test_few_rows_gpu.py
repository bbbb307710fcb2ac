"""Small steps of layer-list models: grouped and strided projections of up to 8 rows (linear_few_kernel), distance-biased attention with
its keys split over clusters and (64 and 128 wide, prompts) in the tcgen05 kernel, against the float64 oracle."""
import numpy as np
import pytest

from oracle import hybrid as oh
from test_hybrid_gpu import check, make_engine, prompt, run_pieces

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("experts,top,width,eff,r_width", [
    (40, 3, 264, 72, 192),         # groups found in the second 32; K that ends inside a piece; blocks of 64 (one chunk for eight warps)
    (5, 1, 64, 136, 216),          # K of one chunk; blocks of 72
    (8, 4, 520, 64, 600),          # two tokens are eight rows, three are more
    (3, 3, 72, 1000, 768),         # every expert has rows; blocks of 256
])
def test_few_rows(kge, tmp_path, experts, top, width, eff, r_width):
    cfg = oh.make_config(width=width, layers=("parallel", "rglru"), mlps=("moe", "moe"), experts=experts, top=top, expert_ff=eff, r_width=r_width)
    W = oh.make_weights(cfg, seed=26)        # a choice of experts that rounding to bfloat16 does not turn
    toks = prompt(cfg, 40)
    want = oh.forward(cfg, W, toks)
    llm = make_engine(kge, tmp_path, cfg, W, "bfloat16")
    check(run_pieces(llm, 0, toks, [1, 2, 3, 4, 7, 8, 9, 1, 1, 1, 1, 2]), want, "bfloat16")
    llm.close()


@pytest.mark.parametrize("chunk,kv,hd,n", [(1024, 2, 64, 1100), (520, 1, 32, 700), (300, 4, 128, 420), (200, 1, 128, 450)])      # clusters of 8, 4, 2 and 1; chunk edges inside pieces
def test_decode_over_clusters(kge, tmp_path, chunk, kv, hd, n):
    cfg = oh.make_config(layers=("parallel",), mlps=(None,), right_scale=0.0, chunk=chunk, scale=3.0 / hd ** 0.5, heads=4, kv_heads=kv, dim=hd, vdim=hd)
    W = oh.make_weights(cfg, seed=31)
    toks = prompt(cfg, n)
    want = oh.forward(cfg, W, toks)
    llm = make_engine(kge, tmp_path, cfg, W, "bfloat16", tokens=2 * n + 64, bs=16)
    head = max(1, chunk - 3)        # decoding from just before the chunk's end into the next chunk (few keys: most CTAs of a cluster have none)
    check(run_pieces(llm, 0, toks, [head] + [1] * 12 + [n - head - 32] + [1] * 20), want, "bfloat16", "decoding over the edge")
    # two requests at once, one of them with a single key
    llm.trace_add(1, toks)
    llm.trace_step([(1, n - 1, [])])
    llm.trace_add(2, toks[:1])
    got = llm.trace_step([(1, 1, [0]), (2, 1, [0])])
    llm.close()
    check(got, want[[n - 1, 0]], "bfloat16", "two requests")


@pytest.mark.parametrize("width", [1024, 1028, 2048, 2052, 4096, 4100])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_sum_and_norm_by_width(kge, tmp_path, dtype, width):
    """The stream's sum and the next layer's norm in one pass: each number of pieces per thread, the first width beyond it."""
    cfg = oh.make_config(width=width, layers=("rglru", "rglru", "rglru"), mlps=("dense", "moe", None), experts=3, top=3)
    W = oh.make_weights(cfg, seed=5)
    toks = prompt(cfg, 11)
    llm = make_engine(kge, tmp_path, cfg, W, dtype)
    check(run_pieces(llm, 0, toks, [9, 1, 1]), oh.forward(cfg, W, toks), dtype)
    llm.close()


@pytest.mark.parametrize("width,blocks,rows", [(480, 3, 257), (512, 2, 300), (48, 3, 400), (288, 2, 385)])
def test_block_diagonal_gates_of_many_rows(kge, tmp_path, width, blocks, rows):
    """Strided slices in 128 x 128 tiles: blocks that end inside a tile (160), fill two (256), leave most warps without outputs (16), and end
    inside a warp's columns (144); rows that end inside a tile."""
    cfg = oh.make_config(layers=("rglru",), mlps=(None,), r_width=width, r_blocks=blocks)
    W = oh.make_weights(cfg, seed=41)
    toks = prompt(cfg, rows)
    llm = make_engine(kge, tmp_path, cfg, W, "bfloat16")
    check(run_pieces(llm, 0, toks, [rows]), oh.forward(cfg, W, toks), "bfloat16")
    llm.close()


@pytest.mark.parametrize("width,blocks,taps", [(64, 2, 4), (192, 3, 3), (256, 2, 4), (480, 3, 4), (320, 2, 2), (512, 2, 4), (66, 2, 4),
                                               (352, 2, 4), (416, 2, 3), (480, 2, 4), (384, 2, 4), (448, 2, 2)])
def test_recurrence_by_tiles(kge, tmp_path, width, blocks, taps):
    """Convolution, gates and coefficients in one kernel (blocks of 32, 64, 128 and 160 channels; others take the general ones), the
    recurrence by tiles of 32 rows: pieces that end before, at and behind a tile's edge and span more tiles than are composed at once;
    many requests that begin and end inside one tile, beside decode rows; then decode steps of more requests than a block has rows, in one
    launch where the columns of a diagonal block can be shared out over at most eight blocks (not 176, 208 and 33)."""
    cfg = oh.make_config(layers=("rglru",), mlps=(None,), r_width=width, r_blocks=blocks, r_conv=taps)
    W = oh.make_weights(cfg, seed=43)
    toks = prompt(cfg, 420)
    want = oh.forward(cfg, W, toks)
    llm = make_engine(kge, tmp_path, cfg, W, "bfloat16", tokens=2048, seqs=24)
    for rid, pieces in enumerate([[420], [31, 1, 32, 33, 2, 64, 65, 127, 62, 3]]):
        check(run_pieces(llm, rid, toks, pieces), want, "bfloat16", f"pieces {pieces}")
        llm.trace_end(rid)
    n = 18
    lens = [1 + 3 * rid for rid in range(n)]
    for rid in range(n):
        llm.trace_add(rid, toks[:lens[rid]])
    got = llm.trace_step([(rid, lens[rid], list(range(lens[rid]))) for rid in range(n)])
    check(got, want[[i for m in lens for i in range(m)]], "bfloat16", "prompts side by side")
    for turn in range(3):
        for rid in range(n):
            llm.trace_add(rid, [toks[lens[rid] + turn]])
        got = llm.trace_step([(rid, 1, [0]) for rid in range(n)])
        check(got, want[[m + turn for m in lens]], "bfloat16", f"decode step {turn}")
    for rid in range(n):                                   # pieces of some beside single tokens of others
        m = 1 + (rid % 3) * 20
        llm.trace_add(rid, toks[lens[rid] + 3:lens[rid] + 3 + m])
    got = llm.trace_step([(rid, 1 + (rid % 3) * 20, list(range(1 + (rid % 3) * 20))) for rid in range(n)])
    check(got, want[[lens[rid] + 3 + i for rid in range(n) for i in range(1 + (rid % 3) * 20)]], "bfloat16", "mixed step")
    llm.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_a_rate_that_is_not_a_number_spreads(kge, tmp_path, dtype):
    """In prompt pieces and in decode steps, whichever kernels take them."""
    cfg = oh.make_config(layers=("rglru",), mlps=(None,), r_width=64, r_blocks=2)
    W = oh.make_weights(cfg, seed=43)
    lam = next(k for k in W if k.endswith("mix.lam"))
    W[lam] = W[lam].clone()
    W[lam][37] = float("nan")
    toks = prompt(cfg, 40)
    llm = make_engine(kge, tmp_path, cfg, W, dtype)
    assert np.isnan(run_pieces(llm, 0, toks, [33, 1, 4, 1, 1])).all()
    llm.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("heads,dim,vdim,requests", [(3, 128, 256, 3), (1, 4, 8, 9), (2, 36, 40, 5), (2, 128, 33, 2), (1, 16, 264, 2)])
def test_matrix_memory_token_by_token(kge, tmp_path, heads, dim, vdim, requests, dtype):
    """Decode steps in one launch: key dimensions that do not fill their warps, value columns that end inside a block and take one to eight
    blocks, the first width beyond (264); requests that start at different steps, so that some states are fresh."""
    cfg = oh.make_config(layers=("parallel",), mlps=(None,), left_scale=0.0, m_heads=heads, m_dim=dim, m_vdim=vdim)
    W = oh.make_weights(cfg, seed=47)
    toks = prompt(cfg, 24)
    want = oh.forward(cfg, W, toks)
    llm = make_engine(kge, tmp_path, cfg, W, dtype, tokens=1024, seqs=16)
    at = [0] * requests
    for turn in range(16):
        live = [r for r in range(requests) if r <= turn and at[r] < 24]
        for r in live:
            llm.trace_add(r, [toks[at[r]]])
        got = llm.trace_step([(r, 1, [0]) for r in live])
        check(got, want[[at[r] for r in live]], dtype, f"step {turn}")
        for r in live:
            at[r] += 1
    llm.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("heads,dim,vdim,requests", [(8, 16, 256, 32), (8, 16, 256, 33), (4, 48, 136, 110), (8, 96, 256, 33)])
def test_matrix_memory_of_many_requests(kge, tmp_path, heads, dim, vdim, requests, dtype):
    """Decode steps on either side of the line between one launch and three (2048 blocks of less than 96 key dimensions)."""
    cfg = oh.make_config(layers=("parallel",), mlps=(None,), left_scale=0.0, m_heads=heads, m_dim=dim, m_vdim=vdim)
    W = oh.make_weights(cfg, seed=47)
    toks = prompt(cfg, 6)
    want = oh.forward(cfg, W, toks)
    llm = make_engine(kge, tmp_path, cfg, W, dtype, tokens=16 * requests, seqs=requests)
    for t in range(6):
        for r in range(requests):
            llm.trace_add(r, [toks[t]])
        check(llm.trace_step([(r, 1, [0]) for r in range(requests)]), want[[t] * requests], dtype, f"step {t}")
    llm.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("experts,top,width", [(16, 2, 512), (17, 4, 2056), (33, 3, 40), (128, 5, 136), (129, 2, 136)])
def test_routing_of_a_few_tokens(kge, tmp_path, experts, top, width, dtype):
    """Scores, choice and grouping in one launch: one row a warp, several, the last count of experts it takes and the first it does not, rows
    longer than what is asked for ahead; one to five tokens (four are the most)."""
    cfg = oh.make_config(width=width, layers=("rglru",), mlps=("moe",), experts=experts, top=top, expert_ff=16)
    W = oh.make_weights(cfg, seed=53)
    toks = prompt(cfg, 15)
    llm = make_engine(kge, tmp_path, cfg, W, dtype)
    check(run_pieces(llm, 0, toks, [1, 2, 3, 4, 5]), oh.forward(cfg, W, toks), dtype)
    llm.close()


@pytest.mark.parametrize("hd", [64, 128])
def test_short_biased_pieces(kge, tmp_path, hd):
    """Pieces around the length from which on prompts run in the tcgen05 kernel: the last whose keys are one tile of the other, and the next."""
    cfg = oh.make_config(layers=("parallel",), mlps=(None,), right_scale=0.0, chunk=1024, scale=3.0 / hd ** 0.5, dim=hd, vdim=hd)
    W = oh.make_weights(cfg, seed=37)
    toks = prompt(cfg, 70)
    want = oh.forward(cfg, W, toks)
    llm = make_engine(kge, tmp_path, cfg, W, "bfloat16", tokens=160)
    for rid, pieces in enumerate([[32, 33, 5], [31, 1, 38], [33, 37], [20, 20, 30]]):
        check(run_pieces(llm, rid, toks, pieces), want, "bfloat16", f"pieces {pieces}")
        llm.trace_end(rid)
    llm.close()


@pytest.mark.parametrize("heads,dim,vdim,lens", [
    (1, 128, 32, [64, 65, 129, 193, 257, 449, 512, 513, 700]),      # one to eight blocks for the same columns
    (2, 48, 72, [1, 130, 1, 64, 321]),                              # requests of one token and of one chunk beside longer ones
    (3, 16, 256, [200, 90]),
    (5, 128, 256, [150, 70, 10, 3]),                                # no room for a second block
    (4, 128, 256, [300, 20]),                                       # norm and gate by a warp a row, a piece a lane
    (4, 16, 128, [200, 200, 200]),                                  # 48 clusters: of two, since 45 of three fit
    (2, 128, 264, [700, 2]), (2, 4, 520, [650]), (9, 32, 40, [135]), (9, 32, 40, [860]),      # (other sums; norm and gate by a warp a row: two and four pieces a lane, less than one)
])
def test_matrix_memory_prompts_in_runs_of_chunks(kge, tmp_path, heads, dim, vdim, lens):
    """A request's chunks shared out over the blocks of a cluster: all requests in one step, first without a state, then on from it, and the
    decode steps behind, which read what the last block wrote; beside the same tokens in pieces of one chunk, which one block takes.
    The two do the same fp32 arithmetic (but for the running maximum, kept in 64 bits within a step): what may differ is a 16-bit
    rounding of a mixer output, 2^-8 of it, at most some 2^-6 of the logits' size.  Against the oracle the middle row of each chunk is held to
    4 x 2^-8 (roundings of q, k, v and the output): a run that went wrong is wrong in all of its rows, while single rows whose normaliser
    cancels magnify the roundings of their q and k (0.063 at one token of 1402, with one block as with eight)."""
    cfg = oh.make_config(layers=("parallel",), mlps=(None,), left_scale=0.0, m_heads=heads, m_dim=dim, m_vdim=vdim)
    W = oh.make_weights(cfg, seed=59)
    n = len(lens)
    P = [prompt(cfg, 2 * m + 2, 60 + r) for r, m in enumerate(lens)]
    llm = make_engine(kge, tmp_path, cfg, W, "bfloat16", tokens=8192, seqs=n + 1)
    got = [[] for _ in range(n)]
    for part in range(4):
        sizes = [m if part < 2 else 1 for m in lens]
        at = [sum(len(x) for x in got[r]) for r in range(n)]
        for r in range(n):
            llm.trace_add(r, P[r][at[r]:at[r] + sizes[r]])
        lg = np.split(llm.trace_step([(r, m, list(range(m))) for r, m in enumerate(sizes)]), np.cumsum(sizes)[:-1])
        for r in range(n):
            got[r].append(lg[r])
    for r in range(n):
        llm.trace_end(r)
    for r, m in enumerate(lens):
        mine = np.concatenate(got[r])
        whole = [min(64, m - i) for i in range(0, m, 64)]
        other = run_pieces(llm, n + r, P[r], whole + whole + [1, 1])
        llm.trace_end(n + r)
        want = oh.forward(cfg, W, P[r]).numpy()
        size = np.sqrt((want ** 2).mean())
        err = np.sqrt(((mine - other) ** 2).mean(-1)) / size
        assert err.max() < 2.0 ** -6, f"request {r}: row {err.argmax()} is {err.max():.3g} of the logits' size from the pieces'"
        err = np.sqrt(((mine - want) ** 2).mean(-1)) / size
        mid = [np.median(err[i:i + 64]) for i in range(0, len(err), 64)]
        assert max(mid) < 2.0 ** -6, f"request {r}: {max(mid):.3g} of the logits' size in chunk {int(np.argmax(mid))}"
    llm.close()
