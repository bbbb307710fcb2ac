"""The barrier protocol of the prompt attention kernel with two query tiles per CTA (csrc/attn_pair.cuh), explored on the CPU over
every order in which its roles can run: no wait may be left behind by its barrier (a parity wait that is sampled a phase late never
ends), none may pass early, and no buffer may be overwritten before its readers are done."""
import os
import re

import pytest

import barrier_explorer

SRC = os.path.join(os.path.dirname(__file__), "..", "kubernetes-gpu-cluster_b200", "csrc", "attn_pair.cuh")

# every barrier operation of the kernel after the barriers' set-up, in the order of the source: what the programs below transcribe
OPS = [
    # producer
    "arrive gathered", "wait item_empty(slot), ((ni >> 1) - 1) & 1", "arrive item_full(slot)",
    "wait is_k ? k_empty(st) : v_empty(st), (nk / NST - 1) & 1",
    "wait q_empty, (ni - 1) & 1", "wait clc_full, nclc & 1", "wait item_empty(slot), ((ni >> 1) - 1) & 1", "arrive item_full(slot)",
    # issuers
    "wait item_full(ni & 1), (ni >> 1) & 1", "arrive item_empty(ni & 1)", "wait q_full, ni & 1",
    "wait k_full(st), ((nk + js) / NST) & 1", "wait s_read(a), (ns - 1) & 1", "commit s_full(a)", "commit k_empty(st)", "commit q_empty",
    "wait v_full(st), ((nk + j) / NST) & 1", "wait v_clean(st), (cleaned >> st) & 1", "arrive v_clean(st)", "wait p_full(a, np), (np >> 1) & 1", "commit o_full(a, np)", "commit v_empty(st)",
    # softmax warps
    "wait item_full(ni & 1), (ni >> 1) & 1", "arrive item_empty(ni & 1)", "wait s_full(a), ns & 1", "arrive s_read(a)",
    "wait o_full(a, ns - 1), ((ns - 1) >> 1) & 1", "wait o_full(a, ns), ((ns - 2) >> 1) & 1", "arrive p_full(a, ns)",
    "wait o_full(a, ns - 1), ((ns - 1) >> 1) & 1",
]


def barrier_ops():
    src = open(SRC).read()
    body = src[src.index("if (warp == 10) {\n"):src.index("}  // namespace atc2")]
    body = re.sub(r"//[^\n]*", "", body)
    out = []
    for m in re.finditer(r"\b(mbar_wait|mbar_arrive|tc_commit)\(", body):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(body[i], 0)
            i += 1
        out.append(m.group(1).replace("mbar_", "").replace("tc_", "") + " " + body[m.end():i - 1])
    return out


def test_transcription_matches_the_kernel():
    assert barrier_ops() == OPS


def programs(items, nst, turns_from=3):
    """Instruction lists of the roles.  items: (key tiles of the first query tile, of the second[, whether they share the key tiles of one
    query tile between them[, whether values beyond the last key are cleared]]).  turns_from: key tiles of the second query tile from
    which on the two groups of softmax threads take turns."""
    def wait(bar, k, optional=False):
        return ("maybe" if optional else "wait", bar, k)
    prod, nk, end = [], 0, len(items)
    items = [(*i, 0, 0)[:4] for i in items]
    tiles = [i[0] + i[1] if i[2] else max(i) for i in items]
    for ni in range(end + 1):
        if ni >= 2:
            prod.append(wait(("item_empty", ni & 1), (ni >> 1) - 1))
        prod.append(("arrive", ("item_full", ni & 1)))
        if ni == end:
            break
        if ni:
            prod.append(wait(("q_empty",), ni - 1))
        prod.append(("load", ("q_full",), ("q",)))
        for _ in range(tiles[ni]):
            for x in "kv":
                if nk >= nst:
                    prod.append(wait((x + "_empty", nk % nst), nk // nst - 1))
                prod.append(("load", (x + "_full", nk % nst), (x, nk % nst)))
            nk += 1
    roles = [prod]
    for a in range(2):
        issue, ns, np, nk, cleaned = [], 0, 0, 0, [0] * nst
        for ni, nn in enumerate(items):
            n, ahead = tiles[ni], 1 + nn[2]
            issue += [wait(("item_full", ni & 1), ni >> 1), ("arrive", ("item_empty", ni & 1)), wait(("q_full",), ni)]
            for j in range(-ahead, n):
                js = j + ahead
                if js < n:
                    st = (nk + js) % nst
                    issue.append(wait(("k_full", st), (nk + js) // nst))
                    if js % 2 == a if nn[2] else js < nn[a]:
                        if ns:
                            issue.append(wait(("s_read", a), ns - 1))
                        issue.append(("mma", [("s_full", a)], [("q",), ("k", st)], [("s", a)]))
                        ns += 1
                    issue.append(("mma", [("k_empty", st)] + ([("q_empty",)] if js + 1 == n else []), [], []))
                if j >= 0:
                    st = (nk + j) % nst
                    issue.append(wait(("v_full", st), (nk + j) // nst))
                    if j % 2 == a if nn[2] else j < nn[a]:
                        both = not nn[2] and nn[0] == nn[1]
                        if nn[3] and j + 1 == n and both and a:
                            issue.append(wait(("v_clean", st), cleaned[st]))
                            cleaned[st] += 1
                        elif nn[3] and j + 1 == n:
                            issue += [("write", ("v", st))] + ([("arrive", ("v_clean", st))] if both else [])
                        issue += [wait(("p_full", a, np & 1), np >> 1),
                                  ("mma", [("o_full", a, np & 1)], [("p", a, np & 1), ("v", st)], [("o", a)])]
                        np += 1
                    issue.append(("mma", [("v_empty", st)], [], []))
            nk += n
        issue.append(wait(("item_full", end & 1), end >> 1))
        roles.append(issue)
    for a in range(2):
        s, ns, joined = [], 0, {}

        def join(bar, meet):
            s.append(("join", (bar,), a))
            if meet:                                             # bar.sync
                s.append(("meet", (bar,), joined.get(bar, 0)))
            joined[bar] = joined.get(bar, 0) + 1
        for ni, nn in enumerate(items):
            s += [wait(("item_full", ni & 1), ni >> 1), ("arrive", ("item_empty", ni & 1))]
            for j in range(nn[a]):
                s += [wait(("s_full", a), ns), ("read", ("s", a)), ("arrive", ("s_read", a))]
                if j:
                    s += [wait(("o_full", a, (ns - 1) & 1), (ns - 1) >> 1, True)]        # only where a row's maximum has grown
                if ns >= 2:
                    s.append(wait(("o_full", a, ns & 1), (ns - 2) >> 1))
                turn = nn[1] >= turns_from and j == 0
                if turn and a:
                    join("bar1", True)
                s.append(("write", ("p", a, ns & 1)))
                if turn and not a:
                    join("bar1", False)
                s.append(("arrive", ("p_full", a, ns & 1)))
                ns += 1
            if nn[a]:
                s += [wait(("o_full", a, (ns - 1) & 1), (ns - 1) >> 1), ("read", ("o", a))]
            if nn[2]:
                join("bar2", True)
                if not a:
                    s.append(("read", ("o", 1)))
                join("bar3", True)
        s.append(wait(("item_full", end & 1), end >> 1))
        roles.append(s)
    return roles


def explore(items, nst, only=None, drop=None, turns_from=3, rings=True):
    """What can go wrong (barrier_explorer).  only: the query tile whose roles are run (the other's arrivals are taken out), which keeps the
    number of states small; so does rings: False, keys and values are always there (more orders than there are, of fewer roles' steps).
    drop: a wait that is left out."""
    roles = programs(items, nst, turns_from)
    need = {"item_empty": 4, "k_empty": 2, "v_empty": 2, "q_empty": 2}
    if only is not None:
        roles = [roles[0], roles[1 + only], roles[3 + only]]
        need = {"item_empty": 2}
        roles = [[op for op in r if op[0] == "mma" or op[1][0][:3] != "bar" and op[1][0] != "v_clean"] for r in roles]
    if drop:
        roles = [[op for op in r if not (op[0] == "wait" and op[1][0] == drop)] for r in roles]
    if not rings:
        ring = {"k_full", "k_empty", "v_full", "v_empty", "v_clean"}
        roles = [[("mma", [b for b in op[1] if b[0] not in ring], *op[2:]) if op[0] == "mma" else op for op in r
                  if op[0] == "mma" or not (op[1][0] in ring or op[0] == "write" and op[1][0] == "v")] for r in roles]
        roles = [[op for op in r if op[0] != "mma" or op[1]] for r in roles]
    return barrier_explorer.explore(roles, need)


@pytest.mark.parametrize("items", [[(1, 0)], [(1, 1)], [(1, 2)], [(1, 0), (1, 1)], [(1, 1, 1), (1, 0)], [(2, 1, 1)], [(3, 3)]], ids=str)
def test_every_wait_ends_in_every_order(items):
    assert not explore(items, 2)


@pytest.mark.parametrize("nst", [2, 4])
@pytest.mark.parametrize("items", [[(5, 6)], [(2, 3), (1, 0), (3, 3)], [(1, 1)] * 4, [(4, 5), (2, 0)], [(3, 2, 1), (2, 2)], [(1, 1, 1)] * 3, [(3, 3, 1), (1, 2)]], ids=str)
@pytest.mark.parametrize("only", [0, 1])
def test_every_wait_of_one_query_tile_ends_in_every_order(items, nst, only):
    assert not explore(items, nst, only)


@pytest.mark.parametrize("drop", ["o_full", "p_full", "s_read", "k_empty", "q_empty"])
def test_the_exploration_finds_a_missing_wait(drop):
    assert explore([(3, 3), (2, 1)], 2, 0, drop)


@pytest.mark.parametrize("items", [[(1, 0, 0, 1)], [(1, 1, 0, 1)], [(1, 2, 0, 1)], [(2, 1, 1, 1)], [(1, 1, 0, 1), (1, 1, 0, 1)], [(3, 3, 0, 1)]], ids=str)
def test_cleared_values_in_every_order(items):
    assert not explore(items, 2)


@pytest.mark.parametrize("nst", [2, 4])
@pytest.mark.parametrize("items", [[(5, 6, 0, 1)], [(2, 3, 0, 1), (1, 0, 0, 1), (3, 3)], [(3, 2, 1, 1), (1, 2, 0, 1)], [(1, 1, 1, 1)] * 3], ids=str)
@pytest.mark.parametrize("only", [0, 1])
def test_cleared_values_of_one_query_tile_in_every_order(items, nst, only):
    assert not explore(items, nst, only)


def test_the_exploration_finds_values_that_are_cleared_too_early_or_not_waited_for():
    assert explore([(3, 3, 0, 1)], 2, 0, "v_full")
    assert explore([(1, 1, 0, 1)], 2, None, "v_clean")


@pytest.mark.parametrize("items", [[(3, 3), (3, 3)], [(1, 3), (4, 3)], [(3, 3), (1, 1), (3, 3)], [(1, 1, 1), (3, 3), (2, 1, 1)], [(1, 1, 1), (1, 1, 1)]], ids=str)
def test_turns_of_items_in_sequence(items):
    assert not explore(items, 4, rings=False)


@pytest.mark.parametrize("turns_from", [1, 2])
def test_the_exploration_finds_turns_that_begin_too_early(turns_from):
    """The first group must not come to its next item's handshake before the second has passed this one."""
    n = turns_from
    assert "arrives twice" in explore([(n, n), (n, n)], 4, turns_from=n, rings=False)
