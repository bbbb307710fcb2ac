"""The barrier protocol of the prompt attention kernel (csrc/attn_tc.cu), explored on the CPU over every order in which its roles
can run: no wait may be left behind by its barrier (a parity wait that is sampled a phase late never ends) and none may pass early."""
import os
import re

import pytest

import barrier_explorer

SRC = os.path.join(os.path.dirname(__file__), "..", "kubernetes-gpu-cluster_b200", "csrc", "attn_tc.cu")

# every barrier operation of the kernel after the barriers' set-up, in the order of the source: what the programs below transcribe
OPS = [
    "wait o_full(j & 1), (uint32_t)((j >> 1) & 1)",                  # wait_o
    # issuer
    "wait k_full(st), (uint32_t)((j >> 1) & 1)", "commit s_full(st)",
    "wait q_full, 0u", "wait_o j - 1", "wait v_full(j & 1), (uint32_t)((j >> 1) & 1)", "wait p_full(j & 1), (uint32_t)((j >> 1) & 1)",
    "commit o_full(j & 1)", "commit v_empty(j & 1)",
    # producer
    "wait s_full(j & 1), (uint32_t)((j >> 1) & 1)", "wait v_empty(j & 1), (uint32_t)((j >> 1) & 1)",
    # softmax threads
    "arrive q_full", "arrive k_full(0)", "wait s_full(j & 1), (uint32_t)((j >> 1) & 1)", "arrive k_full((j + 1) & 1)",
    "wait_o j - 1", "wait_o j - 1", "arrive v_full(j & 1)", "arrive p_full(j & 1)", "wait_o ntiles - 1",
]


def barrier_ops():
    src = open(SRC).read()
    body = src[src.index("__global__ void __launch_bounds__(TMA ? 192 : 160, 2)"):src.index("template <int HD> constexpr int tc_smem()")]
    body = re.sub(r"//[^\n]*", "", body)
    out = []
    for m in re.finditer(r"\b(mbar_wait|mbar_arrive|tc_commit|wait_o)\(", body):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(body[i], 0)
            i += 1
        out.append(m.group(1).replace("mbar_", "").replace("tc_", "") + " " + body[m.end():i - 1])
    return out


def test_transcription_matches_the_kernel():
    assert barrier_ops() == OPS


def programs(n, tma, o_bars, last):
    """Instruction lists of the roles for n key tiles.  o_bars: barriers that P V commits to in turn; last: the tiles that a softmax
    thread waits for at the end."""
    def wait(name, j, turn=2, optional=False):
        return ("maybe" if optional else "wait", (name, j % turn), j // turn)

    def wait_o(j, optional=False):
        return wait("o", j, o_bars, optional)
    issuer, producer, soft = [], [], []

    def issue_s(j):
        issuer.extend([wait("k", j), ("mma", (("s", j % 2),))])
    if tma:
        issuer.append(wait("q", 0, 1))
    issue_s(0)
    for j in range(n):
        if j + 1 < n:
            if j > 0:
                issuer.append(wait_o(j - 1))
            issue_s(j + 1)
        issuer += [wait("v", j), wait("p", j), ("mma", (("o", j % o_bars),) + ((("e", j % 2),) if tma else ()))]
    if tma:
        for t in range(min(n, 2)):
            producer.append(("load", ("k", t)))
        for t in range(min(n, 2)):
            producer.append(("load", ("v", t)))
        for j in range(n - 2):
            producer += [wait("s", j), ("load", ("k", j % 2)), wait("e", j), ("load", ("v", j % 2))]
        soft.append(("arrive", ("q", 0)))
    else:
        soft.append(("arrive", ("k", 0)))
    for j in range(n):
        soft.append(wait("s", j))
        if not tma:
            if j + 1 < n:
                soft.append(("arrive", ("k", (j + 1) % 2)))
            if j > 0:
                soft.append(wait_o(j - 1))
        elif j > 0:
            soft.append(wait_o(j - 1, optional=True))        # only where a row's maximum has grown
        if not tma:
            soft.append(("arrive", ("v", j % 2)))
        soft.append(("arrive", ("p", j % 2)))
    soft += [wait_o(j) for j in last if j >= 0]
    return issuer, producer, soft


def explore(n, tma, o_bars=2, last=None):
    """What can go wrong (barrier_explorer), with two softmax threads."""
    issuer, producer, soft = programs(n, tma, o_bars, [n - 1] if last is None else last)
    roles = [issuer, producer, soft, soft]
    need = {"q": 2, "p": 2, "k": 1 if tma else 2, "v": 1 if tma else 2}
    roles = [[(*op, (), ()) if op[0] == "mma" else (*op, None) if op[0] == "load" else op for op in r] for r in roles]
    return barrier_explorer.explore(roles, need)


@pytest.mark.parametrize("tma", [True, False])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5])
def test_every_wait_ends_in_every_order(n, tma):
    assert not explore(n, tma)


@pytest.mark.parametrize("tma", [True, False])
def test_the_exploration_finds_a_wait_that_can_miss_its_phase(tma):
    """One barrier for all tiles, and waits for the last two phases in turn after everything has been handed over."""
    assert explore(2, tma, o_bars=1, last=[0, 1])
    assert explore(3, tma, o_bars=1, last=[1, 2])
