"""Every order in which the roles of a kernel can run, for the tests of barrier protocols.

A role is a list of operations:
  ("wait", bar, k)     mbarrier.try_wait.parity for phase k;  ("maybe", bar, k): the same, or skipped
  ("arrive", bar)      one arrival;  `need` says how many complete a phase, by the barrier's name bar[0] (one unless told otherwise)
  ("join", bar, g)     group g of threads arrives at a named barrier of two groups (bar.arrive, the first half of bar.sync)
  ("meet", bar, k)     the second half of bar.sync: the phase that the k-th join belongs to is complete
  ("mma", bars, reads, writes)   an MMA that commits to `bars`; those of a role complete in the order of issue
  ("load", bar, buf)   a copy into `buf` (or None) that arrives at `bar`; copies complete in any order
  ("read", buf), ("write", buf)  by threads
"""


def explore(roles, need):
    """What can go wrong, or None: a role that waits for ever, a wait that passes in another phase than its own, a group that arrives twice
    in a phase of a named barrier, or a buffer that is written while an MMA or a copy in flight uses it."""
    def barriers(op):
        return op[1] if op[0] == "mma" else () if op[0] in ("read", "write") else (op[1],)
    bars = sorted({b for r in roles for op in r for b in barriers(op)}, key=str)
    index = {b: i for i, b in enumerate(bars)}
    mmas = [[op for op in r if op[0] == "mma"] for r in roles]
    before = [[sum(op[0] == "mma" for op in r[:i]) for i in range(len(r) + 1)] for r in roles]

    def put(state, bar, value):
        return state[:index[bar]] + (value,) + state[index[bar] + 1:]

    def arrive(state, bar):
        done, got = state[index[bar]]
        return put(state, bar, (done + 1, 0) if got + 1 == need.get(bar[0], 1) else (done, got + 1))

    start = ((0,) * len(roles), ((0, 0),) * len(bars), (0,) * len(roles), ())            # positions, barriers, MMAs done, copies in flight
    seen, todo = {start}, [start]
    while todo:
        pcs, state, done_mma, loads = todo.pop()
        flight = [f for m, d, b, pc in zip(mmas, done_mma, before, pcs) for f in m[d:b[pc]]]
        succ = []
        for r, prog in enumerate(roles):
            if pcs[r] == len(prog):
                continue
            op = prog[pcs[r]]
            nxt = pcs[:r] + (pcs[r] + 1,) + pcs[r + 1:]
            if op[0] in ("wait", "maybe"):
                if op[0] == "maybe":
                    succ.append((nxt, state, done_mma, loads))
                done = state[index[op[1]]][0]
                if (done & 1) != (op[2] & 1):
                    if done != op[2] + 1:
                        return f"wait for phase {op[2]} of {op[1]} passes after {done}"
                    succ.append((nxt, state, done_mma, loads))
            elif op[0] == "arrive":
                succ.append((nxt, arrive(state, op[1]), done_mma, loads))
            elif op[0] == "join":
                done, there = state[index[op[1]]]
                if there & (1 << op[2]):
                    return f"group {op[2]} arrives twice in a phase of {op[1]}"
                there |= 1 << op[2]
                succ.append((nxt, put(state, op[1], (done + 1, 0) if there == 3 else (done, there)), done_mma, loads))
            elif op[0] == "meet":
                if state[index[op[1]]][0] > op[2]:
                    succ.append((nxt, state, done_mma, loads))
            elif op[0] == "load":
                if op[2] is not None and any(op[2] in f[2] for f in flight):
                    return f"copy into {op[2]}, which an MMA reads"
                succ.append((nxt, state, done_mma, tuple(sorted(loads + (op[1:],), key=str))))
            else:
                if op[0] == "read" and any(op[1] in f[3] for f in flight) or op[0] == "write" and any(op[1] in f[2] for f in flight):
                    return f"{op} beside an MMA"
                if op[0] == "write" and any(op[1] == buf for _, buf in loads):
                    return f"{op} beside a copy"
                succ.append((nxt, state, done_mma, loads))
        for r, m in enumerate(mmas):
            if done_mma[r] < before[r][pcs[r]]:
                s = state
                for b in m[done_mma[r]][1]:
                    s = arrive(s, b)
                succ.append((pcs, s, done_mma[:r] + (done_mma[r] + 1,) + done_mma[r + 1:], loads))
        for i, (b, _) in enumerate(loads):
            succ.append((pcs, arrive(state, b), done_mma, loads[:i] + loads[i + 1:]))
        if not succ and any(pcs[r] < len(prog) for r, prog in enumerate(roles)):
            return "waits for ever: " + ", ".join(str(prog[pcs[r]]) for r, prog in enumerate(roles) if pcs[r] < len(prog))
        for s in succ:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None
