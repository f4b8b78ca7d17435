"""The waits of the chunked gated delta rule (``csrc/linear_attn/gdn_chunk.cu``), followed on the CPU.

An mbarrier wait names the parity of a phase.  It is sound only if the phase behind the awaited one cannot complete before the
waiting thread has looked: two phases further on the parity is the same again, and the wait blocks for a phase that may need the
waiter itself.  The roles of the kernel are written down below, in program order; which barrier and which phase every wait and
arrival names is read from the source.  From these follows what happens before what, whatever the timing.
"""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(__file__), "..", "csrc", "linear_attn", "gdn_chunk.cu")

# per role: what it does for chunk n of N, in program order.  A number = the wait with this code; "+x" = an arrival at x; "*x" = a
# commit of the products issued so far (arrives when they are done); "bar" = a barrier of the four warps of prep_a and prep_p;
# (op, -1): for the chunk in front (none at first)
ROLES = {
    "prep_a": [901, 902, "+d0_read", "bar", 905, "+t_ready", "bar"],
    "prep_p": [901, 902, 903, "+d0_read", "bar", 905, "+t_ready", "bar"],
    "chain": [911, "+s_ready", (910, -1), ("+o_read", -1), 912, 913, "+r_ready", 914, 915, "+ut_ready", "+uo_ready", 916],
    "loads": [904, "*raw", 906, "+full"],
    "mma": [921, "*x1", 922, "*x2", 925, "*d0", 923, 924, "*u_full", 926, "*d3", 927, "*y"],
}
# what a chunk at the start does not do, by the first chunk that does; what the last one does not do (it is for the next)
FIRST = {903: 2, 904: 2, 905: 1, 922: 1}
NOT_LAST = (925, "*d0")
TAIL = {"chain": [(910, 0), ("+o_read", 0)]}      # after the last chunk
HEAD = {"mma": [(920, 0), ("*d0", 0)]}            # in front of the first one


def _named(src):
    index = lambda text: text if text else "0"
    waits = {int(code): (name, index(i), phase) for name, i, phase, code in
             re.findall(r"wait(?:_one|_tc)?\(&sm\.(\w+)(?:\[([^\]]+)\])?, ([^,]+), (\d+)\)", src)}
    arrivals = {}
    for name, i in re.findall(r"(?:mbar_expect_tx|arrive|umma_commit)\(&sm\.(\w+)(?:\[([^\]]+)\])?[,)]", src):
        assert arrivals.setdefault(name, index(i)) == index(i), name
    return waits, arrivals


def _events(src, N):
    """Edges (before -> after) between events; (barrier, index, phase) nodes are completions."""
    waits, arrivals = _named(src)
    edges, waited, count, commits = [], [], {}, []

    def value(expr, n, role):
        v = dict(n=n, c=n, st=n & 1)
        return eval(expr.replace("sm.", ""), {}, v)

    def step(role, op, n, prev, uid):
        node = (role, n, str(op), uid)
        if prev is not None:
            edges.append((prev, node))
        if op == "bar":
            edges.extend([(node, ("bar", uid)), (("bar", uid), node + ("passed",)), (node, node + ("passed",))])
            return node + ("passed",)
        if isinstance(op, int):
            name, i, phase = waits[op]
            done = (name, value(i, n, role), value(phase, n, role))
            edges.append((done, node))
            waited.append((node, done, op))
            return node
        name = op[1:]
        i = value(arrivals[name], n, role) if name in arrivals else 0
        key = (name, i, role)
        count[key] = count.get(key, -1) + 1
        done = (name, i, count[key])
        edges.append((node, done))
        if op[0] == "*" and role == "mma":          # commits complete in the order in which they were issued
            if commits:
                edges.append((commits[-1], done))
            commits.append(done)
        return node

    for role, ops in ROLES.items():
        prev, uid = None, 0
        todo = [(op, n) for op, n in HEAD.get(role, [])]
        for n in range(N):
            for op in ops:
                op, d = op if isinstance(op, tuple) else (op, 0)
                if n + d >= FIRST.get(op, 0) and not (op in NOT_LAST and n == N - 1):
                    todo.append((op, n + d))
        todo += [(op, N - 1) for op, _ in TAIL.get(role, [])]
        bars = 0
        for op, n in todo:
            bars += op == "bar"
            prev = step(role, op, n, prev, bars if op == "bar" else f"{role}{uid}")
            uid += 1
    return edges, waited


def _after(edges, start):
    out = {}
    for a, b in edges:
        out.setdefault(a, []).append(b)
    seen, todo = set(), [start]
    while todo:
        for b in out.get(todo.pop(), []):
            if b not in seen:
                seen.add(b)
                todo.append(b)
    return seen


@pytest.mark.parametrize("N", [1, 2, 5])
def test_no_wait_can_be_passed(N):
    src = open(SOURCE).read()
    waits, _ = _named(src)
    used = {op[0] if isinstance(op, tuple) else op for ops in list(ROLES.values()) + list(TAIL.values()) + list(HEAD.values()) for op in ops}
    assert {op for op in used if isinstance(op, int)} == set(waits), "the roles above and the source name different waits"
    edges, waited = _events(src, N)
    happens = {b for _, b in edges} | {a for a, _ in edges}
    for node, (name, i, phase), code in waited:
        assert any(b == (name, i, phase) and a[0] != "bar" for a, b in edges), f"wait {code}: nothing completes {name}[{i}] phase {phase}"
        after = _after(edges, node)
        assert node not in after, f"wait {code} of {node[0]}, chunk {node[1]}: waits for itself"
        follow = (name, i, phase + 1)
        assert follow not in happens or follow in after, \
            f"wait {code} of {node[0]}, chunk {node[1]}: {name}[{i}] may be a phase further before it is looked at"
