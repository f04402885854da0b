"""A host-side model of the CTA-pair attention backward (``csrc/attn_bwd_pair_tcgen05.cu``): its roles' programs, the buffers that
they hand to one another and the mbarriers between them, checked by happens-before.

Two CTAs with some twenty actors have too many interleavings to walk (``pipeline_model.py`` does that for the single-CTA kernel),
and need not be walked: no role ever chooses, so the arrivals that complete a phase and the phase that lets a wait pass are
the same in every interleaving, provided that the graph of one execution shows

* for every arrival, that the phase before the one it counts towards had completed,
* for every wait, that it can neither pass a phase pair early (the parity is the same) nor come a phase too late.

Given that, one execution's graph (program order, the tensor core in issue order, copies from their issue to the bytes' arrival on a
barrier, arrivals to the phase they complete to the waits that it lets pass) orders two accesses exactly if they are ordered in all
of them.  Reported are conditions above that fail, deadlocks, reads that find other contents than they expect, and accesses of
which one writes that the graph does not order.

Scopes.  Shared memory of one CTA that its threads wrote with ordinary stores and that an instruction issued in the other CTA reads has
to be released and acquired at cluster scope somewhere between the two: for such pairs an arrival on the other CTA's barrier orders
what came before the arriving thread's last cluster fence, if the wait for it is of cluster scope, and nothing otherwise.  (Tensor memory is handed over under the tcgen05 fences, copies and
commits complete on barriers at cluster scope.)

The programs are transcribed from the kernel; a change of its synchronisation has to be mirrored here.
"""

from __future__ import annotations

from collections import defaultdict
from dataclasses import dataclass
from typing import Dict, List, Tuple

GROUPS = 4          # softmax warpgroups: 32 queries of a chunk each
P_CELL = (0, 2, 1, 3)               # 16-column cell of T1 that takes group g's P


@dataclass(frozen=True)
class Variant:
    """Switches that re-introduce hazards the kernel's synchronisation exists to prevent (to show the model sees them)."""
    cluster_fence: bool = True          # CTA 1's relay fences at cluster scope behind its softmax warps' half of dS
    cluster_acquire: bool = True        # and the leader acquires there
    wait_last_dq_read: bool = True      # behind the last chunk, dQ waits until the dQ before it has been read
    wait_quad_read: bool = True         # groups 2, 3 store P once groups 0, 1 have read their scores
    wait_dq_before_ds: bool = True      # dS(c) is stored once dQ(c - 1) has been formed


# Operations: ("wait", (barrier, cta), parity, cluster scope?), ("arrive", (barrier, cta), weight), ("fence", "cluster"), ("read" / "write",
# buffer, tag), ("tc", reads, writes, commits) and ("copy", reads, writes, barrier or None, label), ("drained", label): the copy
# with that label has read its source.

def _producer(r: int, n: int) -> List[Tuple]:
    def load(buf, tag, bar):
        return ("copy", [], [((buf, r), tag)], (bar, 0), None)

    def expect(bar):
        return [("arrive", (bar, 0), 1)] if r == 0 else []

    def stats(c):
        return [("arrive", (f"stFull{c & 1}", r), 1), ("copy", [], [((f"stat{c & 1}", r), ("stat", c))], (f"stFull{c & 1}", r), None)]

    ops = expect("kvFull") + [load("KV", "KV", "kvFull")] + stats(0) + (stats(1) if n > 1 else [])
    for c in range(n + 1):
        wpar = (c & 1) ^ 1
        if c < n:
            ops += [("wait", ("qsEmpty", r), wpar, False)] + expect("qsFull") + [load("Qs", ("Qs", c), "qsFull")]
        if c > 0:
            ops += [("wait", ("qkEmpty", r), wpar ^ 1, False)] + expect("qkFull") + [load("Qk", ("Qk", c - 1), "qkFull")]
            if 2 <= c < n:
                ops += stats(c)
        if c < n:
            ops += [("wait", ("dopEmpty", r), wpar, False)] + expect("dopFull") + [load("dOp", ("dOp", c), "dopFull")]
            ops += [("wait", ("dovEmpty", r), wpar, False)] + expect("dovFull") + [load("dOv", ("dOv", c), "dovFull")]
    return ops


def _both(bufs_tags):
    return [((b, r), t) for b, t in bufs_tags for r in (0, 1)]


def _mma(n: int, v: Variant) -> List[Tuple]:
    def wait(bar, parity, cluster=False):
        return ("wait", (bar, 0), parity, cluster)

    def tc(reads, writes, *commits):
        return ("tc", _both(reads), _both(writes), [(b, r) for b in commits for r in (0, 1)])

    def scores(c):
        return [wait("qsFull", c & 1), tc([("KV", "KV"), ("Qs", ("Qs", c))], [(f"T1.{i}", ("S", c)) for i in range(8)], "sFull", "qsEmpty")]

    def dp(c):
        return [wait("dopFull", c & 1), tc([("KV", "KV"), ("dOp", ("dOp", c))], [(f"T2.{i}", ("dP", c)) for i in range(8)], "dpFull", "dopEmpty")]

    def dv(c):
        return [wait("dovFull", c & 1), wait("pReady", c & 1),
                tc([(f"T1.{i}", ("P", c)) for i in range(4)] + [("dOv", ("dOv", c))], [("accV", ("dV", c))], "dovEmpty")]

    ops = [wait("kvFull", 0)] + scores(0) + dp(0) + dv(0) + (scores(1) if n > 1 else [])
    for c in range(n):
        par, more = c & 1, c + 1 < n
        ops += [("arrive", ("exIn", 0), 1), wait("qkFull", par), wait("dsReady", par),
                tc([(f"T2.{2 * g}", ("dS", c)) for g in range(GROUPS)] + [("Qk", ("Qk", c))], [("accK", ("dK", c))], "qkEmpty")]
        if more:
            ops += dp(c + 1) + [wait("sRead", par ^ 1)]
        elif c > 0 and v.wait_last_dq_read:
            ops.append(wait("dqRead", par ^ 1))
        ops += [wait("dsOwn", par), wait("exIn", par), wait("exPeer", par, v.cluster_acquire),
                tc([("dSown", ("dS", c)), ("dSpeer", ("dS", c)), ("KV", "KV")], [(f"T1.{i}", ("dQ", c)) for i in range(4, 8)], "dqFull")]
        if more:
            ops += dv(c + 1)
        if c + 2 < n:
            ops += [wait("dqRead", par)] + scores(c + 2)
    return ops + [tc([], [], "accFinal")]


def _relay(n: int, v: Variant) -> List[Tuple]:
    ops: List[Tuple] = []
    for c in range(n):
        ops += [("arrive", ("exIn", 1), 1), ("wait", ("dsOwn", 1), c & 1, False)] + ([("fence", "cluster")] if v.cluster_fence else [])
        ops += [("wait", ("exIn", 1), c & 1, False), ("arrive", ("exPeer", 0), 1)]
    return ops


def _exchange(r: int, n: int) -> List[Tuple]:
    ops: List[Tuple] = []
    for c in range(n):
        ops += [("wait", ("exStaged", r), c & 1, False),
                ("copy", [(("out", r), ("dS", c))], [(("dSpeer", r ^ 1), ("dS", c))], ("exIn", r ^ 1), None)]
    return ops


def _reducer(r: int, n: int) -> List[Tuple]:
    ops: List[Tuple] = []
    for i in range(2 * n):
        ops += [("wait", ("staged", r), i & 1, False), ("copy", [(("stage", r), ("dQ", i >> 1, i & 1))], [], None, ("red", r, i)),
                ("drained", ("red", r, i)), ("arrive", (f"stageFree{i & 1}", r), 1)]
    return ops


def _drain(r: int, half: int, n: int) -> List[Tuple]:
    ops: List[Tuple] = []
    for c in range(n):
        ops.append(("wait", ("dqFull", r), c & 1, False))
        ops += [("read", (f"T1.{4 + 2 * half + i}", r), ("dQ", c)) for i in (0, 1)]
        ops.append(("arrive", ("dqRead", 0), 4))
        if c > 0 or half > 0:
            ops.append(("wait", (f"stageFree{half ^ 1}", r), (c if half else c - 1) & 1, False))
        ops += [("write", ("stage", r), ("dQ", c, half)), ("arrive", ("staged", r), 4)]
    return ops


def _softmax(r: int, g: int, n: int, v: Variant) -> List[Tuple]:
    mine = (g >> 1) == r
    ops: List[Tuple] = []
    for c in range(n):
        par = c & 1
        ops += [("wait", (f"stFull{par}", r), (c >> 1) & 1, False), ("wait", ("sFull", r), par, False)]
        ops += [("read", (f"T1.{2 * g + i}", r), ("S", c)) for i in (0, 1)]
        if g < 2:
            ops.append(("arrive", ("quadRead", r), 1))
        ops += [("arrive", ("sRead", 0), 4), ("read", (f"stat{par}", r), ("stat", c))]
        if g >= 2 and v.wait_quad_read:
            ops.append(("wait", ("quadRead", r), par, False))
        ops += [("write", (f"T1.{P_CELL[g]}", r), ("P", c)), ("arrive", ("pReady", 0), 4), ("wait", ("dpFull", r), par, False)]
        ops += [("read", (f"T2.{2 * g + i}", r), ("dP", c)) for i in (0, 1)]
        ops += [("read", (f"stat{par}", r), ("stat", c)), ("write", (f"T2.{2 * g}", r), ("dS", c)), ("arrive", ("dsReady", 0), 4)]
        if c > 0 and v.wait_dq_before_ds:
            ops.append(("wait", ("dqFull", r), par ^ 1, False))
        # the two groups of a half write rows of one tile: a buffer each, read together
        ops += [("write", ("dSown" if mine else "out", r, g & 1), ("dS", c)), ("arrive", ("dsOwn" if mine else "exStaged", r), 4)]
    return ops + [("wait", ("accFinal", r), 0, False), ("read", ("accV", r), ("dV", n - 1)), ("read", ("accK", r), ("dK", n - 1))]


def _counts() -> Dict[str, int]:
    """Arrivals that complete a phase: for the barriers of copies the expectation and each CTA's loads, one each."""
    c = {"kvFull": 3, "qsFull": 3, "qkFull": 3, "dopFull": 3, "dovFull": 3, "sRead": 32, "pReady": 32, "dsReady": 32, "dqRead": 16, "exPeer": 1,
         "dsOwn": 8, "exStaged": 8, "staged": 4, "exIn": 2, "quadRead": 2}
    for b in ("qsEmpty", "qkEmpty", "dopEmpty", "dovEmpty", "sFull", "dpFull", "dqFull", "accFinal", "stageFree0", "stageFree1"):
        c[b] = 1
    c["stFull0"] = c["stFull1"] = 2
    return c


def _halves(buf):
    """``dSown`` and ``out`` are read whole and written by halves."""
    return [(buf[0], buf[1], i) for i in (0, 1)] if buf[0] in ("dSown", "out") and len(buf) == 2 else [buf]


class _Graph:
    def __init__(self):
        self.label: List[str] = []
        self.cta: List[int] = []
        self.into: List[List[int]] = []             # all orders
        self.into_cluster: List[List[int]] = []     # those that order ordinary stores for the other CTA
        self.into_late: List[List[int]] = []        # a wait's own predecessors: what is known before the barrier is looked at

    def node(self, label, cta, *preds) -> int:
        self.label.append(label)
        self.cta.append(cta)
        preds = [p for p in preds if p is not None]
        self.into.append(list(preds))
        self.into_cluster.append(list(preds))
        self.into_late.append(list(preds))
        return len(self.label) - 1


def check(chunks: int, variant: Variant = Variant()) -> List[str]:
    """Violations of the kernel's protocol over ``chunks`` query chunks (none: an empty list)."""
    n, counts = chunks, _counts()
    progs: Dict[str, Tuple[int, List[Tuple]]] = {"mma": (0, _mma(n, variant)), "relay": (1, _relay(n, variant))}
    for r in (0, 1):
        progs[f"producer {r}"] = (r, _producer(r, n))
        progs[f"exchange {r}"] = (r, _exchange(r, n))
        progs[f"reducer {r}"] = (r, _reducer(r, n))
        for h in (0, 1):
            progs[f"drain {r}.{h}"] = (r, _drain(r, h, n))
        for g in range(GROUPS):
            progs[f"softmax {r}.{g}"] = (r, _softmax(r, g, n, variant))
    G, out = _Graph(), []
    pending: Dict[Tuple, int] = {}
    phase_arrivals: Dict[Tuple, List[Tuple]] = defaultdict(list)    # barrier -> arrivals of the current phase
    completed: Dict[Tuple, List[int]] = defaultdict(list)                           # barrier -> completion nodes
    foreign: Dict[Tuple, List[List[int]]] = defaultdict(list)                       # ... the fences ahead of arrivals from the other CTA
    complete_with: Dict[Tuple, List[int]] = defaultdict(list)                       # ... and all its arrivals, as a bit set
    arrival_phase: List[Tuple[int, Tuple, int]] = []
    waits: List[Tuple[int, Tuple, int]] = []                                        # node, barrier, phases completed when it passed
    content: Dict[Tuple, object] = {}
    accesses: Dict[Tuple, List[Tuple[int, bool, bool]]] = defaultdict(list)         # node, writes?, by ordinary stores?
    copies: Dict[Tuple, int] = {}

    def arrive(bar, node, weight, cta, fence, asynchronous):
        arrival_phase.append((node, bar, len(completed[bar])))
        phase_arrivals[bar].append((node, asynchronous or cta == bar[1], fence))
        left = pending.get(bar, counts[bar[0]]) - weight
        if left < 0:
            out.append(f"{G.label[node]}: beyond the count of {bar}")
        if left <= 0:
            done = G.node(f"{bar} phase {len(completed[bar])}", bar[1])
            far, arrivals = [], 0
            for a, plain, behind in phase_arrivals.pop(bar):
                arrivals |= 1 << a
                G.into[done].append(a)
                G.into_late[done].append(a)
                if plain:
                    G.into_cluster[done].append(a)
                elif behind is not None:
                    far.append(behind)
            completed[bar].append(done)
            foreign[bar].append(far)
            complete_with[bar].append(arrivals)
            left = counts[bar[0]]
        pending[bar] = left

    def access(node, buf, tag, write, ordinary):
        for b in _halves(buf):
            if write:
                content[b] = tag
            elif content.get(b) != tag:
                out.append(f"{G.label[node]} read {b} expecting {tag}, found {content.get(b)}")
            accesses[b].append((node, write, ordinary))

    pc = {a: 0 for a in progs}
    last: Dict[str, int] = {a: G.node(a, r) for a, (r, _) in progs.items()}
    fences: Dict[str, int] = {}
    last_tc = None
    moved = True
    while moved:
        moved = False
        for a, (r, ops) in progs.items():
            if pc[a] >= len(ops):
                continue
            op = ops[pc[a]]
            name = f"{a} {op[0]} {op[1] if op[0] != 'tc' else op[2]}"
            if op[0] == "wait":
                bar, done = op[1], len(completed[op[1]])
                if (done & 1) == op[2]:
                    continue
                node = G.node(name, r, last[a])
                if done:
                    G.into[node].append(completed[bar][-1])
                    G.into_cluster[node].append(completed[bar][-1])
                    if op[3]:
                        G.into_cluster[node] += foreign[bar][-1]
                waits.append((node, bar, done))
            elif op[0] == "fence":
                node = fences[a] = G.node(name, r, last[a])
            elif op[0] == "drained":
                node = G.node(name, r, last[a], copies[op[1]])
            elif op[0] == "arrive":
                node = G.node(name, r, last[a])
                arrive(op[1], node, op[2], r, fences.get(a), False)
            elif op[0] in ("read", "write"):
                node = G.node(name, r, last[a])
                access(node, op[1], op[2], op[0] == "write", not op[1][0].startswith(("T1", "T2", "acc")))
            elif op[0] == "copy":
                node = G.node(name, r, last[a])
                run = G.node(f"{a} copy {op[1]} -> {op[2]}", r, node)
                for b, t in op[1]:
                    access(run, b, t, False, False)
                for b, t in op[2]:
                    access(run, b, t, True, False)
                if op[3] is not None:
                    arrive(op[3], run, 1, r, None, True)
                if op[4] is not None:
                    copies[op[4]] = run
            else:
                node = G.node(name, r, last[a])
                last_tc = G.node(f"tensor core {op[2][0] if op[2] else op[3][0]}", r, node, last_tc)
                for b, t in op[1]:
                    access(last_tc, b, t, False, False)
                for b, t in op[2]:
                    access(last_tc, b, t, True, False)
                for bar in op[3]:
                    arrive(bar, last_tc, 1, r, None, True)
            last[a] = node
            pc[a] += 1
            moved = True
    stuck = [f"{a} at {ops[pc[a]]}" for a, (_, ops) in progs.items() if pc[a] < len(ops)]
    if stuck:
        return out + ["deadlock: " + ", ".join(stuck)]

    # reachability as bit sets; a node's number is above those of its predecessors
    def reach(into):
        before = [0] * len(into)
        for i, preds in enumerate(into):
            for p in preds:
                before[i] |= before[p] | (1 << p)
        return before

    all_before, cluster_before = reach(G.into), reach(G.into_cluster)
    late_before = [0] * len(G.into)
    for i, preds in enumerate(G.into_late):
        for p in preds:
            late_before[i] |= all_before[p] | (1 << p)

    def known(node, bar, k):        # every arrival of phase k comes before the node looks at the barrier
        return complete_with[bar][k] & ~late_before[node] == 0

    for node, bar, k in arrival_phase:
        if k > 0 and not known(node, bar, k - 1):
            out.append(f"{G.label[node]} for phase {k} may come before phase {k - 1} of {bar} has completed")
    for node, bar, done in waits:
        if done >= 2 and not known(node, bar, done - 2):
            out.append(f"{G.label[node]} may pass on phase {done - 3} of {bar} instead of {done - 1}")
        if done < len(completed[bar]) and not all_before[completed[bar][done]] >> node & 1:
            out.append(f"{G.label[node]} may miss phase {done - 1} of {bar}")
    for buf, list_ in accesses.items():
        for j, (b, wb, _) in enumerate(list_):
            for a, wa, ordinary in list_[:j]:
                if not (wa or wb) or a == b:
                    continue
                scoped = wa and ordinary and G.cta[a] != G.cta[b]
                if not (cluster_before if scoped else all_before)[b] >> a & 1:
                    out.append(f"{G.label[a]} and {G.label[b]} are not ordered on {buf}" + (" at cluster scope" if scoped else ""))
    return sorted(set(out))
