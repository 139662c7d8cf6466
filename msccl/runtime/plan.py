"""Compile a validated MSCCL-IR program into the flat device arrays the executor kernel reads.

Layout contract: ``csrc/msccl_device.h`` (``DevTb`` 64 bytes, ``DevStep`` 32 bytes).  Aliases of
the in-place collectives are resolved here, so the kernel sees plain (buffer, chunk) pairs.

Besides the translation, three analyses run here:

* **direct stores** - the k-th send of a connection is matched with the k-th receive on the peer.  When that
  receive is ``r`` or ``rcs`` the send is marked ``SF_DIRECT_SEND`` with the receiver's slot, and the receive
  ``SF_DIRECT_RECV``: on registered (symmetric) memory the sender then stores into the final slot and only the
  flag travels through the connection (the receive semantics of ``r`` / ``rcs``, reference
  ``msccl/language/rank_dag.py:128-154``).  ``rrc`` / ``rrs`` / ``rrcs`` keep the FIFO: the receiver has to add.
* **opening receive slots** - a sender may only store into a slot once nothing on the receiving GPU touches it
  any more before the receive.  For every receive the earliest such point is worked out from program order and
  the ``depid/deps`` edges: the start of the iteration (nothing touches the slot before the receive), the end of
  an earlier step of the same threadblock (the last one that touches it), or the receive step itself.  A tile
  whose slot is not yet open when the sender gets to it simply takes the FIFO, so this never adds a wait.
* **batched reduces** - a run of ``re`` steps into one destination (with the ``nop`` steps that carry their extra
  dependencies, reference ``msccl/language/ir.py:264-291``) becomes one multi-input add with one store.
"""
import struct
from collections import Counter
from dataclasses import dataclass, field, replace
from itertools import count
from typing import Dict, List

from msccl.xml.loader import AlgoIR, StepIR, TbIR
from msccl.xml.validator import validate

STEP_CODES = {'nop': 0, 's': 1, 'r': 2, 'rcs': 3, 'rrs': 4, 'rrc': 5, 'rrcs': 6, 'cpy': 7, 're': 8}
BUF_CODES = {'i': 0, 'o': 1, 's': 2}
PROTO_CODES = {'Simple': 0, 'LL': 1, 'LL128': 2}
K_MAX_RANKS = 16
K_MAX_CHANNELS = 128
K_MAX_TBS = 128
K_FIFO_SLOTS = 4
K_MAX_BATCH = 8                 # `re` steps fused into one pass (csrc/msccl_device.h kMaxBatch)
K_MAX_STEPS_PER_TB = 4094       # the progress word keeps 12 bits of step + 1 ...
K_MAX_ITERATIONS = 1 << 20      # ... and 20 bits of iteration
SF_DIRECT_SEND, SF_DIRECT_RECV, SF_DIRECT_ALWAYS = 1, 2, 4
_TB = struct.Struct('<4h4i2i2q4i')
_STEP = struct.Struct('<4B2h3i4Bi2H')
assert _TB.size == 64 and _STEP.size == 32


class PlanError(ValueError):
    pass


@dataclass
class HostPlan:
    """Host-side description of a compiled program for a set of local ranks."""
    algo: AlgoIR
    local_ranks: List[int]
    tb_bytes: bytes = b''
    step_bytes: bytes = b''
    first_tb: Dict[int, int] = field(default_factory=dict)     # rank -> index of its first tb
    num_tbs: Dict[int, int] = field(default_factory=dict)
    in_conns: int = 0              # most incoming connections of any rank
    max_cnt: int = 1
    proto: int = 0
    extents: Dict[int, Dict[str, int]] = field(default_factory=dict)   # rank -> physical buffer -> chunks used
    direct_bufs: Dict[int, set] = field(default_factory=dict)          # rank -> buffers ('i','o','s') that direct stores land in
    direct_steps: int = 0          # send steps that may store straight into the receiver's slot
    eager_tbs: int = 0             # threadblocks whose receives are all opened at kernel start
    batched_steps: int = 0         # `re` steps folded into a multi-input add
    single_hop: bool = False       # every tile is stored straight into its final slot and no step waits for another's tile

    def total_tbs(self):
        return sum(self.num_tbs[r] for r in self.local_ranks)


def fifo_index_tables(algo: AlgoIR):
    """For every rank, the incoming connections (src, chan) in a fixed order.  The position of a
    connection in this list selects its slots inside the receiver's FIFO area; sender and
    receiver derive the same table from the same XML."""
    incoming = {g.id: set() for g in algo.gpus}
    for g in algo.gpus:
        for tb in g.tbs:
            if tb.recv != -1 and any(st.is_recv() for st in tb.steps):
                incoming[g.id].add((tb.chan, tb.recv))
    return {r: {conn: i for i, conn in enumerate(sorted(conns))} for r, conns in incoming.items()}


def _match_connections(algo: AlgoIR):
    """Pair the k-th send of every connection with the k-th receive on the peer.  Returns
    ``{(rank, tb index, step index): (peer rank, peer tb index, peer step index)}`` for both directions."""
    sends, recvs = {}, {}
    for g in algo.gpus:
        for ti, tb in enumerate(g.tbs):
            for si, st in enumerate(tb.steps):
                if st.is_send() and tb.send != -1:
                    sends.setdefault((g.id, tb.send, tb.chan), []).append((g.id, ti, si))
                if st.is_recv() and tb.recv != -1:
                    recvs.setdefault((tb.recv, g.id, tb.chan), []).append((g.id, ti, si))
    match = {}
    for conn, ss in sends.items():
        rr = recvs.get(conn, [])
        for a, b in zip(ss, rr):
            match[a] = b
            match[b] = a
    return match


def _slots(algo, rank, st):
    """Resolved (buffer, first chunk, count) ranges a step reads or writes on its own GPU."""
    out = []
    if st.type == 'nop':
        return out
    if st.type in ('s', 'cpy', 're'):
        b, o = algo.resolve(rank, st.srcbuf, st.srcoff)
        out.append((b, o, st.cnt))
    if st.type != 's':
        b, o = algo.resolve(rank, st.dstbuf, st.dstoff)
        out.append((b, o, st.cnt))
    return out


def _open_positions(algo: AlgoIR, match):
    """For every threadblock with receives: ``{(rank, tb index): (opens_at_start, {step: opens_after},
    {step: opens_before}, nrecv, bufmask)}``.

    Position of a receive R at step ``si``: 0 when no step of the GPU touches R's slots unless it is ordered after R;
    ``k + 1`` ("after step k") when all such steps are earlier steps of R's own threadblock, k the last of them;
    otherwise R opens the slots itself when it is reached (after its dependency wait: the other threadblocks'
    accesses must be ordered before it by ``depid/deps``, which the FIFO path relies on just the same).  Slots are
    opened in receive order, so a receive never opens before its predecessors on the connection."""
    result = {}
    for g in algo.gpus:
        rank = g.id
        index_of = {tb.id: ti for ti, tb in enumerate(g.tbs)}
        # successors in the happens-before graph of this GPU: program order plus dependency edges
        waiters = {}
        for ti, tb in enumerate(g.tbs):
            for si, st in enumerate(tb.steps):
                if st.depid >= 0 and st.depid in index_of:
                    waiters.setdefault((index_of[st.depid], st.deps), []).append((ti, si))
        touched = {}
        for ti, tb in enumerate(g.tbs):
            for si, st in enumerate(tb.steps):
                for b, o, c in _slots(algo, rank, st):
                    for k in range(o, o + c):
                        touched.setdefault((b, k), []).append((ti, si))

        def after(ti, si):
            """Earliest step index per threadblock that is ordered after (ti, si)."""
            first = {ti: si + 1}
            todo = [(ti, si)]
            while todo:
                t, s0 = todo.pop()
                for s in range(s0, len(g.tbs[t].steps)):
                    for (t2, s2) in waiters.get((t, s), []):
                        if s2 < first.get(t2, 1 << 30):
                            first[t2] = s2
                            todo.append((t2, s2))
            return first

        for ti, tb in enumerate(g.tbs):
            recv_steps = [(si, st) for si, st in enumerate(tb.steps) if st.is_recv()]
            if not recv_steps or tb.recv == -1:
                continue
            running, at_start, opens_after, opens_before, mask = 0, 0, {}, {}, 0
            for si, st in recv_steps:
                own = 0                               # encoded: 2k = after step k-1 (0: iteration start), 2si+1 = at step si
                capable = st.type in ('r', 'rcs') and (rank, ti, si) in match
                if capable:
                    b, o = algo.resolve(rank, st.dstbuf, st.dstoff)
                    mask |= 1 << BUF_CODES[b]
                    later = after(ti, si)
                    for k in range(o, o + st.cnt):
                        for (t2, s2) in touched.get((b, k), []):
                            if (t2, s2) == (ti, si) or s2 >= later.get(t2, 1 << 30):
                                continue
                            if t2 == ti:
                                own = max(own, 2 * (s2 + 1))
                            else:
                                own = max(own, 2 * si + 1)
                running = max(running, own)
                if running == 0:
                    at_start += 1
                elif running % 2 == 0:
                    opens_after[running // 2 - 1] = opens_after.get(running // 2 - 1, 0) + 1
                else:
                    opens_before[running // 2] = opens_before.get(running // 2, 0) + 1
            result[(rank, ti)] = (at_start, opens_after, opens_before, len(recv_steps), mask)
    return result


def _batches(tb):
    """``{first step index: number of steps}`` for runs of ``re`` steps into one destination (``nop`` steps may sit
    between them) that the kernel executes as one multi-input add: it waits for everything the steps wait for, then adds.
    So behind a step that somebody waits for no step of the run may wait: what it waits for could be ordered after that step
    (the source refilled, say, once the first add has read it), and the add would wait for itself."""
    out = {}
    steps = tb.steps
    i = 0
    while i < len(steps):
        st = steps[i]
        if st.type != 're':
            i += 1
            continue
        j, last_re, sources, awaited = i + 1, i, 1, False
        srcs = {(st.srcbuf, st.srcoff)}
        while j < len(steps) and sources < K_MAX_BATCH and j - i < 2 * K_MAX_BATCH:
            nx = steps[j]
            awaited = awaited or steps[j - 1].hasdep
            if awaited and nx.depid >= 0:
                break
            if nx.type == 'nop':
                j += 1
                continue
            same_dst = nx.type == 're' and (nx.dstbuf, nx.dstoff, nx.cnt, nx.part, nx.parts) == (st.dstbuf, st.dstoff, st.cnt, st.part, st.parts)
            # a source that overlaps the destination must see the partial sum of the steps before it: not batched
            overlaps = nx.type == 're' and nx.srcbuf == st.dstbuf and nx.srcoff < st.dstoff + st.cnt and st.dstoff < nx.srcoff + nx.cnt
            if not same_dst or overlaps:
                break
            srcs.add((nx.srcbuf, nx.srcoff))
            last_re, sources = j, sources + 1
            j += 1
        if sources > 1:
            out[i] = last_re - i + 1
            i = last_re + 1
        else:
            i += 1
    return out


_NOP = StepIR(0, 'nop', 'i', -1, 'o', -1, 0, -1, -1, False)


def occupy_idle_ranks(algo: AlgoIR) -> AlgoIR:
    """The program with a threadblock that does nothing on every rank that has none.  The last threadblock of a rank advances the
    rank's launch epoch, which the packet flags of LL and LL128 are made of: a rank that sat a launch out would never find the
    flags of its peers again."""
    if all(g.tbs for g in algo.gpus):
        return algo
    return replace(algo, gpus=[g if g.tbs else replace(g, tbs=[TbIR(0, -1, -1, 0, [replace(_NOP)])]) for g in algo.gpus])


def _dependencies_exist(gpu):
    """False: the validator will report the program, which is left as it is."""
    return all(st.depid < 0 or (st.depid < len(gpu.tbs) and 0 <= st.deps < len(gpu.tbs[st.depid].steps))
               for tb in gpu.tbs for st in tb.steps)


def split_copies(algo: AlgoIR, most_tbs: int) -> AlgoIR:
    """The program with local copies that nothing depends on in threadblocks of their own.

    A direct all-to-all or all-gather puts the copy of a rank's own block behind one of its sends: with a threadblock per
    connection that one moves twice as much as the others (8 ranks, 32 MB each: done at 133 us, the others at 80;
    101 us for the call with the copies apart, 140 before).  A copy may
    leave its threadblock when it waits for nothing, nobody waits for it, no step of its GPU writes its source and no other
    step touches its destination.  The input is not modified; unchanged if more than ``most_tbs`` threadblocks came out."""
    gpus, total = [], sum(len(g.tbs) for g in algo.gpus)
    for g in algo.gpus:
        gpu = replace(g, tbs=[replace(tb, steps=[replace(st) for st in tb.steps]) for tb in g.tbs])
        gpus.append(gpu)
        if any(tb.id != i for i, tb in enumerate(gpu.tbs)) or not _dependencies_exist(gpu):
            continue
        steps = [(t, i, st) for t, tb in enumerate(gpu.tbs) for i, st in enumerate(tb.steps)]
        waited = {(st.depid, st.deps) for _, _, st in steps if st.depid >= 0}
        written, touched = Counter(), Counter()
        for _, _, st in steps:
            if st.type not in ('s', 'nop'):
                b, o = algo.resolve(gpu.id, st.dstbuf, st.dstoff)
                written.update((b, k) for k in range(o, o + st.cnt))
            touched.update((b, k) for b, o, c in _slots(algo, gpu.id, st) for k in range(o, o + c))
        moved = {}
        for t, i, st in steps:
            if st.type != 'cpy' or st.depid >= 0 or st.hasdep or (t, i) in waited or len(gpu.tbs[t].steps) - len(moved.get(t, ())) < 2:
                continue
            sb, so = algo.resolve(gpu.id, st.srcbuf, st.srcoff)
            db, do = algo.resolve(gpu.id, st.dstbuf, st.dstoff)
            if all(written[(sb, so + k)] == 0 and touched[(db, do + k)] == 1 for k in range(st.cnt)):
                moved.setdefault(t, []).append(i)
        for t, out in moved.items():
            tb = gpu.tbs[t]
            kept = [i for i in range(len(tb.steps)) if i not in out]
            renumber = {i: k for k, i in enumerate(kept)}
            for i in out:
                gpu.tbs.append(replace(tb, id=len(gpu.tbs), send=-1, recv=-1, chan=0, steps=[replace(tb.steps[i], s=0)]))
            tb.steps = [tb.steps[i] for i in kept]
            for other in gpu.tbs:
                for i, st in enumerate(other.steps):
                    st.s = i
                    if st.depid == t:
                        st.deps = renumber[st.deps]
    result = replace(algo, gpus=gpus)
    if result.num_threadblocks() == total or result.num_threadblocks() > most_tbs or result.max_tbs_per_gpu() > K_MAX_TBS:
        return algo
    return result


def _overlap(o1, c1, o2, c2):
    return o1 < o2 + c2 and o2 < o1 + c1


class _Node:
    """A step while its program is rewritten: its neighbours in the threadblock ``tb``, the step it waits for, the steps that wait
    for it, and a ``key`` that orders the steps of a threadblock."""
    __slots__ = ('st', 'tb', 'key', 'prev', 'next', 'dep', 'waiters')

    def __init__(self, st, tb, key):
        self.st, self.tb, self.key = st, tb, key
        self.prev = self.next = self.dep = None
        self.waiters = set()

    def wait_for(self, node):
        if self.dep is not None:
            self.dep.waiters.discard(self)
        self.dep = node
        if node is not None:
            node.waiters.add(self)

    def put_in_front(self, fresh):
        for node in fresh:
            node.prev, node.next = self.prev, self
            self.prev.next = self.prev = node

    def remove(self):
        self.prev.next = self.next
        self.next.prev = self.prev
        self.wait_for(None)


def _linked(gpu):
    """The steps of every threadblock as linked ``_Node``s: the end mark in front of each (another one is behind)."""
    fronts, rows = [], [[_Node(st, t, (i, 0, 0)) for i, st in enumerate(tb.steps)] for t, tb in enumerate(gpu.tbs)]
    for t, row in enumerate(rows):
        front, back = (_Node(replace(_NOP, type='end'), t, (i, 0, 0)) for i in (-1, len(row)))
        front.next, back.prev = back, front
        back.put_in_front(row)
        fronts.append(front)
        for node in row:
            if node.st.depid >= 0:
                node.wait_for(rows[node.st.depid][node.st.deps])
    return fronts


def _chain_to(end, slot, limit):
    """The chain of ``re`` steps into one slot, each in another threadblock and waiting for the one before, that ends with
    ``end`` and may run as one multi-input add at its place: ``[node, ...]``, or None.

    A link may be taken out of its threadblock when nobody but the next link waits for it and whatever follows it in
    its threadblock already waits for the end of the chain: then everything that was ordered after a link is ordered
    after the end, and everything that came before a link is waited for by the end."""
    def alone(node):                                            # not one of a run of adds in its threadblock
        return node.prev.st.type != 're'

    dst = slot(end.st, False)
    if end.st.type != 're' or end.next.st.type == 're':
        return None
    if any(x.st.type == 're' and x.tb != end.tb and slot(x.st, False) == dst and x.next.st.type != 're' for x in end.waiters):
        return None                                             # not the end of its chain
    chain = [end]
    while len(chain) < limit and alone(chain[0]):
        link = chain[0].dep
        if (link is None or any(link.tb == node.tb for node in chain) or link.st.type != 're' or slot(link.st, False) != dst or
                link.st.cnt != end.st.cnt or len(link.waiters) != 1 or not alone(link)):
            break
        behind = link.next
        if behind.st.type != 'end' and (behind.dep is None or behind.dep.tb != end.tb or behind.dep.key < end.key):
            break
        chain.insert(0, link)
    srcs = [slot(node.st, True) for node in chain]
    if len(chain) < 2 or any(b == dst[0] and _overlap(o, end.st.cnt, dst[1], end.st.cnt) for b, o in srcs):
        return None
    return chain


def _fold(chain, fresh_key):
    """Replace ``chain`` by one multi-input add of which each of its threadblocks does a part."""
    end = chain[-1]
    head, pred = {}, {}              # tb -> latest step that must be done before the first add / step that fills a source
    for k, link in enumerate(chain):
        waits = [link.dep] if k == 0 else []
        while link.prev.st.type == 'nop' and not link.prev.waiters and not link.prev.st.hasdep:
            waits.append(link.prev.dep)
            link.prev.remove()
        for dep in waits:
            if dep is not None and (dep.tb not in head or head[dep.tb].key < dep.key):
                head[dep.tb] = dep
        if link.prev.st.type != 'end':
            link.prev.st.hasdep = True
            pred[link.tb] = link.prev

    def nop(in_front_of, dep):
        node = _Node(replace(_NOP), in_front_of.tb, (in_front_of.key[0], in_front_of.key[1] - 1, fresh_key()))
        node.wait_for(dep)
        return node

    groups = []
    for k, link in enumerate(chain):
        first = {tb: dep for tb, dep in head.items() if tb != link.tb}
        adds = []
        for source in chain:
            add = _Node(replace(source.st, hasdep=False, part=k, parts=len(chain)), link.tb, (link.key[0], link.key[1], fresh_key()))
            dep = pred.get(source.tb) if source.tb != link.tb else None
            if dep is not None and source.tb in first:          # one wait per threadblock, the later of the two
                first[source.tb] = max(first[source.tb], dep, key=lambda node: node.key)
            else:
                add.wait_for(dep)
            adds.append(add)
        adds[-1].st.hasdep = True
        groups.append([nop(link, dep) for _, dep in sorted(first.items())] + adds)
    # whoever waited for the end, or came behind it, waits for every part (its own threadblock's is behind it anyway)
    last = {link.tb: group[-1] for link, group in zip(chain, groups)}
    for waiter in sorted(end.waiters, key=lambda node: (node.tb, node.key)):
        parts = [last[link.tb] for link in chain if link.tb != waiter.tb]
        waiter.put_in_front([nop(waiter, dep) for dep in parts[:-1]])
        waiter.wait_for(parts[-1])
    behind = end.next
    if behind.st.type != 'end':
        behind.put_in_front([nop(behind, last[link.tb]) for link in chain[:-1]])
    for link, group in zip(chain, groups):
        link.put_in_front(group)
        link.remove()


def fold_reduce_chains(algo: AlgoIR) -> AlgoIR:
    """The program with chains of local reduces that pass a slot from threadblock to threadblock (n - 1 hops of store,
    fence, flag and poll in the one-shot and two-shot all-reduce) replaced by one multi-input add - same operands, same
    order, same roundings - of which every threadblock of the chain does its part of each chunk.  Whoever waited for the
    end of the chain waits for all parts (two-shot all-reduce of 64 MB over 8 ranks: 848 us with the whole add in the last
    threadblock, 505 in parts).  The input is not modified; a GPU whose threadblocks would get more steps than the interpreter
    takes keeps its chains.  The time grows with the number of steps only, which a program may have thousands of."""
    gpus, changed = [], False
    for g in algo.gpus:
        gpus.append(g)
        gpu = replace(g, tbs=[replace(tb, steps=[replace(st) for st in tb.steps]) for tb in g.tbs])
        if any(tb.id != i for i, tb in enumerate(gpu.tbs)) or not _dependencies_exist(gpu):
            continue
        fronts = _linked(gpu)

        def slot(st, src):
            return algo.resolve(g.id, st.srcbuf, st.srcoff) if src else algo.resolve(g.id, st.dstbuf, st.dstoff)

        fresh_key, found, more = count(1).__next__, False, True
        while more:
            more = False
            for front in fronts:
                node = front.next
                while node.st.type != 'end':
                    behind = node.next
                    chain = _chain_to(node, slot, K_MAX_BATCH)
                    if chain is not None:
                        _fold(chain, fresh_key)
                        found = more = True
                    node = behind
        if not found:
            continue
        for tb, front in zip(gpu.tbs, fronts):
            tb.steps, node = [], front.next
            while node.st.type != 'end':
                node.st.s, node.key = len(tb.steps), len(tb.steps)
                tb.steps.append(node)
                node = node.next
        for tb in gpu.tbs:
            for node in tb.steps:
                node.st.depid, node.st.deps = (-1, -1) if node.dep is None else (node.dep.tb, node.dep.key)
            tb.steps = [node.st for node in tb.steps]
        if max(len(tb.steps) for tb in gpu.tbs) <= K_MAX_STEPS_PER_TB:
            gpus[-1], changed = gpu, True
    return replace(algo, gpus=gpus) if changed else algo


def compile_plan(algo: AlgoIR, local_ranks, slot_bytes: int, check=True, direct=True, batch=True) -> HostPlan:
    if check:
        problems = validate(algo)
        if problems:
            raise PlanError('invalid MSCCL-IR: ' + '; '.join(problems[:5]))
    if algo.proto not in PROTO_CODES:
        raise PlanError(f'unknown protocol {algo.proto}')
    if algo.ngpus > K_MAX_RANKS:
        raise PlanError(f'{algo.ngpus} ranks exceed the executor limit of {K_MAX_RANKS}')
    if algo.nchannels > K_MAX_CHANNELS:
        raise PlanError(f'{algo.nchannels} channels exceed the executor limit of {K_MAX_CHANNELS}')
    if algo.max_tbs_per_gpu() > K_MAX_TBS:
        raise PlanError(f'{algo.max_tbs_per_gpu()} threadblocks per GPU exceed the executor limit of {K_MAX_TBS}')
    longest = max((len(tb.steps) for g in algo.gpus for tb in g.tbs), default=0)
    if longest > K_MAX_STEPS_PER_TB:
        raise PlanError(f'a threadblock has {longest} steps, the executor handles at most {K_MAX_STEPS_PER_TB}')
    tables = fifo_index_tables(algo)
    plan = HostPlan(algo, list(local_ranks), proto=PROTO_CODES[algo.proto], max_cnt=max(algo.max_count(), 1),
                    in_conns=max((len(t) for t in tables.values()), default=0))
    simple = algo.proto == 'Simple'
    match = _match_connections(algo) if (direct and simple) else {}
    opens = _open_positions(algo, match) if match else {}
    for r in range(algo.ngpus):
        plan.direct_bufs[r] = set()
    plan.single_hop = simple
    stride = K_FIFO_SLOTS * slot_bytes
    tb_blob, step_blob = [], []
    nsteps_total = 0
    for rank in plan.local_ranks:
        gpu = algo.gpus[rank]
        plan.first_tb[rank] = len(tb_blob)
        plan.num_tbs[rank] = len(gpu.tbs)
        used = {'i': 0, 'o': 0, 's': 0}
        for ti, tb in enumerate(gpu.tbs):
            sends = any(st.is_send() for st in tb.steps)
            recvs = any(st.is_recv() for st in tb.steps)
            send_peer = tb.send if sends else -1
            recv_peer = tb.recv if recvs else -1
            send_conn = tb.chan * K_MAX_RANKS + send_peer if sends else -1
            recv_conn = tb.chan * K_MAX_RANKS + recv_peer if recvs else -1
            send_off = tables[send_peer][(tb.chan, rank)] * stride if sends else 0
            recv_off = tables[rank][(tb.chan, recv_peer)] * stride if recvs else 0
            batches = _batches(tb) if batch else {}
            at_start, opens_after, opens_before, _, recv_mask = opens.get((rank, ti), (0, {}, {}, 0, 0))
            nrecv = sum(1 for st in tb.steps if st.is_recv()) if recvs else 0
            packed = []
            for si, st in enumerate(tb.steps):
                if st.type not in STEP_CODES:
                    raise PlanError(f'step type {st.type!r} is not executable by the interpreter kernel')
                flags, rbuf, roff = 0, 0, 0
                if st.type == 'nop':
                    sbuf, soff, dbuf, doff, cnt = 'i', 0, 'i', 0, 0
                else:
                    # local operand of receive-type steps is dst; src of s/cpy/re is local too
                    sbuf, soff = algo.resolve(rank, st.srcbuf, st.srcoff)
                    dbuf, doff = algo.resolve(rank, st.dstbuf, st.dstoff)
                    cnt = st.cnt
                    if st.type in ('s', 'cpy', 're'):
                        used[sbuf] = max(used[sbuf], soff + cnt)
                    if st.type != 's':
                        used[dbuf] = max(used[dbuf], doff + cnt)
                    if st.type in ('r', 'rcs', 'rrs', 'rrc', 'rrcs'):
                        sbuf, soff = 'i', 0       # the remote source slot is not addressed by the receiver
                    if st.type == 's':
                        dbuf, doff = 'i', 0       # nor the remote destination by the sender
                    peer = match.get((rank, ti, si))
                    if peer is not None and st.is_send():
                        pr, pt, ps = peer
                        other = algo.gpus[pr].tbs[pt].steps[ps]
                        if other.type in ('r', 'rcs') and other.cnt == st.cnt:
                            pb, po = algo.resolve(pr, other.dstbuf, other.dstoff)
                            flags |= SF_DIRECT_SEND
                            if opens[(pr, pt)][0] == opens[(pr, pt)][3]:
                                flags |= SF_DIRECT_ALWAYS
                            rbuf, roff = BUF_CODES[pb], po
                            plan.direct_bufs[pr].add(pb)
                            plan.direct_steps += 1
                    if peer is not None and st.type in ('r', 'rcs'):
                        pr, pt, ps = peer
                        if algo.gpus[pr].tbs[pt].steps[ps].cnt == st.cnt:
                            flags |= SF_DIRECT_RECV
                            plan.direct_bufs[rank].add(dbuf)
                if st.type not in ('s', 'r', 'cpy') or st.depid >= 0 or (st.type == 's' and (
                        not flags & SF_DIRECT_ALWAYS or any(x.type == 'r' for x in tb.steps[:si]))):
                    plan.single_hop = False
                nb = batches.get(si, 0)
                if nb:
                    plan.batched_steps += sum(1 for k in range(si, si + nb) if tb.steps[k].type == 're')
                packed.append(_STEP.pack(STEP_CODES[st.type], BUF_CODES[sbuf], BUF_CODES[dbuf], int(st.hasdep),
                                         st.depid, st.deps, soff, doff, cnt, flags, rbuf, nb,
                                         st.parts << 4 | st.part if st.parts > 1 else 0, roff,
                                         opens_after.get(si, 0), opens_before.get(si, 0)))
            if nrecv > 0 and recv_mask and at_start == nrecv:
                plan.eager_tbs += 1
            tb_blob.append(_TB.pack(rank, tb.id, send_peer, recv_peer, tb.chan, len(tb.steps), nsteps_total,
                                    len(gpu.tbs), send_conn, recv_conn, send_off, recv_off, at_start, recv_mask, nrecv, 0))
            step_blob.extend(packed)
            nsteps_total += len(tb.steps)
        plan.extents[rank] = used
    plan.tb_bytes = b''.join(tb_blob)
    plan.step_bytes = b''.join(step_blob)
    return plan


def chunk_geometry(algo: AlgoIR, rank: int, input_elems: int):
    """Elements per chunk for a call whose input on ``rank`` has ``input_elems`` elements."""
    g = algo.gpus[rank]
    if algo.inplace and algo.coll == 'allgather':
        chunks = g.o_chunks // algo.ngpus
    else:
        chunks = g.i_chunks
    if chunks <= 0 or input_elems % chunks != 0:
        raise PlanError(f'{input_elems} input elements are not divisible into {chunks} chunks')
    return input_elems // chunks


def access_width(chunk_elems: int, elem_size: int, pointers=()):
    """Bytes per access of the kernel: 16 when every chunk and buffer is a multiple of 16 bytes, else one element."""
    if (chunk_elems * elem_size) % 16 == 0 and all(p % 16 == 0 for p in pointers):
        return 16
    return elem_size


# One-GPU interpreter (csrc/exec_one_gpu.cu).  SLICE_BYTES: a CTA's share of a chunk below which another CTA only adds
# flags (all-reduce of 1 MB over 8 ranks, LL128: 31 us with 4 KB, 29 with 16 KB).  TILE_BYTES: what a slice moves between
# two signals of the Simple protocol; a hop costs a few microseconds beside the movement (256 MB ring all-reduce over 8
# ranks, four slices per CTA: 1.90 ms with 32 KB, 1.56 with 64 KB, 1.52 with 128 KB).  STREAMS: 2.35 ms with one slice per
# CTA, 1.77 with two, 1.52 with four, 1.53 with eight.
ONE_GPU_SLICE_BYTES = 16 << 10
ONE_GPU_TILE_BYTES = 128 << 10
ONE_GPU_STREAMS = 4
K_ONE_GPU_CHANNELS = 1024       # channels x slices that have flags of their own (csrc/msccl_device.h)
K_ONE_GPU_PROGRESS = 4096       # threadblocks of a rank x slices


def one_gpu_geometry(plan: HostPlan, chunk_elems: int, elem_size: int, slot_bytes: int, width: int, proto: int, max_ctas: int,
                     direct=True):
    """(CTAs per threadblock, slices per CTA, slice_elems, tile_elems, slot bytes of a slice) of a launch with every rank
    on one GPU.

    Each chunk is cut into slices of ``slice_elems`` elements (whole 128-byte lines) that run independently of each
    other: as many CTAs per threadblock as fit on the GPU at once, have flags of their own and are worth a CTA, and under
    the Simple protocol up to four slices per CTA as long as each has a whole tile.  A slice moves in tiles of
    ``tile_elems`` through its own FIFO slots; in one tile when every tile is stored straight into its final slot and no
    step waits for it (all-to-all of 32 MB, copies still behind sends: 153 us in tiles of 128 KB, 141 whole)."""
    per_access = width // elem_size
    if chunk_elems < 1:
        raise PlanError('the buffers hold less than one element per chunk')
    if (chunk_elems * elem_size) % width:
        raise PlanError(f'chunks of {chunk_elems * elem_size} bytes are not whole {width}-byte accesses')
    tbs = max(plan.total_tbs(), 1)
    chans = 1 + max((tb.chan for g in plan.algo.gpus for tb in g.tbs), default=0)
    fifo_bytes = {0: width, 1: 32 if width == 16 else 8, 2: 128}[proto]          # one access (LL128: one line) in the FIFO
    least_slot = max(1024, 128 * -(-plan.max_cnt * fifo_bytes // 128))
    most = min(K_ONE_GPU_CHANNELS // chans, K_ONE_GPU_PROGRESS // max(plan.algo.max_tbs_per_gpu(), 1), slot_bytes // least_slot)
    chunk_bytes = chunk_elems * elem_size
    ctas = max(1, min(max_ctas // tbs, most, -(-chunk_bytes // ONE_GPU_SLICE_BYTES)))
    streams = 1
    while proto == 0 and not (plan.single_hop and direct) and streams < ONE_GPU_STREAMS and 2 * streams * ctas <= most and \
            chunk_bytes >= 2 * streams * ctas * ONE_GPU_TILE_BYTES:
        streams *= 2
    line = max(per_access, 128 // elem_size)
    slice_elems = -(-(-(-chunk_elems // (ctas * streams))) // line) * line
    ctas = max(1, -(-chunk_elems // (slice_elems * streams)))
    slot = slot_bytes // (ctas * streams) // 128 * 128
    if proto == 2:
        tile = slot // 128 // plan.max_cnt * 15 // 2 * per_access                # 15 units of 8 bytes per line
    else:
        tile = slot // (plan.max_cnt * fifo_bytes) * per_access
    if tile <= 0:
        raise PlanError('FIFO slot too small for this program')
    if proto == 0 and not (plan.single_hop and direct):
        want = max(per_access, ONE_GPU_TILE_BYTES // plan.max_cnt // elem_size // line * line)
        least = -(-slice_elems // (K_MAX_ITERATIONS - 1))                        # fewer would be too many iterations
        want = max(want, -(-least // per_access) * per_access)
        tile = min(tile, want)
    tile = min(tile, slice_elems)
    if -(-slice_elems // tile) >= K_MAX_ITERATIONS:
        raise PlanError(f'{-(-slice_elems // tile)} iterations through FIFO slots of {slot} bytes exceed the executor limit '
                        f'of {K_MAX_ITERATIONS}: use a larger FIFO area')
    return ctas, streams, slice_elems, tile, slot


def tile_geometry(plan: HostPlan, chunk_elems: int, elem_size: int, slot_bytes: int, width: int = 16, proto=None):
    """(tile_elems, iterations): how many elements of each chunk one iteration moves so that the
    largest step (max_cnt chunks) fits into one FIFO slot.  ``width`` is the access size in bytes
    (``access_width``); ``proto`` overrides the plan's protocol (LL128 programs whose chunks are not
    multiples of 16 bytes run as LL)."""
    proto = plan.proto if proto is None else proto
    per_access = width // elem_size
    if (chunk_elems * elem_size) % width:
        raise PlanError(f'chunks of {chunk_elems * elem_size} bytes are not whole {width}-byte accesses')
    if proto == 2:
        if width != 16:
            raise PlanError('LL128 needs chunks that are multiples of 16 bytes')
        lines = slot_bytes // 128 // plan.max_cnt             # 15 units of 8 bytes per 128-byte line
        tile = (lines * 15 // 2) * per_access
    else:
        fifo_bytes = width if proto == 0 else (32 if width == 16 else 8)
        tile = slot_bytes // (plan.max_cnt * fifo_bytes) * per_access
    if tile <= 0:
        raise PlanError('FIFO slot too small for this program')
    if proto == 0:
        # Simple: a receiver starts on a tile only when the whole tile has landed, so a chunk is cut
        # into at least four tiles (of 256 KB or more) to overlap the two sides.
        quarter = -(-chunk_elems // 4)
        want = max((256 << 10) // (plan.max_cnt * elem_size), quarter)
        want = -(-want // per_access) * per_access
        tile = min(tile, want)
    tile = min(tile, chunk_elems)
    iterations = -(-chunk_elems // tile)
    if iterations >= K_MAX_ITERATIONS:
        raise PlanError(f'{iterations} iterations through FIFO slots of {slot_bytes} bytes exceed the executor limit '
                        f'of {K_MAX_ITERATIONS}: use a larger FIFO area')
    return tile, iterations
