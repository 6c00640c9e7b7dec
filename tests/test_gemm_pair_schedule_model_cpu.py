"""Host-side models of the CTA-pair GEMM (``gemm_bf16_tcgen05_pair_kernel`` in ``csrc/gemm_tcgen05.cu``) with either tile height:
how tile indices, operand stages and accumulators go round between two producers, the MMA warp and the epilogues of both CTAs.

Two things are looked at.  Every interleaving of a small launch is explored (``explore`` of the attention kernels' models): no
deadlock, no wait that passes on an older phase, and no stage, slot or accumulator that is overwritten or read too early.  And the
order is looked at as the PTX memory model grants it: an arrival and a wait order the accesses of two CTAs only if both are of
cluster scope.  Any two accesses to a tile index or an accumulator, one of them a write, have to be ordered that way.
"""
import random

import pytest
from test_attention_schedule_model_cpu import explore

DEPTH = 2  # slots of a CTA's ring (the kernel has four)

# How each signal that crosses the pair is given and awaited; everything else is of CTA scope, within one CTA.
KERNEL = {"mail_full": ("cluster", "cluster"), "mail_empty": ("cluster", "cluster"), "tmem_empty": ("relaxed", "relaxed")}


def pair_programs(row_blocks, tiles, num_kb, stages, drop=(), publish_kb=None):
    """Programs as ``explore`` takes them: ``row_blocks`` 1, tiles of 256 rows with two accumulators; 2, tiles of 512 rows.
    The next index is handed on behind the first ``publish_kb`` loads of a tile, a ring of them unless given."""
    prods, mma, epis = ([], []), [], ([], [])
    publish_kb = min(num_kb, stages) if publish_kb is None else publish_kb
    order = list(range(tiles)) + [-1]
    need = {f"full{s}": 2 for s in range(stages)}  # the bytes of both CTAs
    need.update({f"tmem_empty{a}": 2 for a in (0, 1)})  # an epilogue of each CTA
    need.update({f"slot_empty0{q}": 2 for q in range(DEPTH)})  # the leader's MMA warp and epilogue; the peer has the epilogue only
    for c, prog in enumerate(prods):

        def publish(i):
            q = i % DEPTH
            if "slot_empty" not in drop:
                prog.append(("wait", f"slot_empty{c}{q}", ((i // DEPTH) & 1) ^ 1, i // DEPTH))
            prog.extend([("write", f"slot{c}{q}", order[i]), ("arrive", f"slot_full{c}{q}")])

        def hand_on(i):
            if c == 0:
                publish(i)
                if "mail_empty" not in drop:
                    prog.append(("wait", "mail_empty", (i & 1) ^ 1, i))
                prog.append(("load", "mail", order[i], "mail_full"))  # st.async: lands when it lands
            else:
                prog.extend([("wait", "mail_full", i & 1, i + 1), ("read", "mail", order[i]), ("arrive", "mail_empty")])
                publish(i)

        def blocks(i, lo, hi):
            for kb in range(lo, hi):
                n = i * num_kb + kb
                s = n % stages
                prog.extend([("wait", f"empty{c}{s}", ((n // stages) & 1) ^ 1, n // stages), ("load", f"ops{c}{s}", (i, kb), f"full{s}")])

        hand_on(0)
        for i in range(tiles):
            blocks(i, 0, publish_kb)
            hand_on(i + 1)
            blocks(i, publish_kb, num_kb)

    def take(prog, c, i):
        q = i % DEPTH
        prog.extend([("wait", f"slot_full{c}{q}", (i // DEPTH) & 1, i // DEPTH + 1), ("read", f"slot{c}{q}", order[i]), ("arrive", f"slot_empty{c}{q}")])

    for i in range(tiles + 1):
        take(mma, 0, i)
        for c in (0, 1):
            take(epis[c], c, i)
        if i == tiles:
            break
        uses = [(0, i & 1, i >> 1)] if row_blocks == 1 else [(0, 0, i), (1, 1, i)]  # row block, accumulator, how often it was used before
        for kb in range(num_kb):
            n = i * num_kb + kb
            s = n % stages
            if row_blocks == 1 and kb == 0 and "tmem_empty" not in drop:
                mma.append(("wait", f"tmem_empty{uses[0][1]}", (uses[0][2] & 1) ^ 1, uses[0][2]))
            mma.append(("wait", f"full{s}", (n // stages) & 1, n // stages + 1))
            for h, acc, used in uses:
                if row_blocks == 2 and kb == 0 and "tmem_empty" not in drop:
                    mma.append(("wait", f"tmem_empty{acc}", (used & 1) ^ 1, used))
                mma.append(("mma", ((f"ops0{s}", (i, kb)), (f"ops1{s}", (i, kb))), f"acc{acc}", (i, h, kb)))
                if kb == num_kb - 1:
                    mma.extend(("commit", f"tmem_full{c}{acc}") for c in (0, 1))
            mma.extend(("commit", f"empty{c}{s}") for c in (0, 1))
        for c in (0, 1):
            for h, acc, used in uses:
                epis[c].extend([("wait", f"tmem_full{c}{acc}", used & 1, used + 1), ("read", f"acc{acc}", (i, h, num_kb - 1)), ("arrive", f"tmem_empty{acc}")])
    return [*prods, mma, *epis], need


# K blocks against stages: fewer, as many, more (the ring wraps within a tile and across tiles)
SHAPES = [(1, 3, 1, 2), (1, 2, 2, 2), (1, 2, 3, 2), (2, 3, 1, 1), (2, 2, 2, 2), (2, 2, 3, 2)]


@pytest.mark.parametrize("row_blocks,tiles,num_kb,stages", SHAPES)
def test_pair_schedule_is_safe_and_live(row_blocks, tiles, num_kb, stages):
    problems, deadlocks, states = explore(pair_programs(row_blocks, tiles, num_kb, stages))
    assert states > 100
    assert not problems and deadlocks == 0, (sorted(map(str, problems))[:3], deadlocks)


@pytest.mark.parametrize("row_blocks", [1, 2])
@pytest.mark.parametrize("mistake", ["slot_empty", "mail_empty", "tmem_empty"])
def test_model_notices_a_missing_wait(row_blocks, mistake):
    problems, deadlocks, _ = explore(pair_programs(row_blocks, 3, 1, 1, drop=(mistake,)))
    assert problems or deadlocks


# ---- the order that scopes grant
CTA_OF = [0, 1, 0, 0, 1]  # of the actors that pair_programs returns


def races(programs, signals, seed):
    """Pairs of accesses to an index or an accumulator that nothing orders, in one interleaving chosen by ``seed``.

    Vector clocks: a release of cluster scope, and what completes by itself (a remote store, a commit), reaches every waiter of
    cluster scope; one of CTA scope the waiters of its own CTA.  A relaxed signal of cluster scope orders accumulators only."""
    progs, need = programs
    rng = random.Random(seed)
    n = len(progs)
    zero = (0,) * (n + 1)  # the last component: the tensor pipe
    clocks = {k: [zero] * (n + 1) for k in ("mem", "tmem")}
    arrivals, given = {}, {}  # given: barrier -> clocks released to it, as (kind of place, scope, CTA, clock)
    pcs, pipe, flying, seen, found = [0] * n, [], [], {}, set()

    def join(a, b):
        return tuple(map(max, a, b))

    def tick(kind, who):
        c = clocks[kind][who]
        clocks[kind][who] = c[:who] + (c[who] + 1,) + c[who + 1:]
        return clocks[kind][who]

    def access(kind, who, place, write, now):
        for other, at, other_writes in seen.get(place, []):
            if (write or other_writes) and other != who and now[other] < at:
                found.add((place, other, who))
        seen.setdefault(place, []).append((who, now[who], write))

    def signal(bar, kind, scope, cta, clock):
        given.setdefault(bar, []).append((kind, scope, cta, clock))

    def crossing(bar, side):
        return next((v[side] for k, v in signals.items() if bar.startswith(k)), "cta")

    while True:
        moves = [("run", a) for a in range(n) if pcs[a] < len(progs[a]) and
                 (progs[a][pcs[a]][0] != "wait" or arrivals.get(progs[a][pcs[a]][1], 0) // need.get(progs[a][pcs[a]][1], 1) >= progs[a][pcs[a]][3])]
        moves += [("land", i) for i in range(len(flying))] + ([("pipe", 0)] if pipe else [])
        if not moves:
            assert all(pcs[a] == len(progs[a]) for a in range(n))
            return found
        what, a = rng.choice(moves)
        if what == "land":
            place, bar, clock = flying.pop(a)
            arrivals[bar] = arrivals.get(bar, 0) + 1
            signal(bar, "mem", "cluster", None, clock)
        elif what == "pipe":
            op, issued = pipe.pop(0)
            clocks["tmem"][n] = join(clocks["tmem"][n], issued)
            if op[0] == "mma":
                access("tmem", n, op[2], True, tick("tmem", n))
            else:
                arrivals[op[1]] = arrivals.get(op[1], 0) + 1
                signal(op[1], "tmem", "cluster", None, clocks["tmem"][n])
        else:
            op = progs[a][pcs[a]]
            pcs[a] += 1
            if op[0] == "wait":
                scope = crossing(op[1], 1)
                for kind, rel, cta, clock in given.get(op[1], []):
                    ordered = (rel == "cluster" and scope == "cluster") or (cta == CTA_OF[a] and rel != "relaxed" and scope != "relaxed")
                    if kind == "tmem":  # fenced tcgen05 work: any signal whose scope reaches the waiter; a commit reaches both CTAs
                        ordered = cta is None or cta == CTA_OF[a] or (rel != "cta" and scope != "cta")
                    if ordered:
                        clocks[kind][a] = join(clocks[kind][a], clock)
            elif op[0] == "arrive":
                arrivals[op[1]] = arrivals.get(op[1], 0) + 1
                for kind in ("mem", "tmem"):
                    signal(op[1], kind, crossing(op[1], 0), CTA_OF[a], clocks[kind][a])
            elif op[0] in ("read", "write"):
                kind = "tmem" if op[1].startswith("acc") else "mem"
                access(kind, a, op[1], op[0] == "write", tick(kind, a))
            elif op[0] == "load":
                if op[1] == "mail":
                    access("mem", a, op[1], True, tick("mem", a))  # ordered behind what its sender has waited for
                flying.append((op[1], op[3], clocks["mem"][a]))
            else:
                pipe.append((op, tick("tmem", a)))


@pytest.mark.parametrize("row_blocks,tiles,num_kb,stages", SHAPES + [(1, 6, 3, 4), (2, 5, 3, 4)])
def test_accesses_across_the_pair_are_ordered(row_blocks, tiles, num_kb, stages):
    for seed in range(20):
        assert not races(pair_programs(row_blocks, tiles, num_kb, stages), KERNEL, seed)


@pytest.mark.parametrize("signal,weaker", [("mail_full", ("cluster", "cta")), ("mail_empty", ("cta", "cluster")), ("mail_empty", ("cluster", "cta")),
                                           ("tmem_empty", ("cta", "relaxed")), ("tmem_empty", ("relaxed", "cta"))])
def test_cta_scope_does_not_order_the_two_ctas(signal, weaker):
    """What the kernel gave its hand-out before: arrivals and waits of CTA scope between the CTAs."""
    assert any(races(pair_programs(1, 6, 3, 4), {**KERNEL, signal: weaker}, seed) for seed in range(20))


@pytest.mark.parametrize("row_blocks,tiles,num_kb,stages", [s for s in SHAPES if s[0] == 1] + [(1, 4, 1, 1)])
def test_indices_handed_on_before_the_loads_are_safe_and_live(row_blocks, tiles, num_kb, stages):
    """As the kernel does where the epilogue stores a row per thread."""
    programs = pair_programs(row_blocks, tiles, num_kb, stages, publish_kb=0)
    problems, deadlocks, states = explore(programs)
    assert states > 100
    assert not problems and deadlocks == 0, (sorted(map(str, problems))[:3], deadlocks)
    for seed in range(20):
        assert not races(programs, KERNEL, seed)
