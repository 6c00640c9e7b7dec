"""Exhaustive host-side models of the barrier schedules of the attention kernels: the ping-pong forward
(``csrc/attention_fwd_pingpong.cu``) with either head size, and the two backward kernels (``csrc/attention.cu``).

A model is a set of actors (TMA producer, MMA issuer, groups of softmax warps) that run straight-line programs and are
synchronised by phase-parity mbarriers exactly as in the kernel, plus TMA loads that land at arbitrary later times and the tensor
pipe, which executes what was issued in order, at arbitrary later times.  Every interleaving is explored.  Each piece of memory -
operand stages, score and probability columns, accumulators - carries the step that wrote it, and whoever reads one checks that
it holds the step it means, so a stage or a buffer that is overwritten too early, or read too early, shows as a wrong step in
some interleaving.  Checked besides: no deadlock, and no parity wait that passes on an older phase than the one the waiter means.

The programs cover several work items of one persistent CTA (the barriers' phases run through all of them), among them items
with a single query tile.
"""
import pytest


# Operations of a program:
#   ("wait", barrier, parity, meant)      meant: number of completed phases the waiter relies on
#   ("load", place, version, barrier)     a TMA load; completes a phase of the barrier when it lands
#   ("mma", reads, place, version)        queued on the tensor pipe; reads: ((place, version), ...)
#   ("commit", barrier)                   queued behind the products issued so far
#   ("read", place, version), ("write", place, version), ("arrive", barrier)
def forward_programs(items, sep, rescale, drop=()):
    """items: (n_a, has_b) per item - key tiles of the first query tile, is there a second one (which sees one tile more)."""
    producer, mma, softmax = [], [], ([], [])

    def s_place(t):
        return f"s{t}"

    def p_place(t):
        return f"p{t}" if sep else f"s{t}"

    kt = it_b = 0
    cs, ss = [0, 0], [0, 0]
    for it, (n_a, has_b) in enumerate(items):
        n_kv = n_a + 1 if has_b else n_a
        # ---- producer
        producer += [("wait", "q_empty", (it & 1) ^ 1, it), ("load", "q", it, "q_full")]
        for j in range(n_kv):
            k = kt + j
            st, par = k & 1, ((k >> 1) & 1) ^ 1
            producer += [("wait", f"k_empty{st}", par, k >> 1), ("load", f"k{st}", k, f"k_full{st}"),
                         ("wait", f"v_empty{st}", par, k >> 1), ("load", f"v{st}", k, f"v_full{st}")]

        # ---- MMA issuer
        def issue_s(t, j):
            k = kt + j
            mma.append(("wait", f"k_full{k & 1}", (k >> 1) & 1, (k >> 1) + 1))
            if sep and ss[t] > 0 and "s_read" not in drop:
                mma.append(("wait", f"s_read{t}", (ss[t] - 1) & 1, ss[t]))
            ss[t] += 1
            mma.extend([("mma", (("q", it), (f"k{k & 1}", k)), s_place(t), ("S", it, j)), ("commit", f"s_full{t}")])

        def issue_pv(t, j):
            k = kt + j
            mma.extend([("wait", f"p_full{t}", cs[t] & 1, cs[t] + 1),
                        ("mma", ((p_place(t), ("P", it, j)), (f"v{k & 1}", k)), f"o{t}", (it, j)), ("commit", f"o_done{t}")])
            cs[t] += 1

        mma.append(("wait", "q_full", it & 1, it + 1))
        issue_s(0, 0)
        if has_b:
            issue_s(1, 0)
        mma.append(("commit", f"k_empty{kt & 1}"))
        if n_kv == 1:
            mma.append(("commit", "q_empty"))
        for j in range(n_kv):
            k = kt + j
            mma.append(("wait", f"v_full{k & 1}", (k >> 1) & 1, (k >> 1) + 1))

            def next_scores(t_list):
                for t in t_list:
                    if t == 0 and j + 1 < n_a or t == 1 and has_b and j + 1 < n_kv:
                        issue_s(t, j + 1)
                if 1 in t_list and j + 1 < n_kv:
                    mma.append(("commit", f"k_empty{(k + 1) & 1}"))
                    if j + 2 == n_kv:
                        mma.append(("commit", "q_empty"))

            if sep:
                next_scores((0, 1))
            if j == 0:
                mma.append(("wait", "o_free0", (it & 1) ^ 1, it))
                if has_b:
                    mma.append(("wait", "o_free1", (it_b & 1) ^ 1, it_b))
            if "early_scores" in drop and not sep:  # in place, the next scores must not be issued ahead of the product
                next_scores((0,))
            if j < n_a:
                issue_pv(0, j)
                if not sep and "early_scores" not in drop:
                    next_scores((0,))
            if has_b:
                issue_pv(1, j)
            mma.append(("commit", f"v_empty{k & 1}"))
            if not sep:
                next_scores((1,))
        kt += n_kv
        it_b += has_b
    # ---- softmax groups
    for t in (0, 1):
        c = 0
        for it, (n_a, has_b) in enumerate(items):
            if t == 1 and not has_b:
                continue
            prog = softmax[t]
            for j in range(n_a + t):
                prog += [("wait", f"s_full{t}", c & 1, c + 1), ("read", s_place(t), ("S", it, j))]
                if j > 0 and (sep or rescale):
                    if "o_done" not in drop:
                        prog.append(("wait", f"o_done{t}", (c - 1) & 1, c))
                    if rescale:
                        prog.append(("read", f"o{t}", (it, j - 1)))
                if sep:
                    prog += [("write", p_place(t), ("half", it, j)), ("read", s_place(t), ("S", it, j)), ("arrive", f"s_read{t}")]
                prog += [("write", p_place(t), ("P", it, j)), ("arrive", f"p_full{t}")]
                c += 1
            prog += [("wait", f"o_done{t}", (c - 1) & 1, c), ("read", f"o{t}", (it, n_a + t - 1)), ("arrive", f"o_free{t}")]
    return [producer, mma, *softmax], {}


def backward_programs(items, nbuf, stages, steps_per_load, drop=()):
    """items: steps per item (even).  ``steps_per_load`` 2: the dQ kernel (a K / V tile of 128 keys in two steps), 1: the dK / dV
    kernel (a Q / dO sub-tile per step, whose statistics the softmax warps read from the same stage)."""
    producer, mma, sets = [], [], ([], [])
    jt0 = ut0 = 0
    for it, n in enumerate(items):
        producer += [("wait", "stat_empty", (it & 1) ^ 1, it), ("load", "stat", it, "stat_full")]
        for j in range(n // steps_per_load):
            jt = jt0 + j
            st = jt % stages
            producer += [("wait", f"str_empty{st}", ((jt // stages) & 1) ^ 1, jt // stages), ("load", f"str{st}", jt, f"str_full{st}")]

        def stage(u):
            jt = jt0 + u // steps_per_load
            return jt, jt % stages

        def issue_sp(u):
            jt, st = stage(u)
            buf = (ut0 + u) % nbuf
            if u % steps_per_load == 0:
                mma.append(("wait", f"str_full{st}", (jt // stages) & 1, jt // stages + 1))
            mma.extend([("mma", (("stat", it), (f"str{st}", jt)), f"buf{buf}", ("S", ut0 + u)), ("commit", f"s_full{buf}")])
            if u == n - 1:
                mma.append(("commit", "stat_empty"))

        mma.append(("wait", "stat_full", it & 1, it + 1))
        for u in range(min(nbuf, n)):
            issue_sp(u)
        for u in range(n):
            jt, st = stage(u)
            ut = ut0 + u
            buf = ut % nbuf
            if "early_scores" in drop and u + nbuf < n:
                issue_sp(u + nbuf)
            if u == 0 and "acc_free" not in drop:
                mma.append(("wait", "acc_free", (it & 1) ^ 1, it))
            mma.extend([("wait", f"p_full{buf}", (ut // nbuf) & 1, ut // nbuf + 1),
                        ("mma", ((f"buf{buf}", ("P", ut)), (f"str{st}", jt)), "acc", (it, u))])
            if u % steps_per_load == steps_per_load - 1:
                mma.append(("commit", f"str_empty{st}"))
            if u == n - 1:
                mma.append(("commit", "acc_done"))
            if u + nbuf < n and "early_scores" not in drop:
                issue_sp(u + nbuf)
        for s in (0, 1):
            for u in range(s, n, 2):
                jt, st = stage(u)
                ut = ut0 + u
                buf = ut % nbuf
                sets[s].extend([("wait", f"s_full{buf}", (ut // nbuf) & 1, ut // nbuf + 1), ("read", f"buf{buf}", ("S", ut))])
                if steps_per_load == 1:
                    sets[s].extend([("wait", f"str_full{st}", (jt // stages) & 1, jt // stages + 1), ("read", f"str{st}", jt)])
                sets[s].extend([("write", f"buf{buf}", ("P", ut)), ("arrive", f"p_full{buf}")])
            sets[s].extend([("wait", "acc_done", it & 1, it + 1), ("read", "acc", (it, n - 1)), ("arrive", "acc_free")])
        jt0 += n // steps_per_load
        ut0 += n
    return [producer, mma, *sets], {"acc_free": 2}  # both sets read the accumulators


def _commutes(progs):
    """Per actor and position: a step that neither depends on nor is seen by another actor before the next one of its own kind may
    be taken at once (queueing on the tensor pipe, starting a load after the wait for its stage)."""
    return [[op[0] in ("mma", "commit", "load") for op in prog] for prog in progs]


def explore(programs):
    progs, counts = programs
    names = sorted({op[1] for p in progs for op in p if op[0] in ("wait", "commit", "arrive")} | {op[3] for p in progs for op in p if op[0] == "load"})
    bars = {b: i for i, b in enumerate(names)}
    places = sorted({op[1] for p in progs for op in p if op[0] in ("load", "read", "write")} | {op[2] for p in progs for op in p if op[0] == "mma"})
    slot = {p: i for i, p in enumerate(places)}
    need = [counts.get(b, 1) for b in names]
    at_once = _commutes(progs)
    start = ((0,) * len(progs), (0,) * len(names), frozenset(), (), (None,) * len(places))
    seen, stack = {start}, [start]
    problems, deadlocks = set(), 0

    def put(t, i, v):
        return t[:i] + (v,) + t[i + 1:]

    while stack and len(problems) < 20:
        pcs, arrivals, loads, pipe, mem = stack.pop()
        after = []
        for a, prog in enumerate(progs):
            pc = pcs[a]
            if pc == len(prog):
                continue
            op = prog[pc]
            n_arr, n_loads, n_pipe, n_mem = arrivals, loads, pipe, mem
            if op[0] == "wait":
                i = bars[op[1]]
                done = arrivals[i] // need[i]
                if op[2] == (done & 1):
                    continue
                if done < op[3]:
                    problems.add(("a wait passed on an older phase", a, op, done))
            elif op[0] == "arrive":
                i = bars[op[1]]
                n_arr = put(arrivals, i, arrivals[i] + 1)
            elif op[0] == "read":
                if mem[slot[op[1]]] != op[2]:
                    problems.add(("read another step", a, op, mem[slot[op[1]]]))
            elif op[0] == "write":
                n_mem = put(mem, slot[op[1]], op[2])
                if pc + 1 < len(prog) and prog[pc + 1][0] == "arrive":  # nobody looks at it before the arrival
                    i = bars[prog[pc + 1][1]]
                    n_arr = put(arrivals, i, arrivals[i] + 1)
                    pc += 1
            elif op[0] == "load":
                n_loads = loads | {op[1:]}
            else:
                n_pipe = pipe + ((a, op),)
            pc += 1
            while pc < len(prog) and at_once[a][pc]:
                if prog[pc][0] == "load":
                    n_loads = n_loads | {prog[pc][1:]}
                else:
                    n_pipe = n_pipe + ((a, prog[pc]),)
                pc += 1
            after.append((put(pcs, a, pc), n_arr, n_loads, n_pipe, n_mem))
        for ld in loads:  # a TMA load lands
            i = bars[ld[2]]
            after.append((pcs, put(arrivals, i, arrivals[i] + 1), loads - {ld}, pipe, put(mem, slot[ld[0]], ld[1])))
        for at in {a: k for k, (a, _) in reversed(list(enumerate(pipe)))}.values():  # the tensor pipe completes the oldest entry of an issuer
            op, rest = pipe[at][1], pipe[:at] + pipe[at + 1:]
            if op[0] == "commit":
                i = bars[op[1]]
                after.append((pcs, put(arrivals, i, arrivals[i] + 1), loads, rest, mem))
            else:
                for place, version in op[1]:
                    if mem[slot[place]] != version:
                        problems.add(("a product read another step", op, place, mem[slot[place]]))
                after.append((pcs, arrivals, loads, rest, put(mem, slot[op[2]], op[3])))
        if not after and any(pc < len(p) for pc, p in zip(pcs, progs)):
            deadlocks += 1
        for s in after:
            if s not in seen:
                seen.add(s)
                stack.append(s)
    return problems, deadlocks, len(seen)


# (key tiles of the first query tile, is there a second one): a pair and a single tile in either order, three items
FORWARD_ITEMS = [[(5, True)], [(1, True), (1, False)], [(1, False), (1, True)], [(3, False), (2, True)], [(3, True), (2, True), (1, False), (1, True)]]


@pytest.mark.parametrize("n_kv", [2, 4])
@pytest.mark.parametrize("rescale", [False, True])
def test_pingpong_schedule_is_safe_and_live(n_kv, rescale):
    problems, deadlocks, states = explore(forward_programs([(n_kv - 1, True)], False, rescale))
    assert states > 50
    assert not problems and deadlocks == 0, (sorted(map(str, problems))[:3], deadlocks)


def test_checker_notices_scores_issued_ahead_of_the_product_that_reads_the_probabilities():
    problems, deadlocks, _ = explore(forward_programs([(3, True)], False, False, drop=("early_scores",)))
    assert problems or deadlocks


@pytest.mark.parametrize("items", FORWARD_ITEMS, ids=str)
@pytest.mark.parametrize("rescale", [False, True])
@pytest.mark.parametrize("sep", [False, True], ids=["head128", "head64"])
def test_forward_schedule_is_safe_and_live(items, rescale, sep):
    problems, deadlocks, states = explore(forward_programs(items, sep, rescale))
    assert states > 100
    assert not problems and deadlocks == 0, (sorted(map(str, problems))[:3], deadlocks)


# buffers, stages, steps per load of the four kernels; items long enough that buffers and stages come round
@pytest.mark.parametrize("nbuf,stages,per_load,items", [(3, 4, 2, [8, 4, 2]), (2, 2, 2, [6, 4, 2]), (3, 6, 1, [8, 6, 2]), (2, 4, 1, [8, 4, 2])],
                         ids=["dq64", "dq128", "dkv64", "dkv128"])
def test_backward_schedule_is_safe_and_live(nbuf, stages, per_load, items):
    problems, deadlocks, states = explore(backward_programs(items, nbuf, stages, per_load))
    assert states > 100
    assert not problems and deadlocks == 0, (sorted(map(str, problems))[:3], deadlocks)


@pytest.mark.parametrize("mistake,sep", [("early_scores", False), ("s_read", True), ("o_done", True)])
def test_model_notices_a_wrong_forward(mistake, sep):
    problems, deadlocks, _ = explore(forward_programs([(2, True), (1, True)], sep, True, drop=(mistake,)))
    assert problems or deadlocks


@pytest.mark.parametrize("mistake", ["early_scores", "acc_free"])
@pytest.mark.parametrize("nbuf,stages,per_load", [(3, 4, 2), (2, 4, 1)])
def test_model_notices_a_wrong_backward(mistake, nbuf, stages, per_load):
    problems, deadlocks, _ = explore(backward_programs([4, 4], nbuf, stages, per_load, drop=(mistake,)))
    assert problems or deadlocks


# ---- two issuers: nothing orders the products of one behind those of the other but barriers
def split_backward_programs(items, nbuf, stages, steps_per_load, drop=()):
    """The backward kernels as they issue: score products by one warp, accumulating products by another."""
    (producer, _, *sets), counts = backward_programs(items, nbuf, stages, steps_per_load)
    scores, sums = [], []
    jt0 = ut0 = 0
    for it, n in enumerate(items):
        scores.append(("wait", "stat_full", it & 1, it + 1))
        sums.append(("wait", "acc_free", (it & 1) ^ 1, it))
        for u in range(n):
            jt, ut = jt0 + u // steps_per_load, ut0 + u
            st, buf, last = jt % stages, ut % nbuf, u == n - 1
            if u % steps_per_load == 0:
                scores.append(("wait", f"str_full{st}", (jt // stages) & 1, jt // stages + 1))
            if "buf_free" not in drop:
                scores.append(("wait", f"buf_free{buf}", ((ut // nbuf) & 1) ^ 1, ut // nbuf))
            scores.extend([("mma", (("stat", it), (f"str{st}", jt)), f"buf{buf}", ("S", ut)), ("commit", f"s_full{buf}")])
            sums.extend([("wait", f"p_full{buf}", (ut // nbuf) & 1, ut // nbuf + 1),
                         ("mma", ((f"buf{buf}", ("P", ut)), (f"str{st}", jt)), "acc", (it, u)), ("commit", f"buf_free{buf}")])
            if u % steps_per_load == steps_per_load - 1:
                sums.append(("commit", f"str_empty{st}"))
            if last:
                scores.append(("commit", "stat_empty"))
                sums.append(("commit", "acc_done"))
        jt0 += n // steps_per_load
        ut0 += n
    return [producer, scores, sums, *sets], counts


def split_forward_programs(items, drop=()):
    """The forward with head size 64 as it issues: a warp for each query tile."""
    producer, _, *_ = forward_programs(items, True, False)[0]
    issuers, softmax = ([], []), ([], [])
    for t in (0, 1):
        prog, soft = issuers[t], softmax[t]
        kt0 = c = own = 0
        for it, (n_a, has_b) in enumerate(items):
            n_kv = n_a + 1 if has_b else n_a
            n_own = n_a if t == 0 else (n_kv if has_b else 0)

            def wait_tile(kind, j):
                k = kt0 + j
                return ("wait", f"{kind}_full{k & 1}", (k >> 1) & 1, (k >> 1) + 1)

            prog.append(("wait", "q_full", it & 1, it + 1))
            for j in range(-1, n_own if n_own else -1):
                k = kt0 + j
                if j + 1 < n_own:
                    prog.append(wait_tile("k", j + 1))
                    if c + j + 1 > 0:
                        prog.append(("wait", f"s_read{t}", (c + j) & 1, c + j + 1))
                    prog.extend([("mma", (("q", it), (f"k{(k + 1) & 1}", k + 1)), f"s{t}", ("S", it, j + 1)), ("commit", f"s_full{t}"),
                                 ("commit", f"k_empty{(k + 1) & 1}")])
                    if j + 2 == n_own:
                        prog.append(("commit", "q_empty"))
                if j >= 0:
                    prog.append(wait_tile("v", j))
                    if j == 0:
                        prog.append(("wait", f"o_free{t}", (own & 1) ^ 1, own))
                    prog.extend([("wait", f"p_full{t}", (c + j) & 1, c + j + 1), ("mma", ((f"p{t}", ("P", it, j)), (f"v{k & 1}", k)), f"o{t}", (it, j)),
                                 ("commit", f"o_done{t}"), ("commit", f"v_empty{k & 1}")])
            if n_own == 0:
                prog.append(("commit", "q_empty"))
            for j in range(n_own, n_kv):
                k = kt0 + j
                for kind in "kv":
                    if "pass_wait" not in drop:
                        prog.append(wait_tile(kind, j))
                    prog.append(("commit", f"{kind}_empty{k & 1}"))
            for j in range(n_own):
                soft.extend([("wait", f"s_full{t}", (c + j) & 1, c + j + 1), ("read", f"s{t}", ("S", it, j)), ("arrive", f"s_read{t}")])
                if j > 0:
                    soft.append(("wait", f"o_done{t}", (c + j - 1) & 1, c + j))
                soft.extend([("write", f"p{t}", ("P", it, j)), ("arrive", f"p_full{t}")])
            if n_own:
                c += n_own
                own += 1
                soft.extend([("wait", f"o_done{t}", (c - 1) & 1, c), ("read", f"o{t}", (it, n_own - 1)), ("arrive", f"o_free{t}")])
            kt0 += n_kv
    counts = {"q_empty": 2, "k_empty0": 2, "k_empty1": 2, "v_empty0": 2, "v_empty1": 2}
    return [producer, *issuers, *softmax], counts


@pytest.mark.parametrize("nbuf,stages,per_load,items", [(3, 4, 2, [6, 2, 2]), (2, 2, 2, [4, 2, 2]), (3, 6, 1, [6, 2]), (2, 4, 1, [6, 2])],
                         ids=["dq64", "dq128", "dkv64", "dkv128"])
def test_backward_with_two_issuers_is_safe_and_live(nbuf, stages, per_load, items):
    problems, deadlocks, states = explore(split_backward_programs(items, nbuf, stages, per_load))
    assert states > 100
    assert not problems and deadlocks == 0, (sorted(map(str, problems))[:3], deadlocks)


@pytest.mark.parametrize("items", [[(2, True)], [(1, True), (1, False)], [(1, False), (1, True)], [(2, False), (1, True)]], ids=str)
def test_forward_with_two_issuers_is_safe_and_live(items):
    problems, deadlocks, states = explore(split_forward_programs(items))
    assert states > 100
    assert not problems and deadlocks == 0, (sorted(map(str, problems))[:3], deadlocks)


def test_model_notices_two_issuers_without_their_barriers():
    assert any(explore(split_backward_programs([4, 4], 2, 4, 1, drop=("buf_free",)))[:2])
    assert any(explore(split_forward_programs([(2, True), (1, True)], drop=("pass_wait",)))[:2])


def followed_backward_programs(items, nbuf, stages, steps_per_load):
    """... and the score products of an item wait until the accumulating ones of the item before have been issued."""
    (producer, scores, sums, *sets), counts = split_backward_programs(items, nbuf, stages, steps_per_load)
    after = []
    for op in scores:
        if op[:2] == ("wait", "stat_full") and op[3] > 1:
            after.append(("wait", "acc_issued", (op[3] - 2) & 1, op[3] - 1))
        after.append(op)
    told = [o for op in sums for o in ([op, ("arrive", "acc_issued")] if op == ("commit", "acc_done") else [op])]
    return [producer, after, told, *sets], counts


@pytest.mark.parametrize("nbuf,stages,per_load,items", [(3, 4, 2, [6, 2, 2]), (2, 2, 2, [2, 2, 2]), (3, 6, 1, [6, 2]), (2, 4, 1, [2, 2, 2])],
                         ids=["dq64", "dq128", "dkv64", "dkv128"])
def test_backward_issuers_that_follow_one_another_are_safe_and_live(nbuf, stages, per_load, items):
    programs, counts = followed_backward_programs(items, nbuf, stages, per_load)
    assert sum(op[1] == "acc_issued" for op in programs[1]) == len(items) - 1 and programs[2].count(("arrive", "acc_issued")) == len(items)
    problems, deadlocks, states = explore((programs, counts))
    assert states > 100
    assert not problems and deadlocks == 0, (sorted(map(str, problems))[:3], deadlocks)
