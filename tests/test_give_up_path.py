"""The attention kernel's give-up path, followed on the CPU: where a bounded wait is abandoned, no softmax warp may be left
behind in a named barrier, the one kind of wait of theirs that has no limit.

The sequence of waits, barriers, arrivals and looks at the abort word is read off the kernel's source; a model of two softmax
groups of two warps walks it in every order, any warp abandoning any of its waits at any time.  What the other roles do is taken
to follow at once: a later answer is a warp that is scheduled later, and none at all is an abandoned wait."""
import os
import re

import pytest

from test_kernel_ordering import CSRC, body

GROUPS, WARPS = 2, 2                       # warp 0 of a group publishes the maxima, and in group 0 the row sums
RING, S_BUFS = 4, 3
EVENT = re.compile(r"(?P<wait>MXDSA_WAIT_POLL\(sm\.bar_(?P<on>\w+))|(?P<sync>named_bar_sync\(1 \+ (?P<id>\w+))"
                   r"|(?P<look>MXDSA_LEAVE_IF_ABORTED\(\))|(?P<arrive>mbar_arrive(?:_cluster)?\((?:smem_u32\(&sm\.bar_)?(?P<at>[a-z_]+))")


def role():
    """(events of a tile, events of a pair's end) of a softmax warp, in program order."""
    b = body("attn_sm100.cuh", "mxdsa_attn_kernel")
    r = b[b.index("setmaxnreg_inc<kRegsSoftmax>"): b.index("setmaxnreg_inc<kRegsEpi>")]
    r = r[r.index("while (it.template next<NT>(w))"):]
    tile, end = r[: r.index("gt0 += ntiles;")], r[r.index("gt0 += ntiles;"):]

    def events(text):
        out = []
        for m in EVENT.finditer(text):
            out.append(("wait", m["on"]) if m["wait"] else ("sync", m["id"]) if m["sync"] else ("look", "") if m["look"]
                       else ("arrive", m["at"]))
        return out
    # the tear-down's arrivals in place of a warp that has left
    done = b[b.index("done:"):]
    assert done.count("named_bar_arrive(") == 2 and "(warp - 12) / kGroupWarps" in done and "1 + kGroups" in done
    return events(tile), events(end)


def programs(pairs):
    """The events of every warp over the given tile counts of successive pairs; barriers named by what completes them."""
    tile, end = role()
    assert ("sync", "grp") in tile and ("sync", "kGroups") in end      # otherwise there is nothing to look at
    out = []
    for g in range(GROUPS):
        for i in range(WARPS):
            prog, first = [], 0
            for p, n in enumerate(pairs):
                for gt in range(first, first + n):
                    if gt % GROUPS != g:
                        continue
                    for kind, name in tile:
                        if kind == "wait":
                            at = {"tok_full": gt, "qk_done": gt, "pv_done": gt - S_BUFS, "m_ready": gt - 1}[name]
                            if at >= 0:
                                prog.append(("wait", name, at))
                        elif kind == "arrive":
                            if name != "m_ready" or i == 0:
                                prog.append(("arrive", {"p_empty": "p_empty", "s_full": "s_full"}.get(name, name), gt))
                        else:
                            prog.append((kind, name, g))
                first += n
                for kind, name in end:
                    if kind == "wait" and name == "m_ready":
                        if (first - 1) % GROUPS != g:
                            prog.append(("wait", name, first - 1))
                    elif name == "os_empty":
                        if g == 0 and i == 0 and p >= 2:
                            prog.append(("wait", name, p - 2))
                    elif name == "os_full":
                        if g == 0 and i == 0:
                            prog.append(("arrive", name, p))
                    else:
                        prog.append((kind, name, g))
            out.append(prog)
    return out


def stuck_states(pairs):
    """Reachable states in which warps are left that can do nothing, and the number of states."""
    progs = programs(pairs)
    n = len(progs)
    group = [w // WARPS for w in range(n)]
    first = [sum(pairs[:p]) for p in range(len(pairs))]
    where = [{e: k for k, e in enumerate(prog) if e[0] == "arrive"} for prog in progs]

    def arrived(pos, name, gt, warps):
        return all(where[w][("arrive", name, gt)] < pos[w] for w in warps)

    def of(gt):
        return [w for w in range(n) if group[w] == gt % GROUPS]

    def holds(pos, name, at):
        if name == "tok_full":
            return at < RING or arrived(pos, "tok_empty", at - RING, of(at))
        if name == "qk_done":
            return at < GROUPS or arrived(pos, "p_empty", at - GROUPS, of(at))
        if name == "m_ready":
            return arrived(pos, "m_ready", at, of(at)[:1])
        if name in ("os_full", "os_empty"):
            return arrived(pos, "os_full", at, [0])
        assert name == "pv_done", name
        if not arrived(pos, "s_full", at, of(at)) or not holds(pos, "m_ready", at) or (at > 0 and not holds(pos, "pv_done", at - 1)):
            return False
        return at not in first or at == 0 or holds(pos, "os_full", first.index(at) - 1)      # O drained

    def count(state, bar):                       # arrivals on a named barrier so far
        pos, mode, _ = state
        total = 0
        for w in range(n):
            if bar[0] == "grp" and group[w] != bar[1]:
                continue
            done = pos[w] + (1 if mode[w] > 0 else 0)
            total += sum(1 for k in range(done) if progs[w][k][0] == "sync" and progs[w][k][1] == bar[0])
            total += 1 if mode[w] < 0 else 0     # in the tear-down
        return total

    start = ((0,) * n, (0,) * n, False)          # mode: 0 at an event, > 0 parked until that many arrivals, < 0 in the tear-down
    seen, todo, stuck = {start}, [start], []
    while todo:
        state = todo.pop()
        pos, mode, abort = state
        after = []

        def put(w, p, m, a=abort):
            after.append((pos[:w] + (p,) + pos[w + 1:], mode[:w] + (m,) + mode[w + 1:], a))

        for w in range(n):
            if mode[w] < 0:
                continue
            if pos[w] == len(progs[w]):
                put(w, pos[w], -1)
                continue
            kind, name, at = progs[w][pos[w]]
            if kind == "wait":
                if holds(pos, name, at):
                    put(w, pos[w] + 1, 0)
                put(w, pos[w], -1, True)         # abandoned: the abort word is set ahead of the tear-down's arrivals
            elif kind == "arrive":
                put(w, pos[w] + 1, 0)
            elif kind == "look":
                put(w, pos[w] + (0 if abort else 1), -1 if abort else 0)
            elif mode[w] == 0:
                width = WARPS if name == "grp" else n
                so_far = count(state, (name, at)) + 1
                put(w, pos[w], -(-so_far // width) * width)
            elif count(state, (name, at)) >= mode[w]:
                put(w, pos[w] + 1, 0)
        if not after and any(m >= 0 for m in mode):
            stuck.append(state)
        for s in after:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return stuck, len(seen)


@pytest.mark.parametrize("pairs", [(1, 1, 1), (2, 1), (1, 2), (3,), (1, 3), (1, 1, 1, 1), (4,), (1, 1, 2), (5,)])
def test_no_softmax_warp_is_left_in_a_named_barrier(pairs):
    stuck, states = stuck_states(pairs)
    assert states > 1000
    assert not stuck, (len(stuck), states, stuck[0])


def test_copies_in_flight_get_time_to_land():
    """A role that gives up leaves copies and matrix instructions behind it; the CTA pair may not end, nor give its tensor
    memory back, in the moment it was abandoned.  The warp that gives it back stays, and with it the CTA, for a time that is
    bounded, once no role of either CTA issues any more."""
    done = body("attn_sm100.cuh", "mxdsa_attn_kernel")
    done = done[done.index("done:"):]
    last = re.search(r"if \(warp == 10\) \{\s*if \(\*\(volatile int\*\)&sm\.abort_word != 0\) let_copies_land\(\);\s*tmem_dealloc", done)
    assert last and done.index("cluster_arrive") < done.index("cluster_wait()") < last.start()
    with open(os.path.join(CSRC, "attn_sm100.cuh")) as f:
        text = f.read()
    pause = text[text.index("void let_copies_land()"):]
    pause = pause[: pause.index("\n}\n")]
    assert re.search(r"for \(int i = 0; i < \(1 << 16\) && clock64\(\) - start < 2000000; \+\+i\) __nanosleep", pause)
