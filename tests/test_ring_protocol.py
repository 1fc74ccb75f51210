"""The operand ring of the tensor-core kernel, its waits and arrivals played through on the CPU.

A wait on an mbarrier names the parity of the phase it waits for, so a waiter that is passed by two phases sleeps for
good. Every interleaving of the roles over one ring is walked here; the counts come from the kernels' header.
"""
import os
import re

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ogle_b200", "csrc", "kernels")


def _passers():
    """How many of the arrivals that complete a stage's operand come from the group that does not build it."""
    text = open(os.path.join(KERNELS, "tc_common.cuh")).read()
    m = re.search(r"constexpr uint32_t kXfPassers = (\d+);", text)
    return int(m.group(1)) if m else 0


def _overtaken(stages, chunks, passers_arrive):
    """Whether some order of events lets a split group wait for a phase of bar_full that lies two or more back.
    State: copies landed, chunks multiplied, and per split group the chunk it waits for. Copies of a stage are issued
    once its last multiply is done; the multiply of chunk i waits for group i % 2 to have built its operand - and, where
    both groups arrive, for the other one to have seen the copy - and multiplies run in order."""
    start = (0, 0, 0, 0)
    seen, todo = {start}, [start]
    while todo:
        landed, done, g0, g1 = todo.pop()
        for g in (g0, g1):
            # bar_full of stage g % stages has completed a phase for each landed chunk of that stage
            if g < chunks and (landed - 1 - g) // stages >= 1 and landed > g:
                return True
        nxt = []
        if landed < chunks and landed < done + stages:
            nxt.append((landed + 1, done, g0, g1))
        if g0 < landed:
            nxt.append((landed, done, g0 + 1, g1))
        if g1 < landed:
            nxt.append((landed, done, g0, g1 + 1))
        builder, other = (g0, g1) if done % 2 == 0 else (g1, g0)
        if done < landed and builder > done and (not passers_arrive or other > done):
            nxt.append((landed, done + 1, g0, g1))
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return False


@pytest.mark.parametrize("stages", [2, 3, 4, 5, 8])
def test_no_split_group_is_passed_by_the_ring(stages):
    assert not _overtaken(stages, 3 * stages + 1, _passers() > 0)


def test_the_model_sees_a_group_that_nobody_waits_for():
    assert _overtaken(3, 10, False)


TENSOR_CORE_KERNELS = ["conv_tc2.cu", "conv_tc2_pair.cu", "conv_tc2_t.cu"]


def _teardown_drains(name):
    """Whether the block as a whole waits for the multiplies in flight when a role has given up, not the issuer alone."""
    text = open(os.path.join(KERNELS, name)).read()
    end = text[text.index("-- teardown"):]
    return re.search(r"commit\w*\(&bar_drain\);\s+mbar_wait\(&bar_drain", end[:end.index("tcgen05.dealloc")]) is not None


def _freed_in_flight(chunks, teardown_drains):
    """Whether tensor memory can be freed with multiplies in flight. The issuer issues them all and leaves, or gives up at
    some point and waits for its own; an epilogue waits for the last of them, or gives up; the block frees when both left."""
    start = (0, 0, "runs", "waits")                       # issued, finished, issuer, epilogue
    seen, todo = {start}, [start]
    while todo:
        issued, done, issuer, epilogue = todo.pop()
        gave_up = "gave up" in (issuer, epilogue)
        left = issuer in ("left", "gave up") and epilogue in ("left", "gave up")
        drained = done == issued
        if left and not drained and not (gave_up and teardown_drains) and not issuer == "gave up":
            return True
        nxt = []
        if done < issued:
            nxt.append((issued, done + 1, issuer, epilogue))
        if issuer == "runs":
            nxt.append((issued + 1, done, issuer, epilogue) if issued < chunks else (issued, done, "left", epilogue))
            nxt.append((issued, done, "gave up", epilogue))
        if epilogue == "waits":
            if done == chunks:
                nxt.append((issued, done, issuer, "left"))
            nxt.append((issued, done, issuer, "gave up"))
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return False


@pytest.mark.parametrize("name", TENSOR_CORE_KERNELS)
def test_tensor_memory_is_freed_after_the_last_multiply(name):
    assert not _freed_in_flight(4, _teardown_drains(name))


def test_the_model_sees_an_epilogue_that_gives_up_alone():
    assert _freed_in_flight(4, False)


def _groups_stay_together(name):
    """Whether a thread of an epilogue group that gives up on an accumulator goes on to the group's next barrier instead of
    leaving (waits of the cluster form, whose warps meet at the block's barrier only, are no group's)."""
    text = open(os.path.join(KERNELS, name)).read()
    waits = [m.start() for m in re.finditer(r"wait_\w+\(&bar_acc_full\[as\]", text)]
    assert waits
    return not any("break;" in text[at:at + re.search(r"group_sync\w*\(|group_and\(|bar\.sync", text[at:]).start()] for at in waits)


def _stuck(tiles, stay):
    """Whether some warps of a group can wait at a barrier that others never come to. Each warp sees a tile's accumulator come
    or gives up on it by itself, and then comes to the barrier all the same or leaves."""
    start = ((0, "waits"),) * 4                           # (tile, waits | at the barrier | left) of each warp
    seen, todo = {start}, [start]
    while todo:
        warps = todo.pop()
        nxt = []
        for i, (tile, at) in enumerate(warps):
            put = lambda s: warps[:i] + (s,) + warps[i + 1:]
            if at == "waits" and tile < tiles:
                nxt.append(put((tile, "at the barrier")))
                if not stay:
                    nxt.append(put((tile, "left")))
            elif at == "waits":
                nxt.append(put((tile, "left")))
        at_barrier = [w for w in warps if w[1] == "at the barrier"]
        if len(at_barrier) == 4:
            nxt.append(tuple((tile + 1, "waits") for tile, _ in warps))
        elif at_barrier and not any(w[1] == "waits" for w in warps):
            return True
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return False


@pytest.mark.parametrize("name", TENSOR_CORE_KERNELS)
def test_no_epilogue_group_waits_for_warps_that_gave_up(name):
    assert not _stuck(2, _groups_stay_together(name))


def test_the_model_sees_warps_that_leave_by_themselves():
    assert _stuck(2, False)


def _window_copies_waited_for():
    """When the window kernel's copying thread waits, at its end, for the copies it has asked for."""
    text = open(os.path.join(KERNELS, "conv_window.cu")).read()
    role = text[text.index("-- copies"):text.index("-- multiplies")]
    drain = re.search(r"(if \(!ok\)[^\n]*\n\s*)?for \(int i = issued[^\n]*mbar_wait\(&bar_raw_full", role)
    return "never" if not drain else "when it gave up" if drain.group(1) else "always"


def _lands_in_a_block_that_ended(tiles, stages, waits):
    """Whether a copy can land after the block's roles have left. One role asks for a tile's copy once the tile a ring before
    it has been read; the other reads tiles in order as they land. Each gives up wherever it waits, or goes on."""
    start = (0, 0, 0, "runs", "runs")                     # asked for, landed, read, the copying role, the reading one
    seen, todo = {start}, [start]
    while todo:
        asked, landed, read, copying, reading = todo.pop()
        if copying == reading == "left" and landed < asked:
            return True
        nxt = []
        if landed < asked:
            nxt.append((asked, landed + 1, read, copying, reading))
        if copying == "runs":
            if asked == tiles:
                nxt.append((asked, landed, read, "waits" if waits == "always" else "left", reading))
            elif asked < read + stages:
                nxt.append((asked + 1, landed, read, copying, reading))
            else:
                nxt.append((asked, landed, read, "left" if waits == "never" else "waits", reading))
        if copying == "waits" and landed == asked:
            nxt.append((asked, landed, read, "left", reading))
        if reading == "runs":
            if read < landed:
                nxt.append((asked, landed, read + 1, copying, "runs" if read + 1 < tiles else "left"))
            else:
                nxt.append((asked, landed, read, copying, "left"))
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return False


@pytest.mark.parametrize("tiles", [1, 2, 5])
def test_no_window_lands_in_a_block_that_ended(tiles):
    assert not _lands_in_a_block_that_ended(tiles, 2, _window_copies_waited_for())


def test_the_model_sees_readers_that_give_up_alone():
    assert _lands_in_a_block_that_ended(1, 2, "when it gave up")


def _fp32_ring():
    """What thread 0 of the fp32 contraction does once its wait has run out: whether it asks for further copies, and whether
    it then waits for those in flight from the step that did not come on."""
    text = open(os.path.join(KERNELS, "igemm.cu")).read()
    body = text[text.index("conv_igemm_tma_kernel("):]
    asks = re.search(r"if \(tid == 0 && ([^;]*)t \+ kTmaStages < count\) issue", body).group(1)
    return "came" not in asks, re.search(r"for \(int t = s_stop; t < count && t < s_stop \+ kTmaStages", body) is not None


def _copy_behind_a_copy(count, stages, asks_on, waits_from_stop):
    """Whether thread 0, which asks for a step's copy two steps ahead and may give up at any wait, can ask for a stage that a
    copy is still on its way to, or leave with one in flight. A wait succeeds by its phase's parity."""
    start = (0, None, tuple(1 if i < count else 0 for i in range(stages)), (0,) * stages, None)
    seen, todo = {start}, [start]
    while todo:
        t, stop, asked, landed, drain = todo.pop()
        nxt = []
        for i in range(stages):
            if landed[i] < asked[i]:
                nxt.append((t, stop, asked, landed[:i] + (landed[i] + 1,) + landed[i + 1:], drain))
        came = lambda step: landed[step % stages] % 2 != step // stages % 2
        if t < count:
            for gave_up in ([False] if stop is None and came(t) else []) + [True]:
                now = t if stop is None and gave_up else stop
                ask, i = asked, t % stages
                if (now is None or asks_on) and t + stages < count:
                    if asked[i] > landed[i]:
                        return True
                    ask = asked[:i] + (asked[i] + 1,) + asked[i + 1:]
                nxt.append((t + 1, now, ask, landed, None))
        else:
            first = count if stop is None else stop if waits_from_stop else max(0, count - stages)
            last = min(count, first + stages)
            at = first if drain is None else drain
            if at >= last:
                if asked != landed:
                    return True
            elif came(at):
                nxt.append((t, stop, asked, landed, at + 1))
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return False


@pytest.mark.parametrize("count", [1, 2, 3, 6, 7])
def test_fp32_ring_after_a_wait_that_ran_out(count):
    assert not _copy_behind_a_copy(count, 2, *_fp32_ring())


def test_the_model_sees_copies_asked_for_after_giving_up():
    assert _copy_behind_a_copy(6, 2, True, True) and _copy_behind_a_copy(6, 2, False, False)


def _stem_warps_wait():
    """Whether a warp of the direct stem that gives up waits for the copies that were asked for before it leaves."""
    text = open(os.path.join(KERNELS, "conv_stem.cu")).read()
    body = text[text.index("conv3x3_smallc_kernel("):]
    gives_up = body[body.index("s_abort = 1;"):]
    return re.search(r"mbar_wait\(&bar_full\[i\], \(s_asked\[i\] - 1\) & 1u\)", gives_up[:gives_up.index("break;")]) is not None


def _stem_copies_outlive(tiles, stages, warps, give_up_waits):
    """Whether a copy can land after the block. Every warp reads all tiles in order, each as it lands, or gives up by itself
    and waits for what has been asked for by then; the last to have read a stage's tile asks for its next."""
    start = ((0,) * warps, (-1,) * warps, 0)              # tiles read; -1 runs, 1 left, -2 - x gives up and waits for x; tiles landed (a bit each)
    seen, todo = {start}, [start]
    while todo:
        read, how, landed = todo.pop()
        asked = sum(1 << t for t in range(tiles) if t < stages or t - stages < min(read))
        if all(h == 1 for h in how) and landed != asked:
            return True
        nxt = [(read, how, landed | 1 << t) for t in range(tiles) if asked >> t & 1 and not landed >> t & 1]
        for i in range(warps):
            put = lambda h: how[:i] + (h,) + how[i + 1:]
            if how[i] == -1 and read[i] == tiles:
                nxt.append((read, put(1), landed))
            elif how[i] == -1:
                nxt.append((read, put(-2 - asked if give_up_waits else 1), landed))
                if landed >> read[i] & 1:
                    nxt.append((read[:i] + (read[i] + 1,) + read[i + 1:], how, landed))
            elif how[i] < -1 and (-2 - how[i]) & ~landed == 0:
                nxt.append((read, put(1), landed))
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return False


@pytest.mark.parametrize("tiles", [1, 3, 6])
def test_no_stem_copy_lands_in_a_block_that_ended(tiles):
    assert not _stem_copies_outlive(tiles, 3, 2, _stem_warps_wait())


def test_the_model_sees_a_stem_warp_that_gives_up():
    assert _stem_copies_outlive(6, 3, 2, False)
