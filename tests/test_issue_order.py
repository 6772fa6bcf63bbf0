"""The turns that the two MMA issue warps of the decode kernel take, explored on the CPU.

An mbarrier wait names a phase by its parity alone, so it is only sound where no interleaving lets it pass for another phase.
A small model of the roles (their waits and arrivals, the in-order tensor pipe, the ring of five pair slots) is run through every
interleaving; the order of the PV warp's two waits and of the QK^T warp's two arrivals is read from the kernel's source."""
import re
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "flashinfer_mla_fp4_b200" / "csrc" / "decode_sm100.cu"
RING = 5


def source_order(role, marks):
    """The keys of `marks` in the order in which their texts stand in a role's function."""
    body = re.search(rf"void {role}\(.*?\n}}\n", SOURCE.read_text(), re.S).group(0)
    return sorted(marks, key=lambda k: body.index(marks[k]))


def pv_waits():
    return source_order("pv_role", {"qk_issued": "wait(smem, kBarQkIssued", "p_full": "wait(smem, kBarPFull"})


def qk_arrivals():
    return source_order("qk_role", {"s_full": "umma_commit(bar_addr(smem, bar_s_full", "qk_issued": "mbar_arrive(bar_addr(smem, kBarQkIssued"})


def programs(segments, waits, arrivals):
    """Per role a list of operations: ("wait", barrier, phase), ("arrive", barrier), or ("mma", barriers that its completion arrives at)."""
    qk, pv, soft, tma0, tma1 = [], [], [], [], []
    it = 0
    for seg, n in enumerate(segments):
        if seg:
            pv.append(("wait", "o_free", seg - 1))
        for t in range(n):
            s = f"{it & 1}"
            if it >= 2:
                qk.append(("wait", "s_empty" + s, (it >> 1) - 1))
            if t >= 2:
                qk.append(("wait", "pv_issued", it - 2))
            qk += [("wait", "rope_full", it), ("mma", ("rope_empty",))]
            for pr in range(2):
                pos = 2 * it + pr
                qk.append(("wait", f"kv_full{pos % RING}", pos // RING))
                load = tma1 if pr else tma0
                if pr:
                    load += ([("wait", "rope_empty", it - 1)] if it else []) + [("arrive", "rope_full")]
                load += ([("wait", f"kv_empty{pos % RING}", pos // RING - 1)] if pos >= RING else []) + [("arrive", f"kv_full{pos % RING}")]
            for b in arrivals:  # (of the MMAs issued by now; a commit arrives when those before it have completed)
                qk.append(("mma", ("s_full" + s,)) if b == "s_full" else ("arrive", "qk_issued"))
            for b in waits:
                if b == "p_full":
                    pv.append(("wait", "p_full", it))
                elif t + 1 < n:
                    pv.append(("wait", "qk_issued", it + 1))
            pv += [("mma", (f"kv_empty{2 * it % RING}",)), ("arrive", "pv_issued"), ("mma", (f"kv_empty{(2 * it + 1) % RING}", "pv_done"))]
            soft += [("wait", "s_full" + s, it >> 1), ("arrive", "s_empty" + s)]
            soft += ([("wait", "pv_done", it - 1)] if it else []) + [("arrive", "p_full")]
            it += 1
        soft += [("wait", "pv_done", it - 1), ("arrive", "o_free")]
    return [qk, pv, soft, tma0, tma1]


def explore(segments, waits, arrivals):
    """Every reachable state; returns the faults found."""
    roles = programs(segments, waits, arrivals)
    names = sorted({b for r in roles for op in r for b in ([op[1]] if op[0] != "mma" else op[1])})
    at = {b: i for i, b in enumerate(names)}
    start = ((0,) * len(roles), (0,) * len(names), ())
    seen, todo, faults = {start}, [start], set()
    while todo:
        pcs, done, pipe = todo.pop()
        nexts = []
        if pipe:  # the oldest MMAs complete
            d = list(done)
            for b in pipe[0]:
                d[at[b]] += 1
            nexts.append((pcs, tuple(d), pipe[1:]))
        for r, ops in enumerate(roles):
            if pcs[r] == len(ops):
                continue
            op, d, q = ops[pcs[r]], done, pipe
            if op[0] == "wait":
                phases = done[at[op[1]]]
                if (phases & 1) == (op[2] & 1):  # the phase of this parity is the running one
                    continue
                if phases <= op[2]:
                    faults.add(f"{op[1]} phase {op[2]} passed with {phases} complete")
            elif op[0] == "arrive":
                d = tuple(c + (b == op[1]) for b, c in zip(names, done))
            else:
                q = pipe + (op[1],)
            nexts.append((pcs[:r] + (pcs[r] + 1,) + pcs[r + 1:], d, q))
        if not nexts and any(pc < len(ops) for pc, ops in zip(pcs, roles)):
            faults.add("deadlock")
        for s in nexts:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return faults


@pytest.mark.parametrize("segments", [(1,), (5,), (2, 3), (1, 1, 3), (3, 2)])
def test_no_wait_passes_for_another_phase(segments):
    assert explore(segments, pv_waits(), qk_arrivals()) == set()


@pytest.mark.parametrize("waits,arrivals", [
    (["qk_issued", "p_full"], ["qk_issued", "s_full"]),  # PV(0) asks for a phase that may be two away: it passes, and the parities run apart
    (["p_full", "qk_issued"], ["s_full", "qk_issued"]),  # S, and with it P, may be there before QK^T is reported as issued
])
def test_the_model_finds_the_waits_that_run_ahead(waits, arrivals):
    faults = explore((5,), waits, arrivals)
    assert "qk_issued phase 1 passed with 0 complete" in faults and "deadlock" in faults


def test_proxy_fences_of_the_merge():
    """What no run can be relied on to show: bulk copies of bytes that ordinary stores wrote, or over them, come behind a proxy fence."""
    text = SOURCE.read_text()
    fetch = re.search(r"void tail_fetch\(.*?\n}\n", text, re.S).group(0)
    assert fetch.index("ld_acquire(slot_flag") < fetch.index("fence_proxy_async_global()") < fetch.index("ptx::bulk_load(")
    last = re.search(r"void merge_as_last\(.*?\n}\n", text, re.S).group(0)  # one share after the other through the same buffer
    assert re.search(r"tail_merge\(p, smem, tid, parity\);\s*ptx::fence_proxy_async_smem\(\);[^\n]*\s*__syncthreads\(\);", last)


def test_a_small_poll_budget_does_not_shorten_the_drain():
    """A CTA that gave up stays until its copies have landed, whatever the budget of the waits that ran out."""
    drain = re.search(r"void drain_wait\(.*?\n}\n", SOURCE.read_text(), re.S).group(0)
    assert re.search(r"limit = min\(max\(polls, 1u << 10\), 1u << 20\);", drain) and "i < limit" in drain
