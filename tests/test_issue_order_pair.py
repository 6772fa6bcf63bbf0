"""The waits and arrivals of the decode kernel for pairs of CTAs, explored on the CPU.

As in test_issue_order.py: a model of the roles of both CTAs is run through every interleaving, since a wait that names its phase by
parity is only sound where no interleaving lets it pass for another phase."""
import re
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "flashinfer_mla_fp4_b200" / "csrc" / "decode_pair.cuh"
COUNTS = {"qk_full": 2, "pv_full": 2, "q_full": 2, "s_empty": 2, "p_full": 2, "o_free": 4, "epilogue": 2}  # (a group of softmax warps counts once)


def both_cta_report_k():
    """Whether the K copy warp of CTA 1 arrives at CTA 0's barrier for every tile, as the source has it."""
    role = re.search(r"void pair_tma_role\(.*?\n}\n", SOURCE.read_text(), re.S).group(0)
    return bool(re.search(r"if \([^)]*rank && !which\) ptx::mbar_arrive", role))


def programs(segments, both_copy):
    """Roles: QK^T, PV, Q loads of CTA 1, two softmax groups, a K copy warp (with the scales) and a V copy warp in each CTA."""
    qk, pv, q1, load_v, load_k = [], [], [], [[], []], [[], []]
    soft = [[[], []], [[], []]]  # [CTA][parity of the tile]
    total, it = sum(segments), 0
    for si, n in enumerate(segments):
        if si:
            qk.append(("wait", "q_empty.0", si - 1))
            q1.append(("wait", "q_empty.1", si - 1))
            pv.append(("wait", "o_free", si - 1))
        qk += [("arrive", "q_full"), ("wait", "q_full", si)]
        q1.append(("arrive", "q_full"))
        for t in range(n):
            s, half = it & 1, it >> 1
            if it >= 2:
                qk.append(("wait", f"s_empty{s}", half - 1))
            qk += [("wait", f"qk_full{s}", half), ("mma", tuple(f"{b}{s}.{c}" for b in ("s_full", "qk_empty") for c in (0, 1)))]
            pv += [("wait", f"pv_full{s}", half), ("wait", f"p_full{s}", half)]
            pv += [("seen", "tiles_of.0", it + 1), ("seen", "tiles_of.1", it + 1)]  # (P' of this tile, of both CTAs)
            pv += [("mma", (f"pv_empty{s}.0", f"pv_empty{s}.1"))]
            for c in (0, 1):
                load_k[c] += [("wait", f"qk_empty{s}.{c}", half - 1)] if it >= 2 else []
                load_k[c] += [("arrive", f"qk_full{s}")] * (1 if both_copy else 2 * (1 - c))
                (load_k if it else load_v)[c].append(("arrive", f"scale{it & 3}.{c}"))
                load_v[c] += ([("wait", f"pv_empty{s}.{c}", half - 1)] if it >= 2 else []) + [("arrive", f"pv_full{s}")]
                ops = soft[c][s]
                ops += [("wait", f"scale{it & 3}.{c}", it >> 2), ("wait", f"s_full{s}.{c}", half), ("arrive", f"s_empty{s}")]
                ops += ([("wait", f"ref{1 - s}.{c}", (it - 1) >> 1)] if it else []) + ([("arrive", f"ref{s}.{c}")] if it + 1 < total else [])
                ops += [("wait", f"pv_empty{s}.{c}", half - 1)] if it >= 2 else []
                ops += [("wait", f"pv_empty{1 - s}.{c}", (it - 1) >> 1)] if t else []  # (where O is rescaled)
                ops += [("arrive", f"p_full{s}"), ("arrive", f"tiles_of.{c}")]
            it += 1
        qk.append(("mma", ("q_empty.0", "q_empty.1")))
        for c in (0, 1):
            for ops in soft[c]:
                ops += [("arrive", f"epilogue.{c}"), ("wait", f"epilogue.{c}", si), ("wait", f"pv_empty{(it - 1) & 1}.{c}", (it - 1) >> 1), ("arrive", "o_free")]
    return [qk, pv, q1, *load_v, *load_k, *soft[0], *soft[1]]


def explore(roles):
    """Every reachable state, with a role's arrivals made as soon as it gets to them (a role that is late is late in its wait); the faults."""
    names = sorted({b for r in roles for op in r for b in ([op[1]] if op[0] != "mma" else op[1])})
    at = {b: i for i, b in enumerate(names)}
    count = [next((c for k, c in COUNTS.items() if re.match(rf"{k}\d?(\.\d)?$", b)), 1) for b in names]

    def settle(pcs, done):
        pcs, done = list(pcs), list(done)
        for r, ops in enumerate(roles):
            while pcs[r] < len(ops) and ops[pcs[r]][0] == "arrive":
                done[at[ops[pcs[r]][1]]] += 1
                pcs[r] += 1
        return tuple(pcs), tuple(done)

    start = (*settle((0,) * len(roles), (0,) * len(names)), ())
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
            op, q = ops[pcs[r]], pipe
            if op[0] == "seen":
                if done[at[op[1]]] < op[2] and not ("flag.0" in at and done[at["flag.0"]]):  # (a flagged CTA writes nothing)
                    faults.add(f"{op[1]}: {done[at[op[1]]]} of {op[2]}")
            elif op[0] == "wait":
                phases = done[at[op[1]]] // count[at[op[1]]]
                if (phases & 1) == (op[2] & 1):  # the phase of this parity is the running one
                    continue
                if phases != op[2] + 1:
                    faults.add(f"{op[1]} phase {op[2]} passed with {phases} complete")
            else:
                q = pipe + (op[1],)
            nexts.append((*settle(pcs[:r] + (pcs[r] + 1,) + pcs[r + 1:], done), q))
        if not nexts and any(pc < len(ops) for pc, ops in zip(pcs, roles)):
            faults.add("deadlock")
        for s in nexts:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return faults


@pytest.mark.parametrize("segments", [(1, 1, 1), (5,), (2, 1), (1, 2), (3, 1)])
def test_no_wait_passes_for_another_phase(segments):
    assert explore(programs(segments, both_cta_report_k())) == set()


def test_the_model_finds_a_copy_warp_left_behind():
    """Without an arrival of CTA 1 for tiles of which it copies nothing, CTA 0 runs ahead of that warp's waits."""
    assert "deadlock" in explore(programs((3,), both_copy=False))


@pytest.mark.parametrize("partner_first", [None, False])
def test_a_cta_that_gave_up_takes_its_partner_along(partner_first):
    """Softmax warps of CTA 1 whose waits fail go through the rest of their tiles at once and report them: CTA 0 may take two tiles of theirs
    for one of both CTAs', but only if it has been flagged by then."""
    slow = re.search(r"bool pair_wait_slow\(.*?\n}\n", SOURCE.read_text(), re.S).group(0)
    order = [slow.find(t) for t in ("ptx::st_cluster_u32(", "ptx::fence_cluster()", "flag_timeout(")]
    if partner_first is None:  # as the source has it
        partner_first = -1 < order[0] < order[1] < order[2]
        assert partner_first
    roles = programs((4,), True)
    for ops in roles[-2:]:  # CTA 1's softmax groups
        ops[:] = [("wait", "flag.1", 0)] + [op for op in ops if op[0] == "arrive"]
    flags = [("arrive", "flag.0"), ("seen", "flag.0", 0), ("arrive", "flag.1")]  # (a point at which others may run)
    roles.append(flags if partner_first else flags[::-1])
    assert any(f.startswith("tiles_of.0") for f in explore(roles)) != partner_first


def test_what_passes_between_the_ctas_is_ordered_between_them():
    """What no run can be relied on to show: an arrival at the other CTA's barrier that stands for work done releases at cluster scope, and
    every wait acquires at that scope (without a scope both would hold within a CTA alone)."""
    ptx = (SOURCE.parent / "ptx_sm100.cuh").read_text()
    for op in re.findall(r"mbarrier\.arrive\S*shared::cluster\S*", ptx):
        assert op.startswith(("mbarrier.arrive.release.cluster.", "mbarrier.arrive.relaxed.cluster.")), op
    release = re.search(r"void mbar_arrive_release_cluster\(.*?\n}", ptx, re.S).group(0)
    assert release.index("fence.release.sync_restrict::shared::cta.cluster;") < release.index("mbarrier.arrive.relaxed.cluster")
    assert ".acquire.cluster." in re.search(r"bool mbar_try_wait_cluster\(.*?\n}", ptx, re.S).group(0)
    text = SOURCE.read_text()
    assert "mbar_try_wait(" not in text and not re.search(r"[^_]wait\(smem", text)
    relaxed = re.findall(r".*mbar_arrive_relaxed_cluster.*", text)
    assert len(relaxed) == 1 and "!which" in relaxed[0]  # (a count alone: the copies report for themselves)
