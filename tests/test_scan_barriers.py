"""Waits by parity in the warp-specialised forward scan of the delta rule (``csrc/lsm_delta_tc.cu``): every order in which its warps, its loads and its
products can come is walked, and no barrier may get two phases ahead of a warp that waits for it (which would then wait for ever)."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(__file__), "..", "linear_moe_b200", "csrc", "lsm_delta_tc.cu")


def forward_scan(N, S, ring, keep):
    """Arrivals that complete a phase of every barrier, and per actor its steps in order: ("wait", barrier, phase), ("arrive", barrier), and counts without
    phases, ("count", name) and ("reach", name, number), for what the hardware does behind an instruction.  ``ring``: barriers behind ``o_ready``."""
    need = {"sb_ready": 2, "x_full": 1, "v_ready": 1, "s_full": 1, "o_full": 1, "kept": 1}
    need.update({f"{b}{s}": 1 for b in ("full", "empty") for s in range(S)})
    need.update({f"o_ready{s}": 1 for s in range(ring)})
    a = {k: [] for k in ("ask", "issue", "pipe", "state", "store", "upper", "lower", *(f"load{s}" for s in range(S)))}
    for n in range(N):
        s, ph = n % S, n // S
        o = (f"o_ready{n % ring}", n // ring)
        a["ask"] += [("wait", f"empty{s}", ph - 1), ("count", f"asked{s}")]
        a[f"load{s}"] += [("reach", f"asked{s}", ph + 1), ("arrive", f"full{s}")]
        a["issue"] += [("wait", f"full{s}", ph), ("wait", "sb_ready", n), ("count", "issued"), ("wait", "v_ready", n), ("count", "issued")]
        a["pipe"] += [("reach", "issued", 2 * n + 1), ("arrive", "x_full"), ("reach", "issued", 2 * n + 2), ("arrive", "s_full"), ("arrive", "o_full")]
        if keep:
            a["state"] += [("wait", "sb_ready", n), ("wait", "v_ready", n), ("arrive", "kept")]
        a["store"] += [("wait", *o), ("arrive", f"empty{s}")]
        before = [] if n == 0 else [("wait", "s_full", n - 1)] + [("wait", "kept", n - 1)] * keep
        output = [] if n == 0 else [("wait", "o_full", n - 1), ("arrive", f"o_ready{(n - 1) % ring}")]
        a["upper"] += before + [("arrive", "sb_ready")] + output + [("wait", f"full{s}", ph), ("wait", "x_full", n), ("arrive", "v_ready")]
        a["lower"] += before + [("arrive", "sb_ready")]
    a["upper"] += [("wait", "s_full", N - 1), ("wait", "o_full", N - 1), ("arrive", f"o_ready{(N - 1) % ring}")]
    a["lower"] += [("wait", "s_full", N - 1)]
    return need, [x for x in a.values() if x]


def first_lap(need, actors):
    """The (barrier, awaited phase, completed phases) of a wait that its barrier has left behind, in any order of the steps; None if there is none."""
    names = sorted({x[1] for steps in actors for x in steps})
    at = {n: i for i, n in enumerate(names)}
    start = (tuple(0 for _ in actors), tuple(0 for _ in names))
    seen, todo = {start}, [start]
    while todo:
        pcs, got = todo.pop()
        moved = False
        for i, steps in enumerate(actors):
            if pcs[i] == len(steps):
                continue
            kind, name, *more = steps[pcs[i]]
            j, nxt = at[name], got
            if kind == "wait":
                done = got[j] // need[name]
                if done not in (more[0], more[0] + 1):
                    return name, more[0], done
                if done == more[0]:
                    continue
            elif kind == "reach":
                if got[j] < more[0]:
                    continue
            else:
                nxt = got[:j] + (got[j] + 1,) + got[j + 1:]
            moved = True
            state = (pcs[:i] + (pcs[i] + 1,) + pcs[i + 1:], nxt)
            if state not in seen:
                seen.add(state)
                todo.append(state)
        assert moved or all(p == len(s) for p, s in zip(pcs, actors)), "every actor comes to its end"
    return None


@pytest.mark.parametrize("keep", [False, True])
def test_forward_scan_waits_stay_within_a_phase(keep):
    text = open(SOURCE).read()
    S = int(re.search(r"constexpr int STAGES = (\d+)", text).group(1))
    ring = S if re.search(r"\bo_ready\[STAGES\]", text) else 1
    assert first_lap(*forward_scan(S + 3, S, ring, keep)) is None
    if ring == S and not keep:                           # and the walk does find it with one barrier for all stages
        assert first_lap(*forward_scan(S + 3, S, 1, keep))[0] == "o_ready0"
