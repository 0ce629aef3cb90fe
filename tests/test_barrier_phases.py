"""The waits of the attention backward kernels (``rl_b200/csrc/flash_attention_bwd.cu``) as a model that is searched through all its orders: an
issuer, the tensor pipe and two groups of warps that take the tiles in turn. A wait for a parity passes when the barrier's present phase has the
other one, so also when it is two phases behind the one that was meant."""

import pytest


def _violations(n: int, own_barrier: bool):
    """All orders of n tiles: whether a group ever reads the accumulators before the last product, and whether all of them end."""
    # the issuer: scores one tile ahead, each into the buffer of the tile two before, whose product has to be complete
    issuer = []
    for j in range(-1, n):
        if 0 <= j + 1 < n:
            if j + 1 > 1:
                issuer.append(("wait", f"done{(j + 1) & 1}", ((j - 1) >> 1) & 1))
            issuer.append(("issue", f"scores{(j + 1) & 1}"))
        if j >= 0:
            issuer += [("wait", f"weights{j & 1}", (j >> 1) & 1), ("issue", f"done{j & 1}")]
    groups = []
    for g in (0, 1):
        steps = []
        for j in range(g, n, 2):
            steps += [("wait", f"scores{g}", (j >> 1) & 1), ("arrive", f"weights{g}")]
        steps.append(("wait", "all" if own_barrier else f"done{(n - 1) & 1}", 0 if own_barrier else ((n - 1) >> 1) & 1))
        groups.append(steps)
    programs = [issuer, *groups]
    issued = [i for i, s in enumerate(issuer) if s[0] == "issue"]      # the pipe completes them in this order
    products = [issuer[i][1].startswith("done") for i in issued]

    def phases(state):
        """Completed phases of every barrier."""
        *at, piped = state
        c: dict = {}
        for i in issued[:piped]:
            c[issuer[i][1]] = c.get(issuer[i][1], 0) + 1
        for g in (0, 1):
            for s in groups[g][: at[1 + g]]:
                if s[0] == "arrive":
                    c[s[1]] = c.get(s[1], 0) + 1
        c["all"] = int(piped == len(issued))
        return c

    start, early, ends = (0, 0, 0, 0), False, set()
    seen, todo = {start}, [start]
    while todo:
        state = todo.pop()
        *at, piped = state
        c, nxt = phases(state), []
        for k, steps in enumerate(programs):
            if at[k] == len(steps):
                continue
            s = steps[at[k]]
            if s[0] == "wait":
                if (c.get(s[1], 0) & 1) == s[2]:
                    continue
                if k and at[k] == len(steps) - 1 and sum(products[:piped]) < n:
                    early = True
            nxt.append(tuple(x + (i == k) for i, x in enumerate(at)) + (piped,))
        if piped < sum(i < at[0] for i in issued):
            nxt.append((*at, piped + 1))
        if not nxt:
            ends.add(state)
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return early, ends == {(len(issuer), len(groups[0]), len(groups[1]), len(issued))}


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7])
def test_groups_read_complete_sums(n):
    early, ends = _violations(n, own_barrier=True)
    assert not early and ends


@pytest.mark.parametrize("n", [3, 4, 7])
def test_model_sees_a_phase_two_behind(n):
    """With the last tile's own barrier in its place, the group that did not have that tile can be a phase early: the model has to find it."""
    assert _violations(n, own_barrier=False)[0]
