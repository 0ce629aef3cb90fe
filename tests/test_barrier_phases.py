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


def _programs(kernel: str, n: int, one_ds_barrier: bool = False):
    """Issuer and group of ``n`` tiles that both groups share: ("wait", barrier, parity), ("issue", product, tile), ("touch", what, tile) and
    ("arrive", barrier)."""
    issuer, group = [("issue", "S", 0), ("issue", "dP", 0)], []
    for j in range(n):
        more = j + 1 < n
        if kernel == "dq":
            if more:
                issuer += [("wait", "s_read", j & 1), ("issue", "S", j + 1)]
                issuer += [("wait", "dq", (j - 1) & 1)] if j else []
                issuer += [("issue", "dP", j + 1)]
            ds, parity = ("ds_full", j & 1) if one_ds_barrier else (f"ds_full{j & 1}", (j >> 1) & 1)
            issuer += [("wait", ds, parity), ("issue", "dq", j)]
            group += [("wait", "S", j & 1), ("touch", "S", j), ("arrive", "s_read"), ("wait", f"dP{j & 1}", (j >> 1) & 1), ("touch", "dP", j), ("arrive", ds)]
        else:
            issuer += [("wait", "p_full", j & 1), ("issue", "dv", j)]
            issuer += [("wait", "dp_read", j & 1), ("issue", "S", j + 1)] if more else []
            issuer += [("wait", "ds_full", j & 1), ("issue", "dk", j)]
            issuer += [("wait", "dk", j & 1), ("issue", "dP", j + 1)] if more else []
            group += [("wait", "S", j & 1), ("touch", "S", j), ("arrive", "p_full"), ("wait", "dP", j & 1), ("touch", "dP", j), ("arrive", "dp_read"),
                      ("touch", "dS", j), ("arrive", "ds_full")]
    return issuer, group + [("wait", "all", 0), ("touch", "sums", 0)]


def _shared_tiles(kernel: str, n: int, without=None, one_ds_barrier: bool = False):
    """All orders: the faults that are met (a place written before its readers are done, or read before it is written), and whether all programs end."""
    issuer, group = _programs(kernel, n, one_ds_barrier)
    if without:
        issuer = [s for s in issuer if s != without]
    programs = [issuer, group, group]
    issued = [i for i, s in enumerate(issuer) if s[0] == "issue"]      # the pipe completes them in this order
    index = {issuer[i][1:]: k for k, i in enumerate(issued)}
    # what has to be over before a product may write its place: the groups' steps on it, and products that read it
    if kernel == "dq":
        before = {"S": lambda j: ([("S", j - 1)], []), "dP": lambda j: ([("dP", j - 2)], [("dq", j - 2)]), "dq": lambda j: ([("dP", j)], [])}
    else:
        before = {"S": lambda j: ([("dP", j - 1)], []), "dP": lambda j: ([("dS", j - 1)], [("dv", j - 1), ("dk", j - 1)]),
                  "dv": lambda j: ([("S", j)], []), "dk": lambda j: ([("dS", j)], [])}
    after = {("touch", *k): i for i, s in enumerate(group) if s[0] == "touch" for k in [s[1:]]}
    faults, ends = set(), set()
    start = (0, 0, 0, 0)
    seen, todo = {start}, [start]
    while todo:
        state = todo.pop()
        *at, piped = state
        c: dict = {}
        for i in issued[:piped]:
            name = issuer[i][1] + (str(issuer[i][2] & 1) if kernel == "dq" and issuer[i][1] == "dP" else "")
            c[name] = c.get(name, 0) + 1
        arrivals: dict = {}
        for g in (1, 2):
            for s in group[: at[g]]:
                if s[0] == "arrive":
                    arrivals[s[1]] = arrivals.get(s[1], 0) + 1
        c.update({k: v // 2 for k, v in arrivals.items()}, all=int(piped == len(issued)))
        nxt = []
        for k, steps in enumerate(programs):
            if at[k] == len(steps):
                continue
            s = steps[at[k]]
            if s[0] == "wait" and (c.get(s[1], 0) & 1) == s[2]:
                continue
            if s[0] == "issue":
                touched, done = before[s[1]](s[2])
                if any(t[1] >= 0 and min(at[1:]) <= after[("touch", *t)] for t in touched) or any(t[1] >= 0 and index[t] >= piped for t in done):
                    faults.add(s)
            if s[0] == "touch" and s[1] in ("S", "dP") and index[s[1:]] >= piped or s[:2] == ("touch", "sums") and piped < len(issued):
                faults.add(s)
            nxt.append(tuple(x + (i == k) for i, x in enumerate(at)) + (piped,))
        if piped < sum(i < at[0] for i in issued):
            nxt.append((*at, piped + 1))
        if not nxt:
            ends.add(state)
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return faults, ends == {(len(issuer), len(group), len(group), len(issued))}


@pytest.mark.parametrize("kernel", ["dq", "dkv"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6])
def test_tiles_that_both_groups_share(kernel, n):
    """The waits as they are since both groups take a half of every tile."""
    faults, ends = _shared_tiles(kernel, n)
    assert not faults and ends


@pytest.mark.parametrize("kernel,wait", [("dq", ("wait", "s_read", 0)), ("dq", ("wait", "dq", 0)), ("dq", ("wait", "ds_full1", 0)), ("dkv", ("wait", "p_full", 0)),
                                         ("dkv", ("wait", "dp_read", 1)), ("dkv", ("wait", "ds_full", 0)), ("dkv", ("wait", "dk", 0))])
def test_model_sees_a_missing_wait(kernel, wait):
    assert _shared_tiles(kernel, 5, without=wait)[0]


def test_model_sees_a_group_that_arrives_twice():
    """With one barrier for dS of all tiles, a group that is a tile ahead completes the phase of the one behind: the model has to find it."""
    assert _shared_tiles("dq", 2, one_ds_barrier=True)[0]
