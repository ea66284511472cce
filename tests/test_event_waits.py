"""Hand-offs between warps with one job each in the backward's score kernels: the passes arrive on named barriers (events) and go on, the
issuing and the moving warp wait there.  Such a barrier counts arrivals whoever makes them, so a warp that arrives again before its last
arrival was taken would keep the waiting warp for ever.  On the CPU, from the sources: every role has the events in the same order;
between two arrivals on a barrier lies a wait for a product that is issued after the first was taken; after a wait that ran out a
warp knows how many arrivals lie behind it, and the first it makes then is on a barrier with none that may be untaken.  Then the roles are
played in random order with an abort at any moment.  On the GPU: the same hand-off in a self-test kernel."""
import random
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "lookahead_keys_attention_b200" / "csrc"
WARPS = 16
KERNELS = {   # source, kernel, prefix of the events, function of their barriers, macro that looks at a wait's end
    "bwd64": ("bwd.cu", "castle_bwd_kernel(", "kEv", "bwd_event", "BWD_CHECK", "kEvCount", "bar_z"),
    "kv128": ("bwd128.cu", "castle_bwd128_kv_kernel(", "kKv", "kv_event", "KV_CHECK", "kKvEvents", "kKvZ"),
}


class Kernel:
    """order: the events' names; barrier(k): event k's barrier; issuing: what the issuing warp takes and commits in a step, in its order; passes:
    per warp, what it waits for, looks at and arrives on in a step; moving: the events the moving warp takes, and the warps that arrive."""

    def __init__(self, name):
        file, start, prefix, function, macro, count, self.first = KERNELS[name]
        text = re.sub(r"//[^\n]*", "", (CSRC / file).read_text())
        enum = next(e for e in re.findall(r"enum \w+ \{([^}]*)\}", text) if re.search(r"\b" + count + r"\b", e))
        self.order = [e.strip() for e in enum.split(",")]
        assert self.order.pop() == count
        modulus = int(re.search(function + r"\(int k\) \{ return 1 \+ k % (\d+); \}", text).group(1))
        self.barrier = lambda k: 1 + k % modulus
        kernel = text[text.index(start):]
        helpers, passes = kernel.index("if (warp >= kSplitWorkers / 32) {"), kernel.index("bool failed;")
        mover = kernel.index("(warp == 17)" if name == "bwd64" else "(warp == kSplitWorkers / 32 + 1)", helpers)
        issuer = kernel[helpers:mover]
        issuer = issuer[issuer.index("#pragma unroll 1"):]
        walk = kernel[kernel.index("#define " + macro):kernel.index("#undef " + macro)]
        walk = walk[walk.index("#pragma unroll 1"):]
        if name == "kv128":   # a step without scores: its gate is an event of its own, alternately on two barriers that nothing else uses
            assert re.findall(r"next\w*\(([^;]*)\);", issuer[:issuer.index("continue;")]) == ["kv_gate_alone(n)"]
            issuer = issuer[issuer.index("continue;"):]
            assert walk.index("stored_on(kv_gate_alone(n));") < walk.index("continue;") < walk.index("stored(kKvGate)")
            first, staged = (int(re.search(f + r"\(int \w\) \{ return (\d+) \+ \(\w & 1\); \}", text).group(1)) for f in ("kv_gate_alone", "kv_staged"))
            assert modulus < first and first + 2 == staged and staged + 2 == int(re.search(r"kKvGroups = (\d+);", text).group(1)) <= 12
            self.moving = [("kv_staged(m)", WARPS)]
        else:
            ids = dict(re.findall(r"(kEvDqc|kEvDku|kEvDvu) = (\d+)", text))
            assert sorted(map(int, ids.values())) == [modulus + 1, modulus + 2, modulus + 3]   # and three more in odd steps
            assert re.search(r"kWorkers = (\d+)", text).group(1) == str(modulus + 7) and re.search(r"kEpilogue = (\d+)", text).group(1) == str(modulus + 8)
            taken = re.findall(r"ev_wait\((\w+) \+ odd, (\d+)\)", kernel[mover:passes])
            assert taken[:3] == taken[3:] and kernel.count("+ 3 * (n & 1)") == 2
            self.moving = [(e, int(n) // 32) for e, n in taken[:3]]
        self.issuing = [("take", a) if a else ("commit", b or self.first)
                        for a, b in re.findall(r"next\((\w+)\)|mma_commit\(&?(?:bars \+ )?(\w+)\)|issue_z\(", issuer) if b not in ("bar_end", "kKvEnd")]

        def program(part, staged):
            out = []
            for wait, check, arrive, moved in re.findall(r"\bwait\(&?(\w+), ph\w*\)|" + macro + r"\(([^)]*)\)|(?:read|stored)\((k\w+)\)|(ev_arrive)\(", part):
                out.append(("wait", wait) if wait else ("check", check) if check else ("arrive", arrive or staged))
            return out

        if name == "bwd64":
            split = walk.index("if (cc == 1 || cc == 2) {")
            other = walk.index("} else {", split)
            last = {0: "kEvDvu", 1: "kEvDqc", 2: "kEvDku", 3: "kEvDvu"}
            assert "cc == 1 ? kEvDqc : cc == 2 ? kEvDku : kEvDvu" in walk
            self.passes = {w: program(walk[:split], None) + program(walk[split:other] if w // 4 in (1, 2) else walk[other:], last[w // 4]) for w in range(WARPS)}
        else:
            at = walk.index("if (cc >= 2) {")
            end = walk.index("}", at)
            self.passes = {w: program(walk if w // 4 >= 2 else walk[:at] + walk[end:], "kv_staged(m)") for w in range(WARPS)}
        self.behind = {e: k for k, e in enumerate(self.order)} | {count: len(self.order), count + " + 1": len(self.order) + 1}


@pytest.fixture(scope="module", params=sorted(KERNELS))
def kernel(request):
    return Kernel(request.param)


def test_every_role_has_the_same_order(kernel):
    assert [e for kind, e in kernel.issuing if kind == "take"] == kernel.order
    for program in kernel.passes.values():
        arrivals = [e for kind, e in program if kind == "arrive"]
        assert arrivals[:-1] == kernel.order and arrivals[-1] in dict(kernel.moving)
        done = pending = 0
        for kind, what in program:
            if kind == "check":
                assert kernel.behind[what] == done
            assert kind != "arrive" or not pending, what   # a wait is looked at before the next arrival
            done += kind == "arrive"
            pending = kind == "wait" or pending and kind != "check"
        assert not pending
    for event, warps in kernel.moving:
        assert sum(("arrive", event) in p for p in kernel.passes.values()) == warps


def test_untaken_arrivals(kernel):
    steps = 3
    issued = [("commit", kernel.first)] + kernel.issuing * steps
    place = [i for i, t in enumerate(issued) if t[0] == "take"]
    n = len(kernel.order)
    for program in kernel.passes.values():
        seen, made, proven, pending = {}, [], -1, []   # proven: the place up to which a wait that ended well has shown the issuing warp
        for step in range(steps):
            done = 0
            for kind, what in program:
                if kind == "wait":
                    commits = [i for i, t in enumerate(issued) if t == ("commit", what)]
                    seen[what] = seen.get(what, -1) + 1
                    pending.append(commits[seen[what]] if commits else -1)   # (nothing is known of what the moving warp answers)
                elif kind == "check":
                    first = step * n + done if done < n else (step + 1) * n   # made next if one of these waits ran out
                    if done != n:   # (else it is one that the moving warp takes)
                        untaken = {kernel.barrier(k % n) for k in made if place[k] >= proven}
                        assert kernel.barrier(first % n) not in untaken, (what, step)
                    proven = max([proven, *pending])
                    pending = []
                elif done < n:
                    assert what == kernel.order[done]
                    k = step * n + done
                    assert not any(kernel.barrier(j % n) == kernel.barrier(done) and place[j] >= proven for j in made), (what, step)
                    made.append(k)
                    done += 1
                else:
                    done += 1


class _Barrier:
    def __init__(self, need):
        self.need, self.count, self.generation = need, 0, 0

    def arrive(self):
        self.count += 1
        if self.count == self.need:
            self.count, self.generation = 0, self.generation + 1


def _play(kernel, steps, seed, sound=True):
    """All roles in random order, an abort at a random moment: whether all of them end.  Not sound: warps go on arriving as if nothing were."""
    rng = random.Random(seed)
    n = len(kernel.order)
    bars = {kernel.barrier(k): _Barrier(WARPS + 1) for k in range(n)}
    bars.update({(e, odd): _Barrier(w + 1) for e, w in kernel.moving for odd in (0, 1)})
    commits = {kernel.first: 1}
    products = {b for kind, b in kernel.issuing if kind == "commit"}
    state = {"abort": False, "events": 0}

    def sync(bar):
        at = bar.generation
        bar.arrive()
        while bar.generation == at:
            yield
        state["events"] += 1

    def issuing():
        for _ in range(steps):
            k = 0
            for kind, what in kernel.issuing:
                if kind == "take":
                    yield from sync(bars[kernel.barrier(k)])
                    k += 1
                elif not state["abort"] or rng.random() < 0.5:   # products that never end among them
                    commits[what] = commits.get(what, 0) + 1
                yield

    def moving():
        for step in range(steps):
            for event, _ in kernel.moving:
                yield from sync(bars[event, step & 1])
                yield

    def passes(program):
        stopped = failed = False
        for step in range(steps):
            k = 0
            for kind, what in program:
                if kind == "wait" and not stopped:
                    while what in products and commits.get(what, 0) <= step:
                        if state["abort"]:
                            failed = True
                            break
                        yield
                elif kind == "check":
                    stopped = stopped or failed and sound
                    failed = False
                elif kind == "arrive":
                    bar = bars[kernel.barrier(k)] if k < n else bars[what, step & 1]
                    if stopped:
                        yield from sync(bar)
                    else:
                        bar.arrive()
                    k += 1
                yield

    roles = [issuing(), moving(), *map(passes, kernel.passes.values())]
    when, tick, last = rng.randrange(60 * steps * WARPS), 0, (0, None)
    while roles:
        tick += 1
        state["abort"] = state["abort"] or tick >= when
        role = rng.choice(roles)
        try:
            next(role)
        except StopIteration:
            roles.remove(role)
        if (state["events"], len(roles)) != last[1]:
            last = tick, (state["events"], len(roles))
        if tick - last[0] > 20000:
            return False
    return True


def test_all_roles_end_whenever_a_wait_runs_out(kernel):
    assert all(_play(kernel, 3, seed) for seed in range(40))
    # the model does show the fault
    assert not all(_play(kernel, 3, seed, sound=False) for seed in range(40))


@pytest.mark.gpu
@pytest.mark.parametrize("rounds", [1, 2, 5, 16, 17, 400])
@pytest.mark.parametrize("form", [0, 1, 2])
def test_self_test_of_the_events(rounds, form):
    import torch
    from lookahead_keys_attention_b200 import _lib as L, check_status
    from lookahead_keys_attention_b200.ops import status_word
    lib = L.load()
    check_status()
    st = status_word(torch.device("cuda", torch.cuda.current_device()))
    result = torch.full((2,), -1, dtype=torch.int32, device="cuda")
    L.check(lib.castle_selftest_event_timeout(65536 if form == 1 else 1024, rounds, form, result.data_ptr(), st.data_ptr(), None), "event_timeout")
    torch.cuda.synchronize()             # the kernel returned
    assert result.tolist() == [int(form == 1), 2 * rounds]
    if form != 1:
        with pytest.raises(RuntimeError, match="bounded wait"):
            check_status()
    check_status()


@pytest.mark.gpu
def test_event_self_test_rejects_bad_arguments():
    import torch
    from lookahead_keys_attention_b200 import _lib as L
    lib = L.load()
    z = torch.zeros(2, dtype=torch.int32, device="cuda").data_ptr()
    for limit, rounds, form, result, st in ((0, 1, 0, z, z), (65537, 1, 0, z, z), (16, 0, 0, z, z), (16, 1025, 0, z, z), (16, 1, 3, z, z),
                                            (16, 1, -1, z, z), (16, 1, 0, None, z), (16, 1, 0, z, None)):
        assert lib.castle_selftest_event_timeout(limit, rounds, form, result, st, None) < 0
