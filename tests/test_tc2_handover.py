"""k_corr_tc2's hand-over between its fetch warp, main warps and patch warp, explored exhaustively.

The kernel's waits on mbarriers are bounded, its barriers are not. So whatever wait runs out, and
whenever, every warp has to reach the barrier that ends the block, and a point whose output was left
out has to reach the status word. The model has two main threads (thread 0 and one of the polling
warp), the fetch warp, the patch warp and the tensor core; a wait may give up at any moment
before its phase completes, whatever the others do, and every interleaving is followed. `shared_flag`
is the form in which the patch warp told the main warps to leave by a plain shared word.
"""

import re
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parents[1] / "autorift.jl_b200" / "csrc" / "ar_track.cu"

MAIN, PROD, END = "main", "prod", "end"
MEMBERS = {MAIN: (0, 1), PROD: (0, 1, 2), END: (0, 1, 2, 3)}  # threads 0, 1: main, 2: patch, 3: fetch


def explore(points, shared_flag):
    """The reachable final states and the number of states; raises on a deadlock."""
    # Shared: phases completed of full, free, out[0], out[1] and the products; arrivals at out[*];
    # the points in the two slots; s_more; the flag; the status; outputs written.
    sh0 = dict(full=0, free=0, out=(0, 0), arr=(0, 0), issued=0, prods=0, pt=(None, None),
               more=(1, 1), fail=0, lost=0, status=0, written=0)
    main0 = dict(pc="full", b=0, ph=0, mb=0, got=0, ok=1, failed=0, phase=0)
    local0 = (dict(main0), dict(main0), dict(pc="bar", b=0, ph=0, then="more"),
              dict(pc="fetch", b=0, ph=0, n=0))

    def freeze(sh, ls):
        return tuple(sorted(sh.items())), tuple(tuple(sorted(v.items())) for v in ls)

    def put(t, i, v):
        return t[:i] + (v,) + t[i + 1:]

    def done(count, parity):  # try_wait.parity: the phase of that parity has completed
        return count % 2 != parity

    def step(i, sh, me):
        """The next (shared, local) states of thread i; None when it waits at a barrier."""
        sh, me = dict(sh), dict(me)
        pc = me["pc"]
        if i < 2:
            if pc == "full":
                res = []
                if done(sh["full"], me["ph"]):
                    k = sh["pt"][me["b"]]
                    res.append((sh, dict(me, got=1, pc="last" if k < 0 else "seen")))
                else:
                    res.append((dict(sh, fail=1), dict(me, got=0, pc="seen")))
                return res
            if pc == "read":
                if sh["fail"]:
                    return [(sh, dict(me, failed=1, pc="leave"))]
                if i == 0:
                    sh["more"] = put(sh["more"], me["mb"], 1)
                return [(sh, dict(me, pc="products"))]
            if pc == "issue":
                if i == 1:
                    sh["issued"] += 1
                return [(sh, dict(me, ok=1, pc="poll"))]
            if pc == "poll":
                if i == 0 or done(sh["prods"], me["phase"]):
                    return [(sh, dict(me, pc="or"))]
                return [(sh, dict(me, ok=0, pc="or"))]
            if pc == "free":
                if i == 0:
                    sh["free"] += 1
                return [(sh, dict(me, pc="epilogue"))]
            if pc == "out":
                mb = me["mb"]
                a = sh["arr"][mb] + 1
                if a == 2:
                    a = 0
                    sh["out"] = put(sh["out"], mb, sh["out"][mb] + 1)
                sh["arr"] = put(sh["arr"], mb, a)
                return [(sh, dict(me, mb=mb ^ 1, b=me["b"] ^ 1, ph=me["ph"] ^ 1, pc="full"))]
            if pc == "leave":
                if i == 0:
                    if me["failed"]:
                        sh["status"] = 1
                    sh["more"] = put(sh["more"], me["mb"], 0)
                return [(sh, dict(me, pc="last products"))]
            return None
        if i == 2:
            if pc == "more":
                return [(sh, dict(me, pc="wait" if sh["more"][me["b"]] else "end"))]
            if pc == "wait":
                b = me["b"]
                nxt = dict(me, b=b ^ 1, ph=me["ph"] ^ b, pc="bar")
                if done(sh["out"][b], me["ph"]):
                    return [(dict(sh, written=sh["written"] + 1), nxt)]
                return [(sh, dict(me, pc="gave up"))]  # its store comes any time later
            if pc == "gave up":
                nxt = dict(me, b=me["b"] ^ 1, ph=me["ph"] ^ me["b"], pc="bar")
                return [(dict(sh, **{"fail" if shared_flag else "lost": 1}), nxt)]
            return None
        if pc == "fetch":
            sh["pt"] = put(sh["pt"], me["b"], me["n"] if me["n"] < points else -1)
            sh["full"] += 1
            return [(sh, dict(me, n=me["n"] + 1, b=me["b"] ^ 1, pc="free" if me["n"] < points else "end"))]
        if pc == "free":
            if done(sh["free"], me["ph"]):
                return [(sh, dict(me, ph=me["ph"] ^ 1, pc="fetch"))]
            return [(sh, dict(me, pc="end"))]
        return None

    # Where a thread at a barrier goes on, and which barrier it is.
    bars = {"seen": (MAIN, "read"), "last": (MAIN, "leave"), "products": (PROD, "issue"),
            "or": (MAIN, "free"), "epilogue": (MAIN, "out"), "last products": (PROD, "end"),
            "bar": (PROD, "more"), "end": (END, "gone")}

    seen, stack, finals = set(), [(sh0, local0)], []
    while stack:
        sh, ls = stack.pop()
        key = freeze(sh, ls)
        if key in seen:
            continue
        seen.add(key)
        nxt = []
        for i, me in enumerate(ls):
            for s2, m2 in step(i, sh, me) or []:
                nxt.append((s2, put(ls, i, m2)))
        if sh["prods"] < sh["issued"]:  # the tensor core
            nxt.append((dict(sh, prods=sh["prods"] + 1), ls))
        for name, who in MEMBERS.items():
            if all(bars.get(ls[i]["pc"], (None,))[0] == name for i in who):
                l2 = list(ls)
                bad = any(ls[i]["pc"] == "or" and not ls[i]["ok"] for i in who)
                for i in who:
                    m = dict(ls[i])
                    if m["pc"] == "or":
                        m["phase"] ^= 1
                        if bad:  # the products' wait ran out: this point's barrier is past
                            m.update(failed=1, mb=m["mb"] ^ 1, pc="leave")
                        else:
                            m["pc"] = "free"
                    else:
                        m["pc"] = bars[m["pc"]][1]
                    l2[i] = m
                nxt.append((dict(sh), tuple(l2)))
        if all(m["pc"] == "gone" for m in ls):
            finals.append(dict(sh, status=sh["status"] | sh["lost"]))  # thread 0, after the last barrier
        elif not nxt:
            raise AssertionError("deadlock: " + ", ".join(m["pc"] for m in ls))
        stack.extend(nxt)
    return finals, len(seen)


@pytest.mark.parametrize("points", [0, 1, 2, 3])
def test_every_wait_may_run_out(points):
    finals, states = explore(points, shared_flag=False)
    assert any(f["written"] == points and not f["status"] for f in finals)
    assert all(f["written"] == points or f["status"] for f in finals), "a lost point went unreported"
    assert points == 0 or any(f["status"] for f in finals)


def test_the_model_finds_the_shared_flags_fault():
    with pytest.raises(AssertionError, match="deadlock"):
        explore(2, shared_flag=True)


def test_kernel_follows_the_model():
    """The patch warp keeps a wait that ran out in a word of its own, which reaches the status after the
    barrier that ends the block; only main warps touch the flag that makes the main warps leave."""
    text = SRC.read_text()
    body = text[text.index("k_corr_tc2(const TcArgs A) {"):]
    body = re.sub(r"// [A-Za-z][^\n]*", "", body[:body.index("__global__")])
    patch = body[body.index("} else if (warp == 9) {"):]
    patch = patch[:patch.index("// ---", 200)]
    assert "s_fail" not in patch
    gave_up = patch[patch.index("if (!__all_sync(kFull, tc::mbar_wait(&s_outb[b]"):]
    assert "s_lost = 1" in gave_up[:gave_up.index("continue;")]
    assert body.count("s_lost") == 4
    last = body.rindex("__syncthreads();")
    assert "if (tid == 0 && s_lost) atomicExch(A.status, 1);" in body[last:]
