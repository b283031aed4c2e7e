"""Order of the lockstep chain's hand-overs, walked through on the CPU.  A buffer of its exchange is marked unwritten while other
CTAs run on, and comes round again some uses later; that no reader finds it marked too early or too late cannot be shown by
running it, since microseconds lie between."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qwen3-tts-native_b200", "csrc")

CLUSTERS, RANKS, LAYERS, HEADS = 32, 4, 5, 8
CTAS = CLUSTERS * RANKS


class Walk:
    """What each group of threads (a CTA's I/O warps; a row's norm warps) knows of the others, from what it has polled alone.
    cause[g, o]: events of o that lie before g's now in time.  knows[g, o]: those that g may rely on by the memory model.  A thread's
    fence vouches for what its group had at the barrier before (its own marks among that), and takes in what it has polled since;
    the group has that from its next barrier on.  `buffers`: how many of each kind of value take turns."""

    def __init__(self, rows, buffers):
        self.rows, self.buffers = rows, buffers
        self.mt = 16 * -(-rows // 16)
        n = CTAS + rows
        self.cause, self.knows, self.met, self.said, self.heard, self.fenced = (np.zeros((n, n), dtype=np.int32) for _ in range(6))
        self.use = dict.fromkeys(buffers, 0)                      # uses published so far
        self.made, self.marked, self.read = {}, {}, {}           # of a (value, use): by whom and when
        self.faults = set()

    def tick(self, g):
        self.cause[g, g] += 1
        return self.cause[g, g]

    def barrier(self, g):
        self.tick(g)
        np.maximum(self.knows[g], self.fenced[g], out=self.knows[g])
        self.knows[g, g] = self.cause[g, g]
        self.met[g] = self.knows[g]

    def fence(self, g):
        self.tick(g)
        np.maximum(self.fenced[g], self.heard[g], out=self.fenced[g])
        self.said[g] = self.met[g]

    def publish(self, value, groups):
        self.use[value] += 1
        made = self.made[value, self.use[value]] = {}
        for g in groups:
            self.tick(g)
            made[g] = self.cause[g].copy(), self.said[g].copy()

    def poll(self, value, g, writers):
        use = self.use[value]
        at = self.tick(g)
        made, marked, old = self.made[value, use], self.marked.get((value, use), {}), self.marked.get((value, use - self.buffers[value]), {})
        for w in writers:
            if w in marked:
                self.faults.add((value, "early"))
            if use > self.buffers[value] and self.knows[g, w] < old.get(w, 1 << 30):
                self.faults.add((value, "late"))
            cause, said = made[w]
            np.maximum(self.cause[g], cause, out=self.cause[g])
            np.maximum(self.heard[g], said, out=self.heard[g])
            self.read.setdefault((value, use, w), []).append((g, at))

    def mark(self, value, g):
        use = self.use[value] - 1
        if g not in self.made.get((value, use), {}):
            return
        for reader, at in self.read.get((value, use, g), []):
            if self.cause[g, reader] < at:
                self.faults.add((value, "early"))
        self.marked.setdefault((value, use), {})[g] = self.tick(g)

    # who has what
    def owners(self, clusters, sharers, row=None):
        """ranks that finish rows (that row) of the clusters' tiles; the tiles of a pair of ranks: both"""
        share = self.mt // sharers
        rows = range(self.rows) if row is None else (row,)
        some = sorted({r // share for r in rows})
        return [c * RANKS + r + 2 * t for c in clusters for t in range(RANKS // sharers) for r in some]

    def units(self, heads, rows=None):
        return sorted({(r * HEADS + h) % CTAS for r in (range(self.rows) if rows is None else rows) for h in heads})

    def project(self, clusters, sharers, source, publishes):
        """clusters' ranks poll, their slices meet, results out"""
        ctas = [c * RANKS + r for c in clusters for r in range(RANKS)]
        for g in ctas:
            if source:
                source(g)
        for c in clusters:
            for first in range(0, RANKS, sharers):
                group = [c * RANKS + first + r for r in range(sharers)]
                most = self.cause[group].max(axis=0)
                self.cause[group] = most
        for g in ctas:
            self.barrier(g)
            self.barrier(g)
        self.publish(publishes, self.owners(clusters, sharers))

    def norm(self, value):
        for r in range(self.rows):
            g = CTAS + r
            self.poll(value, g, self.owners(range(16, 32), 4, r))
            self.barrier(g)
            self.barrier(g)
        self.publish("vNormed", range(CTAS, CTAS + self.rows))
        for g in range(CTAS, CTAS + self.rows):
            self.mark("vNormed", g)
            self.fence(g)

    def normed(self, g):
        self.poll("vNormed", g, range(CTAS, CTAS + self.rows))

    def all_fence(self):
        for g in range(CTAS):
            self.fence(g)

    def position(self, p):
        every, late = range(CLUSTERS), range(16, 32)
        tokens = lambda g: self.poll("vTokens", g, [2 * r + 1 for r in range(self.rows)])
        self.project(late, 4, tokens if p >= 2 else None, "vIn")
        for g in self.owners(late, 4):
            self.mark("vIn", g)
        self.all_fence()
        for layer in range(LAYERS):
            self.norm("vIn")
            self.project(every, 4, self.normed, "vQkv")
            ends = p == 0 and layer == LAYERS - 1
            for g in self.units(range(HEADS)):
                for unit in range(g, self.rows * HEADS, CTAS):
                    r, h = divmod(unit, HEADS)
                    self.poll("vQkv", g, self.owners((2 * h, 2 * h + 1, 16 + h, 24 + h), 4, r))
            if not ends:
                self.publish("vAtt", self.units(range(HEADS)))
                self.project(late, 4, lambda g: self.poll("vAtt", g, self.units((2 * (g % 4), 2 * (g % 4) + 1))), "vMid")
                self.norm("vMid")
                self.project(range(24), 2, self.normed, "vAct")
                self.project(late, 4, lambda g: self.poll("vAct", g, self.owners(range(6 * (g % 4), 6 * (g % 4) + 6), 2)), "vIn")
            for g in self.owners(every, 4):
                self.mark("vQkv", g)
            if ends:
                self.all_fence()
                return
            for g in self.units(range(HEADS)):
                self.mark("vAtt", g)
            for g in self.owners(late, 4):
                self.mark("vMid", g)
            for g in self.owners(range(24), 2):
                self.mark("vAct", g)
            for g in self.owners(late, 4):
                self.mark("vIn", g)
            self.all_fence()
        if p == 0:
            return
        self.norm("vIn")
        self.project(range(16), 4, self.normed, "vLogits")
        draws = [2 * r + 1 for r in range(self.rows)]
        for r, g in enumerate(draws):
            self.poll("vLogits", g, self.owners(range(16), 4, r))
            self.barrier(g)
        self.publish("vTokens", draws)
        for g in draws:
            self.mark("vTokens", g)
            self.fence(g)
            self.barrier(g)
        for g in self.owners(range(16), 4):
            self.mark("vLogits", g)
        self.all_fence()


def source():
    with open(os.path.join(CSRC, "lockstep_chain.cu")) as f:
        return f.read()


def buffers():
    kinds = re.search(r"enum Value \{ ([^}]*), kValues \};", source()).group(1).split(", ")
    rule = re.search(r"constexpr int turns_of\(int v\) \{ return v == vNormed \? (\d+) : \(v == vLogits \|\| v == vTokens \? (\d+) : (\d+)\); \}", source())
    normed, few, others = (int(n) for n in rule.groups())
    return {k: normed if k == "vNormed" else few if k in ("vLogits", "vTokens") else others for k in kinds}


def faults(rows, buffers, positions):
    walk = Walk(rows, buffers)
    for p in positions:
        walk.position(p)
    return walk.faults


@pytest.mark.parametrize("rows", [9, 15, 16, 17, 33, 64])
def test_no_place_is_marked_too_early_or_comes_round_too_soon(rows):
    assert faults(rows, buffers(), range(5)) == set()


def test_the_walk_sees_what_it_is_for():
    """One buffer less of any kind, and 8 rows, of which position 0 leaves nothing that everybody has waited for."""
    for kind, count in buffers().items():
        less = faults(9, {**buffers(), kind: count - 1}, range(5))
        assert less == {(kind, "late")} or (count == 3 and not less), (kind, less)
    assert ("vNormed", "early") in faults(8, buffers(), range(2))


def test_the_source_is_what_the_walk_follows():
    text = source()
    # who takes part
    part = text[text.index("bool takes_part("):text.index("int tile_of(")]
    assert "if (kind == kQkv) return true;" in part and "kGateUp) return cluster < 24;" in part
    assert "kHead) return cluster < 16;" in part and "return cluster >= 16;" in part
    # a norm marks its last use behind its new one, and fences; the I/O warps mark at a layer's end and fence there
    norm = text[text.index("// ---- norms: the row of this CTA"):text.index("// ---- dequantisers")]
    assert norm.index("turns.at<vNormed>() + to") < norm.index("turns.before<vNormed>() + to, mark()") < norm.index("marks_stand();")
    walk = text[text.index("projections(a, [&](int kind, int layer, int p) {\n            if (is_narrow(kind)) project("):]
    end = walk[walk.index("else if (kind == kDown || (kind == kQkv && ends_early))"):walk.index("else if (kind == kHead && a.draws != 0)")]
    order = [end.index(what) for what in ("turns.before<vQkv>()", "turns.before<vAtt>()", "turns.before<vMid>()", "turns.before<vAct>()",
                                          "turns.before<vIn>()", "marks_stand();")]
    assert order == sorted(order)
    assert walk.index("turns.before<vIn>()") < walk.index("marks_stand();") < walk.index("else if (kind == kDown")
    # and a projection has its barriers behind its polls
    project = text[text.index("auto project = "):text.index("auto mark_again = ")]
    assert project.index("bring_in(") < project.index("io_barrier();") < project.rindex("io_barrier();") < project.index("put_piece(to")


def test_every_word_of_a_piece_is_looked_at():
    """A piece of 16 bytes counts as written when none of its four words is the mark any more: nothing rests on its arriving at
    once.  (One that came in parts would be multiplied as NaN, which a run on a GPU has microseconds not to see.)"""
    text = source()
    poll = text[text.index("void poll("):text.index("int4 mark()")]
    for word in "xyzw":
        assert "(uint32_t)v[i].%s" % word in poll


def test_no_launch_for_rows_that_the_hand_overs_are_not_ordered_for():
    text = source()
    rule = text[text.index("bool lockstep_chain_available("):text.index("bool make_lockstep_map(")]
    assert "rows <= kChainRows" in rule and "lockstep_chain_available(c.rows)" in text[text.index("cudaError_t launch_lockstep_chain("):]


def test_a_frame_sees_whether_it_is_alone_and_is_seen_in_one_step():
    """Between the look at the census and the entry into it a prompt or a chain could have come in, unseen and not seeing."""
    with open(os.path.join(CSRC, "engine.cu")) as f:
        text = f.read()
    large = text[text.index("InFlight(Traffic* traffic, const Workspace& w, int rows, Large)"):]
    large = large[:large.index("    }\n")]
    assert large.count("lock_guard") == 1 and large.index("lock_guard") < large.index("->alone(") < large.index("->enter(")
    assert text.count("->alone(workspace_)") == 1 and "traffic->alone(" not in text


def test_no_launch_has_the_number_of_none():
    """Launches are numbered in 32 bits, and a frame may be sixteen of them: the number that stands for "none was given up" comes up
    after some twelve days, and the launch that bore it would give up."""
    text = source()
    assert "constexpr uint32_t kNoLaunch = ~0u;" in text and "threadIdx.x == 1 ? kNoLaunch : 0u" in text
    following = re.search(r"\*state = wt\.base >= kNoLaunch - 1 \? 0 : wt\.base \+ 1;", text)
    assert following and text.count("*state = ") == 1
