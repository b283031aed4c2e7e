"""Order of the decode chain's hand-overs, read from its source: what orders one CTA's cache rows before another's
loads cannot be shown by running it, since the stores have microseconds to land."""
import os
import re

import numpy as np

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qwen3-tts-native_b200", "csrc")


def body(source, signature):
    """Text of the function whose signature contains `signature`, comments taken out."""
    at = source.index(signature)
    start = source.index("{", at)
    depth = 0
    for i in range(start, len(source)):
        depth += {"{": 1, "}": -1}.get(source[i], 0)
        if depth == 0:
            return re.sub(r"//[^\n]*", "", source[start:i + 1])
    raise AssertionError(signature)


def test_cache_rows_are_released_by_their_writer_and_acquired_by_their_readers():
    """The predictor's K/V rows are appended in a layer's attention by one warp and read by other CTAs at the next position.
    So that warp has to release a flag behind its appends, and every reading warp has to acquire it before its first load."""
    with open(os.path.join(CSRC, "decode_chain.cu")) as f:
        source = f.read()
    assert "st.release.gpu" in body(source, "void put_behind(") and "ld.acquire.gpu" in body(source, "uint32_t get_ahead(")
    # the appending warp says so itself, in program order behind the position's layers
    attention = body(source, "void predictor_attention(")
    assert re.search(r"if \(rank == r\) append\(", attention) and "const int r = warp;" in attention
    say = body(source, "void say_appended(")
    assert re.search(r"warp < rows && rank == warp && lane == 0\) put_behind\(at, appended_flag\)", say)
    positions = body(source, "void run()")
    positions = positions[positions.index("p < kCodebooks"):]
    assert 0 < positions.index("layer(l, p,") < positions.index("say_appended(")
    # and no load of cache rows comes before the look at the flag
    layer = body(source, "void layer(int index, int pos")
    assert layer.count("page::load(") == 1
    assert re.search(r"if \(walk\.any\) \{\s*if \(!TALKER && index == 0 && pos > 0\) await_appended\(\);\s*page::load\(", layer)
    wait = body(source, "void await_appended(")
    assert wait.index("get_ahead(") < wait.rindex("__syncwarp()")


class Exchanges:
    """What each of the 8 x 16 CTAs knows of the others' progress, from what it has read alone: known[c, o] is the last exchange
    that c knows o to have read to its end.  A buffer may be written again once the writer knows that of all who read it."""

    SLICES, RANKS = 8, 16

    def __init__(self):
        n = self.SLICES * self.RANKS
        self.known = np.zeros((n, n), dtype=np.int64)
        self.number = 0
        self.last_use = {}                                   # (kind, buffer) -> number of the exchange and its readers
        self.slice, self.rank = np.arange(n) // self.RANKS, np.arange(n) % self.RANKS

    def readers(self, scope):
        """[writer, reader]"""
        if scope == "group":
            return self.slice[:, None] == self.slice[None, :]
        if scope == "rank":
            return self.rank[:, None] == self.rank[None, :]
        return np.ones_like(self.known, dtype=bool)

    def exchange(self, kind, buffer, scope):
        reads = self.readers(scope)
        before = self.last_use.get((kind, buffer))
        if before is not None:
            number, readers = before
            assert (self.known[readers] >= number).all(), f"{kind} {buffer}: exchange {self.number + 1} may overwrite {number}"
        self.number += 1
        self.last_use[(kind, buffer)] = (self.number, reads)
        sent = self.known.copy()
        for reader in range(len(sent)):
            self.known[reader] = sent[reads[:, reader]].max(axis=0)
        np.fill_diagonal(self.known, self.number)


def hand_overs(source):
    """A layer's hand-overs in source order: buffers taken, exchanges, the early end."""
    layer = body(source, "void layer(int index, int pos")
    return re.findall(r"flip\(k\w+\)|\breturn;|\bcollect_group\(|\bmma_slice\(", layer)


def walk_predictor(source, one_hop, ends_early, positions=16, layers=5):
    net, flips = Exchanges(), {}

    def flip(kind):
        flips[kind] = flips.get(kind, 1) ^ 1
        return flips[kind]

    def layer(index, position):
        for half in range(2):
            for what in hand_overs(source):
                if what.startswith("flip"):
                    flip(what[5:-1])
                elif what == "return;":
                    if half == 0 and ends_early and position == 0 and index + 1 == layers:
                        return
                elif what == "collect_group(":
                    net.exchange("kGroup", flips["kGroup"], "group")
                else:
                    net.exchange("kPart", flips["kPart"], "all" if one_hop else "rank")
                    if not one_hop:
                        net.exchange("kHid", flip("kHid"), "group")

    for position in range(positions):
        for index in range(layers):
            layer(index, position)
        if position > 0:
            net.exchange("kLogits", flip("kLogits"), "all")
    return net.number


def test_no_buffer_is_written_before_its_readers_are_known_to_have_read_it():
    """Walks the predictor's hand-overs in the order of the source, with and without the early end of position 0."""
    with open(os.path.join(CSRC, "decode_chain.cu")) as f:
        source = f.read()
    assert sorted(set(hand_overs(source))) == ["collect_group(", "flip(kGroup)", "flip(kPart)", "mma_slice(", "return;"]
    assert "flip(kHid)" in body(source, "void collect_partials(")
    assert walk_predictor(source, one_hop=True, ends_early=False) == 16 * 5 * 4 + 15
    assert walk_predictor(source, one_hop=False, ends_early=False) == 16 * 5 * 6 + 15
    assert walk_predictor(source, one_hop=False, ends_early=True) == 16 * 5 * 6 + 15 - 5


def test_setting_up_the_chain_allocates_through_the_engine_alone():
    """A chain that finds no memory is done without; only the engine's own buffers report that as what it is."""
    for name in ("decode_chain.cu", "chain_places.cu"):
        with open(os.path.join(CSRC, name)) as f:
            assert not re.search(r"\bcuda(Malloc|HostAlloc|Free)\w*\(", f.read()), name
