"""Order of the decode chain's hand-overs, read from its source: what orders one CTA's cache rows before another's
loads cannot be shown by running it, since the stores have microseconds to land."""
import os
import re

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
