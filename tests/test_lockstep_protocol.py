"""Hand-overs of the lockstep chain, read from its source."""
import os

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qwen3-tts-native_b200", "csrc")


def source():
    with open(os.path.join(CSRC, "lockstep_chain.cu")) as f:
        return f.read()


def test_every_word_of_a_piece_is_looked_at():
    """A piece of 16 bytes counts as written when none of its four words is the mark any more: nothing rests on its arriving at
    once.  (One that came in parts would be multiplied as NaN, which a run on a GPU has microseconds not to see.)"""
    text = source()
    poll = text[text.index("void poll("):text.index("int4 mark()")]
    for word in "xyzw":
        assert "(uint32_t)v[i].%s" % word in poll
