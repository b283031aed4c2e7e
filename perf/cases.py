"""What the speed of this library is judged by: the calls its users make, at the sizes they make them.

Five kinds of case, all through public entry points:

  utterance    one request served alone: reset, prompt, then a few streamed frames, the host reading every
               frame's codes (qwen3_tts_session_reset / _prefill / _next_frame)
  decode       one frame for each of `sessions` running utterances, alone (_next_frame) or in lockstep
               (qwen3_tts_model_batch_next_frame_begin_v2 + qwen3_tts_session_next_frame_finish_v2), ragged contexts
  prompt       one prompt up to its first semantic token (_reset / _prefill)
  projections  the operator-level int8 projections of a few talker layers, as a host with its own decoder loop calls
               them (q3t_launch_int8_gemm_rows, q3t_launch_int8_gate_up_silu_rows)
  attention    the operator-level decode attention over contiguous bf16 caches, ragged lengths
               (q3t_launch_batch_causal_gqa_attention_fast)

Weights are synthetic (no checkpoint is at hand), of the real architecture and loaded once per process, as a serving
process does.  Their output heads are tied to the embeddings so that the logits are as peaked as a trained model's: with
unrelated random heads the two best logits are closer than one bf16 rounding and every token would hang on the last bit.
"""
import ctypes as C
import importlib
import math
import zlib

import numpy as np
import torch

q3t = importlib.import_module("qwen3-tts-native_b200")
synth = importlib.import_module("qwen3-tts-native_b200.synth")

HIDDEN, INTER, QKV, VOCAB, SEMANTIC = 2048, 6144, 4096, 3072, 2048
LAYERS, PREDICTOR_LAYERS, GROUPS = 28, 5, 15
Q_HEADS, KV_HEADS, HEAD_DIM = 16, 8, 128
LAYER_WEIGHTS = QKV * HIDDEN + HIDDEN * HIDDEN + 2 * INTER * HIDDEN + HIDDEN * INTER       # int8 bytes of a talker layer
TALKER_WEIGHTS = LAYERS * LAYER_WEIGHTS + VOCAB * HIDDEN + 2 * HIDDEN * HIDDEN
PREDICTOR_LAYER = 4096 * 1024 + 1024 * 2048 + 2 * 3072 * 1024 + 1024 * 3072
PREDICTOR_WEIGHTS = PREDICTOR_LAYERS * PREDICTOR_LAYER + GROUPS * 2048 * 1024 + 1024 * 2048
PREDICTOR_FLOPS = 2 * (16 * (PREDICTOR_LAYERS * PREDICTOR_LAYER + 1024 * 2048) + GROUPS * 2048 * 1024)
KV_TOKEN = LAYERS * 2 * KV_HEADS * HEAD_DIM * 2                                            # bytes of one cached position
MAX_SEQUENCE = 8192
TEXT_IDS = 151936
OP_LAYERS = 4            # 201 MB of int8 weights: more than the L2 holds, as in a decoder that streams them


def listed():
    return [
        # the first packet of audio of a short line: time to first sound (four frames are one codec packet)
        {"name": "packet_short_prompt", "kind": "utterance", "prompt": 24, "frames": 4},
        # two seconds of a streamed answer after an ordinary prompt
        {"name": "stream_128", "kind": "utterance", "prompt": 128, "frames": 25},
        # one listener, far into a long reading
        {"name": "decode_1_long", "kind": "decode", "sessions": 1, "shortest": 3000, "longest": 3000},
        # a few users on one GPU
        {"name": "decode_3", "kind": "decode", "sessions": 3, "shortest": 64, "longest": 1024},
        # the largest lockstep batch of the reference host
        {"name": "decode_8", "kind": "decode", "sessions": 8, "shortest": 64, "longest": 1024},
        # an odd, half-filled server
        {"name": "decode_23", "kind": "decode", "sessions": 23, "shortest": 64, "longest": 2048},
        # a full one: the batched benchmark configuration
        {"name": "decode_64", "kind": "decode", "sessions": 64, "shortest": 64, "longest": 2048},
        # a voice description and a sentence
        {"name": "prompt_150", "kind": "prompt", "prompt": 150},
        # a long passage with its instructions
        {"name": "prompt_1500", "kind": "prompt", "prompt": 1500},
        # the single-session projections, one activation row
        {"name": "projections_1", "kind": "projections", "rows": 1},
        # and those of a well-filled batch
        {"name": "projections_48", "kind": "projections", "rows": 48},
        # attention of the full batch, one layer
        {"name": "attention_64", "kind": "attention", "rows": 64, "shortest": 64, "longest": 2048},
    ]


def _log_uniform(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["utterance", "decode", "decode", "decode", "prompt", "projections", "attention"])
    if kind == "utterance":
        return {"kind": kind, "prompt": _log_uniform(rng, 12, 256), "frames": rng.randint(1, 25)}
    if kind == "decode":
        sessions = rng.choice([1, _log_uniform(rng, 1, 64)])
        shortest = _log_uniform(rng, 16, 1024)
        longest = _log_uniform(rng, shortest, 4096 if sessions <= 8 else 2048)
        return {"kind": kind, "sessions": sessions, "shortest": shortest, "longest": longest}
    if kind == "prompt":
        return {"kind": kind, "prompt": _log_uniform(rng, 12, 1500)}
    if kind == "projections":
        return {"kind": kind, "rows": _log_uniform(rng, 1, 64)}
    shortest = _log_uniform(rng, 16, 1024)
    return {"kind": kind, "rows": _log_uniform(rng, 1, 64), "shortest": shortest, "longest": _log_uniform(rng, shortest, 2048)}


# ---- the model, loaded once --------------------------------------------------------------------------------------------

_loaded = None


def _tensors():
    """(name, bf16 bits) of all 404 tensors: the distributions of the package's synthetic checkpoint, except that layer outputs
    carry the usual 1/sqrt(2 layers), embeddings have unit scale (the codec's twice that) and each head row points along the
    embedding of the token that it follows."""
    device = torch.device("cuda")
    shapes = synth.tensor_shapes(128)
    generator = torch.Generator(device=device)

    def normal(name):
        generator.manual_seed(zlib.crc32(name.encode()) & 0x7FFFFFFF)
        return torch.randn(shapes[name], generator=generator, device=device)

    def unit(rows):
        return rows / rows.square().mean(1, keepdim=True).sqrt()

    def matrix(name):
        generator.manual_seed(zlib.crc32(name.encode()) & 0x7FFFFFFF)
        rows, cols = shapes[name]
        q = torch.randint(-127, 128, (rows, cols), generator=generator, device=device, dtype=torch.int8).float()
        scale = (0.5 + torch.rand((rows, 1), generator=generator, device=device)) / (73.6 * cols ** 0.5)
        if name.endswith(("o_proj.weight", "down_proj.weight")):
            scale = scale / (2 * (PREDICTOR_LAYERS if "code_predictor" in name else LAYERS)) ** 0.5
        return q * scale

    codec = "talker.model.codec_embedding.weight"
    mtp = "talker.code_predictor.small_to_mtp_projection.weight"
    follows = (torch.arange(SEMANTIC, device=device) * 1021 + 7) % SEMANTIC        # token t comes after follows[t]

    def embedding(group):                                                         # 0: the codec's, 1..15: the predictor's
        name = codec if group == 0 else "talker.code_predictor.model.codec_embedding.%d.weight" % (group - 1)
        return normal(name) * (2.0 if group == 0 else 1.0)

    for name in shapes:
        if name == codec:
            t = embedding(0)
        elif ".codec_embedding." in name:
            t = embedding(int(name.split(".")[-2]) + 1)
        elif name == "talker.codec_head.weight":
            t = 0.0005 * normal(name)                                             # reserved tokens and the end of speech: unlikely
            t[:SEMANTIC] += unit(embedding(0)[:SEMANTIC])[follows] * 0.015
        elif ".lm_head." in name:
            group = int(name.split(".")[-2])
            t = unit(embedding(group)[:SEMANTIC] @ matrix(mtp).T)[follows] * 0.018
        elif name.endswith("norm.weight") or name.endswith("layernorm.weight"):
            t = 1.0 + 0.02 * normal(name)
        elif name.endswith(".bias") or "embedding" in name:
            t = 0.02 * normal(name)
        else:
            t = matrix(name)
        yield name, t.to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16)


def _model():
    global _loaded
    if _loaded is None:
        _loaded = q3t.NativeTalkerModel.load(0, _tensors())
        torch.cuda.empty_cache()
    return _loaded


TALKER_SAMPLING = q3t.SamplingConfig(True, 50, 0.9, 0.9, 1.05)
PREDICTOR_SAMPLING = q3t.SamplingConfig(True, 50, 0.9, 0.9, 1.0)


def _session(capacity, seed):
    s = _model().create_session(capacity, seed)
    s.talker_sampling, s.predictor_sampling = TALKER_SAMPLING, PREDICTOR_SAMPLING
    return s


# ---- inputs ------------------------------------------------------------------------------------------------------------

def _prompt_state(case, seed):
    rng = np.random.default_rng(seed)
    n = case["prompt"]
    text = [int(t) for t in rng.integers(0, TEXT_IDS, size=n)]
    codec = [-1] * n                                       # text positions, then the codec's opening tokens
    for i in range(max(1, n - 4), n):
        codec[i] = int(rng.integers(0, SEMANTIC))
    frames = case.get("frames", 0)
    capacity = max(16, (n + frames + 15) // 16 * 16)
    return {"case": case, "seed": 1 + seed % (1 << 40), "session": _session(capacity, 1 + seed), "text": text, "codec": codec,
            "trailing": [int(t) for t in rng.integers(0, TEXT_IDS, size=frames)]}


def _lengths(rng, case, count):
    return [int(v) for v in rng.integers(case["shortest"], case["longest"] + 1, size=count)]


def _decode_state(case, seed):
    rng = np.random.default_rng(seed)
    n = case["sessions"]
    lengths = _lengths(rng, case, n)
    room = 4096 if n <= 8 else 1024
    state = {"case": case, "lengths": lengths, "trailing": [int(t) for t in rng.integers(0, TEXT_IDS, size=n)], "codes": None,
             "taken": None, "left": 0, "seeds": [1 + (seed * 131 + i) % (1 << 40) for i in range(n)]}
    state["room"] = min(min(room, MAX_SEQUENCE - v) for v in lengths)
    state["sessions"] = [_session((v + state["room"] + 15) // 16 * 16, s) for v, s in zip(lengths, state["seeds"])]
    _start_contexts(state)
    return state


def _start_contexts(state):
    """Every session at its context length, its cache filled with N(0, 1) values (also when the caches have run full)."""
    for s, length, seed in zip(state["sessions"], state["lengths"], state["seeds"]):
        s.reset(seed)
        s.synthetic_prefill(length, seed)
    state["left"] = state["room"] - 1


class _Codes:
    """A session's sixteen codes where they lie on the device, for torch to look at."""

    def __init__(self, address):
        self.__cuda_array_interface__ = {"shape": (16,), "typestr": "<i2", "data": (address, False), "version": 2}


def _projection_state(case, seed):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    rows = case["rows"]

    def int8(n, k):
        w = torch.randint(-127, 128, (n, k), generator=generator, device="cuda", dtype=torch.int8)
        s = (0.5 + torch.rand((n,), generator=generator, device="cuda")) / (73.6 * k ** 0.5)
        return w, s

    def out(n):
        return torch.zeros((rows, n), dtype=torch.bfloat16, device="cuda")

    lib = q3t.library()
    keep, calls, outputs = [], [], []
    for _ in range(OP_LAYERS):
        for fn, n, k, matrix_rows in ((lib.q3t_launch_int8_gemm_rows, QKV, HIDDEN, QKV), (lib.q3t_launch_int8_gemm_rows, HIDDEN, HIDDEN, HIDDEN),
                                      (lib.q3t_launch_int8_gate_up_silu_rows, INTER, HIDDEN, 2 * INTER),
                                      (lib.q3t_launch_int8_gemm_rows, HIDDEN, INTER, HIDDEN)):
            w, s = int8(matrix_rows, k)
            x = torch.randn((rows, k), generator=generator, device="cuda").to(torch.bfloat16)
            y = out(n)
            keep += [w, s, x]
            outputs.append(y)
            calls.append((fn, C.c_void_p(w.data_ptr()), C.c_void_p(s.data_ptr()), C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), k, n))
    return {"case": case, "keep": keep, "calls": calls, "outputs": outputs}


def _attention_state(case, seed):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    rows, width = case["rows"], KV_HEADS * HEAD_DIM
    lengths = _lengths(rng, case, rows)
    capacity = (max(lengths) + 63) // 64 * 64

    def normal(*shape):
        return torch.randn(shape, generator=generator, device="cuda", dtype=torch.bfloat16)

    q, k, v = normal(rows, Q_HEADS * HEAD_DIM), normal(rows, capacity, width), normal(rows, capacity, width)
    stride = capacity * width * 2
    bases = [torch.tensor([t.data_ptr() + r * stride for r in range(rows)], dtype=torch.int64, device="cuda") for t in (k, v)]
    positions = torch.tensor([n - 1 for n in lengths], dtype=torch.int32, device="cuda")
    y = torch.zeros((rows, Q_HEADS * HEAD_DIM), dtype=torch.bfloat16, device="cuda")
    size = int(q3t.library().q3t_attention_scratch_bytes(rows, Q_HEADS, KV_HEADS, HEAD_DIM, capacity))
    scratch = torch.empty((max(size, 16),), dtype=torch.uint8, device="cuda")
    p = [C.c_void_p(t.data_ptr()) for t in (q, bases[0], bases[1], positions, y)]
    return {"case": case, "keep": [q, k, v, positions, scratch, bases], "output": y,
            "call": (*p, rows, Q_HEADS, KV_HEADS, HEAD_DIM, capacity, C.c_void_p(scratch.data_ptr()), C.c_size_t(size), None)}


def prepare(case, seed):
    if case["kind"] in ("utterance", "prompt"):
        return _prompt_state(case, seed)
    if case["kind"] == "decode":
        return _decode_state(case, seed)
    return _projection_state(case, seed) if case["kind"] == "projections" else _attention_state(case, seed)


# ---- one pass ----------------------------------------------------------------------------------------------------------

def _floats(bits):
    return (bits.astype(np.uint32) << 16).view(np.float32)


def _must(status):
    if status != 0:
        raise RuntimeError("launch returned %d" % status)


def run(state):
    kind = state["case"]["kind"]
    if kind in ("utterance", "prompt"):
        s = state["session"]
        s.reset(state["seed"])
        s.prefill(state["text"], state["codec"])
        tokens, codes = [s.current_semantic_token], []
        for trailing in state["trailing"]:
            frame = s.next_frame(trailing)
            codes.append(frame.codes)
            tokens.append(frame.next_semantic_token)
        hidden, _, _ = s.read_state()                       # the session's state, as a checkpoint of it would keep it
        return {"tokens": np.array(tokens), "codes": np.array(codes, dtype=np.int64), "hidden": _floats(hidden)}
    if kind == "decode":
        if state["left"] < 1:
            _start_contexts(state)
        state["left"] -= 1
        sessions = state["sessions"]
        if len(sessions) == 1:
            frame = sessions[0].next_frame(state["trailing"][0])
            return {"tokens": np.array([frame.next_semantic_token]), "codes": np.array([frame.codes])}
        if state["taken"] is not None:
            state["taken"].synchronize()                     # the codec has taken the codes of the frame before
        pending = _model().batch_begin_device_frames(sessions, state["trailing"])
        if state["codes"] is None:
            state["codes"] = [torch.as_tensor(_Codes(p.device_codes), device="cuda") for p in pending]
            state["taken"] = torch.cuda.Event()
        tokens = [p.finish().next_semantic_token for p in pending]
        codes = torch.stack(state["codes"])                  # what the codec reads: [sessions][16]
        state["taken"].record()
        return {"tokens": np.array(tokens), "codes": codes}
    if kind == "projections":
        rows = state["case"]["rows"]
        for fn, w, s, x, y, k, n in state["calls"]:
            _must(fn(w, s, x, y, k, n, rows, None))
        return state["outputs"]
    _must(q3t.library().q3t_launch_batch_causal_gqa_attention_fast(*state["call"]))
    return state["output"]


# ---- what a pass cannot do without -------------------------------------------------------------------------------------

def _frame_work(rows, context_sum):
    bytes_ = TALKER_WEIGHTS + PREDICTOR_WEIGHTS + KV_TOKEN * context_sum
    flops = rows * (2 * TALKER_WEIGHTS + PREDICTOR_FLOPS) + LAYERS * 4 * Q_HEADS * HEAD_DIM * context_sum
    return bytes_, flops


def work(case):
    kind = case["kind"]
    mean = (case.get("shortest", 0) + case.get("longest", 0)) / 2
    if kind == "decode":
        b, f = _frame_work(case["sessions"], mean * case["sessions"])
        return {"bytes": b, "flops": f}
    if kind in ("utterance", "prompt"):
        n = case["prompt"]
        b = TALKER_WEIGHTS + KV_TOKEN * n + 2 * HIDDEN * n
        f = 2 * n * (LAYERS * LAYER_WEIGHTS + 2 * HIDDEN * HIDDEN) + 2 * VOCAB * HIDDEN + LAYERS * 2 * Q_HEADS * HEAD_DIM * n * n
        for i in range(case.get("frames", 0)):
            more = _frame_work(1, n + i + 1)
            b, f = b + more[0], f + more[1]
        return {"bytes": b, "flops": f}
    rows = case["rows"]
    if kind == "projections":
        per = LAYER_WEIGHTS + 4 * (QKV + 2 * HIDDEN + 2 * INTER) + 2 * rows * (3 * HIDDEN + INTER + QKV + 2 * HIDDEN + INTER)
        return {"bytes": OP_LAYERS * per, "flops": OP_LAYERS * 2 * rows * LAYER_WEIGHTS}
    return {"bytes": rows * (mean * 2 * KV_HEADS * HEAD_DIM * 2 + 2 * Q_HEADS * HEAD_DIM * 2), "flops": rows * mean * 4 * Q_HEADS * HEAD_DIM}


def tolerance(case):
    """bf16 operators: one rounding of the result each, so 2^-8 of a value at most, 1e-2 with the sums inside; a hidden state after 28
    layers of them gathers a few such roundings.  Tokens are drawn from peaked distributions: a draw on an edge may fall the other way."""
    if case["kind"] in ("utterance", "prompt"):
        return {"rel": 2e-2, "max": 0.2, "differ": 0.01}
    if case["kind"] == "decode":
        return {"rel": 0.0, "differ": 0.01}
    return {"rel": 1e-2, "max": 0.1}
