"""Sessions, caches and models that are made while the default stream is busy.

The engine's streams do not wait for the default stream, so nothing that a frame reads may be set up there: a session's state
that is cleared after its random state was set draws other tokens, a table of slabs that is filled too late points nowhere."""
import importlib

import pytest

pytestmark = pytest.mark.gpu

TEXT, CODEC = [1501, 77, 151935, -1, 9000, 42, 31337, 8, 5, 6, 7, 8], [-1, 2148, 3, 2049, -1, 100, 7, 2000, -1, -1, -1, -1]


def run(q3t, model, capacity, batch):
    """Sessions made now: prompt, four frames alone and, where `batch`, four in lockstep."""
    model.set_option("mask_eos", 1)
    out, ss = [], []
    for i in range(3 if batch else 1):
        t = q3t.SamplingConfig(True, 50, 0.9, 0.9, 1.05)
        s = model.start_prompt(TEXT, CODEC, capacity, 70 + i, t, q3t.SamplingConfig(True, 50, 1.0, 0.9, 1.0))
        out.append(s.current_semantic_token)
        out += [(f.codes, f.next_semantic_token) for f in (s.next_frame(3 + k) for k in range(4))]
        ss.append(s)
    for k in range(4 if batch else 0):
        out.append([p.finish_without_consumer().next_semantic_token for p in model.batch_begin_device_frames(ss, [9 + k] * len(ss))])
    out += [s.read_state()[2] for s in ss]
    for s in ss:
        s.close()
    return out


def test_sessions_made_while_the_default_stream_is_busy(q3t, gpu_model):
    import torch
    want = run(q3t, gpu_model, 64, True)
    for capacity in (64, 4096):                       # the latter needs another slab of the cache
        torch.cuda._sleep(1_000_000_000)              # on the default stream: half a second
        assert run(q3t, gpu_model, capacity, True) == want
    torch.cuda.synchronize()


def test_model_finalised_while_the_default_stream_is_busy(q3t, gpu_model, checkpoint):
    import torch
    dp = importlib.import_module("qwen3-tts-native_b200.dp")
    want = run(q3t, gpu_model, 64, True)
    replica = q3t.NativeTalkerModel.create(0)
    try:
        dp.copy_weight_image(gpu_model, replica, list(checkpoint.keys()))
        torch.cuda._sleep(1_000_000_000)
        replica.finalize()
        torch.cuda._sleep(1_000_000_000)
        assert run(q3t, replica, 64, True) == want
        torch.cuda.synchronize()
    finally:
        replica.close()
