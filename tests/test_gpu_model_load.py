"""What a model makes of its weights when it is finalised, and what it does without when memory is short."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def replica_of(q3t, model, names, delay_cycles=0):
    """A second model, not yet finalised, whose storage is being filled from the first one's on torch's stream."""
    import torch
    dp = importlib.import_module("qwen3-tts-native_b200.dp")
    replica = q3t.NativeTalkerModel.create(0)
    if delay_cycles:
        torch.cuda._sleep(delay_cycles)
    for name in names:
        for (src, n), (dst, _) in zip(dp.image_spans(model.tensor_image(name)), dp.image_spans(replica.tensor_image(name))):
            dp.device_bytes(dst, n, 0).copy_(dp.device_bytes(src, n, 0))
        replica.adopt_tensor(name)
    return replica


def frames(q3t, model, sessions=1, count=2, seed=11):
    """(codes, next tokens, hidden row) of `count` frames of sessions that start on synthetic contexts."""
    model.set_option("mask_eos", 1)
    ss = []
    for i in range(sessions):
        s = model.create_session(128, seed + i)
        s.talker_sampling = q3t.SamplingConfig(True, 50, 0.9, 0.9, 1.05)
        s.predictor_sampling = q3t.SamplingConfig(True, 50, 1.0, 0.9, 1.0)
        s.synthetic_prefill(40 + i, seed + i)
        ss.append(s)
    out = []
    for f in range(count):
        if sessions == 1:
            ss[0].next_frame(7 + f)
        else:
            for p in model.batch_begin_device_frames(ss, [7 + f] * sessions):
                p.finish_without_consumer()
        out += [(s.current_semantic_token, *(np.array(x) for x in s.read_state()[:2])) for s in ss]
    for s in ss:
        s.close()
    return out


def same(a, b):
    return all(x[0] == y[0] and np.array_equal(x[1], y[1]) and np.array_equal(x[2], y[2]) for x, y in zip(a, b))


def test_weights_that_are_still_being_filled(q3t, gpu_model, checkpoint):
    """Adopted storage is filled by work that the caller has enqueued and not waited for: finalize makes its streams of the
    weights that will be there, not of what lies there when it is called."""
    want = frames(q3t, gpu_model), frames(q3t, gpu_model, 3)
    replica = replica_of(q3t, gpu_model, checkpoint.keys(), delay_cycles=1_000_000_000)
    try:
        replica.finalize()
        assert same(frames(q3t, replica), want[0]) and same(frames(q3t, replica, 3), want[1])
    finally:
        replica.close()


def test_without_memory_for_the_chain_and_for_long_passes(q3t, gpu_model, checkpoint):
    """The decode chain's second image of the weights is optional: where it cannot be allocated the model loads all the same and
    its frames run launch by launch (hundreds of kernels instead of a dozen), with the codes that the chain gives."""
    lib = q3t.library()
    want = frames(q3t, gpu_model, 2, count=1)
    replica = replica_of(q3t, gpu_model, checkpoint.keys())
    try:
        lib.q3t_test_fail_allocation_after(6)          # behind what every model needs (the table of embeddings, the rotations)
        replica.finalize()
        lib.q3t_test_fail_allocation_after(0)
        before = replica.kernel_launches()
        got = frames(q3t, replica, 2, count=1)
        assert replica.kernel_launches() - before > 300
        before = gpu_model.kernel_launches()
        frames(q3t, gpu_model, 2, count=1)
        assert gpu_model.kernel_launches() - before < 30
        for a, b in zip(got, want):
            assert np.array_equal(a[2], b[2])

        # likewise the workspace of prompts in one pass: without it they run in passes of 64
        rng = np.random.default_rng(3)
        text, codec = [int(t) for t in rng.integers(0, 151936, size=150)], [-1] * 150

        def prompt(model):
            s = model.create_session(160, 5)
            s.prefill(text, codec)
            out = s.current_semantic_token, s.read_state()[0], s.read_kv(27, 0, 150)
            s.close()
            return out

        gpu_model.set_option("prefill_chunk", 64)
        want = prompt(gpu_model)
        gpu_model.set_option("prefill_chunk", 2048)
        import torch
        s = replica.create_session(160, 5)
        free = torch.cuda.mem_get_info()[0]
        lib.q3t_test_fail_allocation_after(1)
        s.prefill(text, codec)
        lib.q3t_test_fail_allocation_after(0)
        # the workspace is 3 MB, the attention's scratch 4, with what the driver adds 12: no exchange of 7.6 MB for frames that never run here
        assert free - torch.cuda.mem_get_info()[0] <= 14 << 20
        s.close()
        got = prompt(replica)
        assert got[0] == want[0] and np.array_equal(got[1], want[1]) and all(np.array_equal(a, b) for a, b in zip(got[2], want[2]))
    finally:
        gpu_model.set_option("prefill_chunk", 2048)
        lib.q3t_test_fail_allocation_after(0)
        replica.close()


def test_without_memory_for_the_lockstep_chains_table(q3t, gpu_model, checkpoint):
    """The lockstep chain's table of tensor maps is optional too: without it large frames run launch by launch, with the same bits."""
    lib = q3t.library()
    want = frames(q3t, gpu_model, 12, count=1)
    replica = replica_of(q3t, gpu_model, checkpoint.keys())
    try:
        lib.q3t_test_fail_allocation_after(17)         # two that every model needs, fourteen of the decode chain, then this one
        replica.finalize()
        lib.q3t_test_fail_allocation_after(0)
        before = replica.kernel_launches()
        assert same(frames(q3t, replica, 12, count=1), want)
        assert replica.kernel_launches() - before > 600
        before = replica.kernel_launches()
        frames(q3t, replica, 2, count=1)
        assert replica.kernel_launches() - before < 30
    finally:
        lib.q3t_test_fail_allocation_after(0)
        replica.close()


def test_two_models_on_one_device(q3t, gpu_model, checkpoint):
    """Two replicas that decode at the same time from threads of their own, in large batches (tensor cores, norms as launches of
    their own) and in small ones (decode chain), decode what each decodes alone: nothing that a frame writes is shared."""
    import threading
    replica = replica_of(q3t, gpu_model, checkpoint.keys())
    try:
        replica.finalize()
        for sessions in (12, 3):
            want = frames(q3t, gpu_model, sessions, count=25)
            for _ in range(3):
                got = {}
                threads = [threading.Thread(target=lambda i=i, m=m: got.__setitem__(i, frames(q3t, m, sessions, count=25)))
                           for i, m in enumerate((gpu_model, replica))]
                for t in threads:
                    t.start()
                for t in threads:
                    t.join()
                assert same(got[0], want) and same(got[1], want)
    finally:
        replica.close()
