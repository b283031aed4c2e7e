"""The lockstep chain (the predictor's part of 9 to 64 sessions in one cooperative launch) against the frame made launch by
launch: the same sums in the same order, so the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def model(gpu_model):
    gpu_model.set_option("mask_eos", 1)
    yield gpu_model
    gpu_model.set_option("decode_chain", 1)


def frames(q3t, model, rows, chain, count, predictor=None):
    model.set_option("decode_chain", chain)
    sessions = []
    for i in range(rows):
        length = 1 + (37 * i) % 90
        s = model.create_session((length + count + 32) // 16 * 16, 100 + i)
        s.talker_sampling = q3t.SamplingConfig(True, 50, 0.9, 0.9, 1.05)
        s.predictor_sampling = predictor(i) if predictor else q3t.SamplingConfig(True, 50, 1.0, 0.9, 1.0)
        s.synthetic_prefill(length, 1000 + i)
        sessions.append(s)
    launches = model.kernel_launches()
    out = []
    for f in range(count):
        for p in model.batch_begin_device_frames(sessions, [7 + f] * rows):
            p.finish_without_consumer()
        out.append([(s.read_state()[1].tolist(), s.current_semantic_token) for s in sessions])
    ends = [(s.read_state()[0], s.read_state()[2]) for s in sessions]
    for s in sessions:
        s.close()
    return out, ends, model.kernel_launches() - launches


# every tile, with rows that fill it and rows that leave its last share of four empty or nearly so
@pytest.mark.parametrize("rows", [9, 12, 13, 16, 17, 23, 32, 33, 48, 49, 50, 64])
def test_lockstep_chain_equals_launch_by_launch(q3t, model, rows):
    chained, launched = frames(q3t, model, rows, 1, 3), frames(q3t, model, rows, 0, 3)
    assert chained[0] == launched[0]
    for (ha, ra), (hb, rb) in zip(chained[1], launched[1]):
        assert np.array_equal(ha, hb) and ra == rb
    assert launched[2] > 2000 and chained[2] < launched[2] / 2, (chained[2], launched[2])
    assert q3t.library().q3t_kernel_error_count() == 0


@pytest.mark.parametrize("inside", [True, False])
def test_every_draw(q3t, model, inside):
    """Draws that differ between the rows of a frame: greedy, a few and many, which the chain makes itself, and more than it
    ranks, with which the sampler runs between its positions."""
    kinds = [q3t.SamplingConfig.greedy(), q3t.SamplingConfig(True, 1, 1.0, 0.9, 1.0), q3t.SamplingConfig(True, 128, 0.8, 1.1, 1.0)]
    if not inside:
        kinds += [q3t.SamplingConfig(True, 300, 0.9, 1.0, 1.0), q3t.SamplingConfig(True, 0, 1.0, 1.0, 1.0)]
    pick = lambda i: kinds[i % len(kinds)]
    chained, launched = frames(q3t, model, 20, 1, 2, pick), frames(q3t, model, 20, 0, 2, pick)
    assert chained[0] == launched[0]
    assert all(np.array_equal(a[0], b[0]) and a[1] == b[1] for a, b in zip(chained[1], launched[1]))
    # and the frames were made the way this is about: one launch for all positions, or one for each with a draw behind it
    whole = frames(q3t, model, 20, 1, 2)[2]
    assert chained[2] == whole + (0 if inside else 2 * (15 + 15)) and chained[2] < launched[2] / 2, (chained[2], whole, launched[2])
    assert q3t.library().q3t_kernel_error_count() == 0


def test_row_counts_in_turn(q3t, model):
    """The chain's places are marked for one row count: another count, and the first again, start with all of them marked."""
    want = {n: frames(q3t, model, n, 0, 1) for n in (12, 40, 9)}
    for n in (12, 40, 9, 40, 12):
        got = frames(q3t, model, n, 1, 1)
        assert got[0] == want[n][0] and got[2] < want[n][2] / 2
    assert q3t.library().q3t_kernel_error_count() == 0


class Batch:
    """Sessions that are stepped frame by frame, with draws of one kind or another."""

    def __init__(self, q3t, model, rows, chain):
        model.set_option("decode_chain", chain)
        self.q3t, self.model, self.frame = q3t, model, 0
        self.sessions = [model.create_session(256, 100 + i) for i in range(rows)]
        for i, s in enumerate(self.sessions):
            s.talker_sampling = q3t.SamplingConfig(True, 50, 0.9, 0.9, 1.05)
            s.synthetic_prefill(1 + (37 * i) % 90, 1000 + i)

    def step(self, top_k=50):
        """(what came of it, kernels launched)"""
        for s in self.sessions:
            s.predictor_sampling = self.q3t.SamplingConfig(True, top_k, 1.0, 0.9, 1.0)
        self.frame += 1
        before = self.model.kernel_launches()
        for p in self.model.batch_begin_device_frames(self.sessions, [7 + self.frame] * len(self.sessions)):
            p.finish_without_consumer()
        return [tuple(np.array(x).tobytes() for x in s.read_state()) for s in self.sessions], self.model.kernel_launches() - before

    def close(self):
        for s in self.sessions:
            s.close()


def test_ways_in_turn(q3t, model):
    """One launch for a frame, one for each position, launch by launch and back, at one row count: nothing is marked anew between them."""
    kinds = [50, 300, 50, 50, 0, 300, 128, 50]
    launched = Batch(q3t, model, 13, 0)
    want = [launched.step(k) for k in kinds]
    launched.close()
    mixed = Batch(q3t, model, 13, 1)
    for i, k in enumerate(kinds):
        model.set_option("decode_chain", 0 if i == 3 else 1)
        got, count = mixed.step(k)
        assert got == want[i][0], i
        assert (count < want[i][1] / 2) == (i != 3)
    mixed.close()
    assert q3t.library().q3t_kernel_error_count() == 0


def test_after_a_wait_that_ran_out(q3t, model):
    """Device errors that have been counted since the last frame: the chain starts with every place marked, and gives the same bits."""
    launched = Batch(q3t, model, 13, 0)
    want = [launched.step()[0] for _ in range(4)]
    launched.close()
    chained = Batch(q3t, model, 13, 1)
    for i in range(4):
        got, count = chained.step()
        assert got == want[i] and count < 400, i
        if i % 2 == 0:
            assert q3t.library().q3t_test_report_device_wait_failure(0) == 0
    chained.close()


@pytest.mark.parametrize("rows", [12, 40])
def test_beside_other_work(q3t, model, rows):
    """Prompts that come while a batch decodes, and kernels of the host's that hold SMs, few and more than a launch leaves: every frame
    and every prompt is what it is on a quiet device."""
    import ctypes as C
    import threading
    import torch
    lib = q3t.library()
    lib.q3t_test_hold_sms.argtypes = [C.c_int32, C.c_uint64, C.c_void_p]
    rng = np.random.default_rng(rows)
    prompts = [([int(t) for t in rng.integers(0, 151936, size=n)], [-1] * n) for n in (24, 150)]
    steps = 16

    def prompt(which):
        s = model.create_session(192, 3)
        s.prefill(*prompts[which])
        out = s.current_semantic_token, s.read_state()[0].tobytes()
        s.close()
        return out

    def decode(held=0, ns=0):
        batch, stream, out = Batch(q3t, model, rows, 1), torch.cuda.Stream(), []
        for _ in range(steps):
            if held:
                assert lib.q3t_test_hold_sms(held, ns, stream.cuda_stream) == 0
            out.append(batch.step()[0])
        torch.cuda.synchronize()
        batch.close()
        return out

    want, wanted = decode(), [prompt(0), prompt(1)]
    for held, ns in ((4, 3_000_000), (20, 1_000_000), (60, 1_000_000), (148, 100_000)):
        assert decode(held, ns) == want, held
    got, prompted, done = [], [], threading.Event()

    def others():
        i = 0
        while not done.is_set():
            prompted.append((i % 2, prompt(i % 2)))
            done.wait(0.004 * (i % 4))
            i += 1

    thread = threading.Thread(target=others)
    thread.start()
    try:
        for _ in range(3):
            got.append(decode())
    finally:
        done.set()
        thread.join()
    assert all(g == want for g in got) and len(prompted) > 4 and all(out == wanted[which] for which, out in prompted)
    assert lib.q3t_kernel_error_count() == 0


def test_without_graphs_launch_by_launch(q3t, model):
    """With "use_graphs" 0 a frame is made launch by launch, as the header has it: the 600th of its launches is there to fail."""
    lib = q3t.library()
    model.set_option("decode_chain", 1)
    model.set_option("use_graphs", 0)
    sessions = []
    try:
        for i in range(12):
            s = model.create_session(64, 1 + i)
            s.synthetic_prefill(20 + i, 1 + i)
            sessions.append(s)
        lib.q3t_test_fail_launch_after(600)
        with pytest.raises(q3t.NativeTalkerStatusError):
            model.batch_begin_device_frames(sessions, [7] * 12)
    finally:
        lib.q3t_test_fail_launch_after(0)
        model.set_option("use_graphs", 1)
        for s in sessions:
            s.close()
