"""The decode chain (frames of up to eight sessions as two cooperative launches) against the frame made
launch by launch, at the context lengths where its page walk and merges change."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one page and its edges, the first page of a second class (16 x 16 tokens), several pages per warp
POSITIONS = [1, 15, 16, 17, 255, 256, 700, 2100]


@pytest.fixture(scope="module")
def model(gpu_model):
    gpu_model.set_option("mask_eos", 1)
    yield gpu_model
    gpu_model.set_option("decode_chain", 1)


def frame(q3t, model, positions, chain, predictor=None, frames=1):
    """(codes, next tokens, hidden rows, layer-0 and layer-1 K/V rows of the new token) after `frames` frames."""
    model.set_option("decode_chain", chain)
    sessions = []
    for i, p in enumerate(positions):
        s = model.create_session((p + frames + 32) // 16 * 16, 100 + i)
        s.talker_sampling = q3t.SamplingConfig(True, 50, 0.9, 0.9, 1.05)
        s.predictor_sampling = predictor or q3t.SamplingConfig(True, 50, 1.0, 0.9, 1.0)
        s.synthetic_prefill(p, 1000 + i)
        sessions.append(s)
    for f in range(frames):
        if len(sessions) == 1:
            sessions[0].next_frame(7 + f)
        else:
            for p in model.batch_begin_device_frames(sessions, [7 + f] * len(sessions)):
                p.finish_without_consumer()
    out = []
    for s, p in zip(sessions, positions):
        hidden, tokens, rng = s.read_state()
        kv = [np.stack(s.read_kv(layer, p, 1)) for layer in (0, 1)]
        out.append((tokens, s.current_semantic_token, hidden, kv, rng))
        s.close()
    return out


@pytest.mark.parametrize("rows", [1, 2, 3, 5, 8])
def test_chain_equals_launch_by_launch(q3t, orc, model, rows):
    """The predictor's part is the same to the bit (codes, random state); so is the new token's K/V of layer 0.  The
    talker merges a long context page by page instead of in chunks of 64 tokens: fp32 sums in another order.  From
    there to layer 1's K lie eight bf16 roundings (attention, o, gate/up, down, q/k/v, norm twice, rotation), each of
    which may fall the other way by an ulp, 2^-8 to 2^-7 of a value, in part of the elements: 8 x 2^-9 = 2^-6 at most.
    After 28 layers: a direction within 0.995.  Within one page: to the bit."""
    positions = POSITIONS[:rows] if rows != 3 else POSITIONS[5:8]
    chained, launched = frame(q3t, model, positions, 1), frame(q3t, model, positions, 0)
    for p, a, b in zip(positions, chained, launched):
        assert np.array_equal(a[0], b[0]), p
        assert np.array_equal(a[3][0], b[3][0])
        if p < 16:
            assert a[1] == b[1] and np.array_equal(a[2], b[2]) and a[4] == b[4]
        ka, kb = orc.from_bf16(a[3][1]).ravel(), orc.from_bf16(b[3][1]).ravel()
        assert np.linalg.norm(ka - kb) <= 2.0 ** -6 * np.linalg.norm(kb)
        ha, hb = orc.from_bf16(a[2]).ravel(), orc.from_bf16(b[2]).ravel()
        assert float(ha @ hb / np.sqrt((ha @ ha) * (hb @ hb))) > 0.995
    assert q3t.library().q3t_kernel_error_count() == 0


@pytest.mark.parametrize("rows", [2, 4, 7, 8])
def test_row_does_not_depend_on_its_batch(q3t, model, rows):
    together = frame(q3t, model, POSITIONS[-rows:], 1, frames=2)
    for i, p in enumerate(POSITIONS[-rows:]):
        # the same session alone: its seeds are those of its place in the batch
        model.set_option("decode_chain", 1)
        s = model.create_session((p + 34) // 16 * 16, 100 + i)
        s.talker_sampling = q3t.SamplingConfig(True, 50, 0.9, 0.9, 1.05)
        s.predictor_sampling = q3t.SamplingConfig(True, 50, 1.0, 0.9, 1.0)
        s.synthetic_prefill(p, 1000 + i)
        for f in range(2):
            s.next_frame(7 + f)
        hidden, tokens, rng = s.read_state()
        assert np.array_equal(tokens, together[i][0]) and np.array_equal(hidden, together[i][2]) and rng == together[i][4]
        s.close()


@pytest.mark.parametrize("config", [(False, 0, 1.0), (True, 1, 1.0), (True, 128, 0.5), (True, 129, 0.9), (True, 0, 1.0)])
def test_draws_inside_and_outside_the_chain(q3t, model, config):
    """Greedy and top-k up to 128 are drawn inside the chain, the rest launch by launch: the codes are the same."""
    do_sample, top_k, top_p = config
    predictor = q3t.SamplingConfig(do_sample, top_k, top_p, 0.9, 1.0)
    for positions in ([9], [9, 40, 3]):
        for a, b in zip(frame(q3t, model, positions, 1, predictor), frame(q3t, model, positions, 0, predictor)):
            assert np.array_equal(a[0], b[0])


@pytest.mark.parametrize("used,given_up", [(2 ** 31 - 1024, 2 ** 32 - 1), (2 ** 31 - 1023, 2 ** 31 - 1023), (2 ** 32 - 300, 2 ** 32 - 300)])
def test_exchange_numbers_start_again(q3t, model, used, given_up):
    """Exchanges are numbered in 32 bits.  At the last frame before a restart, at the first behind it, and where numbers
    would come round within a frame; the latter two where the run that was once given up bore the next run's number."""
    lib = q3t.library()
    lib.q3t_test_set_chain_numbers.argtypes = [C.c_void_p, C.c_uint64, C.c_uint32]
    want = frame(q3t, model, [40, 9, 700], 1, frames=3)
    assert lib.q3t_test_set_chain_numbers(model._handle, used, given_up) == 0
    got = frame(q3t, model, [40, 9, 700], 1, frames=3)
    for a, b in zip(got, want):
        assert np.array_equal(a[0], b[0]) and a[1] == b[1] and np.array_equal(a[2], b[2]) and a[4] == b[4]
    assert lib.q3t_kernel_error_count() == 0


@pytest.mark.parametrize("rows", [1, 2, 3, 5, 8])
def test_launches_in_the_chains_place(q3t, model, rows):
    """Where the device is shared a frame is made launch by launch instead of as a chain: the same bits, for contexts of one
    page, one slot, several slots and several pages to a class (2,048 tokens and more), and for the frames that follow."""
    positions = POSITIONS[-rows:]
    for a, b in zip(frame(q3t, model, positions, 2, frames=3), frame(q3t, model, positions, 1, frames=3)):
        assert np.array_equal(a[0], b[0]) and a[1] == b[1] and np.array_equal(a[2], b[2]) and a[4] == b[4]
        assert all(np.array_equal(x, y) for x, y in zip(a[3], b[3]))
    assert q3t.library().q3t_kernel_error_count() == 0


def test_frames_do_not_depend_on_what_else_runs(q3t, model):
    """Sessions stepped alone from threads of their own, a lockstep batch and prompts, all at once: every session decodes what
    it decodes on a quiet device, whichever way its frames were made."""
    import threading
    model.set_option("decode_chain", 1)
    rng = np.random.default_rng(8)
    prompts = {n: ([int(t) for t in rng.integers(0, 151936, size=n)], [-1] * n) for n in (70, 300)}
    steps = 12

    def session(seed, position):
        s = model.create_session(position + steps + 32, seed)
        s.talker_sampling = q3t.SamplingConfig(True, 50, 0.9, 0.9, 1.05)
        s.predictor_sampling = q3t.SamplingConfig(True, 50, 1.0, 0.9, 1.0)
        s.synthetic_prefill(position, seed)
        return s

    def alone(seed, position):
        s = session(seed, position)
        out = [s.next_frame(5 + i) for i in range(steps)]
        out = [(f.codes, f.next_semantic_token) for f in out] + [s.read_state()[0].tobytes()]
        s.close()
        return out

    def together(count, seed):
        ss = [session(seed + i, 100 + 50 * i) for i in range(count)]
        out = []
        for i in range(steps):
            out.append([p.finish_without_consumer().next_semantic_token for p in model.batch_begin_device_frames(ss, [5 + i] * count)])
        out.append([s.read_state()[0].tobytes() for s in ss])
        for s in ss:
            s.close()
        return out

    def prompt(n):
        out = []
        for _ in range(4):
            s = model.create_session(n + 16, 3)
            s.prefill(*prompts[n])
            out.append((s.current_semantic_token, s.read_state()[0].tobytes()))
            s.close()
        return out

    jobs = [lambda i=i: alone(300 + i, 20 + 150 * i) for i in range(4)] + [lambda: together(3, 400), lambda: prompt(70), lambda: prompt(300)]
    quiet = [job() for job in jobs]
    assert all(len(set(q)) == 1 for q in quiet[-2:])
    for some in ([0, 1], [0, 1, 2, 3], [0, 4], [0, 1, 2, 4], [0, 5], [4, 6], list(range(len(jobs)))):
        got = {}
        threads = [threading.Thread(target=lambda i=i: got.__setitem__(i, jobs[i]())) for i in some]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for i in some:
            assert got.get(i) == quiet[i], (some, i)
    assert q3t.library().q3t_kernel_error_count() == 0


@pytest.mark.parametrize("rows", [1, 3, 12])
def test_frame_loop_behind_other_frames(q3t, model, rows):
    """A frame loop whose stream has to wait for frames of other sessions: its rows start where they are, not where the host,
    which is done enqueueing by then, has counted them to."""
    model.set_option("decode_chain", 1)

    def run(others):
        busy = []
        for i in range(others):
            b = model.create_session(256, 800 + i)
            b.synthetic_prefill(200, 800 + i)
            busy.append((b, b.begin_device_frame(3)))
        ss = []
        for i in range(rows):
            s = model.create_session(64 + 40 * i + 32, 60 + i)
            s.synthetic_prefill(20 + 40 * i, 60 + i)
            ss.append(s)
        for b, p in busy:
            p.finish_without_consumer()
        pending = [b.begin_device_frame(3) for b, _ in busy]
        model.run_frames(ss, 9, 11)
        out = [tuple(np.array(x).tobytes() for x in s.read_state()) for s in ss]
        for p in pending:
            p.finish_without_consumer()
        for s in ss + [b for b, _ in busy]:
            s.close()
        return out

    quiet = run(0)
    assert run(1) == quiet and run(2) == quiet and run(4) == quiet


def set_places(q3t, model, die_of_sm=None, pages=None, grid=128):
    lib = q3t.library()
    lib.q3t_test_set_chain_places.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int32]
    die = None if die_of_sm is None else np.ascontiguousarray(die_of_sm, dtype=np.uint8)
    page = None if pages is None else np.ascontiguousarray(pages, dtype=np.uint32)
    return lib.q3t_test_set_chain_places(model._handle, None if die is None else die.ctypes.data, None if page is None else page.ctypes.data, grid)


@pytest.mark.parametrize("rows", [1, 2, 3, 8])
def test_places_change_no_bit(q3t, model, rows):
    """Wherever the CTAs and the buffers are taken to lie, and however many CTAs more than needed there are, every place is
    taken once and a frame has the same bits: all SMs on either die, one SM, a third and half of them on the other."""
    rng = np.random.default_rng(rows)
    positions = POSITIONS[-rows:]
    want = frame(q3t, model, positions, 1, frames=2)
    sms = np.arange(256)
    try:
        for die, pages, grid in ((0 * sms, np.arange(992), 128), (0 * sms, np.arange(992), 148), (0 * sms + 1, np.arange(2303, 1311, -1), 128),
                                 (0 * sms + 1, np.arange(992), 140), (sms == 17, rng.permutation(2304)[:992], 128), (sms != 17, np.arange(992), 148),
                                 (sms % 3 == 0, np.arange(992), 128), (sms % 3 == 0, np.arange(992), 133),
                                 (rng.integers(0, 2, 256), rng.permutation(2304)[:992], 128), (rng.integers(0, 2, 256), np.arange(992), 148)):
            assert set_places(q3t, model, die, pages, grid) == 0
            for a, b in zip(frame(q3t, model, positions, 1, frames=2), want):
                assert np.array_equal(a[0], b[0]) and a[1] == b[1] and np.array_equal(a[2], b[2]) and a[4] == b[4]
        assert set_places(q3t, model, 0 * sms + 2, np.arange(992)) != 0
        assert set_places(q3t, model, 0 * sms, np.arange(992), 127) != 0 and set_places(q3t, model, 0 * sms, np.arange(992), 149) != 0
        assert set_places(q3t, model, 0 * sms, np.zeros(992)) != 0 and set_places(q3t, model, 0 * sms, np.arange(1313, 2305)) != 0
    finally:
        assert set_places(q3t, model) == 0
    for a, b in zip(frame(q3t, model, positions, 1, frames=2), want):
        assert np.array_equal(a[0], b[0]) and a[1] == b[1] and np.array_equal(a[2], b[2]) and a[4] == b[4]
    assert q3t.library().q3t_kernel_error_count() == 0


@pytest.mark.parametrize("rows", [1, 3])
def test_frames_beside_a_kernel_that_holds_sms(q3t, model, rows):
    """A launch of 128 CTAs needs as many SMs.  What a host runs on some of the others (its codec) does not hold a frame up,
    whichever die it lies on, and changes none of its bits."""
    import time
    import torch
    lib = q3t.library()
    lib.q3t_test_hold_sms.argtypes = [C.c_int32, C.c_uint64, C.c_void_p]
    model.set_option("decode_chain", 1)
    stream = torch.cuda.Stream()

    def run(held):
        ss = []
        for i in range(rows):
            s = model.create_session(256, 40 + i)
            s.talker_sampling = q3t.SamplingConfig(True, 50, 0.9, 0.9, 1.05)
            s.predictor_sampling = q3t.SamplingConfig(True, 50, 1.0, 0.9, 1.0)
            s.synthetic_prefill(60 + 30 * i, 40 + i)
            ss.append(s)
        done = torch.cuda.Event()
        torch.cuda.synchronize()
        if held:
            assert lib.q3t_test_hold_sms(held, 500_000_000, stream.cuda_stream) == 0
            done.record(stream)
            time.sleep(0.02)
        out = []
        for f in range(4):
            if rows == 1:
                out.append(ss[0].next_frame(7 + f).codes)
            else:
                out.append([p.finish_without_consumer().next_semantic_token for p in model.batch_begin_device_frames(ss, [7 + f] * rows)])
        assert not held or not done.query()
        torch.cuda.synchronize()
        out.append([tuple(np.array(x).tobytes() for x in s.read_state()) for s in ss])
        for s in ss:
            s.close()
        return out

    want = run(0)
    try:
        assert set_places(q3t, model, np.arange(256) // 2 % 2, np.arange(992), 128) == 0
        for held in (1, 7, 20):
            assert run(held) == want
    finally:
        assert set_places(q3t, model) == 0
    assert lib.q3t_kernel_error_count() == 0
