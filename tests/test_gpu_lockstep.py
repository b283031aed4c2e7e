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


def test_row_counts_in_turn(q3t, model):
    """The chain's places are marked for one row count: another count, and the first again, start with all of them marked."""
    want = {n: frames(q3t, model, n, 0, 1)[0] for n in (12, 40, 9)}
    for n in (12, 40, 9, 40, 12):
        assert frames(q3t, model, n, 1, 1)[0] == want[n]
    assert q3t.library().q3t_kernel_error_count() == 0


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
