"""Prompt passes of more rows than a lockstep batch: the row-blocked and wide tensor-core GEMMs and the
attention that shares its passes over the cache, against the position-by-position path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,chunk", [(n, 2048) for n in (9, 33, 65, 128, 129, 257, 300, 385, 641, 1201)] + [(450, 200), (150, 141)])
def test_prompt_pass_tracks_single_positions(q3t, orc, gpu_model, n, chunk):
    """Lengths around the row blocks (64, 128), the attention blocks (32 or 64 positions, 64 tokens) and the changes of GEMM kernel
    (gate/up after 64 rows, q/k/v after 256, the others after 576), and passes behind a longer one, the last of 50 or of 9
    rows.  Layer 0's keys and values have one GEMM chain behind them (text projection, q/k/v) whose fp32 sums differ in order
    only: relative error below one bf16 rounding, 2^-8.  From there to layer 1's lie eight bf16 roundings (attention, o,
    gate/up, down, q/k/v, norm twice, rotation), each of which may fall the other way by an ulp, 2^-8 to 2^-7 of a value, in
    part of the elements: 8 x 2^-9 = 2^-6 at most, at every position.  28 layers on they have spread: direction within 0.995, as for the passes
    of 64."""
    rng = np.random.default_rng(n)
    text = [int(t) for t in rng.integers(0, 151936, size=n)]
    codec = [int(c) if i % 3 == 0 else -1 for i, c in enumerate(rng.integers(0, 2048, size=n))]

    def run(chunk, tc_min_rows):
        gpu_model.set_option("prefill_chunk", chunk)
        gpu_model.set_option("tc_min_rows", tc_min_rows)
        try:
            s = gpu_model.create_session((n + 31) // 16 * 16, 5)
            s.prefill(text, codec)
            hidden = orc.from_bf16(s.read_state()[0]).ravel()
            kv = [[orc.from_bf16(x).reshape(n, -1) for x in s.read_kv(layer, 0, n)] for layer in (0, 1, 27)]
            s.close()
            return hidden, kv
        finally:
            gpu_model.set_option("prefill_chunk", 2048)
            gpu_model.set_option("tc_min_rows", 9)

    want_hidden, want = run(8, 65)            # passes of 8 rows: what one position alone gives, bit for bit
    hidden, got = run(chunk, 9)
    again, _ = run(chunk, 9)
    assert np.array_equal(hidden, again)
    for a, b in zip(got[0], want[0]):
        assert np.linalg.norm(a - b) <= 2.0 ** -8 * np.linalg.norm(b)
    for a, b in zip(got[1], want[1]):
        assert (np.linalg.norm(a - b, axis=1) <= 2.0 ** -6 * np.linalg.norm(b, axis=1)).all()
    for a, b in zip([hidden] + got[2], [want_hidden] + want[2]):
        a, b = a.ravel(), b.ravel()
        assert float(a @ b / np.sqrt((a @ a) * (b @ b))) > 0.995
    assert q3t.library().q3t_kernel_error_count() == 0
