"""Device memory that a context holds for its capacities: on the 16-bit paths none
at all (activations and outputs stay on chip or go to the caller's arrays), on the
FP32 path a query's raw output row and a record's input row, kept activations and
deltas, and no more."""
import pytest

pytestmark = pytest.mark.gpu


def held(nmg, queries, batch, **over):
    f = nmg.GuidingField(nmg.config(1, **over), max_queries=queries, max_batch=batch)
    try:
        return f.device_bytes, f.info
    finally:
        f.close()


@pytest.mark.parametrize("path", [1, 2], ids=["bf16", "fp16"])
def test_16_bit_paths_hold_nothing_per_query(nmg, path):
    assert held(nmg, 1 << 20, 1 << 18, path=path)[0] == held(nmg, 1, 1, path=path)[0]


def test_fp32_path(nmg):
    one, info = held(nmg, 64, 0, path=0)
    row = 4 * info.n_output_padded
    assert held(nmg, 1 << 20, 0, path=0)[0] - one == ((1 << 20) - 64) * row
    hidden, enc, out = 3 * 64, info.n_encoded_padded, info.n_output_padded
    # input row, encoded row, activations, deltas of every layer, dL/draw, raw outputs, a record
    record = 4 * (info.n_input + enc + hidden + hidden + out + out + out + 8)
    a, b = held(nmg, 0, 64, path=0)[0], held(nmg, 0, 1 << 16, path=0)[0]
    assert b - a == ((1 << 16) - 64) * record
