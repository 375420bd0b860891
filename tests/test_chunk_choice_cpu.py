"""Which steps bring the recurrences' chunk kernels, and how much scratch: the requests' own lengths where the host may go by them, the
most that a step of the shape can have where a step graph is recorded."""

import numpy as np
import pytest

from tokasaurus_b200.kernels import ops


@pytest.mark.parametrize("lengths,chunks", [([191] * 40, 0), ([192], 3), ([128] * 64, 0), ([1, 193, 5, 256, 257, 100], 4 + 4 + 5), ([], 0),
                                            ([1] * 300, 0), ([0, 500, 0], 8)])
def test_chunks_of_known_requests(lengths, chunks):
    assert ops.decay_chunk_count(sum(lengths), len(lengths), np.asarray(lengths, dtype=np.int32)) == chunks
    assert ops.decay_chunk_count(sum(lengths), len(lengths), lengths) == chunks


def test_chunks_of_any_request_of_a_shape():
    rng = np.random.default_rng(1)
    assert ops.decay_chunk_count(191, 1) == ops.decay_chunk_count(256, 256) == ops.decay_chunk_count(100, 1) == 0
    for _ in range(300):  # a graph's padded shape holds every step that fits it, requests without a token among them
        n = int(rng.integers(1, 8))
        lengths = rng.integers(0, 700, n) * (rng.random(n) < 0.8)
        T = int(lengths.sum()) + int(rng.integers(0, 100))
        if T > n:
            bound = ops.decay_chunk_count(T, n)
            assert bound >= ops.decay_chunk_count(T, n, lengths) and (bound > 0 or T < ops.DECAY_CHUNKS_FROM)


def test_a_step_graph_does_not_go_by_its_first_step_s_lengths():
    from tokasaurus_b200.engine.batch import StepContext

    ctx = StepContext.__new__(StepContext)
    ctx.host = type("Host", (), dict(seq_q_len=np.asarray([5, 200])))
    ctx.plan_caps = None
    assert ctx.lengths.tolist() == [5, 200]
    ctx.plan_caps = {}
    assert ctx.lengths is None
