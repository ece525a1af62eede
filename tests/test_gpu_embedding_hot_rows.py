"""The gradient of a table whose rows are read a number of times around the edges of the block-wide
path: 32 occurrences are a warp's, 33 the block's, whose indices are read two chunks of 32 ahead of
their rows. The sum is the sequential one, bit for bit, so the oracle's bits are expected."""
import numpy as np
import pytest

from helpers import ProgramText, assert_bits_equal, run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [4, 33, 132])
@pytest.mark.parametrize("counts", [(31, 32, 33), (63, 64, 65), (95, 96, 97, 1), (127, 128, 129, 161)])
def test_a_row_read_around_the_edges_of_a_chunk(device, counts, h):
    r = np.random.default_rng(h + sum(counts))
    rows = 2 * len(counts) + 1
    ids = np.concatenate([np.full(c, 2 * k + 1, np.int32) for k, c in enumerate(counts)])
    ids = ids[r.permutation(len(ids))]
    p = ProgramText()
    i = p.input("ids", "i32", [len(ids)]); g = p.input("g", "f32", [len(ids), h]); dense = p.input("dense", "f32", [rows, h])
    alone = p.op("EmbeddingGrad", [rows, h], [i, g], attr="[%d]" % rows)
    made = p.op("Mul", [rows, h], [dense, dense])
    again = p.op("EmbeddingGrad", [rows, h], [i, g], attr="[%d]" % rows)
    in_place = p.op("Add", [rows, h], [made, again])
    p.output(alone); p.output(in_place)
    res = run_both(device, p.text(), {"ids": ids, "g": r.standard_normal((len(ids), h)).astype(np.float32),
                                      "dense": r.standard_normal((rows, h)).astype(np.float32)},
                   outputs=[(alone, rows * h), (in_place, rows * h)])
    for cpu, gpu in res:
        assert_bits_equal(gpu, cpu)
