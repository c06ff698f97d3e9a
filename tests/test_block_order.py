"""The order of a tile's pair words inside the library: 16 blocks of 8 x 8
atoms, lane l and bit 8 J + 4 e + I standing for the pair i = 8 I + (l & 7),
j = 8 J + (4 e ^ (l & 4)) + (l >> 3). Restated here from the kernels' shuffles
(blockOrder), the precise kernel's decoding of a live word's bit, and the
export's way back to the interface's order (bit t of lane i <-> j = (i + t) & 31).
This pins the arithmetic of the order; that the kernels follow it is what the
pair-set tests check on a GPU, whose exported masks went through the order and
back, and the force tests."""
import numpy as np
import pytest

LANES = np.arange(32)


def block_order(words):
    """blockOrder of the kernels: four shuffles, then the nibble swap."""
    w = np.asarray(words, dtype=np.uint32)
    out = np.zeros(32, dtype=np.uint32)
    for I in range(4):
        out |= ((w[8 * I + (LANES & 7)] >> (LANES >> 3).astype(np.uint32)) & np.uint32(0x11111111)) << np.uint32(I)
    swapped = ((out >> np.uint32(4)) & np.uint32(0x0F0F0F0F)) | ((out & np.uint32(0x0F0F0F0F)) << np.uint32(4))
    return np.where(LANES & 4, swapped, out).astype(np.uint32)


def pair_of(lane, bit):
    I, e, J = bit & 3, (bit >> 2) & 1, bit >> 3
    return 8 * I + (lane & 7), 8 * J + ((4 * e) ^ (lane & 4)) + (lane >> 3)


def test_every_pair_of_a_tile_has_one_lane_and_bit():
    seen = {pair_of(l, b) for l in range(32) for b in range(32)}
    assert seen == {(i, j) for i in range(32) for j in range(32)}
    for l in range(32):  # the precise kernel's decoding
        for t in range(32):
            assert pair_of(l, t) == (((t & 3) << 3) | (l & 7), ((t & 28) ^ (l & 4)) | (l >> 3))


@pytest.mark.parametrize("density", [0.0, 1.0 / 1024, 0.2, 0.9, 1.0])
def test_rows_to_blocks_and_back(density):
    rng = np.random.default_rng(7)
    tile = rng.random((32, 32)) < density          # [i, j]
    rows = (tile.astype(np.uint64) << np.arange(32, dtype=np.uint64)).sum(1).astype(np.uint32)
    words = block_order(rows)
    for l in range(32):
        for b in range(32):
            assert bool((words[l] >> np.uint32(b)) & 1) == bool(tile[pair_of(l, b)])
    assert np.array_equal(block_order(words), rows)
    # the lanes of one block share a bit pair: a block without pairs is skipped by all
    live = np.bitwise_or.reduce(words)
    for I in range(4):
        for J in range(4):
            assert bool((int(live) >> (8 * J)) & (0x11 << I)) == tile[8 * I:8 * I + 8, 8 * J:8 * J + 8].any()
