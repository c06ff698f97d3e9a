"""Export of the tile lists (needs a B200) on a stream that does not wait for
the default one."""
import numpy as np
import pytest

import nbk
from helpers import ALL, PARAMS, mixed_box

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def packed():
    return nbk.Packed(mixed_box(seed=4, natoms=50003))


def _export(p, stream):
    """The pairs of an export; ten more exports of the same lists are the same."""
    nb = nbk.Nonbonded(PARAMS, p.system.lj_table())
    nb.setup(p, stream=stream)
    nb.build_tile_lists(p, stream=stream)
    nb.force(p, ALL | nbk.NBK_PAIRLIST, xyzq=p.xyzq, stream=stream)
    tl, ja, ex = first = nb.export_tile_lists(stream=stream)
    assert len(tl) > 10000
    # packed: list after list, without gaps
    assert np.array_equal(tl[1:, 1], tl[:-1, 2] + 1) and tl[0, 1] == 0 and tl[-1, 2] == len(ja) - 1
    for _ in range(10):
        for again, once in zip(nb.export_tile_lists(stream=stream), first):
            assert np.array_equal(again, once)
    nb.close()
    return nbk.pairs_from_tile_lists(tl, ja, ex, p.atomStorageSize)


def test_export_on_a_non_blocking_stream(packed):
    """torch's streams are non-blocking. The kernel that packs the tiles writes
    where the uploaded offsets say: the pairs are those of the default stream."""
    import torch
    got = _export(packed, torch.cuda.Stream().cuda_stream)
    assert np.array_equal(got, _export(packed, None))
