"""Tokens grouped by expert on the device: offsets, row and pair maps, and the tile list, for few experts and for more than a block has threads."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("E,with_tiles,P,rows", [(1, 1, 1, 128), (5, 5, 7, 4), (32, 32, 4000, 128), (33, 20, 900, 16), (1024, 1024, 3000, 2), (1025, 1000, 5000, 1),
                                                 (3000, 2999, 300, 64)])
def test_groups_and_tiles(E, with_tiles, P, rows):
    from kestrel_llm_b200.csrc import ops
    ids = np.random.default_rng(E).integers(0, E, size=P).astype(np.int32)
    ids[: P // 3] = ids[0]                                             # one expert with many rows, some with none
    dev = torch.from_numpy(ids).to(DEV)
    tiles = -(-P // rows) + E
    new = lambda n: torch.full((n,), -1, dtype=torch.int32, device=DEV)
    offsets, row_pair, pair_row, tile_expert, tile_row0, n_tiles = new(E + 1), new(P), new(P), new(tiles), new(tiles), new(1)
    rc = ops.library().kestrel_moe_group_some(dev.data_ptr(), P, E, with_tiles, rows, offsets.data_ptr(), row_pair.data_ptr(), pair_row.data_ptr(),
                                              tile_expert.data_ptr(), tile_row0.data_ptr(), n_tiles.data_ptr(), ops._stream())
    assert rc == 0
    counts = np.bincount(ids, minlength=E)
    off = np.concatenate([[0], np.cumsum(counts)])
    assert offsets.cpu().tolist() == off.tolist()
    want = [(e, off[e] + r) for e in range(with_tiles) for r in range(0, counts[e], rows)]
    n = int(n_tiles)
    assert list(zip(tile_expert[:n].tolist(), tile_row0[:n].tolist())) == want
    pairs = row_pair.cpu().numpy()
    assert sorted(pairs.tolist()) == list(range(P))                    # each pair a row of its own, among its expert's
    assert (pair_row.cpu().numpy()[pairs] == np.arange(P)).all() and (np.repeat(np.arange(E), counts) == ids[pairs]).all()
