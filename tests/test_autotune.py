"""What the ragged autotuner times and reuses, with a batch that only records its
calls (no GPU)."""
import json

import pytest


class _Batch:
    def __init__(self):
        self.warp_min, self.blocks, self.runs = set(), set(), 0

    def run(self, items, parents_dev=None, blocks_per_sm=2):
        self.warp_min |= {it[4] for it in items}
        self.blocks.add(blocks_per_sm)
        self.runs += 1
        return None, None, None, 1.0


@pytest.mark.parametrize("n,warp_min,blocks,runs", [(1 << 12, {32}, {1, 2}, 2 * (4 + 2)), (1 << 19, {32}, {1, 2}, 2 * (4 + 2)),
                                                    ((1 << 19) + 1, {32, 64, 128}, {1, 2, 3}, 2 * (12 + 3))])
def test_only_what_the_kernels_read_is_swept(nwg, tmp_path, n, warp_min, blocks, runs):
    from nwgr_b200.ragged import Autotuner

    batch = _Batch()
    params, bps = Autotuner(str(tmp_path / "c.json")).tune(batch, [(n, 8 * n)] * 3, [[0]] * 3)
    assert batch.warp_min == warp_min and batch.blocks == blocks and batch.runs == runs
    assert bps == 1 and [p.warp_min for p in params.values()] == [32]


def test_values_of_earlier_kernels_are_tuned_again(nwg, tmp_path):
    from nwgr_b200.ragged import Autotuner, shape_class

    path = tmp_path / "c.json"
    tuner = Autotuner(str(path))
    earlier = "|".join(tuner.key.split("|")[:2])  # GPU and library version
    assert earlier != tuner.key
    cls = shape_class(4096, 32768)
    old = {"classes": {cls: {"warp_min": 128, "alpha": 60, "beta": 36}}, "blocks_per_sm": 1}
    path.write_text(json.dumps({earlier: old}))
    batch, again = _Batch(), Autotuner(str(path))
    assert again.class_params(cls) is None
    params, _ = again.tune(batch, [(4096, 32768)], [[0]])
    assert batch.runs > 0 and params[cls].warp_min == 32
    saved = json.loads(path.read_text())
    assert saved[earlier] == old and saved[again.key]["classes"][cls]["warp_min"] == 32
    batch = _Batch()
    Autotuner(str(path)).tune(batch, [(4096, 32768)], [[0]])
    assert batch.runs == 0
