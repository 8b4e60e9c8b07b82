"""The tuner on the CPU: CTA sizes are tried only where they choose anything."""
import pytest

from map_folding_gb300 import autotune


class _Batch:
    tried = []

    def __init__(self, shapes, depths, cfg):
        self.tried.append((tuple(depths), cfg.block_threads, cfg.node_budget))

    def run(self):
        return [1], type("Stats", (), {"kernel_s": 1.0})

    def close(self):
        pass


@pytest.mark.parametrize("shapes,sizes", [
    ([(4, 5), (1, 14)], {0}),          # a last row on masks: the launch's own size
    ([(1, 14), (2, 2, 4), (2, 7)], {128, 256}),
    ([(7, 7)], {128, 256}),            # over 41 leaves
])
def test_cta_sizes_tried(monkeypatch, tmp_path, shapes, sizes):
    monkeypatch.setenv("MF_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(autotune.api, "LunnonBatch", _Batch)
    _Batch.tried = []
    best = autotune.tune_lunnon_batch(shapes, depth_offsets=(0,), periods=(32, 64), repeats=1)
    assert {t for _, t, _ in _Batch.tried} == sizes
    assert len(_Batch.tried) == len(set(_Batch.tried)) == 2 * len(sizes)
    assert autotune.as_config(best).block_threads in sizes


def test_square_rows():
    assert autotune.sym_rows(7, 24) and autotune.sym_rows(7, 42) and autotune.sym_rows(5, 3)
    assert not autotune.sym_rows(7, 43) and not autotune.sym_rows(4, 3)
