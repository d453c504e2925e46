"""Stencil features (GPU): a cell's row is the same bits whether its block holds the box of
neighbours at once or goes row by row, and for output rows of any alignment."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _model(shape, split, precision):
    from wellbalanced_b200 import MHD3D
    from wellbalanced_b200.mesh import AMRHierarchy

    model = MHD3D(AMRHierarchy(shape, periodic=(True,) * 3, split=split), precision=precision)
    k = 2.0 * np.pi
    model.set_state(lambda x, y, z: 1.0 + 0.5 * np.sin(k * (x + 2.0 * y + 3.0 * z)), (0.2, -0.1, 0.3),
                    lambda x, y, z: 1.0 + 0.4 * np.cos(k * (3.0 * z - x)),
                    vector_potential=(lambda x, y, z: 0.1 * np.sin(k * z), 0.0, lambda x, y, z: 0.1 * np.cos(k * x)))
    return model


def _by_cell(model, rows, starts):
    out = torch.zeros((*model.hierarchy.shape, 16), device=rows.device)
    for patch, start in zip(model.hierarchy.patches, starts):
        block = rows[int(start) : int(start) + int(np.prod(patch.shape))].reshape(*patch.shape, 16)
        out[tuple(slice(lo, hi) for lo, hi in patch.box)] = block
    return out


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("shape, split", [
    ((6, 10, 700), (1, 2, 4)),    # lines longer than a block's box | shorter ones
    ((4, 100, 100), (2, 10, 10)),  # blocks that straddle large planes | whole small patches
    ((5, 7, 510), (1, 1, 2)),     # the longest line the box takes
    ((4, 4, 4), (2, 2, 2)),
])
def test_features_do_not_depend_on_the_blocks(shape, split, precision):
    from wellbalanced_b200 import _lib
    from wellbalanced_b200.tagger import LearnedTagger

    tagger = LearnedTagger()
    tagger.mean += 0.25
    tagger.inv_std *= 1.5
    whole, parts = _model(shape, None, precision), _model(shape, split, precision)
    rows, starts = tagger.features(whole)
    assert torch.isfinite(rows).all()
    assert int((rows.std(dim=0) > 0.0).sum()) >= 8  # |B| does not vary along y, nor much on 4 cells
    assert torch.equal(_by_cell(whole, rows, starts), _by_cell(parts, *tagger.features(parts)))
    # output rows 4 bytes off a 16-byte boundary
    eng = whole.engine
    flat = torch.zeros(rows.numel() + 1, device=rows.device)
    row_start = torch.zeros(1, dtype=torch.int64, device=rows.device)
    _lib.call("wb_tag_features", eng.precision, eng.state.data_ptr(), eng.patches.data_ptr(), eng.chunk_patch.data_ptr(),
              eng.chunk_start.data_ptr(), eng.nchunks, row_start.data_ptr(), 0.0, 0.0, 0.0, eng.gamma,
              tagger.mean.data_ptr(), tagger.inv_std.data_ptr(), flat.data_ptr() + 4,
              torch.cuda.current_stream().cuda_stream)
    assert torch.equal(flat[1:].reshape(rows.shape), rows)


def test_a_ranks_rows_are_those_of_its_own_patches():
    from types import SimpleNamespace

    from wellbalanced_b200.distributed import LocalCluster
    from wellbalanced_b200.tagger import LearnedTagger

    whole = _model((16, 12, 20), (3, 2, 2), 64)
    patches = whole.hierarchy.patches
    tagger = LearnedTagger()
    rows, starts = tagger.features(whole)
    owner = [0, 1, 1, 0, 1, 0, 0, 1, 1, 1, 0, 1]
    cluster = LocalCluster(whole.engine.layout, owner, precision=64, limiter=whole.engine.limiter)
    for rank, engine in enumerate(cluster.engines):
        mine = [k for k, r in enumerate(owner) if r == rank]
        for local, k in enumerate(mine):
            for f in range(8):
                engine.view(engine.state, patches[k], f).copy_(whole.engine.view(whole.engine.state, patches[k], f))
        got, first = tagger.features(SimpleNamespace(engine=engine, hierarchy=whole.hierarchy))
        assert got.shape[0] == sum(int(np.prod(patches[k].shape)) for k in mine) and len(first) == len(mine)
        for local, k in enumerate(mine):
            n = int(np.prod(patches[k].shape))
            assert torch.equal(got[int(first[local]) :][:n], rows[int(starts[k]) :][:n])
