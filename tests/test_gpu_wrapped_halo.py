"""2D patches that wrap onto themselves (GPU): the stage kernel writes the halo that the fill
would, and patches of fewer than three cells an axis, walls or neighbours keep the fill."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _model(shape, precision, periodic=True, split=None, **options):
    from wellbalanced_b200 import MHD2D, MHD3D
    from wellbalanced_b200.mesh import AMRHierarchy

    ndim = len(shape)
    mesh = AMRHierarchy(shape, periodic=(periodic,) + (True,) * (ndim - 1), split=split)
    model = (MHD2D if ndim == 2 else MHD3D)(mesh, precision=precision, limiter="mc", **options)
    k = 2.0 * np.pi
    potential = (lambda x, y: 0.1 * np.cos(k * x) + 0.05 * np.sin(k * y)) if ndim == 2 else (
        lambda x, y, z: 0.1 * np.sin(k * z), lambda x, y, z: 0.1 * np.cos(k * x), lambda x, y, z: 0.1 * np.sin(k * y))
    model.set_state(lambda x, y, *z: 1.0 + 0.2 * np.sin(k * (x + y)), (0.3, -0.2, 0.1),
                    lambda x, y, *z: 1.0 + 0.1 * np.cos(k * y), vector_potential=potential)
    return model


@pytest.mark.parametrize("precision", [32, 64, "mixed"])
@pytest.mark.parametrize("shape, options", [
    ((3, 3), {}), ((4, 37), {}), ((33, 65), {}), ((40, 24), {"resistivity": 1e-3, "conduction": (0.01, 0.0)}),
])
def test_the_stages_leave_a_filled_halo(shape, options, precision):
    model = _model(shape, precision, **options)
    eng = model.engine
    assert eng.layout.wraps
    model.advance(2)
    for pool in (eng.state, eng.stage_pool):
        before = pool.clone()
        eng.fill(pool)
        assert torch.equal(pool, before)
    # and the steps with the fills launched as well end on the same state
    other = _model(shape, precision, **options)
    other.engine.layout.wraps = False
    other.advance(2)
    assert torch.equal(eng.state, other.engine.state)


@pytest.mark.parametrize("shape, options", [((2, 8), {}), ((8, 12, 8), {}), ((16, 16), {"periodic": False}),
                                            ((16, 16), {"split": (2, 1)})])
def test_other_patches_keep_the_fill(shape, options):
    model = _model(shape, 32, **options)
    assert not model.engine.layout.wraps
    model.advance(2)
    before = model.engine.state.clone()
    model.engine.fill(model.engine.state)
    assert torch.equal(model.engine.state, before)


def test_a_batch_wraps_instance_by_instance():
    from wellbalanced_b200 import Batch

    batch = Batch.orszag_tang(6, seed=2)
    assert batch.engine.layout.wraps
    batch.advance(3)
    before = batch.engine.state.clone()
    batch.engine.fill(batch.engine.state)
    assert torch.equal(batch.engine.state, before)


@pytest.mark.parametrize("precision", [32, 64, "mixed"])
@pytest.mark.parametrize("shape, options", [((2, 8), {}), ((8, 2), {}), ((1, 5), {}), ((5, 1), {}),
                                            ((16, 16), {"periodic": False})])
def test_the_flag_is_ignored_where_an_image_has_no_single_writer(shape, options, precision):
    """Fewer than three cells an axis, or a last node plane of the patch's own: the stage leaves
    the halo to the fill, with the flag as without it."""
    from wellbalanced_b200 import _lib
    from wellbalanced_b200.engine import _device_bytes
    from wellbalanced_b200.mesh import WRAP

    eng = _model(shape, precision, **options).engine
    eng.dt.fill_(1e-4)
    pools = []
    for flag in (0, WRAP):
        rows = eng.layout.rows.copy()
        rows["flags"] |= flag
        eng.patches = _device_bytes(rows, eng.device, _lib.PATCH)
        eng.stage_pool.fill_(7.0)
        eng.stage(eng.state, None, eng.stage_pool)
        pools.append(eng.stage_pool.clone())
    assert torch.equal(*pools)
