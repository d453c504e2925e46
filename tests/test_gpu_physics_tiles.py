"""Non-ideal terms set on the engine of a model whose stage tiles were chosen by its grid's
size (GPU): the stage runs on the default tiles, as in a model built with the terms."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _state(*x):
    return 1.0 + 0.2 * np.cos(2 * np.pi * x[0])


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("ndim", [2, 3])
def test_terms_set_later_run_on_the_default_tiles(ndim, precision):
    from wellbalanced_b200.mesh import AMRHierarchy
    from wellbalanced_b200.mhd import MHD2D
    from wellbalanced_b200.mhd3d import MHD3D

    stages, shapes = [], []
    for later in (False, True):
        mesh = AMRHierarchy((40, 24, 20)[:ndim], periodic=(True,) * ndim)
        solver = MHD2D if ndim == 2 else MHD3D
        model = solver(mesh, precision=precision, resistivity=0.0 if later else 1e-3)
        zero = 0.0 if ndim == 2 else (lambda *x: 0.0 * x[0])
        potential = (lambda x, y: 0.05 * np.sin(2 * np.pi * x) * np.cos(2 * np.pi * y)) if ndim == 2 else (
            zero, zero, lambda x, y, z: 0.05 * np.sin(2 * np.pi * x) * np.cos(2 * np.pi * y) + 0.0 * z)
        model.set_state(_state, (0.3, -0.2, 0.1), _state, vector_potential=potential)
        eng = model.engine
        shapes.append(tuple(eng.layout.tile_shape))
        if later:
            eng.physics = (1e-3, 0.0, 0.0, 0.0, 0.0) if ndim == 2 else (1e-3, 0.0, 0.0, 0.0)
        assert tuple(eng.layout.tile_shape) == tuple(eng.layout.default_tile)
        eng.dt.fill_(1e-4)
        eng.stage(eng.state, None, eng.stage_pool)
        stages.append(eng.stage_pool.clone())
    assert shapes[1] != shapes[0]  # the ideal model had chosen another shape
    assert torch.equal(*stages)
