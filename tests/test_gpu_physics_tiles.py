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


@pytest.mark.parametrize("precision, sides", [(32, (32, 48, 64)), (64, (64, 80, (48, 33)))])
def test_terms_set_on_a_batch_run_on_the_default_tiles(precision, sides):
    from wellbalanced_b200 import Batch

    stages, shapes = [], []
    for tile in (None, "default"):
        batch = Batch(sides, precision=precision)
        shapes.append(tuple(batch.layout.tile_shape))
        if tile == "default":
            batch = Batch(sides, precision=precision, tile=batch.layout.default_tile)
        for k, (nx, ny) in enumerate(batch.sides):
            x, y = np.meshgrid((np.arange(nx) + 0.5) / nx, (np.arange(ny) + 0.5) / ny, indexing="ij")
            xn, yn = np.meshgrid(np.arange(nx + 1) / nx, np.arange(ny + 1) / ny, indexing="ij")
            rho = 1.0 + 0.1 * k + 0.2 * np.cos(2 * np.pi * x)
            batch.set_instance(k, (rho, 0.3 * rho, -0.2 * rho * np.cos(2 * np.pi * y), 0.0 * rho, 2.0 + rho, 0.1 * rho),
                               0.05 * np.sin(2 * np.pi * xn) * np.cos(2 * np.pi * yn))
        batch.finish_state()
        batch.engine.physics = (1e-3, 0.0, 0.0, 0.0, 0.0)
        assert tuple(batch.layout.tile_shape) == tuple(batch.layout.default_tile)
        batch.advance(2)
        stages.append(batch.engine.state.clone())
    assert shapes[0] != tuple(batch.layout.default_tile)  # the ideal batch had chosen another shape
    assert torch.equal(*stages)


def test_a_captured_step_keeps_its_work_list():
    """Terms set after a step was captured cut other tiles; the graph replays the ideal step with
    the list it was captured with, whatever the allocator does with the memory of dropped ones."""
    from wellbalanced_b200 import Batch

    captured, ideal = Batch.orszag_tang(4, seed=3), Batch.orszag_tang(4, seed=3)
    captured.capture()
    tiles = captured.engine.tiles
    assert captured._graph.tiles is tiles
    captured.engine.physics = (1e-3, 0.0, 0.0, 0.0, 0.0)
    assert captured.engine.tiles is not tiles
    kept = tiles.data_ptr()
    del tiles
    others = [torch.zeros(captured.engine._ideal_tiles.numel(), dtype=torch.uint8, device="cuda") for _ in range(8)]
    assert all(t.data_ptr() != kept for t in others)
    captured.advance(2)
    ideal.advance(3)
    torch.cuda.synchronize()
    assert torch.equal(captured.engine.state, ideal.engine.state)
