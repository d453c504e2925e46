"""Steps issued from a launch list (GPU): bit for bit the steps launched one by one, after
settings that a list depends on have changed, on another stream and from a CUDA graph."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _refined(ndim, **options):
    from wellbalanced_b200 import MHD2D, MHD3D
    from wellbalanced_b200.mesh import AMRHierarchy

    mesh = AMRHierarchy((24, 32, 16)[:ndim], periodic=(True, False, True)[:ndim])
    mesh.add_patch(1, ((12, 36), (16, 44), (8, 24))[:ndim])
    model = (MHD2D if ndim == 2 else MHD3D)(mesh, limiter="mc", **options)
    fields = {"vector_potential": lambda x, y: 0.1 * np.cos(2.0 * np.pi * x), "bz": 0.2} if ndim == 2 else {
        "vector_potential": (0.0, 0.0, lambda x, y, z: 0.1 * np.cos(2.0 * np.pi * x))}
    model.set_state(lambda x, y, *z: 1.0 + 0.3 * np.exp(-((x - 0.5) ** 2 + (y - 0.5) ** 2) / 0.02), (0.3, 0.4, 0.1), 1.0,
                    **fields)
    return model


def _one_by_one(model, steps):
    """The launches of the steps without a list (as timed stages issue them)."""
    eng = model.engine
    eng.stage_events = []
    model.advance(steps)
    eng.stage_events = None


@pytest.mark.parametrize("ndim, options", [(2, {"precision": 32}), (2, {"precision": 64, "resistivity": 1e-3}),
                                           (2, {"precision": "mixed", "conduction": (0.1, 0.01)}), (3, {"precision": 32})])
def test_listed_steps_equal_single_launches(ndim, options):
    listed, single = _refined(ndim, **options), _refined(ndim, **options)

    def same():
        torch.cuda.synchronize()
        assert torch.equal(listed.engine.state, single.engine.state)
        assert torch.equal(listed.engine.status[1:], single.engine.status[1:])

    launches = listed.engine.launches
    listed.advance(3)
    launches = listed.engine.launches - launches
    before = single.engine.launches
    _one_by_one(single, 3)
    assert single.engine.launches - before == launches
    same()
    # a setting a list holds
    for model in (listed, single):
        model.engine.overlap_fluxes = False
        model.engine.staged_fluxes = False
    assert not listed.engine._lists
    listed.advance(1)
    _one_by_one(single, 1)
    same()
    # another stream, then one step at a time
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        listed.advance(2)
    torch.cuda.current_stream().wait_stream(stream)
    _one_by_one(single, 2)
    same()
    dt = listed.step()
    single.engine.stage_events = []
    assert single.step() == dt
    single.engine.stage_events = None
    same()
    assert listed.time == single.time


def test_captured_steps_equal_listed_ones():
    captured, listed = _refined(2, precision=32), _refined(2, precision=32)
    captured.capture()
    captured.advance(3)
    listed.advance(captured.steps)
    torch.cuda.synchronize()
    assert torch.equal(captured.engine.state, listed.engine.state)
    assert captured.time == listed.time


def test_a_bad_cell_is_counted_in_the_step_that_meets_it():
    model = _refined(2, precision=32)
    model.engine.state[model.engine.layout.rows[0]["off"] + 3 * int(model.engine.layout.rows[0]["pitch0"]) + 4] = -1.0
    with pytest.raises(FloatingPointError):
        model.step()
    model = _refined(2, precision=32)
    model.engine.bad.fill_(7)  # of an earlier call: each step counts its own
    model.step()


@pytest.mark.parametrize("ndim", [2, 3])
def test_a_cfl_of_its_own_each_step_takes_one_list(ndim):
    listed, single = _refined(ndim, precision=32), _refined(ndim, precision=32)
    for k in range(6):
        for model in (listed, single):
            model.cfl = 0.3 - 0.02 * k
        listed.advance(1)
        _one_by_one(single, 1)
        assert len(listed.engine._lists) == 1
        torch.cuda.synchronize()
        assert torch.equal(listed.engine.state, single.engine.state)
        assert torch.equal(listed.engine.status[1:], single.engine.status[1:])
