"""The one-launch stable step (GPU): keys and dt bit for bit those of the rate and dt launches,
on one cell row, chunk remainders, many instances and levels, and again on the scratch a
launch leaves behind."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _plane(shape, precision, **options):
    from wellbalanced_b200 import MHD2D
    from wellbalanced_b200.mesh import AMRHierarchy

    model = MHD2D(AMRHierarchy(shape, periodic=(True, True)), precision=precision, **options)
    model.set_state(lambda x, y: 1.0 + 0.3 * np.sin(6.0 * x) * np.cos(9.0 * y), (0.4, -0.3, 0.1), 0.7,
                    vector_potential=lambda x, y: 0.1 * np.cos(2.0 * np.pi * x), bz=0.2)
    return model.engine


def _refined(precision):
    from wellbalanced_b200 import MHD2D
    from wellbalanced_b200.mesh import AMRHierarchy

    mesh = AMRHierarchy((32, 48), periodic=(True, False))
    mesh.add_patch(1, ((16, 40), (20, 60)))
    mesh.add_patch(2, ((40, 60), (50, 90)))
    model = MHD2D(mesh, precision=precision, conduction=(0.5, 0.1), resistivity=1e-3)
    model.set_state(lambda x, y: 0.2 + x + y, (0.1, 0.2, 0.3), 1.0, bz=0.3)
    assert model.engine.per_level_dt
    return model.engine


def _box(shape, precision):
    from wellbalanced_b200 import MHD3D
    from wellbalanced_b200.mesh import AMRHierarchy

    model = MHD3D(AMRHierarchy(shape, periodic=(True,) * 3), precision=precision)
    model.set_state(lambda x, y, z: 1.0 + 0.4 * np.sin(7.0 * x + 5.0 * y - 3.0 * z), (0.3, 0.2, -0.1), 0.5,
                    vector_potential=(0.0, 0.0, lambda x, y, z: 0.1 * np.sin(2.0 * np.pi * x)))
    return model.engine


def _batch(precision):
    from wellbalanced_b200 import Batch

    return Batch.orszag_tang(300, seed=3, precision=precision).engine


CASES = {
    "one chunk": lambda p: _plane((4, 5), p),
    "remainders": lambda p: _plane((131, 67), p),
    "resistive": lambda p: _plane((64, 40), p, resistivity=2e-2),
    "levels": _refined,
    "thin box": lambda p: _box((5, 4, 7), p),
    "box": lambda p: _box((41, 29, 53), p),
    "instances": _batch,
}


@pytest.mark.parametrize("precision", [32, 64, "mixed"])
@pytest.mark.parametrize("name", CASES)
def test_one_launch_equals_rate_and_dt(name, precision):
    engine = CASES[name](precision)
    eta, kappa = (2e-2, 0.5) if name in ("resistive", "levels") else (0.0, 0.0)
    engine.time.fill_(0.25)
    engine.rate()
    engine.finalize_dt(0.4, eta, kappa, advance=True)
    expect = [t.clone() for t in (engine.keys, engine.dt, engine.time, engine.level_keys)]
    assert bool(torch.isfinite(engine.dt).all()) and float(engine.dt.min()) > 0.0
    scratch = engine.dt_scratch.clone()
    for _ in range(2):
        engine.keys.zero_()
        engine.dt.zero_()
        engine.time.fill_(0.25)
        if engine.per_level_dt:
            engine.level_keys.zero_()
        engine.stable_dt(0.4, eta, kappa, advance=True)
        for got, want in zip((engine.keys, engine.dt, engine.time, engine.level_keys), expect):
            assert torch.equal(got, want)
        assert torch.equal(engine.dt_scratch, scratch)


def test_overlapping_launches_leave_the_scratch_whole():
    """Stable steps of one engine on two streams at once may spoil each other's dt, never a
    later one: the ticket and the keys are back at their start once both are done."""
    engine = _plane((700, 500), 32)
    engine.stable_dt(0.4)
    torch.cuda.synchronize()
    expect, scratch = engine.dt.clone(), engine.dt_scratch.clone()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(200):
        for stream in streams:
            with torch.cuda.stream(stream):
                engine.stable_dt(0.4)
    torch.cuda.synchronize()
    assert torch.equal(engine.dt_scratch, scratch)
    engine.stable_dt(0.4)
    assert torch.equal(engine.dt, expect)


@pytest.mark.parametrize("count", [255, 256, 257, 513])
@pytest.mark.parametrize("precision", [32, 64])
def test_every_count_of_instances_has_the_same_dt(count, precision):
    """One launch up to 256 instances, the rate and dt launches above."""
    from wellbalanced_b200 import Batch
    from wellbalanced_b200.problems import orszag_tang_2d

    batch = Batch([(8, 20, 48)[k % 3] for k in range(count)], precision=precision)
    for k, (n, _) in enumerate(batch.sides):
        batch.set_instance(k, *orszag_tang_2d(n, 0.5 + k / count, 1.5 - k / count))
    batch.finish_state()
    engine = batch.engine
    engine.rate()
    engine.finalize_dt(0.4)
    expect, keys = engine.dt.clone(), engine.keys.clone()
    scratch = engine.dt_scratch.clone()
    engine.dt.zero_()
    engine.stable_dt(0.4)
    assert torch.equal(engine.dt, expect) and torch.equal(engine.keys, keys)
    assert torch.equal(engine.dt_scratch, scratch) and float(expect.min()) > 0.0
