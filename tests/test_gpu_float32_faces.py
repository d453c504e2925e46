"""float32 faces at their edges (GPU): no star state on a cold supersonic face, vanishing
normal fields and star denominators, slopes of either sign and none, against float64 faces."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _uniform(ndim, axis, speed, pressure, precision):
    """A uniform flow along `axis` (density 1, no field) set by its conserved values."""
    from wellbalanced_b200 import MHD2D, MHD3D
    from wellbalanced_b200.mesh import AMRHierarchy

    shape = (20, 12, 9)[:ndim]
    mesh = AMRHierarchy(shape, periodic=(True,) * ndim)
    model = (MHD2D if ndim == 2 else MHD3D)(mesh, precision=precision, limiter="mc")
    cells = [np.ones(shape)] + [np.full(shape, speed if a == axis else 0.0) for a in range(3)]
    cells.append(np.full(shape, 1.5 * pressure + 0.5 * speed**2))
    if ndim == 2:
        model.set_conserved([*cells, np.zeros(shape)], np.zeros((21, 13)))
    else:
        nodes = [tuple(n + (a != c) for a, n in enumerate(shape)) for c in range(3)]
        model.set_conserved(cells, [np.zeros(n) for n in nodes])
    return model


@pytest.mark.parametrize("ndim, axis", [(2, 0), (2, 1), (3, 0), (3, 1), (3, 2)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_a_cold_flow_keeps_the_upwind_flux(ndim, axis, sign):
    """The fast speed (1.8e-7) is below half the spacing of float32 numbers at the velocity, so
    S = S_M and no star state exists; the flux differences of the uniform flow are exact zeros."""
    model = _uniform(ndim, axis, sign * 4.125, 2e-14, "mixed")
    before = model.engine.state.clone()
    model.step()
    assert torch.equal(model.engine.state, before)


@pytest.mark.parametrize("ndim, axis", [(2, 0), (2, 1), (3, 0), (3, 1), (3, 2)])
def test_a_flow_without_pressure_stays_finite(ndim, axis):
    model = _uniform(ndim, axis, 1.0, 0.0, 32)
    before = model.engine.state.clone()
    model.advance(1, check=False)
    assert int(model.engine.bad.item()) > 0  # no valid state, and counted as that
    assert torch.equal(model.engine.state, before)


@pytest.mark.parametrize("ndim, axis", [(2, 0), (2, 1), (3, 0), (3, 1), (3, 2)])
def test_a_negative_pressure_beside_a_cold_flow_keeps_the_upwind_flux(ndim, axis):
    """Two cold supersonic streams, the faster one with a (bad) negative pressure: where they part
    its star denominator is zero in float32, and the flux is that of the slower stream, as in
    float64. Bound: float32 rounding of a flux (1e-6 of its scale) on the two faces of a cell."""
    from wellbalanced_b200 import MHD2D, MHD3D
    from wellbalanced_b200.mesh import AMRHierarchy

    shape, ratio = (24, 24, 24)[:ndim], 0.02
    fast = np.broadcast_to(np.moveaxis((np.arange(24) >= 12).reshape(24, *(1,) * (ndim - 1)), 0, axis), shape)
    v = [np.full(shape, 0.5), np.full(shape, 0.25), np.full(shape, -0.75)]
    v[axis] = np.where(fast, 6.0, 2.0)
    cells = [np.ones(shape), *v, 1.5 * np.where(fast, -2e-14, 4e-15) + 0.5 * sum(c * c for c in v)]
    results = []
    for precision in (64, "mixed"):
        mesh = AMRHierarchy(shape, periodic=(True,) * ndim)
        model = (MHD2D if ndim == 2 else MHD3D)(mesh, precision=precision, limiter="minmod")
        if ndim == 2:
            model.set_conserved([*cells, np.zeros(shape)], np.zeros((25, 25)))
        else:
            model.set_conserved(cells, [np.zeros(tuple(24 + (a != c) for a in range(3))) for c in range(3)])
        eng = model.engine
        eng.dt.fill_(ratio / 24)
        eng.stage(eng.state, None, eng.stage_pool)
        results.append([model._read(mesh.patches[0], f, pool=eng.stage_pool).cpu().numpy() for f in range(5)])
    scale = float(np.abs(cells[4]).max()) * 6.0
    for want, got in zip(*results, strict=True):
        assert np.isfinite(got).all()
        assert np.abs(got - want).max() <= 2 * ratio * 1e-6 * scale


@pytest.mark.parametrize("limiter", ["minmod", "vanleer", "mc"])
@pytest.mark.parametrize("speed", [0.3, 4.0])
@pytest.mark.parametrize("field", ["none", "normal", "across", "out"])
@pytest.mark.parametrize("unit", [1.0, 2.0**-33])
def test_faces_agree_with_float64(unit, field, speed, limiter):
    """Random cells with constant stripes (slopes of both signs, and zero) under a field that is
    absent, along x (B_n = 0 on the y-faces, a vanishing star denominator on the x-faces, whose
    fast speed is the Alfven speed), along y, or along z (B_n = 0 everywhere); and the same in units
    in which the speeds are 1e-10 (their fourth powers are subnormal, good to 1e-6).

    Bound: a float32 flux is good to 2e-3 of its scale (star denominators are used down to 1e-3
    of their terms, with 1e-6 of rounding in them), four faces change a cell by dt / dx = 0.02 of
    their errors each; the scale of a flux is the largest conserved value times the largest
    signal speed."""
    from wellbalanced_b200 import MHD2D
    from wellbalanced_b200.mesh import AMRHierarchy

    shape, ratio = (24, 40), 0.02
    rng = np.random.default_rng(5)
    stripes = (np.arange(shape[0]) // 4 % 3 == 0)[:, None]
    draw = lambda lo, hi: np.where(stripes, 0.5 * (lo + hi), rng.uniform(lo, hi, shape))  # noqa: E731
    rho, p = draw(0.6, 1.4), draw(0.6, 1.4) * unit**2
    velocity = [draw(-speed, speed) * unit for _ in range(3)]
    mean, bz = {"none": ((0.0, 0.0), 0.0), "normal": ((2.0, 0.0), 0.0), "across": ((0.0, -2.0), 0.0),
                "out": ((0.0, 0.0), 1.5)}[field]
    mean, bz = (mean[0] * unit, mean[1] * unit), bz * unit
    b2 = mean[0] ** 2 + mean[1] ** 2 + bz**2
    energy = 1.5 * p + 0.5 * rho * sum(v * v for v in velocity) + 0.5 * b2
    results = []
    for precision in (64, "mixed"):
        mesh = AMRHierarchy(shape, ((0.0, 0.6), (0.0, 1.0)), periodic=(True, True))
        model = MHD2D(mesh, precision=precision, limiter=limiter, mean_field=mean)
        model.set_conserved([rho, *(rho * v for v in velocity), energy, np.full(shape, bz)], np.zeros((25, 41)))
        eng = model.engine
        eng.dt.fill_(ratio * 0.025 / unit)
        eng.bad.zero_()
        eng.stage(eng.state, None, eng.stage_pool)
        assert int(eng.bad.item()) == 0
        (patch,) = mesh.patches
        results.append([model._read(patch, f, node=f == 6, pool=eng.stage_pool).cpu().numpy() for f in range(7)])
    signal = speed + np.sqrt((5.0 / 3.0 * 1.4 + b2 / unit**2) / 0.6)
    bound = 4 * ratio * 2e-3 * float(np.abs(energy).max()) / unit**2 * signal
    scales = (1.0, unit, unit, unit, unit**2, unit, unit)
    for want, got, scale in zip(*results, scales, strict=True):
        assert np.isfinite(got).all()
        assert np.abs(got - want).max() <= bound * scale


@pytest.mark.parametrize("ndim", [2, 3])
def test_the_stable_step_in_units_of_small_speeds(ndim):
    """Speeds of 1e-10: the discriminants (6e-40) keep 18 bits, their roots 2e-6, the step half
    of that of its fast speed; 1e-5 with the float32 rounding around them."""
    from wellbalanced_b200 import MHD2D, MHD3D
    from wellbalanced_b200.mesh import AMRHierarchy

    unit = 2.0**-33
    steps = []
    for precision in (64, 32):
        mesh = AMRHierarchy((20, 12, 9)[:ndim], periodic=(True,) * ndim)
        model = (MHD2D if ndim == 2 else MHD3D)(mesh, precision=precision)
        model.set_state(lambda x, *y: 1.0 + 0.3 * np.sin(6.0 * x), (0.3 * unit, -0.2 * unit, 0.1 * unit), 0.8 * unit**2)
        steps.append(model.stable_step())
    assert abs(steps[1] - steps[0]) <= 1e-5 * steps[0]
