"""float64 quotients of zero, infinite and NaN operands (GPU): the per-kernel interface gives
what the reference's divisions give, and a cell of infinite energy leaves no stable step."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

INF = float("inf")


def _fields():
    rng = np.random.default_rng(4)
    shape = (12, 11)
    fields = [rng.uniform(0.5, 1.5, shape)] + [rng.normal(size=shape) for _ in range(3)]
    fields += [rng.uniform(6.0, 9.0, shape), 0.3 * rng.normal(size=shape)]
    return fields, 0.02 * rng.normal(size=(13, 12))


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def test_primitives_are_the_reference_quotients():
    from oracle import kernels as oracle
    from wellbalanced_b200.kernels import KERNELS

    fields, az = _fields()
    # (row, value) in cells of their own, a field value beside each
    for k, (row, value) in enumerate([(0, 0.0), (0, -0.0), (0, INF), (1, INF), (2, -INF), (3, np.nan), (4, INF), (5, -INF)]):
        fields[row][k + 1, 2 * (k % 5) + 1] = value
    fields[0][10, 9], fields[1][10, 9] = 0.0, 0.0
    az[11, 3] = INF
    nx, ny = fields[0].shape
    shapes = ((8, nx, ny), (nx + 1, ny), (nx, ny + 1), (nx, ny))
    expect = [np.empty(s) for s in shapes]
    args = (0.1, 0.2, 0.3, -0.4, 5.0 / 3.0)
    with np.errstate(all="ignore"):
        count = oracle.mhd_primitive(*fields, az, *args, *expect)
    got = [torch.empty(s, dtype=torch.float64, device="cuda") for s in shapes]
    assert KERNELS["mhd_primitive"](*map(_dev, fields), _dev(az), *args, *got) == count
    for g, e in zip(got, expect, strict=True):
        np.testing.assert_allclose(g.cpu().numpy(), e, rtol=1e-13, atol=1e-13)


def test_the_rate_of_an_infinite_energy():
    from wellbalanced_b200.kernels import KERNELS

    fields, az = _fields()
    fields[4][6, 5] = INF
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    KERNELS["mhd_rate"](*map(_dev, fields), _dev(az), 2, 0.1, 0.2, 0.3, -0.4, 5.0 / 3.0, out)
    assert out[0].item() == INF and out[1].item() == fields[0][2:-2, 2:-2].min()


@pytest.mark.parametrize("ndim", [2, 3])
def test_an_infinite_energy_leaves_no_stable_step(ndim):
    from wellbalanced_b200 import MHD2D, MHD3D
    from wellbalanced_b200.mesh import AMRHierarchy

    shape = (12, 10, 8)[:ndim]
    cells = [np.ones(shape), np.full(shape, 0.3), np.zeros(shape), np.zeros(shape), np.full(shape, 2.0)]
    cells[4][(5, 4, 3)[:ndim]] = INF
    mesh = AMRHierarchy(shape, periodic=(True,) * ndim)
    mean = (0.2, -0.1, 0.3)[:ndim]
    model = (MHD2D if ndim == 2 else MHD3D)(mesh, precision=64, mean_field=mean)
    if ndim == 2:
        model.set_conserved([*cells, np.full(shape, 0.1)], np.zeros((13, 11)))
    else:
        model.set_conserved(cells, [np.zeros(tuple(n + (a != c) for a, n in enumerate(shape))) for c in range(3)])
    assert model.stable_step() == 0.0
