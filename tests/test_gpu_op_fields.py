"""Halo interpolation and copy kernels over field ranges the layouts do and do not use (GPU):
the code for the layouts' field counts and the general one against the NumPy emulation."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _layout(ndim, precision):
    from wellbalanced_b200.mesh import AMRHierarchy, Layout

    mesh = AMRHierarchy((12, 16, 8)[:ndim], periodic=(True, False, True)[:ndim])
    mesh.add_patch(1, ((6, 18), (8, 22), (4, 12))[:ndim])
    mesh.add_patch(1, ((18, 24), (8, 16), (2, 12))[:ndim])
    return Layout(mesh, precision=precision)


def _run(name, ops, layout, precision, host):
    from wellbalanced_b200 import _lib
    from wellbalanced_b200.engine import _device_bytes

    dtype = _lib.INTERP_OP if name == "wb_interp_ops" else _lib.COPY_OP
    pool = torch.from_numpy(host.astype(np.float32 if precision == 32 else np.float64)).cuda()
    rows = _device_bytes(layout.rows, pool.device, _lib.PATCH)
    device_ops = _device_bytes(ops, pool.device, dtype)
    _lib.call(name, precision, pool.data_ptr(), rows.data_ptr(), device_ops.data_ptr(), int(ops.size),
              torch.cuda.current_stream().cuda_stream)
    return pool.cpu().numpy().astype(np.float64)


def _pool(layout, seed, precision):
    values = np.random.default_rng(seed).uniform(-1.0, 1.0, layout.pool_size)
    return values.astype(np.float32).astype(np.float64) if precision == 32 else values


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("fields", [None, (0, 1), (1, 4), (0, 7)])
def test_interpolation_over_field_ranges(precision, ndim, fields):
    from tests import _emulate

    layout = _layout(ndim, precision)
    host = _pool(layout, 1, precision)
    # at most 64 terms of magnitude 1, weights adding up to (5/4)^3 < 2: rounding of the
    # weights' products and of the sum
    tolerance = 2.0 * 70.0 * (2.0**-24 if precision == 32 else 2.0**-53)
    for mask in np.unique(layout.interp_levels[1]["node_mask"]):
        ops = layout.interp_levels[1][layout.interp_levels[1]["node_mask"] == mask].copy()
        if fields is not None:
            ops["field_lo"], ops["field_hi"] = fields
        got = _run("wb_interp_ops", ops, layout, precision, host)
        # a node on the periodic seam lies in the reach of two ops (its parent and the parent's
        # image), which agree on a state but not on random numbers: either value is right there
        error = np.abs(got - host)
        written = np.zeros(host.size, dtype=bool)
        for k in range(ops.size):
            expect = host.copy()
            _emulate.apply_interp(expect, layout.rows, ops[k : k + 1])
            mine = expect != host
            error[mine] = np.where(written[mine], np.minimum(error[mine], np.abs(got - expect)[mine]),
                                   np.abs(got - expect)[mine])
            written |= mine
        assert written.any()
        assert np.max(error) <= tolerance


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("fields", [None, (0, 1), (1, 4), (0, 7)])
@pytest.mark.parametrize("weights", [(1.0, 0.0, -1), (1.0, 0.0, 1), (0.5, 2.0, 2)])
def test_copies_over_field_ranges(precision, ndim, fields, weights):
    """Through the fill launch (one point per thread) and the copy launch (two)."""
    from tests import _emulate
    from wellbalanced_b200 import _lib
    from wellbalanced_b200.engine import _device_bytes

    layout = _layout(ndim, precision)
    host = _pool(layout, 2, precision)
    same = layout.copy_phases[1][0]
    ops = same[same["field_lo"] == 0].copy()
    if fields is not None:
        ops["field_lo"], ops["field_hi"] = fields
    ops["w1"], ops["w2"], ops["negate"] = weights
    ops["src2"], ops["s2"], ops["m2"] = ops["src1"], ops["s1"], ops["m1"]
    expect = host.copy()
    _emulate.apply_copy(expect, layout.rows, ops)
    assert not np.array_equal(expect, host)
    # w1 x + w2 x with exact weights: one rounding of the sum (magnitude < 3)
    tolerance = 4.0 * (2.0**-24 if precision == 32 else 2.0**-53)
    got = _run("wb_copy_ops", ops, layout, precision, host)
    assert np.max(np.abs(got - expect)) <= tolerance
    pool = torch.from_numpy(host.astype(np.float32 if precision == 32 else np.float64)).cuda()
    rows = _device_bytes(layout.rows, pool.device, _lib.PATCH)
    device_ops = _device_bytes(ops, pool.device, _lib.COPY_OP)
    _lib.call("wb_fill_ops", precision, pool.data_ptr(), rows.data_ptr(), None, 0, device_ops.data_ptr(), int(ops.size),
              torch.cuda.current_stream().cuda_stream)
    assert np.max(np.abs(pool.cpu().numpy() - expect)) <= tolerance
