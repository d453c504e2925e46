"""Launch lists (CPU): every name has a code, arguments land in their slots."""

import numpy as np
import pytest

from wellbalanced_b200 import _lib, build


def test_slots_hold_integers_pointers_and_double_bits():
    build.build()
    calls = [("wb_reflux_apply", (32, 11, 12, 13, 14, 15, 16), None), ("record_event", (77,), 5),
             ("wb_copy_ops", (64, 1, 2, None, 0), 0)]
    name, types = "wb_stable_dt", _lib.SIGNATURES["wb_stable_dt"]
    calls.append((name, tuple(0.5 + k if t is _lib.c_double else k for k, t in enumerate(types[:-1])), None))
    entries = _lib.launch_list(calls)
    assert len(set(entries["code"].tolist())) == 4
    assert entries["args"][0][:7].tolist() == [32, 11, 12, 13, 14, 15, 16]
    assert entries["own_stream"].tolist() == [0, 1, 1, 0] and entries["stream"].tolist() == [0, 5, 0, 0]
    assert entries["args"][2][:5].tolist() == [64, 1, 2, 0, 0]
    for k, t in enumerate(types[:-1]):
        slot = entries["args"][3][k]
        assert slot.view(np.float64) == 0.5 + k if t is _lib.c_double else slot == k


def test_the_slots_of_the_dt_parameters():
    """cfl, eta and kappa, which a step's list takes anew when they change."""
    from wellbalanced_b200.engine import _DT_SLOTS

    build.build()
    types = _lib.SIGNATURES["wb_stable_dt"][:-1]
    doubles = [k for k, t in enumerate(types) if t is _lib.c_double]
    assert doubles[-3:] == list(range(_DT_SLOTS.start, _DT_SLOTS.stop))
    assert len(doubles) == 7  # the mean field and gamma before them


def test_wrong_names_and_counts_are_refused():
    build.build()
    with pytest.raises(_lib.WBError, match="no launch named"):
        _lib.launch_list([("wb_version", (), None)])
    with pytest.raises(ValueError, match="arguments"):
        _lib.launch_list([("wb_copy_ops", (32, 1), None)])
    assert _lib.load().wb_launch_code(b"no such launch") < 0
    bad = np.zeros(1, dtype=_lib.LAUNCH)
    bad["code"] = 1000
    assert _lib.load().wb_run_launches(bad.ctypes.data, 1, 1, None) < 0
