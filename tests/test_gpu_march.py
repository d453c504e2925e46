"""The x-planes per tile of the 3D stage kernel (GPU): `lx` bounds them, `march` says and sets
how many run, and on one tile shape no choice changes a bit."""

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64, "mixed"])
def test_the_march_is_readable_bounded_and_settable(precision):
    from wellbalanced_b200 import MHD3D

    chosen = MHD3D.turbulence(24, seed=2, precision=precision, lx=32)
    assert 1 <= chosen.march <= 32 and chosen.march == chosen.engine.layout.march
    chosen.advance(2)
    for planes in (1, 5, 32):
        exact = MHD3D.turbulence(24, seed=2, precision=precision)
        exact.capture()
        exact.load(MHD3D.turbulence(24, seed=2, precision=precision).save())
        exact.march = planes
        assert exact.march == planes and exact.engine.layout.march == planes and exact._graph is None
        assert int(exact.engine.layout.tiles["x0"].max()) == (24 - 1) // planes * planes
        exact.engine.time.zero_()
        exact.advance(2)
        torch.cuda.synchronize()
        assert torch.equal(exact.engine.state, chosen.engine.state)
    for planes in (0, -4):
        with pytest.raises(ValueError, match="at least one plane"):
            chosen.march = planes


def test_a_tuned_model_runs_what_was_measured():
    from wellbalanced_b200 import MHD3D

    tuned = MHD3D.turbulence(20, seed=2, precision=32, lx="auto")
    assert tuned.march == tuned.lx
