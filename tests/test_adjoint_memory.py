"""The first backward pass allocates nothing on the device: tg_forward has taken its
buffers (an allocation there would count against the backward pass's time)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("n_side,leaf,ewald", [(16, 64, True), (24, 16, True), (20, 128, True), (20, 32, False)])
def test_first_backward_allocates_nothing(precision, n_side, leaf, ewald):
    import tigergrav_b200 as tg
    from tigergrav_b200 import ics
    x = ics.clustered(n_side, 3)
    w = np.random.default_rng(4).standard_normal((len(x), 3))
    with tg.GravitySolver(len(x), theta=0.7, leaf_max=leaf, ewald=ewald, precision=precision) as s:
        s.set_particles(x).forward(1e-3, 2)
        before = s.memory()
        s.backward(w, w)
        assert s.memory() == before
