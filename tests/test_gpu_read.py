"""Populations read between steps, materialised in the same pass: the values of
the materialised state, bit for bit, and no trace in the steps that follow."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,sr", [(0, None), (1, None), (2, None), (1, 5), (3, None)])
@pytest.mark.parametrize("nx,ny", [(3, 3), (33, 5), (128, 4), (257, 67)])
@pytest.mark.parametrize("edge", ["ref", "channel"])
def test_read_between_steps_equals_the_materialised_state(lbm, cuda_ok, storage, sr, nx, ny, edge):
    rng = np.random.default_rng(nx + ny)
    mask = (rng.random((ny, nx)) < 0.15).astype(np.uint8)
    if edge == "channel":
        mask[0] = mask[-1] = 1

    def lattice():
        lat = lbm.Lattice(nx, ny, 1.3, lbm.EDGE_REF if edge == "ref" else lbm.EDGE_CHANNEL, storage)
        if edge == "channel":
            lat.set_inlet_velocity(0.05)
        lat.init_equilibrium(1.0, 0.05, 0.0, 1e-2, 7)
        lat.draw_mask(mask)
        if sr is not None:
            lat.set_rounding(lbm.ROUND_STOCHASTIC, sr)
        return lat

    a, b = lattice(), lattice()  # a is read, b is not
    for n in (1, 4, 7):
        a.iterate(n)
        b.iterate(n)
        pulled = a.populations(f64=storage == 3)
        np.testing.assert_array_equal(a.populations(f64=storage == 3), pulled)  # from memory
    a.iterate(2)
    a.populations()
    a.iterate(3)
    b.iterate(5)
    np.testing.assert_array_equal(np.frombuffer(a.checkpoint(), np.uint8), np.frombuffer(b.checkpoint(), np.uint8))
    a.close()
    b.close()
