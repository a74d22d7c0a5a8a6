"""Reference-mode steps of the default kernel (two cells per lane) against the
CPU oracle, bit for bit: the lattice's edge cells, its columns' remainders by
64, rows by four, solid cells in runs and alone, and the storage options."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,inlet,sr", [(0, False, None), (1, False, None), (2, True, None), (1, True, 5)])
@pytest.mark.parametrize("nx,ny", [(3, 3), (4, 5), (63, 6), (64, 7), (65, 9), (66, 4), (129, 31), (300, 70),
                                   (1100, 130)])
@pytest.mark.parametrize("walls", [True, False])
def test_pair_steps_match_the_oracle(lbm, cuda_ok, oracle_mod, storage, inlet, sr, nx, ny, walls):
    P = oracle_mod
    rng = np.random.default_rng(nx * 100 + ny)
    omega = float(np.float32(rng.uniform(0.8, 1.7)))
    mask = (rng.random((ny, nx)) < 0.15).astype(np.uint8)
    if walls:
        mask[0] = mask[-1] = 1
    lat = lbm.Lattice(nx, ny, omega, lbm.EDGE_REF, storage)
    o = P.Oracle(nx, ny, omega, P.EDGE_REF, storage)
    if inlet:
        lat.set_storage_reference(True)
        o.set_storage_reference(True)
    lat.init_equilibrium(1.0, 0.1, 0.0, 1e-2, 7)
    o.init_equilibrium(1.0, float(np.float32(0.1)), 0.0, float(np.float32(1e-2)), 7)
    lat.draw_mask(mask)
    o.set_mask(mask)
    if sr is not None:
        lat.set_rounding(lbm.ROUND_STOCHASTIC, sr)
        o.set_rounding(1, sr)
    for n in (3, 6, 1, 6):
        lat.iterate(n)
        o.step(n)
    pairs = np.stack([rng.integers(0, nx * ny, 12), rng.integers(0, 2, 12)], 1).astype(np.uint32)
    lat.draw_points(pairs)  # single points among the packed mask words
    o.barrier_pairs(pairs)
    np.testing.assert_array_equal(lat.mask(), o.mask())
    lat.iterate(20)
    o.step(20)
    pops, rho, jx, jy = o.state()
    for name, want in (("rho", rho), ("jx", jx), ("jy", jy)):
        np.testing.assert_array_equal(lat.field(name), want.astype(np.float32))
    np.testing.assert_array_equal(lat.populations(), pops.astype(np.float32))
    lat.close()
