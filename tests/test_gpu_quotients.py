"""The collision's shared-reciprocal quotients against the CPU oracle's
divisions, bit for bit: densities with a mantissa of all ones (1 - 2^-24 is the
one next to rest) under momenta that are powers of two, and densities out of the
quotients' range in a column that a tile advances without storing it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CX = (-1, 0, 1, -1, 0, 1, -1, 0, 1)
CY = (1, 1, 1, 0, 0, 0, -1, -1, -1)  # populations move from row y + CY to row y
HOLD = float(np.float32(2.0 ** -120))  # a collision at this rate leaves the populations as they are


def streamed_to(want):
    """The populations that pull to `want` [9, ny, nx] (periodic)."""
    out = np.empty_like(want)
    for q in range(9):
        out[q] = np.roll(want[q], (CY[q], -CX[q]), (0, 1))
    return out


def both(lbm, P, edge, pops, omega, steps):
    ny, nx = pops.shape[1:]
    lat = lbm.Lattice(nx, ny, HOLD, lbm.EDGE_REF if edge else lbm.EDGE_CHANNEL, lbm.F32)
    o = P.Oracle(nx, ny, HOLD, P.EDGE_REF if edge else P.EDGE_CHANNEL, P.P_F32)
    lat.reset_barrier()
    mask = np.zeros((ny, nx), np.uint8)
    lat.draw_mask(mask)
    o.set_mask(mask)
    lat.write_populations(pops)
    o.put_state(pops)
    lat.iterate(1)  # collides in place
    o.step(1)
    lat.update_omega_buffer(omega)
    o.set_omega(omega)
    lat.iterate(steps)
    o.step(steps)
    got, want = lat.populations(), o.state()[0].astype(np.float32)
    lat.close()
    np.testing.assert_array_equal(got, want)


# k_step_tile, k_step_multi, k_step_pair
@pytest.mark.parametrize("edge,nx,ny", [(0, 300, 40), (0, 730, 560), (1, 300, 40)])
@pytest.mark.parametrize("scale", [0, -40, 30])
def test_all_ones_densities_with_power_of_two_momenta(lbm, cuda_ok, oracle_mod, edge, nx, ny, scale):
    """Every cell's density 1 - 2^-24, whose reciprocal lies next to a tie, and
    its momenta 0 or a power of two: all sums are exact in f32, so the quotients
    are what the density and the momenta say."""
    rng = np.random.default_rng(nx + scale)
    one = 1 << 24
    n = rng.integers(one // 16, one // 12, (9, ny, nx))
    # the momenta through the axis pairs, the density through the rest population
    for axis, (plus, minus), others in ((0, (5, 3), ((2, 1), (8, 1), (0, -1), (6, -1))),
                                        (1, (1, 7), ((2, 1), (0, 1), (8, -1), (6, -1)))):
        power = rng.integers(10, 21, (ny, nx))
        j = rng.integers(-1, 2, (ny, nx)) * (1 << power)
        n[plus] = n[minus] + j - sum(s * n[q] for q, s in others)
    n[4] = 0
    n[4] = one - 1 - n.sum(0)
    assert np.abs(n).max() < one
    want = n.astype(np.float64) * 2.0 ** (scale - 24)
    assert np.array_equal(want, want.astype(np.float32))
    both(lbm, oracle_mod, edge, streamed_to(want.astype(np.float32)), 1.25, 4)


def test_a_density_out_of_range_in_a_column_not_stored(lbm, cuda_ok, oracle_mod):
    """One cell at column 120, which the tile of columns 60 to 119 advances for
    its neighbours' sake: its density is above 2^126 (the reciprocal is a
    denormal, read as zero) and its populations are such that, with a zero
    velocity, nothing of it moves west, north, south or stays."""
    nx, ny, y = 181, 2300, 13
    m = np.float32(2.0 ** 122)
    want = np.empty((9, ny, nx), np.float32)
    want[:] = (np.array([1, 4, 1, 4, 16, 4, 1, 4, 1], np.float32) * np.float32(2.0 ** 40 / 36))[:, None, None]
    cell = np.array([1.75, 7, -5, 7, 28, -15.5, 1.75, 7, -5], np.float32)
    assert np.float32(27) * np.float32(1 / 9) == 3 and cell.sum() == 27
    want[:, y, 120] = cell * m
    both(lbm, oracle_mod, 0, streamed_to(want), 1.75, 4)
