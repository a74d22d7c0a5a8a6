"""Calls that take three steps per launch (the default kernel in channel
mode) against the CPU oracle, bit for bit, and against the one-step kernels:
the stored state of both buffer sets and the moments are the same bytes."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# k_step_multi, just above the 400,000 cells (250,000 in 16-bit storage) from
# which it runs: around one and two warps' 60 columns, the narrowest and the
# lowest, bands that end unevenly
# (stochastic rounding: four times the rows, as it starts at 900,000)
SIZES = [(7, 60000), (60, 6667), (61, 6601), (62, 6452), (121, 3311), (133400, 3), (57200, 7), (1100, 370), (2521, 161)]
# k_step_tile: tiles of 60 columns and 8 rows, or 4 where 8 leave multiprocessors idle
SMALL = [(3, 3), (5, 4), (59, 3), (60, 8), (61, 9), (62, 12), (63, 31), (121, 40), (600, 5), (130, 700), (1200, 70),
         (9000, 25)]


def pair(lbm, P, nx, ny, storage, seed, inlet=False, sr=None, density=0.12):
    rng = np.random.default_rng(seed)
    omega = float(np.float32(rng.uniform(0.7, 1.8)))
    mask = (rng.random((ny, nx)) < density).astype(np.uint8)
    u = float(np.float32(0.06))
    lat = lbm.Lattice(nx, ny, omega, lbm.EDGE_CHANNEL, storage)
    o = P.Oracle(nx, ny, omega, P.EDGE_CHANNEL, storage)
    if inlet:
        lat.set_storage_reference(True)
        o.set_storage_reference(True)
    lat.set_inlet_velocity(u)
    o.set_inlet(u, apply=False)
    lat.init_equilibrium(1.0, u, 0.0, 1e-2, seed)
    o.init_equilibrium(1.0, u, 0.0, float(np.float32(1e-2)), seed)
    lat.draw_mask(mask)
    o.set_mask(mask)
    if sr is not None:
        lat.set_rounding(lbm.ROUND_STOCHASTIC, sr)
        o.set_rounding(1, sr)
    return lat, o


def same(lat, o):
    pops, rho, jx, jy = o.state()
    for name, want in (("rho", rho), ("jx", jx), ("jy", jy)):
        np.testing.assert_array_equal(lat.field(name), want.astype(np.float32))
    np.testing.assert_array_equal(lat.populations(), pops.astype(np.float32))


@pytest.mark.parametrize("storage,inlet,sr", [(0, False, None), (1, False, None), (2, True, None), (1, False, 7),
                                              (2, True, 9)])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_three_step_launches_match_the_oracle(lbm, cuda_ok, oracle_mod, storage, inlet, sr, nx, ny):
    if sr is not None:
        nx, ny = (4 * nx, ny) if 4 * ny > 65535 else (nx, 4 * ny)
    lat, o = pair(lbm, oracle_mod, nx, ny, storage, 31 * nx + ny, inlet, sr)
    for n in (5, 4, 7, 7, 1, 9):  # plain launches, then captured calls from each parity
        lat.iterate(n)
        o.step(n)
    same(lat, o)
    assert lat.get_compute_num() == 33
    lat.close()


@pytest.mark.parametrize("storage,inlet,sr", [(0, False, None), (1, False, None), (2, True, None), (1, False, 7),
                                              (2, True, 9)])
@pytest.mark.parametrize("nx,ny", SMALL)
def test_three_step_tiles_match_the_oracle(lbm, cuda_ok, oracle_mod, storage, inlet, sr, nx, ny):
    lat, o = pair(lbm, oracle_mod, nx, ny, storage, 31 * nx + ny, inlet, sr)
    for n in (5, 4, 7, 7, 7, 1, 24, 83):  # plain launches, then captured calls from each parity, then runs
        lat.iterate(n)
        o.step(n)
    same(lat, o)
    assert lat.get_compute_num() == 138
    lat.close()


@pytest.mark.parametrize("storage,sr,nx,ny", [(0, None, 61, 33), (0, None, 700, 640), (1, None, 300, 90),
                                              (2, 5, 190, 57)])
def test_closure_records_in_three_step_tiles(lbm, cuda_ok, storage, sr, nx, ny):
    """The closure's per-cell rates and fallbacks: the same words and the same
    count as the one-step kernel's, with some cells over the drift bound."""
    rng = np.random.default_rng(nx)
    n_par = 19969
    w = (rng.uniform(-0.3, 0.3, n_par)).astype(np.float32)
    mask = (rng.random((ny, nx)) < 0.06).astype(np.uint8)
    L = lbm.load_library()
    got = []
    for tuned in (False, True):
        lat = lbm.Lattice(nx, ny, 1.4, lbm.EDGE_CHANNEL, storage)
        lat.set_inlet_velocity(0.06)
        lat.init_equilibrium(1.0, 0.06, 0.0, 2e-2, 4)
        lat.draw_mask(mask)
        if sr is not None:
            lat.set_rounding(lbm.ROUND_STOCHASTIC, sr)
        if tuned:
            lat.set_tuning(2, 3 if storage == 0 else 7)
        lbm._check(L.lbm_closure_set_weights(lat.handle, w.ctypes.data, w.size))
        lbm._check(L.lbm_closure_enable(lat.handle, 0.2))
        counts = []
        for n in (3, 20, 20, 7):
            lbm._check(L.lbm_closure_infer(lat.handle))
            lat.iterate(n)
            c = ctypes.c_uint64()
            lbm._check(L.lbm_closure_fallback_count(lat.handle, ctypes.byref(c), 1))
            counts.append(c.value)
        got.append((counts, lat.checkpoint(), lat.field("jx"), lat.field("rho")))
        lat.close()
    assert got[0][0] == got[1][0] and max(got[0][0]) > 0
    assert got[0][1] == got[1][1]
    np.testing.assert_array_equal(got[0][2], got[1][2])
    np.testing.assert_array_equal(got[0][3], got[1][3])


@pytest.mark.parametrize("storage,inlet,sr", [(0, False, None), (1, True, 5)])
def test_long_calls_replay_runs_of_captured_steps(lbm, cuda_ok, oracle_mod, storage, inlet, sr):
    lat, o = pair(lbm, oracle_mod, 700, 2400, storage, 3, inlet, sr)
    for n in (67, 83):
        lat.iterate(n)
        o.step(n)
    same(lat, o)
    lat.close()


@pytest.mark.parametrize("storage,sr", [(0, None), (1, None), (1, 3)])
def test_edits_between_three_step_launches(lbm, cuda_ok, oracle_mod, storage, sr):
    """Solid cells drawn into and cleared from a moving flow, a new inlet
    velocity, a new omega, and column 0 made solid in places."""
    lat, o = pair(lbm, oracle_mod, 700, 2400, storage, 5, sr=sr)
    rng = np.random.default_rng(8)
    for k in range(4):
        lat.iterate(10 + k)
        o.step(10 + k)
        idx = rng.integers(0, 700 * 2400, 400)
        if k == 2:
            idx[:40] = 700 * rng.integers(0, 2400, 40)
        pairs = np.stack([idx, rng.integers(0, 2, 400)], 1).astype(np.uint32)
        lat.draw_points(pairs)
        o.barrier_pairs(pairs)
        if k == 1:
            lat.set_inlet_velocity(0.05)
            o.set_inlet(float(np.float32(0.05)))
        if k == 2:
            lat.update_omega_buffer(1.25)
            o.set_omega(1.25)
    lat.iterate(29)
    o.step(29)
    same(lat, o)
    lat.close()


@pytest.mark.parametrize("storage,inlet,sr", [(0, False, None), (1, True, None), (2, False, 4)])
@pytest.mark.parametrize("ny", [61, 2661])
def test_both_buffer_sets_are_those_of_single_steps(lbm, cuda_ok, oracle_mod, storage, inlet, sr, ny):
    """The checkpoint holds every stored word: the bytes after calls of any
    length equal those of a lattice kept on the one-step kernel, before and
    after edits, and the steps after loading it continue the same."""
    lats = [pair(lbm, oracle_mod, 637, ny, storage, 17, inlet, sr)[0] for _ in range(2)]
    lats[1].set_tuning(2, 3 if storage == 0 else 7)
    for n in (9, 23, 4, 70):
        for lat in lats:
            lat.iterate(n)
        a, b = (lat.checkpoint() for lat in lats)
        assert a == b
        pts = np.array([[40 * 637 + 50 + n, 1], [10 * 637 + 30, n & 1]], np.uint32)
        for lat in lats:
            lat.draw_points(pts)
    for lat in lats:
        lat.iterate(12)
    ck = lats[0].checkpoint()
    lats[0].iterate(15)
    again = lbm.Lattice(637, ny, 1.0, lbm.EDGE_CHANNEL, storage)
    again.restore(ck)
    again.iterate(15)
    lats[1].iterate(15)
    np.testing.assert_array_equal(again.populations(), lats[1].populations())
    np.testing.assert_array_equal(lats[0].populations(), lats[1].populations())
    for lat in lats + [again]:
        lat.close()


def test_inlet_rows_written_to_one_buffer_set(lbm, cuda_ok):
    """lbm_rows_write can leave different words in column 0 of the two buffer
    sets; the steps after it then follow the one-step rule."""
    lats = [lbm.Lattice(800, 520, 1.3, lbm.EDGE_CHANNEL, lbm.F32) for _ in range(2)]
    lats[1].set_tuning(2, 3)
    for lat in lats:
        lat.init_equilibrium(1.0, 0.05, 0.0, 1e-2, 3)
        lat.iterate(11)
        rows = lat.read_rows(7, 4, range(8))
        lat.write_rows(7, list(range(8)), rows * np.float32(1.01))
        lat.iterate(20)
    np.testing.assert_array_equal(lats[0].populations(), lats[1].populations())
    assert lats[0].checkpoint() == lats[1].checkpoint()
    for lat in lats:
        lat.close()


def test_non_finite_density_is_reported(lbm, cuda_ok):
    lat = lbm.Lattice(1030, 400, 1.2, lbm.EDGE_CHANNEL, lbm.F32)
    lat.iterate(4)
    lat.synchronize()
    pops = lat.populations()
    pops[4, 20, 60] = np.nan
    lat.write_populations(pops)
    lat.iterate(8)
    with pytest.raises(lbm.LBMError):
        lat.synchronize()
    lat.close()


@pytest.mark.parametrize("scale", [-110, -63, -60, 0, 58, 63, 100])
@pytest.mark.parametrize("ny", [30, 601])
def test_densities_of_any_scale(lbm, cuda_ok, oracle_mod, scale, ny):
    """Densities inside, at the edge of and outside the range of the
    shared-reciprocal quotients (and zero momenta) divide as IEEE does."""
    P = oracle_mod
    nx = 727
    rng = np.random.default_rng(2)
    pops = rng.uniform(0.01, 0.2, (9, ny, nx)).astype(np.float32)
    pops[:, 5] = np.float32(1.0 / 9.0)
    pops *= np.float32(2.0 ** scale)
    lat = lbm.Lattice(nx, ny, 1.1, lbm.EDGE_CHANNEL, lbm.F32)
    o = P.Oracle(nx, ny, float(np.float32(1.1)), P.EDGE_CHANNEL, P.P_F32)
    lat.write_populations(pops)
    o.put_state(pops)
    lat.iterate(5)
    o.step(5)
    np.testing.assert_array_equal(lat.populations(), o.state()[0].astype(np.float32))
    lat.close()


@pytest.mark.parametrize("storage,inlet,sr,nx,ny", [(0, False, None, 121, 4865), (1, False, None, 1270, 769),
                                                    (2, True, 6, 190, 4861)])
def test_bands_of_twelve_rows_and_a_remainder(lbm, cuda_ok, oracle_mod, storage, inlet, sr, nx, ny):
    """Lattices whose 12-row bands fill half of the chip: the last band is short."""
    lat, o = pair(lbm, oracle_mod, nx, ny, storage, nx, inlet, sr)
    for n in (4, 7):
        lat.iterate(n)
        o.step(n)
    same(lat, o)
    lat.close()


@pytest.mark.parametrize("storage,sr,nx,ny", [(0, None, 200, 64), (0, None, 121, 3400), (1, 9, 200, 64)])
@pytest.mark.parametrize("before", [4, 7])
def test_a_callers_graph_survives_other_steps(lbm, cuda_ok, oracle_mod, storage, sr, nx, ny, before):
    """Ten steps and a population read captured by the caller, replayed around
    plain calls: the graph keeps reading the rest plane that holds the state
    (before: an odd or an even number of three-step launches precedes it)."""
    import torch
    from lbm_gb300 import load_library
    lat, o = pair(lbm, oracle_mod, nx, ny, storage, 5, False, sr)
    s = torch.cuda.Stream()
    lat.set_stream(s.cuda_stream)
    lat.iterate(before)
    o.step(before)
    lat.populations()
    out = torch.zeros(9, ny, nx, device="cuda")
    torch.cuda.synchronize()

    def ten():
        lat.iterate(10)
        lbm._check(load_library().lbm_read_populations_device(lat.handle, ctypes.c_void_p(out.data_ptr())))

    s.synchronize()
    ten()  # the state is now as a replay leaves it
    o.step(10)
    lat.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        ten()
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        o.step(10)
        np.testing.assert_array_equal(out.cpu().numpy(), o.state()[0].astype(np.float32))
    lat.iterate(10)
    lat.populations()
    lat.synchronize()
    o.step(10)
    g.replay()
    torch.cuda.synchronize()
    o.step(10)
    same(lat, o)
    lat.close()


def test_a_callers_captured_inlet_change_survives_other_steps(lbm, cuda_ok, oracle_mod):
    """An inlet change captured by the caller and replayed after plain steps
    sets the column of the rest plane that holds the state."""
    import torch
    lat, o = pair(lbm, oracle_mod, 200, 64, 0, 5, False, None)
    s = torch.cuda.Stream()
    lat.set_stream(s.cuda_stream)
    lat.iterate(10)
    lat.populations()
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        lat.set_inlet_velocity(0.12)
    lat.iterate(13)
    lat.populations()
    lat.synchronize()
    g.replay()
    torch.cuda.synchronize()
    lat.iterate(7)
    o.step(23)
    o.set_inlet(0.12)
    o.step(7)
    same(lat, o)
    lat.close()


@pytest.mark.parametrize("storage,nx,ny,three", [(0, 700, 640, True), (0, 1024, 512, False), (1, 450, 400, True),
                                                 (2, 512, 400, False)])
def test_closure_steps_share_launches_on_small_lattices_only(lbm, cuda_ok, storage, nx, ny, three):
    """With the closure on, three steps share a launch on small lattices; larger
    ones step one by one, which is faster there."""
    L = lbm.load_library()
    lat = lbm.Lattice(nx, ny, 1.4, lbm.EDGE_CHANNEL, storage)
    w = np.zeros(19969, np.float32)
    lbm._check(L.lbm_closure_set_weights(lat.handle, w.ctypes.data, w.size))
    lbm._check(L.lbm_closure_enable(lat.handle, 0.2))
    lat.iterate(2)
    lbm._check(L.lbm_closure_infer(lat.handle))
    before = lat.launch_count()
    lat.iterate(20)
    assert lat.launch_count() - before == (8 if three else 20)
    lat.close()
