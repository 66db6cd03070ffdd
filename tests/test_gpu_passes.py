"""The neighbour passes at the sizes where their variants change, bit for bit
against the oracle: eight threads per particle up to 9,472 particles (148 SMs x 4
blocks x 16), the search with eight threads up to 40,960 (16,384 in
cells of h), and the layout for a device that is not full up to 113,664 threads (148 SMs x 3 blocks x 256), a particle
taking one, two or four threads with one or two, four and eight pair lanes. Also
the searched lists where rows leave the grid, for cells from h/3 to 3h/2, and
s_corr exponents other than four, which have kernels of their own; and the warm
start's first pass, one launch up to 75,776 particles (148 SMs x 2 x 256) and two
above."""
import numpy as np
import pytest
import torch

from pbf_b200 import Solver, autotune, learned, scenes

from test_gpu_parity import assert_substep_bitexact, make_pair, mismatch

pytestmark = pytest.mark.gpu


def block_of(n, iters=2):
    """n particles of a dam break large enough to hold them."""
    side = int(np.ceil(n ** (1.0 / 3.0)))
    sc = scenes.dam_break(side, (int(1.3 * side) + 4, side + 4, side + 4), stable=True, iterations=iters)
    sc.pos, sc.vel = sc.pos[:n].copy(), sc.vel[:n].copy()
    sc.para.nParticles = n
    return sc


@pytest.mark.parametrize("n,lanes,cell", [(9472, 2, 0.5), (9473, 2, 0.5), (9472, 1, 1.0), (9473, 1, 1.0),
                                          (9473, 4, 0.5), (9473, 8, 0.5), (45056, 2, 0.5), (45057, 2, 1.0),
                                          (16384, 2, 1.0), (16385, 2, 1.0), (40960, 2, 0.5), (40961, 2, 0.5),
                                          (56833, 4, 0.5), (28417, 8, 0.5), (113664, 2, 0.5), (113665, 2, 0.5),
                                          (113665, 1, 1.0), (113664, 1, 0.5)])
def test_variant_boundaries_bitexact(n, lanes, cell):
    sc = block_of(n)
    s, orc = make_pair(sc, pair_lanes=lanes, cell_scale=cell,
                       grid_dims=autotune.dims_for_scale(sc.ext_overrides["grid_dims"], cell))
    s.step(1)
    orc.substep()
    assert_substep_bitexact(s, orc)
    s.close()
    orc.close()


@pytest.mark.parametrize("n,lanes,cell", [(9472, 2, 0.5), (9473, 2, 0.5), (9472, 1, 1.0), (9473, 1, 1.0),
                                          (9473, 4, 0.5), (9473, 8, 0.5), (16385, 2, 1.0), (40961, 2, 0.5),
                                          (56833, 4, 0.5), (28417, 8, 0.5), (113664, 2, 0.5), (113665, 2, 0.5),
                                          (113665, 1, 1.0), (113664, 1, 0.5)])
def test_variant_boundaries_of_released_kernels_bitexact(n, lanes, cell):
    """The same sizes without debug fields, as users run them: other instances of the
    kernels, launched programmatically dependent on one another, the graph of one substep
    replayed after itself."""
    sc = block_of(n)
    s, orc = make_pair(sc, debug=0, pair_lanes=lanes, cell_scale=cell,
                       grid_dims=autotune.dims_for_scale(sc.ext_overrides["grid_dims"], cell))
    s.step(3)
    orc.substep(3)
    assert s.stats()["error_bits"] == 0
    assert np.array_equal(s.fetch("perm"), orc.get("perm"))
    for f in ("x", "v", "curl"):
        assert mismatch(s.fetch(f)[:, :3], orc.get(f))[0] == 0, f
    s.close()
    orc.close()


@pytest.mark.parametrize("n", [1200, 46000])
def test_no_corrections_bitexact(n):
    """A substep without corrections keeps the predicted velocities, over several
    substeps (the scan's status words outlive each)."""
    sc = block_of(n, iters=0)
    s, orc = make_pair(sc)
    s.step(3)
    for _ in range(3):
        orc.substep()
    for f in ("x", "v", "curl"):
        assert mismatch(s.fetch(f)[:, :3], orc.get(f))[0] == 0, f
    assert np.array_equal(s.fetch("perm"), orc.get("perm"))
    s.close()
    orc.close()


@pytest.mark.parametrize("tol", [1e-9, 0.02])
@pytest.mark.parametrize("max_it", [1, 2, 3, 5, 6])
@pytest.mark.parametrize("n", [1200, 12000])
def test_adaptive_loop_ends_bitexact(n, max_it, tol):
    """The correction loop, two corrections per body, ended by its cap or by the
    tolerance after even and odd numbers of corrections."""
    sc = block_of(n, iters=1)
    s, orc = make_pair(sc, adaptive=1, density_tol=tol, max_iterations=max_it, debug=0)
    for _ in range(3):
        s.step(1)
        want = orc.substep_adaptive(float(np.float32(tol)), 1, max_it)
        assert s.stats()["last_iterations"] == want
        for f in ("x", "v"):
            assert mismatch(s.fetch(f)[:, :3], orc.get(f))[0] == 0, f
    s.close()
    orc.close()


@pytest.mark.parametrize("exponent", [1.0, 3.0, 3.5])
@pytest.mark.parametrize("n", [1200, 12000])
def test_scorr_exponents_bitexact(n, exponent):
    """Whole exponents are repeated products; 3.5 goes through powf, whose last bit
    is not the host's, so its corrections are compared within 1e-6 of their scale."""
    sc = block_of(n)
    sc.para.n = exponent
    s, orc = make_pair(sc)
    s.step(1)
    orc.substep()
    if exponent == 3.5:
        want = orc.get("dp")
        assert np.abs(s.fetch("dp")[:, :3] - want).max() <= 1e-6 * np.abs(want).max()
    else:
        assert_substep_bitexact(s, orc)


@pytest.mark.parametrize("lanes", [1, 2, 8])
@pytest.mark.parametrize("n", [1200, 12000])
def test_scorr_negative_exponent(n, lanes):
    """A negative exponent makes an entry of weight 0 infinite: none but the list's own
    entries may enter the sums. powf is good for 4 ulp there and 1 here, and the sums
    of up to 63 terms follow: 5e-7 + 63 * 6e-8 < 5e-6 of the terms' magnitudes."""
    sc = block_of(n, iters=1)
    sc.pos += np.random.RandomState(9).uniform(-0.004, 0.004, size=sc.pos.shape).astype(np.float32)
    sc.para.n = -0.25
    s, orc = make_pair(sc, pair_lanes=lanes)
    s.step(1)
    orc.substep()
    want, x, lam = orc.get("dp"), orc.get("xpred").astype(np.float64), orc.get("lambda").astype(np.float64)
    nbr = orc.get("nbr").reshape(n, -1)
    j = np.where(nbr < 0, np.arange(n)[:, None], nbr)
    r = np.linalg.norm(x[:, None] - x[j], axis=2)
    h = float(sc.para.h)
    w = np.maximum(h * h - r * r, 1e-30) ** 3 / (h * h - float(sc.para.deltaq) ** 2) ** 3
    size = np.abs(lam[:, None]) + np.abs(lam[j]) + float(sc.para.k) * w ** -0.25 * s.ext.scorr_scale
    g = 45.0 / (np.pi * h ** 6) * np.maximum(h - r, 0.0) ** 2
    terms = np.where(nbr >= 0, size * g, 0.0).sum(1) / float(sc.para.restRho)
    assert np.isfinite(want).all()
    assert (np.abs(s.fetch("dp")[:, :3] - want).max(1) <= 5e-6 * terms + 1e-7 * np.abs(want).max(1) + 1e-12).all()
    s.close()
    orc.close()


@pytest.mark.parametrize("cell", [1.0 / 3.0, 0.5, 0.7, 1.0, 1.5])
@pytest.mark.parametrize("n", [2100, 46000])
def test_search_around_the_grid_bitexact(cell, n):
    """Particles in and around a grid smaller than their box, on every side and far
    away, with clumps beyond the neighbour cap."""
    rng = np.random.RandomState(5)
    sc = scenes.dam_break(4, (60, 60, 60), stable=True, iterations=1)
    side = 0.05 * n ** (1.0 / 3.0)
    pos = rng.uniform(0.0, side + 0.8, size=(n, 3))
    pos[: n // 7] = 0.5 * side + rng.uniform(0.0, 0.25, size=(n // 7, 3))
    pos[-3:] = [[5.9, 0.3, 0.3], [0.3, 5.9, 0.3], [0.3, 0.3, 5.9]]
    sc.pos, sc.vel = pos.astype(np.float32), np.zeros((n, 3), np.float32)
    sc.para.nParticles = n
    sc.grid_space = [0.25, 0.2, 0.15, 6.0, 6.0, 6.0]
    dims = [int(np.ceil((side + 0.3) / (0.1 * cell)))] * 3
    s, orc = make_pair(sc, cell_scale=cell, grid_dims=dims)
    s.step(1)
    orc.substep()
    cnt = orc.get("ncnt")
    assert (cnt == 63).any() and (orc.get("cell") < 0).any()
    assert_substep_bitexact(s, orc)
    s.close()
    orc.close()


@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
@pytest.mark.parametrize("cap", [1, 5, 64, 127])
@pytest.mark.parametrize("n,cell", [(2100, 0.5), (12000, 1.0), (46000, 0.5), (46000, 1.0)])
def test_neighbour_caps_bitexact(n, cell, cap, lanes):
    """Lists cut at caps from 1 to 127, in a cloud with about 150 particles within h: the
    padding goes past the cap into rows of its own, and the eight-thread kernels size
    their shared memory by it (more than 48 KB from 81 entries on)."""
    rng = np.random.RandomState(cap)
    side = (4.19e-3 * n / 150.0) ** (1.0 / 3.0)
    sc = scenes.dam_break(4, (24, 24, 24), stable=True, iterations=2)
    sc.pos = rng.uniform(0.2, 0.2 + side, size=(n, 3)).astype(np.float32)
    sc.vel = np.zeros((n, 3), np.float32)
    sc.para.nParticles = n
    s, orc = make_pair(sc, pair_lanes=lanes, cell_scale=cell, max_neighbors=cap,
                       grid_dims=autotune.dims_for_scale(sc.ext_overrides["grid_dims"], cell))
    s.step(1)
    orc.substep()
    assert (orc.get("ncnt") == cap).any()
    assert_substep_bitexact(s, orc)
    s.close()
    orc.close()


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("persistent", [0, 1])
@pytest.mark.parametrize("cell", [0.4, 0.5, 1.0])
def test_search_far_from_the_grids_corner_bitexact(cell, persistent, axis):
    """A row of particles around the origin of a grid whose corner lies 1,000,000 h away
    along the row, where keys are rounded by up to 4e-2 h. persistent = 1 takes the
    search with one thread per particle."""
    n, far = 1500, 100000.0
    rng = np.random.RandomState(11)
    sc = scenes.dam_break(4, (1, 1, 1), stable=True, iterations=1)
    pos = rng.uniform(0.049, 0.051, size=(n, 3))
    pos[:, axis] = rng.uniform(-4.0, 4.0, size=n)
    sc.pos, sc.vel = pos.astype(np.float32), np.zeros((n, 3), np.float32)
    sc.para.nParticles = n
    sc.grid_space[axis], sc.boundary[axis], sc.boundary[3 + axis] = -far, -4.2, 4.2
    dims = [int(np.ceil(1 / cell))] * 3
    dims[axis] = int((far + 4.5) / (0.1 * cell))
    s, orc = make_pair(sc, cell_scale=cell, grid_dims=dims, persistent=persistent)
    s.step(1)
    orc.substep()
    assert_substep_bitexact(s, orc)
    s.close()
    orc.close()


@pytest.mark.parametrize("n,lanes,block,persistent,record", [(75776, 2, 256, 0, 0), (75777, 2, 256, 0, 1),
                                                             (75777, 1, 128, 0, 0), (80001, 8, 256, 0, 1),
                                                             (80001, 4, 64, 1, 0), (160000, 2, 256, 0, 0)])
def test_warm_pass_in_two_launches_bitexact(n, lanes, block, persistent, record):
    """lambda0, the total lambda and the state of the first pass with packed rows
    between its launches against the path with FP32 features, bit for bit."""
    sc = block_of(n)
    rng = np.random.RandomState(n)
    feat = torch.from_numpy(rng.normal(size=(2048, 12)).astype(np.float32)).cuda()
    target = torch.from_numpy(rng.normal(size=2048).astype(np.float32)).cuda()
    tr, _ = learned.train(feat, target, epochs=1, batch=1024, lr=2e-3)
    _, b32, w16 = tr.params()
    tr.close()
    runs = []
    for unfused in (0, 1):
        s = Solver(sc.para, sc.grid_space, sc.boundary,
                   sc.ext(warm_start=1, warm_unfused=unfused, pair_lanes=lanes, block_size=block,
                          persistent=persistent, warm_clamp=0.0, record_features=record))
        learned.install(s, w16, b32)
        s.upload(sc.pos, sc.vel)
        s.step(3)
        assert s.stats()["error_bits"] == 0
        runs.append({k: s.fetch(k) for k in ("lambda0", "lambda_total", "x", "v", "curl")})
        s.close()
    for k in runs[0]:
        assert np.array_equal(runs[0][k].view(np.uint32), runs[1][k].view(np.uint32)), k
    assert np.count_nonzero(runs[0]["lambda0"]) > n // 2
