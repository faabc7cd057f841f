"""A non-finite rest population at one cell through the refinement coupling:
seeding, fill and restriction multiply every population by its lattice
velocity, and 0 times NaN or infinity is NaN, so each value formed from such a
cell is NaN in all 19 populations (lbm_refine.cu:70-97, 226-330)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS, BOX = (32, 24, 6), (6, 26, 5, 19)   # box: x0, x1, y0, y1
BAD = [np.nan, np.inf]


@pytest.fixture(scope="module")
def fc(built_lib):
    import foil_cfd_gb300 as fc
    return fc


def fields(factor):
    nx, ny, nz = DIMS
    x0, x1, y0, y1 = BOX
    flags = np.zeros((nz, ny, nx), np.uint8)
    flags[:, 0, :], flags[:, -1, :], flags[:, :, 0], flags[:, 1:-1, -1] = 5, 4, 2, 3
    fine = np.zeros((nz * factor, (y1 - y0) * factor, (x1 - x0) * factor), np.uint8)
    fine[:, :2, :] = fine[:, -2:, :] = 8
    fine[:, :, :2] = fine[:, :, -2:] = 8
    return flags, fine


def state(oracle_mod, dims):
    n = int(np.prod(dims))
    rng = np.random.default_rng(n)
    return oracle_mod.equilibrium(1 + 0.01 * rng.standard_normal(n), 0.05 + 0.01 * rng.standard_normal(n),
                                  0.01 * rng.standard_normal(n), 0.01 * rng.standard_normal(n)).reshape(
                                      19, *dims[::-1]).astype(np.float32)


def solver(fc, storage, f, flags, fine, factor):
    s = fc.LBMSolver()
    s.init(DIMS, fc.scaling_direct(0.55, 0.05), flags.ravel(), storage=storage, les_cs=0.1)
    s.set_startup_ramp_enabled(False)
    s.reset()
    s.import_f32(f.ravel())
    s.init_refinement(fc.Box(BOX[0], BOX[2], BOX[1], BOX[3]), factor, fine.ravel())
    return s


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("storage", ["fp32", "fp16"])
@pytest.mark.parametrize("factor", [2, 3])
def test_seeding_spreads_a_bad_rest_population(fc, oracle_mod, storage, factor, bad):
    flags, fine = fields(factor)
    f = state(oracle_mod, DIMS)
    X, Y, Z = 12, 9, 0                                    # plane 0: its corners wrap
    f[0, Z, Y, X] = bad
    s = solver(fc, storage, f, flags, fine, factor)
    got = np.isnan(s.export_fine_f32().reshape(19, *fine.shape))

    def reads(i, c, lo, n=0):                             # fine indices with cell c among their two along an axis
        g = np.floor(lo + (np.arange(i) + 0.5) / factor - 0.5).astype(int)
        a, b = (g, g + 1) if n == 0 else (g % n, (g + 1) % n)
        return (a == c) | (b == c)

    want = (reads(fine.shape[0], Z, 0, DIMS[2])[:, None, None] & reads(fine.shape[1], Y, BOX[2])[None, :, None]
            & reads(fine.shape[2], X, BOX[0])[None, None, :])
    # Where the corner's weight is 0 (odd factors) 0 times it is NaN as well.
    assert want.any() and np.array_equal(got, np.broadcast_to(want, got.shape))


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("storage", ["fp32", "fp16"])
@pytest.mark.parametrize("factor", [2, 3])
def test_restriction_spreads_a_bad_rest_population(fc, oracle_mod, storage, factor, bad):
    """The parent of a fine cell and that parent's 18 neighbours, whose filter
    reads its record; in the velocity field too."""
    flags, fine = fields(factor)
    s = solver(fc, storage, state(oracle_mod, DIMS), flags, fine, factor)
    ff = s.export_fine_f32().reshape(19, *fine.shape)
    X, Y, Z = 16, 12, 3
    ff[0, factor * Z, factor * (Y - BOX[2]), factor * (X - BOX[0])] = bad
    s.import_fine_f32(ff.ravel())
    assert s.step_n(1) == 0
    f = s.export_f32().reshape(19, *DIMS[::-1])
    u = s.download_macro()[1].reshape(DIMS[::-1])
    from oracle.oracle import CX, CY, CZ
    for q in range(19):
        z, y, x = Z + CZ[q], Y + CY[q], X + CX[q]
        assert np.isnan(f[:, z, y, x]).all() and np.isnan(u[z, y, x]), q


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
def test_fill_spreads_a_bad_rest_population(fc, oracle_mod, storage):
    """A coarse cell under the patch's edge: the filled shell cells are NaN in
    the moving populations, which the fluid cells beside them pull."""
    flags, fine = fields(2)
    s = solver(fc, storage, state(oracle_mod, DIMS), flags, fine, 2)
    f = s.export_f32().reshape(19, *DIMS[::-1])
    f[0, 3, 12, BOX[0]] = np.nan
    s.import_f32(f.ravel())
    assert s.step_n(1) == 0
    got = s.export_fine_f32().reshape(19, *fine.shape)
    assert np.isnan(got[1:, fine == 0]).any()
