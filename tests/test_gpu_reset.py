"""Cold start of the levels: the seeding of a refined level from its parent
against the oracle on every cell that is not solid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fc(built_lib):
    import foil_cfd_gb300 as fc
    return fc


@pytest.mark.parametrize("factor", [2, 3, 4])
@pytest.mark.parametrize("dims,box", [((14, 13, 1), (3, 12, 2, 11)), ((14, 13, 2), (2, 13, 3, 12)), ((45, 20, 5), (4, 41, 3, 16))])
def test_seeding(fc, oracle_mod, dims, box, factor):
    """One and two planes (both neighbours of a plane wrap), rows of less than
    and more than a block, solid corners and targets inside the solid."""
    nx, ny, nz = dims
    x0, x1, y0, y1 = box
    flags = np.zeros((nz, ny, nx), np.uint8)
    flags[:, 0, :], flags[:, -1, :], flags[:, :, 0], flags[:, 1:-1, -1] = 5, 4, 2, 3
    cx, cy = (x0 + x1) // 2, (y0 + y1) // 2
    flags[:, cy - 1:cy + 2, cx - 1:cx + 2] = 1
    fine = np.repeat(np.repeat(np.repeat(flags, factor, 0), factor, 1), factor, 2)[:, y0 * factor:y1 * factor,
                                                                                  x0 * factor:x1 * factor].copy()
    fine[:, :1, :] = fine[:, -1:, :] = 8
    fine[:, :, :1] = fine[:, :, -1:] = 8
    n = nx * ny * nz
    rng = np.random.default_rng(nz)
    f0 = oracle_mod.equilibrium(1 + 0.01 * rng.standard_normal(n), 0.05 + 0.01 * rng.standard_normal(n),
                                0.01 * rng.standard_normal(n), 0.01 * rng.standard_normal(n))
    s = fc.LBMSolver()
    s.init(dims, fc.scaling_direct(0.55, 0.05), flags.ravel(), les_cs=0.1)
    s.set_startup_ramp_enabled(False)
    s.reset()
    s.import_f32(f0)
    s.init_refinement(fc.Box(x0, y0, x1, y1), factor, fine.ravel())
    o = oracle_mod.OracleSolver(dims, flags.ravel(), np.float32(0.55), np.float32(0.05), cs=0.1)
    o.set_state(f0)
    o.enable_refinement([x0, y0, x1, y1], factor, fine.ravel())
    keep = fine.ravel() != 1
    assert np.array_equal(s.export_fine_f32().reshape(19, -1)[:, keep], o.fine["f"].reshape(19, -1)[:, keep])
