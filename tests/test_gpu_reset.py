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


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("dims", [(5, 5, 1), (7, 5, 3), (13, 7, 2), (33, 17, 8), (40, 31, 9)])
def test_edits_of_odd_cell_counts(fc, oracle_mod, dims, device):
    """Cell counts with every remainder of four, edits in the first and the last
    cell, from host and device memory (also at an odd address), back and forth."""
    torch = pytest.importorskip("torch")
    n = int(np.prod(dims))
    rng = np.random.default_rng(n)
    a = (rng.random(n) < 0.1).astype(np.uint8)
    b = (rng.random(n) < 0.1).astype(np.uint8)
    b[0], b[-1] = 1 - a[0], 1 - a[-1]
    s = fc.LBMSolver()
    s.init(dims, fc.scaling_direct(0.55, 0.05), a, les_cs=0.1)
    f = oracle_mod.equilibrium(np.ones(n), np.full(n, 0.03), np.zeros(n), np.zeros(n))
    s.import_f32(f)
    s.mirror_buffers()
    state, old = f.reshape(19, n).astype(np.float32).copy(), a
    for new in (b, b, a):
        arg = new
        if device:
            t = torch.zeros(n + 1, dtype=torch.uint8, device="cuda")
            t[1:] = torch.from_numpy(new)
            arg = t[1:]
        assert s.apply_edited_flags(arg) == int(((old == 1) != (new == 1)).sum())
        mask = np.where((new == 1) & (old != 1), 1, np.where((old == 1) & (new != 1), 2, 0))
        oracle_mod.apply_flag_edits(dims, state, state.copy(), new, mask)
        assert np.array_equal(s.export_f32().reshape(19, n), state)
        old = new
