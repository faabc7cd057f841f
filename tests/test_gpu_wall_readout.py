"""The wall-model readout's counts of one list build (cells left out for a
link to a vane, cells without a normal) against the host builder's, whatever
the list's memory held before: a first build, one that needs more room, one
that fits, and the same on a refined level."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fc(built_lib):
    import foil_cfd_gb300 as fc
    return fc


DIMS = (96, 48, 8)


def field(height, vanes, slots):
    """A slab of `height` rows; vanes on it (in the active field only) and
    one-cell slots between equal blocks, whose cells have no normal."""
    clean = np.zeros(DIMS[::-1], np.uint8)
    clean[:, :height, :] = 1
    for k in range(slots):
        x = 52 + 12 * k
        clean[:, 30:37, x:x + 3] = clean[:, 30:37, x + 4:x + 7] = 1
    active = clean.copy()
    for k in range(vanes):
        active[:, height:height + 4, 10 + 6 * k:12 + 6 * k] = 1
    return active.ravel(), clean.ravel()


def counts(s):
    r = s.wall_model_readout()
    return r.from_fine, r.excluded_vg, r.degenerate


def expected(fc, dims, active, clean, sample):
    st = fc.build_wall_list(dims, active, clean, sample)["stats"]
    assert st["listed"] > 0 and st["excluded_vg"] > 0 and st["degenerate"] > 0
    return st["excluded_vg"], st["degenerate"]


def test_counts_survive_first_growing_and_fitting_builds(fc):
    small, clean = field(8, 2, 1)
    s = fc.LBMSolver()
    s.init(DIMS, fc.scaling_direct(0.55, 0.05), small, les_cs=0.1)
    s.set_startup_ramp_enabled(False)
    assert s.set_surface_reference(clean) == 0
    s.set_wall_model_enabled(True)                        # first build
    assert counts(s) == (0, *expected(fc, DIMS, small, clean, 2))
    large, clean2 = field(8, 4, 3)
    n0, n1 = (fc.build_wall_list(DIMS, a, c, 2)["stats"]["listed"] for a, c in ((small, clean), (large, clean2)))
    assert n1 > n0
    s.apply_edited_flags(large)
    assert s.set_surface_reference(clean2) == 0           # a longer list
    assert counts(s) == (0, *expected(fc, DIMS, large, clean2, 2))
    assert s.set_flags(small) == 0
    assert s.set_surface_reference(clean) == 0            # fits the block of the longer one
    assert counts(s) == (0, *expected(fc, DIMS, small, clean, 2))
    s.set_wall_model_enabled(False)                       # gives the block back
    s.set_wall_model_enabled(True)
    assert counts(s) == (0, *expected(fc, DIMS, small, clean, 2))


def test_counts_of_a_refined_level(fc):
    active, clean = field(8, 3, 2)
    s = fc.LBMSolver()
    s.init(DIMS, fc.scaling_direct(0.55, 0.05), active, les_cs=0.1)
    s.set_startup_ramp_enabled(False)
    s.set_wall_model_enabled(True)
    x0, x1, y0, y1 = 4, 92, 4, 44
    fd = (2 * (x1 - x0), 2 * (y1 - y0), 2 * DIMS[2])

    def fine(f):
        g = np.repeat(np.repeat(np.repeat(f.reshape(DIMS[::-1]), 2, 0), 2, 1), 2, 2)
        g = g[:, 2 * y0:2 * y1, 2 * x0:2 * x1].copy()
        g[:, :2, :] = g[:, -2:, :] = 8
        g[:, :, :2] = g[:, :, -2:] = 8
        # Slots of two fine cells have normals; one of a single cell has none.
        g[:, 60:70, 20:24] = g[:, 60:70, 25:29] = 1
        return g.ravel()

    fa, fcl = fine(active), fine(clean)
    s.init_refinement(fc.Box(x0, y0, x1, y1), 2, fa)      # first build, no reference yet
    st = fc.build_wall_list(fd, fa, None, 3)["stats"]
    assert st["degenerate"] > 0 and counts(s) == (1, 0, st["degenerate"])
    assert s.set_refined_surface_reference(fcl) == 0
    assert counts(s) == (1, *expected(fc, fd, fa, fcl, 3))
