"""The tables a level derives from its flags (bit planes, kind bytes, link
classes, lists) on rows shorter than, equal to and longer than a word of 32
cells, aligned and not, spans of one cell up: the device lists against the host
builders and plain numpy, and the step of a lattice of random walls against
the oracle. All exact."""
import numpy as np
import pytest

from conftest import written_mask

pytestmark = pytest.mark.gpu

DIMS = [(3, 3, 1), (5, 4, 3), (31, 7, 3), (32, 6, 4), (33, 9, 2), (64, 5, 5), (100, 37, 6), (616, 20, 4)]
C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0), (1, 0, 1),
     (-1, 0, -1), (0, 1, 1), (0, -1, -1), (1, -1, 0), (-1, 1, 0), (1, 0, -1), (-1, 0, 1), (0, 1, -1), (0, -1, 1)]


@pytest.fixture(scope="module")
def fc(built_lib):
    import foil_cfd_gb300 as fc
    return fc


@pytest.fixture(scope="module")
def geo(fc):
    from foil_cfd_gb300 import geometry
    return geo_check(geometry)


def geo_check(geometry):
    import torch
    assert torch.cuda.is_available()
    return geometry


def walls(dims, seed, values=(0, 1)):
    """Random flags: blocks of solid, single cells, and the other values sprinkled in."""
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    f = np.zeros((nz, ny, nx), np.uint8)
    f[rng.random(f.shape) < 0.06] = 1
    if nx > 8 and ny > 6:
        f[:, ny // 3 : ny // 3 + 2, nx // 4 : nx // 2] = 1
    for v in values[2:]:
        f[rng.random(f.shape) < 0.04] = v
    return f


def dev(f):
    import torch
    return torch.from_numpy(np.ascontiguousarray(f).ravel()).cuda()


@pytest.mark.parametrize("dims", DIMS)
def test_force_links_vs_numpy(geo, dims):
    f = walls(dims, 1, (0, 1, 2, 3, 8))
    mask = np.zeros(f.shape, np.uint32)
    for q in range(1, 19):
        x, y, z = C[q]
        mask |= (np.roll(f, (-z, -y, -x), (0, 1, 2)) == 1).astype(np.uint32) << np.uint32(q)
    mask = np.where(f == 0, mask, 0).ravel()
    cells, masks = geo.force_links(dims, dev(f))
    want = np.flatnonzero(mask)
    assert np.array_equal(cells.cpu().numpy().view(np.uint32), want.astype(np.uint32))
    assert np.array_equal(masks.cpu().numpy().view(np.uint32), mask[want])


# The host builder wraps z once, so its normals (z +- 2) need two planes.
@pytest.mark.parametrize("vanes", [False, True])
@pytest.mark.parametrize("dims", [d for d in DIMS if d[2] > 1])
def test_wall_list_vs_host(fc, geo, dims, vanes):
    from foil_cfd_gb300.solver import build_wall_list
    active = walls(dims, 2)
    clean = active.copy()
    if vanes:
        clean[np.random.default_rng(3).random(clean.shape) < 0.03] = 0
    host = build_wall_list(dims, active.ravel(), clean.ravel(), 2)
    got = geo.wall_list(dims, dev(active), dev(clean) if vanes else None, 2)
    assert got["stats"] == host["stats"]
    for k in ("cell", "sample", "mask"):
        assert np.array_equal(got[k].cpu().numpy().view(np.uint32), host[k].astype(np.uint32)), k
    for k in ("nx", "ny", "nz", "ys"):
        assert np.array_equal(got[k].cpu().numpy(), host[k]), k


@pytest.mark.parametrize("dims", DIMS)
def test_patch_box_vs_host(fc, geo, dims):
    from foil_cfd_gb300.solver import derive_patch_box
    f = np.zeros((dims[2], dims[1], dims[0]), np.uint8)
    f[-1, 1 : dims[1] // 2 + 1, dims[0] // 3 : dims[0] - 1] = 1
    assert geo.derive_patch_box(dims, dev(f), 1, 2, 1, 2, 1) == derive_patch_box(dims, f.ravel(), 1, 2, 1, 2, 1)


@pytest.mark.parametrize("dims", DIMS)
def test_step_among_random_walls_vs_oracle(fc, oracle_mod, dims):
    f = walls(dims, 4, (0, 1, 4, 5, 6, 7)).ravel()
    n = f.size
    rng = np.random.default_rng(5)
    f0 = oracle_mod.equilibrium(1 + 0.01 * rng.standard_normal(n), 0.05 + 0.01 * rng.standard_normal(n),
                                0.01 * rng.standard_normal(n), 0.01 * rng.standard_normal(n))
    s = fc.LBMSolver()
    s.init(dims, fc.scaling_direct(0.6, 0.05), f, les_cs=0.1)
    s.set_startup_ramp_enabled(False)
    s.reset()
    s.import_f32(f0)
    s.mirror_buffers()
    o = oracle_mod.OracleSolver(dims, f, np.float32(0.6), np.float32(0.05), cs=0.1)
    o.set_state(f0)
    o.g = o.f.copy()
    assert s.step_n(4) == 0
    o.step_n(4)
    m = written_mask(f)
    assert np.array_equal(s.export_f32().reshape(19, -1)[:, m], o.f.reshape(19, -1)[:, m])
