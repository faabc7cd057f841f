"""The collide's tile codes and staged tiles: lattices whose rows, planes and
cell counts do not fit 32-cell warps, 128-cell tiles or 16-byte runs, with
walls, vanes, inlet and outlet. FP32 against the oracle on every cell a step
writes, bit for bit; FP16 staged against the one-cell kernel, whose cells run
the same body on the same values."""
import numpy as np
import pytest

from conftest import written_mask

pytestmark = pytest.mark.gpu

# Below the size from which codes are used: smaller than a warp, rows of a
# block, of one more and of one less. Above it (FP32 2.5, FP16 4 million
# cells): the same, and cell counts that are and are not a multiple of 8.
DIMS = [(5, 4, 3), (128, 9, 8), (129, 8, 6), (41, 23, 17), (128, 160, 200), (129, 160, 200), (333, 121, 101),
        (640, 80, 81)]


@pytest.fixture(scope="module")
def fc(built_lib):
    import foil_cfd_gb300 as fc
    return fc


def channel(dims, periodic):
    nx, ny, nz = dims
    f = np.zeros((nz, ny, nx), np.uint8)
    if not periodic:
        f[:, 0, :] = 5
        f[:, -1, :] = 4
        f[:, :, 0] = 2
        f[:, 1:-1, -1] = 3
    f[nz // 2, ny // 2, nx // 3 : nx // 3 + 2] = 1
    if nx > 64:
        f[:, ny // 2 : ny // 2 + 2, 60:64] = 1
    return f.ravel()


def start(oracle_mod, dims):
    n = int(np.prod(dims))
    rng = np.random.default_rng(n)
    return oracle_mod.equilibrium(1 + 0.01 * rng.standard_normal(n), 0.05 + 0.01 * rng.standard_normal(n),
                                  0.01 * rng.standard_normal(n), 0.01 * rng.standard_normal(n))


def solver(fc, dims, flags, f0, storage, kernel="auto"):
    s = fc.LBMSolver()
    s.init(dims, fc.scaling_direct(0.55, 0.05), flags, storage=storage, les_cs=0.1, kernel=kernel)
    s.set_startup_ramp_enabled(False)
    s.reset()
    s.import_f32(f0)
    return s


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("dims", DIMS)
def test_fp32_vs_oracle(fc, oracle_mod, dims, periodic):
    flags, f0 = channel(dims, periodic), start(oracle_mod, dims)
    s = solver(fc, dims, flags, f0, "fp32")
    o = oracle_mod.OracleSolver(dims, flags, np.float32(0.55), np.float32(0.05), cs=0.1)
    o.set_state(f0)
    assert s.step_n(5) == 0
    o.step_n(5)
    m = written_mask(flags)
    assert np.array_equal(s.export_f32().reshape(19, -1)[:, m], o.f.reshape(19, -1)[:, m])


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("dims", DIMS)
def test_fp16_staged_vs_one_cell(fc, oracle_mod, dims, periodic):
    flags, f0 = channel(dims, periodic), start(oracle_mod, dims)
    a, b = (solver(fc, dims, flags, f0, "fp16", k) for k in ("auto", "cell"))
    assert a.step_n(5) == 0 and b.step_n(5) == 0
    assert np.array_equal(a.export_f32(), b.export_f32())
    for x, y in zip(a.download_macro(), b.download_macro()):
        assert np.array_equal(x, y)
