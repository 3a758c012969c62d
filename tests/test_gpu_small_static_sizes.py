"""gpx_cap_solve_small_static at the sizes of its 32-column panels, 32 x 32
update tiles and 8-column back substitution, against numpy's dense solve of the
library's own potential matrix (1e-9 of the largest entry, the bar of the
entry point's other tests)."""
import numpy as np
import pytest

from gpurify_b200 import _lib

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ctx():
    c = _lib.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n,ncond", [(1, 1), (2, 2), (31, 3), (32, 8), (33, 9), (64, 1), (65, 16), (96, 64), (300, 17),
                                     (511, 33), (512, 64)])
def test_sizes_at_block_edges(ctx, n, ncond):
    rng = np.random.default_rng(1000 * n + ncond)
    # separate horizontal squares of uneven sizes, in random order
    cells = rng.permutation(24 * 24)[:n]
    side = rng.uniform(0.2, 0.9, n) * 1e-6
    x, y, z = (cells % 24) * 1e-6, (cells // 24) * 1e-6, rng.integers(0, 3, n) * 0.4e-6
    v = np.stack([x, y, z, x + side, y, z, x + side, y + side, z, x, y + side, z], axis=1)
    cond = np.concatenate([np.arange(ncond) % ncond, rng.integers(0, ncond, max(0, n - ncond))])[:n].astype(np.int32)
    centre = np.stack([x + side / 2, y + side / 2, z], axis=1)
    on = (cond[:, None] == np.arange(ncond)[None, :]).astype(float)
    ref = (on * (side**2)[:, None]).T @ np.linalg.solve(ctx.potential_matrix(v, centre), on)
    dv, dc = torch.from_numpy(v).cuda(), torch.from_numpy(cond).cuda()
    out = torch.full((ncond, ncond), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.cap_solve_small_static(n, dv.data_ptr(), dc.data_ptr(), ncond, out.data_ptr())
    assert np.abs(out.cpu().numpy() - ref).max() <= 1e-9 * np.abs(ref).max()


def _square(x, y, z, s):
    return [x, y, z, x + s, y, z, x + s, y + s, z, x, y + s, z]


def _nearly_touching(n, gap, rng):
    """Pairs of plates a gap of 1 to 7 times `gap` apart."""
    v = []
    for k in range(n // 2):
        x, y, s = (k % 16) * 1.2e-6, (k // 16) * 1.2e-6, rng.uniform(0.3, 1.0) * 1e-6
        v += [_square(x, y, 0.0, s), _square(x, y, gap * (1 + k % 7), s)]
    return np.array(v)


def _stack(n, gap, rng):
    """One stack of n plates, `gap` apart."""
    return np.array([_square(rng.uniform(-1, 1) * 1e-9, 0.0, k * gap, 1e-6 * (1 + 0.1 * (k % 3))) for k in range(n)])


def _uneven(n, decades, rng):
    """Squares of sides over `decades` powers of ten."""
    cells, side = rng.permutation(24 * 24)[:n], 10 ** rng.uniform(-decades, -0.1, n) * 1e-6
    return np.array([_square((q % 24) * 1e-6, (q // 24) * 1e-6, 1e-9 * (k % 3), side[k]) for k, q in enumerate(cells)])


@pytest.mark.parametrize("shape,n,size", [("touching", 300, 1e-8), ("touching", 512, 1e-11), ("stack", 128, 1e-8),
                                          ("stack", 64, 1e-10), ("uneven", 300, 3), ("uneven", 511, 6)])
def test_nearly_touching_and_uneven_panels(ctx, shape, n, size):
    """Systems of a condition number up to 1e6, whose small pivots lie in the
    32 x 32 diagonal blocks of U that are inverted, against numpy's solve (the
    same bar)."""
    rng = np.random.default_rng(n)
    v = {"touching": _nearly_touching, "stack": _stack, "uneven": _uneven}[shape](n, size, rng)
    ncond = 8
    cond = rng.integers(0, ncond, n).astype(np.int32)
    q = v.reshape(n, 4, 3)
    area = np.linalg.norm(np.cross(q[:, 1] - q[:, 0], q[:, 3] - q[:, 0]), axis=1)
    on = (cond[:, None] == np.arange(ncond)[None, :]).astype(float)
    ref = (on * area[:, None]).T @ np.linalg.solve(ctx.potential_matrix(v, q.mean(axis=1)), on)
    dv, dc = torch.from_numpy(v).cuda(), torch.from_numpy(cond).cuda()
    out = torch.full((ncond, ncond), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.cap_solve_small_static(n, dv.data_ptr(), dc.data_ptr(), ncond, out.data_ptr())
    assert np.abs(out.cpu().numpy() - ref).max() <= 1e-9 * np.abs(ref).max()
