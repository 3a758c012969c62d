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
