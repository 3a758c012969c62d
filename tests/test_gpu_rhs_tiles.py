"""Operator applies at right-hand-side counts around the kernels' column tiles
(multiples of 8 up to 64, chunks beyond) against the oracle's apply: the same
tree and the same compressed operators, FP64 reassociation only (1e-11, the bar
of the operator parity tests)."""
import numpy as np
import pytest

from gpurify_b200 import _lib, layouts

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = _lib.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("order,nrhs", [(2, 8), (3, 20), (4, 9), (4, 16), (4, 64), (5, 17), (5, 33), (5, 40), (5, 56),
                                        (5, 65), (5, 130), (6, 24), (6, 33), (6, 64), (6, 256)])
def test_apply_at_column_tile_edges(ctx, orc, order, nrhs):
    lay = layouts.two_wires(length_nm=6000)
    p = _lib.bridge_panelize(lay.store.arrays(), lay.deck.layer_table(), 1.0, lay.net_of_poly, mesh_max_edge_m=0.3e-6,
                             max_panels=-1)
    sig = np.random.default_rng(order * 1000 + nrhs).standard_normal((len(p["verts"]), nrhs))
    y, rep = ctx.operator_apply(p["verts"], sig, order=order, max_level=4, dense_below=-1)
    assert rep["m2l_pairs"] > 0 and rep["dense"] == 0
    for j in sorted({0, nrhs // 2, 7, 8, 63, 64, nrhs - 1} & set(range(nrhs))):
        yo, _ = orc.fmm_cap_apply(p["verts"], sig[:, j], order, 4)
        assert np.linalg.norm(y[:, j] - yo) / np.linalg.norm(yo) < 1e-11


@pytest.mark.parametrize("order,m2l,far_tc,cols", [(4, 2, 0, 3), (4, 0, 1, 16), (5, 3, 0, 5), (5, 3, 1, 17), (5, 2, 1, 32),
                                                   (5, 0, 0, 33), (6, 3, 0, 12), (6, 0, 0, 64)])
def test_mixed_apply_at_row_padding_edges(ctx, order, m2l, far_tc, cols):
    """The FP32 far field pads the right-hand sides to 16, 32 or a multiple of
    64 rows per box and groups 4 or 2 boxes per tensor-core item: a column's
    result does not depend on how many columns are applied with it (the kernels
    sum every output in the same order), so the columns of a 130-column apply
    (three chunks of 64) agree bit for bit."""
    lay = layouts.two_wires(length_nm=6000)
    p = _lib.bridge_panelize(lay.store.arrays(), lay.deck.layer_table(), 1.0, lay.net_of_poly, mesh_max_edge_m=0.3e-6,
                             max_panels=-1)
    sig = np.random.default_rng(order + cols).standard_normal((len(p["verts"]), 130))
    kw = dict(order=order, max_level=4, dense_below=-1, precision=_lib.PREC_MIXED, mixed_m2l=m2l, mixed_far_tc=far_tc,
              far_quad=1)
    wide, rep = ctx.operator_apply(p["verts"], sig, **kw)
    assert rep["m2l_pairs"] > 0 and rep["dense"] == 0
    few, _ = ctx.operator_apply(p["verts"], sig[:, :cols], **kw)
    assert np.isfinite(few).all() and np.array_equal(few, wide[:, :cols])


@pytest.mark.parametrize("nets", [1, 2, 5])
@pytest.mark.parametrize("panels_um", [1.2, 0.3])
def test_device_loop_matches_host_loop_at_reduction_sizes(ctx, nets, panels_um):
    """Column reductions below and above the size where the last block adds the
    partials itself, and Givens steps with their loop control: the device-side
    loop and the host-driven one run the same sums (bit-identical matrices, same
    iterations), for column counts whose rows do not divide the block."""
    lay = layouts.routing_window(nets, 8.0, seed=5, len_um=(0.5, 4.0))
    p = _lib.bridge_panelize(lay.store.arrays(), lay.deck.layer_table(), 1.0, lay.net_of_poly,
                             mesh_max_edge_m=panels_um * 1e-6, max_panels=-1)
    nc = len(p["nets"]) + 1
    kw = dict(order=4, max_level=3, dense_below=300, precond=1)
    a, ra = ctx.cap_solve(p["verts"], p["cond"], nc, **kw)
    b, rb = ctx.cap_solve(p["verts"], p["cond"], nc, no_graphs=1, **kw)
    assert np.array_equal(a, b) and ra["iterations"] == rb["iterations"] > 1


@pytest.mark.parametrize("near", [0, 2, 3])
@pytest.mark.parametrize("cols", [4, 16, 20, 32, 36, 64])
def test_mixed_near_apply_at_column_tile_edges(ctx, near, cols):
    """The tensor-core near apply copies 16, 32 or 64 columns of X per item: a
    column's sums do not depend on the tile it is in, so the columns of a
    132-column apply (tiles of 64 and a remainder) agree bit for bit."""
    lay = layouts.two_wires(length_nm=6000)
    p = _lib.bridge_panelize(lay.store.arrays(), lay.deck.layer_table(), 1.0, lay.net_of_poly, mesh_max_edge_m=0.3e-6,
                             max_panels=-1)
    sig = np.random.default_rng(10 * near + cols).standard_normal((len(p["verts"]), 132))
    kw = dict(order=4, max_level=3, dense_below=-1, precision=_lib.PREC_MIXED, mixed_m2l=2, far_quad=1, mixed_near=near)
    wide, _ = ctx.operator_apply(p["verts"], sig, **kw)
    few, _ = ctx.operator_apply(p["verts"], np.ascontiguousarray(sig[:, :cols]), **kw)
    assert np.isfinite(few).all() and np.array_equal(few, wide[:, :cols])


@pytest.mark.parametrize("n", [255, 512, 513, 770])
def test_capacitance_sums_over_row_slices(ctx, orc, n):
    """The capacitance sums run over slices of 256 rows or more: one slice up to
    511 panels, then two and three, the last one ragged, with a conductor whose
    panels all lie in one slice, against the oracle's dense solve (1e-9, the bar
    of the parity tests at this solver tolerance)."""
    lay = layouts.two_wires(length_nm=6000)
    p = _lib.bridge_panelize(lay.store.arrays(), lay.deck.layer_table(), 1.0, lay.net_of_poly, mesh_max_edge_m=0.15e-6,
                             max_panels=-1)
    verts = np.ascontiguousarray(p["verts"][:n])
    assert len(verts) == n
    cond = (np.arange(n) % 2).astype(np.int32)
    cond[-5:] = 2
    C, rep = ctx.cap_solve(verts, cond, 3, tol=1e-12, dense_below=2**31 - 1)  # every pair near: the oracle's matrix
    assert rep["dense"] == 1
    ref = orc.cap_dense(verts, cond, 3)
    assert np.abs(C - ref).max() / np.abs(ref).max() < 1e-9


@pytest.mark.parametrize("tol,above", [(1e-7, False), (1e-8, True)])
def test_back_substitution_of_a_long_cycle(ctx, tol, above):
    """A restart may be longer than the 1,024 columns of H whose solution the
    back substitution keeps in shared memory; longer ones are solved in global
    memory.  Nearly touching plates take some 980 and 1,080 steps in one cycle;
    the residual is formed from the solution, so that the cycle converges only
    with the right one."""
    k = np.arange(1300)
    x, y, gap = (k % 37) * 1.2e-6, (k // 37) * 1.2e-6, 1e-6 * 10 ** np.linspace(-4.2, -0.7, 1300)
    verts = np.concatenate([np.stack([x, y, z, x + 1e-6, y, z, x + 1e-6, y + 1e-6, z, x, y + 1e-6, z], axis=1)
                            for z in (0 * gap, gap)])
    cond = np.random.default_rng(0).integers(0, 2, 2600).astype(np.int32)
    _, rep = ctx.cap_solve(verts, cond, 2, tol=tol, restart=1400, max_restarts=1, max_level=2, dense_below=-1)
    assert rep["converged"] == 1 and rep["max_rel_residual"] <= tol and rep["restart_used"] == 1400
    assert (rep["iterations"] > 1024) == above


def _squares(n, seed):
    """n separate horizontal squares, one per micron of a 3-D grid, in random order."""
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** (1 / 3)))
    cell = rng.permutation(side**3)[:n]
    x, y, z = (1e-6 * (cell // d % side) for d in (1, side, side * side))
    s = rng.uniform(0.05, 0.35, n) * 1e-6
    return np.stack([x, y, z, x + s, y, z, x + s, y + s, z, x, y + s, z], axis=1)


# work items of the near assembly: below 256 they are split over 64 blocks of
# their sources, above 16,384 not at all
@pytest.mark.parametrize("n,depth", [(1, 1), (65, 1), (4097, 1), (2500, 3), (20000, 6)])
def test_near_assembly_at_item_splits(ctx, orc, n, depth):
    v = _squares(n, n)
    sig = np.random.default_rng(n).standard_normal((n, 1))
    far = dict(order=2, max_level=depth, dense_below=-1) if depth > 1 else dict(dense_below=2**31 - 1)
    y, rep = ctx.operator_apply(v, sig, **far)
    if depth > 1:
        yo, _ = orc.fmm_cap_apply(v, sig[:, 0], 2, depth)
    else:  # the library's own kernel for single potentials: the oracle's form of the integral cancels at far pairs
        yo = ctx.potential_matrix(v, v.reshape(n, 4, 3).mean(axis=1)) @ sig[:, 0]
    assert rep["dense"] == (depth == 1)
    assert np.linalg.norm(y[:, 0] - yo) / np.linalg.norm(yo) < 1e-11


@pytest.mark.parametrize("n,depth", [(64, 1), (65, 1), (300, 1), (2500, 3), (18000, 6)])
def test_near_derivative_at_item_splits(ctx, n, depth):
    """Capacitance scales with length: along the velocity field x (panels that
    grow) dC = C, and along a common translation dC = 0.  With every pair
    exact that holds to the solver's tolerance of 1e-10; with a far field, whose
    boxes do not move, to its truncation, about 1e-3 at order 5 of panels a
    leaf's size (a block of sources left out is an error of its share of C)."""
    v = _squares(n, n)
    cond = np.where(v[:, 0] > np.median(v[:, 0]), 1, 0).astype(np.int32)
    vel = np.stack([v * 1e6, np.tile([1.0, -2.0, 0.5], (n, 4))])  # per um; translation
    far = dict(order=5, max_level=depth, dense_below=-1, far_quad=1) if depth > 1 else dict(dense_below=2**31 - 1)
    C, dC, rep = ctx.cap_sensitivity(v, cond, 2, vel, tol=1e-10, **far)
    assert rep["dense"] == (depth == 1) and rep["converged"] == 1
    bar = 5e-3 if depth > 1 else 1e-8
    assert np.abs(dC[0] * 1e-6 - C).max() < bar * np.abs(C).max()
    assert np.abs(dC[1] * 1e-6).max() < bar * np.abs(C).max()


@pytest.mark.parametrize("order,m2l", [(4, 1), (4, 2), (5, 1), (5, 2), (5, 3), (6, 1), (6, 3)])
@pytest.mark.parametrize("cols", [4, 16, 20, 32])
def test_mixed_apply_of_few_columns_close_to_fp64(ctx, order, m2l, cols):
    """The FP32 operator at 16 and 32 rows per box, column by column against
    FP64, at the bars of the 64-column tests: 1e-3 with TF32 products, 2e-3 in
    the shared basis, 5e-5 with the FP32 near apply and the factored M2L."""
    lay = layouts.two_wires(length_nm=6000)
    p = _lib.bridge_panelize(lay.store.arrays(), lay.deck.layer_table(), 1.0, lay.net_of_poly, mesh_max_edge_m=0.3e-6,
                             max_panels=-1)
    sig = np.random.default_rng(order + cols).standard_normal((len(p["verts"]), cols))
    kw = dict(order=order, max_level=4, dense_below=-1)
    ref, rep = ctx.operator_apply(p["verts"], sig, **kw)
    y, _ = ctx.operator_apply(p["verts"], sig, precision=_lib.PREC_MIXED, mixed_m2l=m2l, mixed_near=1 if m2l == 1 else 0,
                              **kw)
    assert rep["m2l_pairs"] > 0
    err = np.linalg.norm(y - ref, axis=0) / np.linalg.norm(ref, axis=0)
    assert err.max() < {1: 5e-5, 2: 1e-3, 3: 2e-3}[m2l]
