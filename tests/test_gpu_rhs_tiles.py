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
