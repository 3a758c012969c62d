"""The device M2L tables a context keeps: what a first call of an order uploads
beyond a second one, and the tables the workers of a batch share."""
import numpy as np
import pytest

from gpurify_b200 import _lib, layouts

pytestmark = pytest.mark.gpu


def panels(nets, side, seed, edge=0.5e-6):
    lay = layouts.routing_window(nets, side, seed=seed, len_um=(0.5, 4.0))
    p = _lib.bridge_panelize(lay.store.arrays(), lay.deck.layer_table(), 1.0, lay.net_of_poly, mesh_max_edge_m=edge,
                             max_panels=-1)
    return p["verts"], p["cond"], len(p["nets"]) + 1


@pytest.mark.parametrize("order", [2, 3, 5, 6])
def test_first_call_uploads_only_tables_some_kernel_reads(order):
    """Compressed operators: the factors of rank 32 with rows of the node
    stride in FP64 (and FP32 from order 4), the TF32 operators of orders 4 and
    5, and the ranks.  The unpadded factors and the dense FP64 operators, 384
    MB at order 6, are not among them."""
    v, c, nc = panels(3, 8.0, 5)
    ns = (order**3 + 31) // 32 * 32
    tables = 2 * 343 * 32 * ns * (8 + (4 if order >= 4 else 0)) + (343 * ns * ns * 4 if order in (4, 5) else 0) + 343 * 4
    ctx = _lib.Context(0)
    try:
        up = []
        for _ in range(2):
            _, rep = ctx.cap_solve(v, c, nc, order=order, max_level=3, dense_below=-1)
            assert rep["m2l_pairs"] > 0
            up.append(rep["h2d_bytes"])
    finally:
        ctx.close()
    assert up[0] - up[1] <= tables


@pytest.mark.parametrize("order", [5, 6])
def test_batch_on_a_fresh_context_equals_separate_solves(order):
    """Eight workers meet no table of the order: one builds it while the others
    wait, and with mixed_m2l 3 one of them adds the shared basis to the table
    the others already hold.  Window by window the matrices have the bits of
    separate calls on a context of their own."""
    probs = [panels(n, 8.0, 7 + n) for n in (2, 3, 4, 5, 3, 4, 2, 5)]
    kw = dict(order=order, max_level=3, dense_below=-1, precision=_lib.PREC_MIXED, mixed_m2l=3, far_quad=1, precond=1)
    for _ in range(2):
        ctx = _lib.Context(0)
        try:
            res = ctx.cap_solve_batched(probs, batch_streams=8, **kw)
        finally:
            ctx.close()
        one = _lib.Context(0)
        try:
            for (v, c, nc), (C, rep) in zip(probs, res):
                C1, rep1 = one.cap_solve(v, c, nc, **kw)
                assert rep["m2l_pairs"] > 0 and rep["converged"] == 1 and rep["iterations"] == rep1["iterations"]
                assert np.array_equal(C, C1)
        finally:
            one.close()
