"""Performance cases of the capacitance extractor, through its public entry
points: layouts to per-net capacitances (``pex.run_pex_by_net_checked``), panel
problems to Maxwell matrices (``Context.cap_solve``, plain, with one
permittivity per panel, batched, and without allocation), one operator apply,
and the adjoint sensitivities.

Layouts come from ``gpurify_b200.layouts`` with the sizes of the benchmark's
workloads and of the tests, drawn from the seed.  A case is a dict of plain
values:

* ``api``        ``static`` | ``extract`` | ``maxwell`` | ``media`` | ``batch`` |
                 ``operator`` | ``sensitivity``
* ``layout``     ``window`` (``nets``, ``side_um``), ``wires`` or ``bus``
* ``edge_um``    maximum panel edge; 0 is the reference's own mesh rule
* ``precision``, ``order``, ``depth``, ``quad``, ``precond``, ``m2l``, ``far_tc``: solver
  options (depth -1 is the library's own choice)
* ``count``      windows of a batch, columns of an operator apply, or
                 parameters of a sensitivity
* ``panels``, ``rhs``, ``applies``: the usual panels, right-hand sides and
  operator applies of the case, for ``work``
"""
import math
import random

import numpy as np
import torch

from gpurify_b200 import _lib, layouts, pex, sensitivity

EPS0 = 8.854187812800e-12
UM = 1e-6


def _case(name=None, **kw):
    case = dict(api="maxwell", layout="window", nets=16, side_um=15.0, edge_um=0.4, precision="fp64", order=5, depth=-1,
                quad=1, precond=2, m2l=0, far_tc=0, count=0, panels=6000, rhs=16, applies=70)
    case.update(kw)
    return dict(case, name=name) if name else case


def listed():
    return [
        # A cell-sized problem whose panels already are in device memory, as a
        # caller with its own device pool solves in a loop: the smallest call.
        _case("static_3nets", api="static", nets=3, side_um=6.0, edge_um=0.0, panels=330, rhs=4, applies=1),
        # The default per-net call on a cell of three nets: the reference's mesh
        # and options, below 500 panels, so every pair is exact.
        _case("extract_3nets_default", api="extract", nets=3, side_um=6.0, edge_um=0.0, order=0, quad=0, precond=0,
              panels=330, rhs=4, applies=50),
        # The benchmark's first configuration: two met1 wires, the reference's
        # mesh and options (order 4, depth 4, diagonal preconditioner).
        _case("extract_wires_default", api="extract", layout="wires", nets=2, edge_um=0.0, order=0, quad=0, precond=0,
              panels=513, rhs=3, applies=40),
        # A small window in a stack of several dielectric constants, reference options.
        _case("media_8nets", api="media", nets=8, side_um=10.0, edge_um=0.5, order=4, quad=0, precond=0, panels=1750,
              rhs=9, applies=60),
        # The routing window of the parity tests in plain FP64 and in mixed
        # precision with the library's default engines.
        _case("maxwell_16nets_fp64", panels=6000, rhs=16, applies=45),
        _case("maxwell_16nets_mixed", precision="mixed", precond=1, panels=6000, rhs=16, applies=75),
        # One operator apply (set-up included) with an odd number of columns, as
        # accuracy checks and outer solvers written by users call it.
        _case("operator_37cols", api="operator", nets=24, side_um=25.0, edge_um=0.3, order=4, count=37, panels=17000,
              rhs=37, applies=1),
        # The bus of the benchmark: capacitances and gradients along width,
        # spacing, thickness and height, mixed precision.
        _case("sensitivity_bus_mixed", api="sensitivity", layout="bus", nets=12, edge_um=0.2, precision="mixed",
              precond=1, m2l=3, count=4, panels=21000, rhs=12, applies=200),
        # Entry-wise accuracy of weak couplings needs order 6.
        _case("maxwell_24nets_order6", nets=24, side_um=25.0, edge_um=0.3, order=6, panels=17000, rhs=24, applies=55),
        # The benchmark's headline window at its depth 5, plain and mixed; mixed
        # from polygons to per-net values.
        _case("maxwell_64nets_fp64", nets=64, side_um=40.0, edge_um=0.25, depth=5, panels=70000, rhs=64, applies=72),
        _case("extract_64nets_mixed", api="extract", nets=64, side_um=40.0, edge_um=0.25, depth=5, precision="mixed",
              precond=1, m2l=3, far_tc=1, panels=70000, rhs=64, applies=125),
        # Many uneven windows in one call, as a full-chip run cuts its layout.
        _case("batch_8windows_mixed", api="batch", nets=48, side_um=60.0, edge_um=0.25, precision="mixed", precond=1,
              m2l=3, count=8, panels=120000, rhs=12, applies=110),
    ]


def draw(rng):
    def log_between(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    api = rng.choice(["static", "extract", "extract", "maxwell", "maxwell", "maxwell", "maxwell", "media", "batch",
                      "operator", "sensitivity"])
    if api == "static":
        return _case(api=api, nets=rng.randint(2, 4), side_um=round(rng.uniform(4.0, 6.5), 2), edge_um=0.0, panels=300,
                     rhs=4, applies=1)
    if api == "media":
        nets = int(round(log_between(2, 20)))
        side = round(rng.uniform(5.0, 14.0), 2)
        return _case(api=api, nets=nets, side_um=side, edge_um=round(rng.uniform(0.4, 0.7), 3), order=rng.choice([3, 4]),
                     quad=0, precond=0, panels=220 * nets, rhs=nets + 1, applies=60)
    if api == "operator":
        nets = int(round(log_between(2, 30)))
        return _case(api=api, nets=nets, side_um=round(rng.uniform(8.0, 30.0), 2), edge_um=round(rng.uniform(0.25, 0.5), 3),
                     order=rng.choice([2, 3, 4, 5, 6]), quad=rng.choice([0, 1]), count=rng.randint(1, 64),
                     panels=700 * nets, rhs=32, applies=1)
    if api == "sensitivity":
        mixed = rng.random() < 0.5
        return _case(api=api, layout="bus", nets=12, edge_um=round(rng.uniform(0.2, 0.45), 3), order=rng.choice([4, 5]),
                     precision="mixed" if mixed else "fp64", precond=1 if mixed else 2, m2l=3 if mixed else 0,
                     count=rng.randint(1, 4), panels=10000, rhs=12, applies=160)
    if api == "batch":
        mixed = rng.random() < 0.7
        return _case(api=api, nets=rng.randint(8, 40), side_um=round(rng.uniform(10.0, 50.0), 2), edge_um=0.25,
                     precision="mixed" if mixed else "fp64", precond=1, m2l=3 if mixed else 0, count=rng.randint(2, 6),
                     panels=60000, rhs=10, applies=100)
    if api == "extract" and rng.random() < 0.5:  # the reference's mesh and options, by default
        nets = int(round(log_between(2, 24)))
        return _case(api=api, nets=nets, side_um=round(rng.uniform(5.0, 20.0), 2), edge_um=0.0, order=0, quad=0,
                     precond=0, panels=120 * nets, rhs=nets + 1, applies=60)
    mixed = rng.random() < 0.5
    order = rng.choice([4, 5, 5, 6])
    nets = int(round(log_between(2, 24 if order == 6 else 60)))
    side = round(rng.uniform(max(5.0, 3.0 * math.sqrt(nets)), 38.0), 2)
    edge = round(rng.uniform(0.3 if order == 6 else 0.25, 0.5), 3)
    m2l = rng.choice([0, 3]) if mixed else 0
    depth = rng.choice([-1, -1, 4]) if side < 20.0 else -1
    return _case(api=api, nets=nets, side_um=side, edge_um=edge, precision="mixed" if mixed else "fp64", order=order,
                 depth=depth, quad=1, precond=rng.choice([1, 2]), m2l=m2l, far_tc=rng.choice([0, 1]) if mixed and order < 6 else 0,
                 panels=int(1050 * nets * (0.25 / edge) ** 1.5), rhs=nets, applies=120 if mixed else 65)


# ---- inputs ----


def _layout(case, seed):
    r = random.Random(seed)
    if case["layout"] == "wires":
        return layouts.two_wires(length_nm=50 * r.randint(390, 410), spacing_nm=10 * r.randint(14, 20))
    if case["layout"] == "bus":
        return layouts.bus_crossing(length_nm=100 * r.randint(290, 305), cross_w_nm=20 * r.randint(18, 22))
    if case["api"] == "operator":
        seed = 11  # one mesh: a seed changes the densities
    side = case["side_um"]
    return layouts.routing_window(case["nets"], side, seed=seed, len_um=(0.5, min(8.0, side / 3)))


def _batch_layouts(case, seed):
    """Windows like ``layouts.window_batch``'s: conductors log-uniform, sides uniform."""
    r = random.Random(case["nets"])  # the windows' sizes are the case's, their wires the seed's
    out = []
    for i in range(case["count"]):
        nets = int(round(math.exp(r.uniform(math.log(2), math.log(case["nets"])))))
        side = max(3.0 * math.sqrt(nets), r.uniform(5.0, case["side_um"]))
        out.append(layouts.routing_window(nets, side, seed=seed * 1009 + i, len_um=(0.5, min(8.0, side / 3))))
    return out


def _mesh(case):
    return dict(mesh_max_edge_m=case["edge_um"] * UM, max_panels=-1)


def _panels(case, lay):
    p = _lib.bridge_panelize(lay.store.arrays(), lay.deck.layer_table(), lay.deck.dbu_nm, lay.net_of_poly, **_mesh(case))
    return p["verts"], p["cond"], len(p["nets"]) + 1, p["nets"]


def _options(case):
    """Solver options as keyword arguments; none for the reference's defaults."""
    if case["order"] == 0:
        return {}
    kw = dict(order=case["order"], max_level=case["depth"], far_quad=case["quad"], precond=case["precond"], skip_ground_rhs=1,
              precision=_lib.PREC_MIXED if case["precision"] == "mixed" else _lib.PREC_FP64)
    if case["precision"] == "mixed":
        kw.update(mixed_m2l=case["m2l"], mixed_far_tc=case["far_tc"])
    if case["api"] == "media":
        kw.update(skip_ground_rhs=0)
    return kw


def _parameters(case, lay):
    z0, z1 = sensitivity.layer_span(lay.deck, "met2")
    return [("width", 3), ("spacing", 4), ("thickness", z0, z1), ("height", z0, z1)][: case["count"]]


def _media(verts, seed):
    """Relative permittivity of every panel by the height of its centre."""
    r = np.random.default_rng(seed)
    k = r.uniform(2.5, 4.5, 4)
    z = verts.reshape(-1, 4, 3)[:, :, 2].mean(1)
    return k[np.searchsorted([0.9e-6, 2.4e-6, 3.6e-6], z)]


def prepare(case, seed):
    state = dict(case=case, ctx=pex.default_context(), options=_options(case))
    api = case["api"]
    if api == "batch":
        state["problems"] = [_panels(case, lay)[:3] for lay in _batch_layouts(case, seed)]
        return state
    lay = _layout(case, seed)
    if api == "extract":
        state["layout"] = lay
        return state
    verts, cond, ncond, nets = _panels(case, lay)
    state.update(verts=verts, cond=cond, ncond=ncond)
    if api == "static":
        state["d_verts"] = torch.from_numpy(verts).cuda()
        state["d_cond"] = torch.from_numpy(cond).cuda()
        state["d_out"] = torch.zeros(ncond, ncond, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()  # the call runs on the context's own stream
    elif api == "media":
        state["eps"] = _media(verts, seed)
    elif api == "operator":
        state["sigma"] = np.random.default_rng(seed).standard_normal((len(verts), case["count"]))
    elif api == "sensitivity":
        state["velocities"] = sensitivity.velocity_fields(verts, cond, nets, _parameters(case, lay))
    return state


# ---- one pass ----


def run(state):
    api, ctx, kw = state["case"]["api"], state["ctx"], state["options"]
    if api == "static":
        ctx.cap_solve_small_static(len(state["verts"]), state["d_verts"].data_ptr(), state["d_cond"].data_ptr(),
                                   state["ncond"], state["d_out"].data_ptr())
        return state["d_out"]
    if api == "extract":
        lay = state["layout"]
        got = pex.run_pex_by_net_checked(lay.store, lay.deck, lay.net_of_poly, ctx=ctx, **_mesh(state["case"]), **kw)
        nets = sorted(got)
        return dict(nets=np.array(nets), cap_af=np.array([got[n].cap_af for n in nets]),
                    r_ohm=np.array([got[n].r_ohm for n in nets]))
    if api == "batch":
        return [c for c, _ in ctx.cap_solve_batched(state["problems"], **kw)]
    if api == "operator":
        kw = {k: v for k, v in kw.items() if k not in ("skip_ground_rhs", "precond")}
        return ctx.operator_apply(state["verts"], state["sigma"], **kw)[0]
    if api == "sensitivity":
        c, dc, _ = ctx.cap_sensitivity(state["verts"], state["cond"], state["ncond"], state["velocities"], **kw)
        return dict(maxwell=c, gradients=dc)
    return ctx.cap_solve(state["verts"], state["cond"], state["ncond"], eps=state.get("eps"), **kw)[0]


def work(case):
    """What a solve cannot do without: the panels read and the result written
    once; per operator apply the near entries (about 1,800 per panel, 8 bytes,
    or 4 in mixed precision) and the densities in and out; per Krylov step the
    earlier basis vectors read once.  Flops: the near product, the two ends of
    the far field (n^3 nodes) and about 250 per near entry's closed form."""
    n, r, a = float(case["panels"]), float(case["rhs"]), float(case["applies"])
    near = n * min(n, 1800.0)
    nodes = float(max(case["order"], 4) ** 3)
    if case["api"] == "static":
        return dict(bytes=100.0 * n + 8.0 * r * r, flops=n ** 3 * 2.0 / 3.0 + 250.0 * n * n)
    w = 4.0 if case["precision"] == "mixed" else 8.0
    io = 100.0 * n + (16.0 * n * r if case["api"] == "operator" else 8.0 * r * r)
    basis = 8.0 * n * r * a * a / 2.0 if a > 1 else 0.0
    flops = a * (2.0 * near * r + 4.0 * n * r * nodes) + 250.0 * near
    extra = case["count"] * (near * 8.0 + 100.0 * n) if case["api"] == "sensitivity" else 0.0
    return dict(bytes=io + near * w + a * (near * w + 16.0 * n * r) + basis + extra, flops=flops)


# ---- the same in plain torch, 64 bits ----

MOST_EXACT = 40000  # panels of a direct solve


def _integral(x, y, z):
    """Antiderivative of 1/r over a rectangle's corner offsets (x, y) at height z."""
    tiny = 1e-150
    rx = torch.sqrt(x * x + z * z).clamp_min(tiny)
    ry = torch.sqrt(y * y + z * z).clamp_min(tiny)
    r = torch.sqrt(x * x + y * y + z * z)
    return x * torch.asinh(y / rx) + y * torch.asinh(x / ry) - z * torch.atan2(x * y, z * r)


def _block(points, centre, half, axis):
    """Integral of 1/r over axis-aligned rectangles (normal ``axis``) at points, in um."""
    u, v = (axis + 1) % 3, (axis + 2) % 3
    d = [points[:, None, k] - centre[None, :, k] for k in range(3)]
    z = d[axis].abs()
    out = 0.0
    for su in (1.0, -1.0):
        for sv in (1.0, -1.0):
            out = out + su * sv * _integral(d[u] + su * half[None, :, u], d[v] + sv * half[None, :, v], z)
    return out


def _rectangles(verts):
    q = torch.as_tensor(verts, dtype=torch.float64, device="cuda").reshape(-1, 4, 3) / UM
    lo, hi = q.amin(1), q.amax(1)
    half = 0.5 * (hi - lo)
    axis = half.argmin(1)
    return 0.5 * (lo + hi), half, axis


def _area(half, axis):
    """Areas in m^2."""
    u, v = (axis + 1) % 3, (axis + 2) % 3
    return 4.0 * half.gather(1, u[:, None])[:, 0] * half.gather(1, v[:, None])[:, 0] * UM * UM


def _rows(centre, half, axis, i0, i1):
    """Rows [i0, i1) of the potential matrix (volts per C/m^2)."""
    out = torch.empty(i1 - i0, len(centre), dtype=torch.float64, device="cuda")
    for a in range(3):
        sel = (axis == a).nonzero()[:, 0]
        if len(sel):
            out[:, sel] = _block(centre[i0:i1], centre[sel], half[sel], a)
    return out * (UM / (4.0 * math.pi * EPS0))


def _chunks(n):
    step = max(1, 40_000_000 // n)
    return [(i, min(n, i + step)) for i in range(0, n, step)]


def _matrix(centre, half, axis):
    n = len(centre)
    p = torch.empty(n, n, dtype=torch.float64, device="cuda")
    for i0, i1 in _chunks(n):
        p[i0:i1] = _rows(centre, half, axis, i0, i1)
    return p


def _solve(verts, cond, ncond, columns):
    """Densities of unit-potential columns, the charge weights (conductor by
    panel) and the factors; None above the size of a direct solve."""
    centre, half, axis = _rectangles(verts)
    c = torch.as_tensor(cond, device="cuda").long()
    on = torch.zeros(len(c), ncond, dtype=torch.float64, device="cuda")
    on[torch.arange(len(c), device="cuda"), c] = 1.0
    lu, piv = torch.linalg.lu_factor(_matrix(centre, half, axis))
    sigma = torch.linalg.lu_solve(lu, piv, on[:, :columns].contiguous())
    return sigma, on * _area(half, axis)[:, None], (lu, piv)


def _by_symmetry(c, ncond):
    """The substrate's column from its row, its own entry unknown."""
    full = np.full((ncond, ncond), np.nan)
    full[:, : ncond - 1] = c
    full[: ncond - 1, ncond - 1] = c[ncond - 1]
    return full


def _maxwell(verts, cond, ncond):
    if len(verts) > MOST_EXACT:
        return None
    sigma, q, _ = _solve(verts, cond, ncond, ncond - 1)
    return _by_symmetry((q.T @ sigma).cpu().numpy(), ncond)


def _gradient(verts, cond, ncond, velocities):
    import torch.autograd.forward_ad as fwd

    sigma, q, (lu, piv) = _solve(verts, cond, ncond, ncond - 1)
    lam = torch.linalg.lu_solve(lu, piv, q[:, : ncond - 1].contiguous(), adjoint=True)
    centre, half, axis = _rectangles(verts)
    out = []
    for vel in velocities:
        v = torch.as_tensor(vel, dtype=torch.float64, device="cuda").reshape(-1, 4, 3)
        x = torch.as_tensor(verts, dtype=torch.float64, device="cuda").reshape(-1, 4, 3) / UM
        # an axis-aligned rectangle stays one: its faces move with their vertices
        top = torch.gather(v, 1, x.argmax(1, keepdim=True))[:, 0]
        low = torch.gather(v, 1, x.argmin(1, keepdim=True))[:, 0]
        dcentre, dhalf = 0.5 * (top + low), 0.5 * (top - low)
        # in um of panel per um of parameter
        with fwd.dual_level():
            dc, dh = fwd.make_dual(centre, dcentre), fwd.make_dual(half, dhalf)
            darea = fwd.unpack_dual(_area(dh, axis)).tangent
            ps = torch.zeros_like(sigma)
            for i0, i1 in _chunks(4 * len(centre)):
                i0, i1 = i0, min(i1, len(centre))
                if i0 >= i1:
                    break
                for a in range(3):
                    sel = (axis == a).nonzero()[:, 0]
                    if len(sel):
                        blk = fwd.unpack_dual(_block(dc[i0:i1], dc[sel], dh[sel], a)).tangent
                        ps[i0:i1] += (blk * (UM / (4.0 * math.pi * EPS0))) @ sigma[sel]
        on = (q[:, : ncond - 1] != 0).to(torch.float64)
        g = ((on * darea[:, None]).T @ sigma - lam.T @ ps) / UM  # per metre of parameter
        full = np.full((ncond, ncond), np.nan)
        full[: ncond - 1, : ncond - 1] = g.cpu().numpy()
        out.append(full)
    return _by_symmetry((q.T @ sigma).cpu().numpy(), ncond), np.stack(out)


def exact(case, seed):
    api = case["api"]
    if api == "batch":
        got = [_maxwell(*_panels(case, lay)[:3]) for lay in _batch_layouts(case, seed)]
        return got if any(g is not None for g in got) else None
    lay = _layout(case, seed)
    verts, cond, ncond, nets = _panels(case, lay)
    if api == "operator":
        sigma = torch.from_numpy(np.random.default_rng(seed).standard_normal((len(verts), case["count"]))).cuda()
        rect = _rectangles(verts)
        return torch.cat([_rows(*rect, i0, i1) @ sigma for i0, i1 in _chunks(len(verts))]).cpu().numpy()
    if len(verts) > MOST_EXACT:
        return None
    if api == "sensitivity":
        c, dc = _gradient(verts, cond, ncond, sensitivity.velocity_fields(verts, cond, nets, _parameters(case, lay)))
        return dict(maxwell=c, gradients=dc)
    if api in ("static", "media"):
        sigma, q, _ = _solve(verts, cond, ncond, ncond)
        if api == "media":
            q = q * torch.as_tensor(_media(verts, seed), device="cuda")[:, None]
        c = q.T @ sigma
        return c if api == "static" else c.cpu().numpy()
    c = _maxwell(verts, cond, ncond)
    if api == "extract":
        k = next(iter(lay.deck.pex.values())).dielectric_k
        return dict(nets=None, cap_af=np.diag(c)[: ncond - 1] * k * 1e18, r_ohm=None)
    return c
