"""Kernels at the sizes where their tiles, remainders and selection rules can
go wrong, against the CPU oracle or a plain float64 restatement."""

import math

import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a = np.asarray(a, np.float64).ravel()
    b = np.asarray(b, np.float64).ravel()
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _grid(nodes, graded):
    from easyfsi_b200.grid import CartesianGrid
    from easyfsi_b200.scenarios import graded_axis_widths

    if not graded:
        return CartesianGrid.uniform(bounds_min_m=(0.0, 0.0, 0.0), bounds_max_m=(1.0, 1.0, 1.0), grid_nodes=nodes)
    return CartesianGrid(bounds_min_m=(0.0, 0.0, 0.0), cell_widths_x_m=graded_axis_widths(nodes[0], 0.0, 1.0, 0.3, 0.7),
                         cell_widths_y_m=graded_axis_widths(nodes[1], 0.0, 1.0, 0.3, 0.7),
                         cell_widths_z_m=graded_axis_widths(nodes[2], 0.0, 1.0, 0.2, 0.8))


# ---------------------------------------------------------------------------
# far nodes of the immersed-boundary search
# ---------------------------------------------------------------------------


def _closed_surface(bands, slivers):
    """A UV sphere's markers and triangles; with `slivers`, also triangles
    that the distance bound must not judge: nearly collinear ones, tiny ones
    and degenerate ones, on and inside the sphere."""
    from easyfsi_b200.geometry import UvSphereResolution, make_uv_sphere

    mesh = make_uv_sphere(UvSphereResolution(bands, 2 * bands), 0.33)
    x = mesh.vertices + 0.5
    n = mesh.vertices / 0.33
    tri = [tuple(int(v) for v in f) for f in mesh.faces]
    if slivers:
        rng = np.random.default_rng(bands)
        base = len(x)
        extra, normals = [], []
        for q in range(12):
            u = rng.normal(size=3)
            u /= np.linalg.norm(u)
            v = np.cross(u, rng.normal(size=3))
            v /= np.linalg.norm(v)
            c = 0.5 + 0.33 * u
            size = 0.05 if q % 3 == 0 else 1.0e-4
            off = np.cross(u, v) * size * (1.0e-4 if q % 2 else 0.5)
            extra += [c, c + size * v, c + 0.5 * size * v + off]
            normals += [u] * 3
            tri.append((base + 3 * q, base + 3 * q + 1, base + 3 * q + 2))
        tri += [(base, base, base + 1), (base, base + 1, base)]  # degenerate
        x = np.concatenate([x, np.asarray(extra)])
        n = np.concatenate([n, np.asarray(normals)])
    return x.astype(np.float32), n.astype(np.float32), np.asarray(tri, np.int32)


@pytest.mark.parametrize("bands,slivers,triangles,nodes", [
    (3, False, True, (9, 11, 13)),     # few triangles: looked at by the node's own thread
    (4, True, True, (12, 10, 15)),     # ill-shaped and degenerate ones among them
    (8, False, False, (13, 16, 11)),   # few markers
    (5, True, True, (10, 9, 16)),      # a few more, on both sides of the line
    (5, False, False, (10, 9, 16)),
    (6, True, True, (17, 9, 21)),      # one tile of items, ill-shaped triangles
    (12, False, False, (16, 16, 19)),  # markers without triangles
    (16, True, True, (20, 23, 31)),    # several tiles with a remainder
])
def test_far_nodes_match_the_all_pairs_oracle(bands, slivers, triangles, nodes):
    """Kinds, nearest markers and projection indices identical to the oracle's
    loop over every item; distances and points within 1e-6 (the same f32
    expressions)."""
    from easyfsi_b200.hibm_mpm import HibmMpmIbNodeSearch, HibmMpmSurfaceMarkers

    x, n, tri = _closed_surface(bands, slivers)
    mk = HibmMpmSurfaceMarkers(marker_capacity=len(x), projection_triangle_capacity=len(tri))
    mk.load_markers(positions_m=x.tolist(), velocities_mps=np.zeros_like(x).tolist(), normals=n.tolist(),
                    areas_m2=[1.0] * len(x), region_ids=[1] * len(x))
    if triangles:
        mk.set_projection_triangles(tri.tolist())
    search = HibmMpmIbNodeSearch(grid_nodes=nodes, bounds_min_m=(0.0, 0.0, 0.0), bounds_max_m=(1.0, 1.0, 1.0),
                                 marker_capacity=len(x))
    rep = search.search_and_classify(mk, search_radius_m=0.03, interior_probe_distance_m=0.02,
                                     classify_far_internal_nodes=True)
    ref = orc.ib_node_search(grid_nodes=nodes, markers_x=mk.x_gamma_m.to_numpy(), markers_n=mk.n_gamma.to_numpy(),
                             triangles=tri if triangles else None, search_radius=0.03, interior_probe_distance=0.02,
                             sign_tolerance=search._default_sign_tolerance_m(), classify_far=True,
                             bounds_min=(0.0, 0.0, 0.0), spacing=search.spacing_m)
    assert rep.__dict__ == ref["report"]
    assert rep.internal_node_count > 0
    np.testing.assert_array_equal(search.node_kind_code.to_numpy(), ref["kind"])
    np.testing.assert_array_equal(search.nearest_marker.to_numpy(), ref["nearest_marker"])
    np.testing.assert_array_equal(search.node_projection_marker_indices.to_numpy(), ref["projection_indices"])
    for got, key in ((search.node_signed_distance_m, "signed_distance"), (search.node_boundary_point_m, "boundary_point"),
                     (search.node_interior_fluid_point_m, "interior_point"),
                     (search.node_projection_marker_weights, "projection_weights")):
        np.testing.assert_allclose(got.to_numpy(), ref[key], rtol=0.0, atol=1e-6, err_msg=key)


@pytest.mark.parametrize("edge", [2.0e-3, 5.0e-4, 1.0e-4])
def test_far_nodes_of_a_fine_patch_match_the_all_pairs_oracle(edge):
    """A patch of 1,152 irregular triangles with edges of a thousandth of the
    nodes' distance and less, on a sphere that holds every node: each node is
    internal, with the nearest of all triangles by the same f32 distances."""
    from easyfsi_b200.hibm_mpm import HibmMpmIbNodeSearch, HibmMpmSurfaceMarkers

    rng = np.random.default_rng(int(1.0 / edge))
    m, nodes = 25, (7, 6, 9)
    u, v = np.meshgrid(*[edge * (np.arange(m) - m / 2)] * 2, indexing="ij")
    u, v = (q + 0.3 * edge * rng.uniform(-1.0, 1.0, (m, m)) for q in (u, v))
    n = np.stack([u + 0.5, v + 0.3, np.full_like(u, 0.8)], axis=-1).reshape(-1, 3)
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    x = (0.5 + 0.95 * n).astype(np.float32)
    at = np.arange(m * m).reshape(m, m)
    a, b, c, d = (q.ravel() for q in (at[:-1, :-1], at[1:, :-1], at[1:, 1:], at[:-1, 1:]))
    tri = np.concatenate([np.stack([a, b, c], 1), np.stack([a, c, d], 1)]).astype(np.int32)
    mk = HibmMpmSurfaceMarkers(marker_capacity=len(x), projection_triangle_capacity=len(tri))
    mk.load_markers(positions_m=x.tolist(), velocities_mps=np.zeros_like(x).tolist(), normals=n.tolist(),
                    areas_m2=[1.0] * len(x), region_ids=[1] * len(x))
    mk.set_projection_triangles(tri.tolist())
    search = HibmMpmIbNodeSearch(grid_nodes=nodes, bounds_min_m=(0.0, 0.0, 0.0), bounds_max_m=(1.0, 1.0, 1.0),
                                 marker_capacity=len(x))
    rep = search.search_and_classify(mk, search_radius_m=0.02, interior_probe_distance_m=0.02,
                                     classify_far_internal_nodes=True)
    ref = orc.ib_node_search(grid_nodes=nodes, markers_x=mk.x_gamma_m.to_numpy(), markers_n=mk.n_gamma.to_numpy(),
                             triangles=tri, search_radius=0.02, interior_probe_distance=0.02,
                             sign_tolerance=search._default_sign_tolerance_m(), classify_far=True,
                             bounds_min=(0.0, 0.0, 0.0), spacing=search.spacing_m)
    assert rep.__dict__ == ref["report"]
    assert rep.internal_node_count == math.prod(nodes)
    np.testing.assert_array_equal(search.nearest_marker.to_numpy(), ref["nearest_marker"])
    np.testing.assert_array_equal(search.node_projection_marker_indices.to_numpy(), ref["projection_indices"])
    for got, key in ((search.node_signed_distance_m, "signed_distance"), (search.node_boundary_point_m, "boundary_point"),
                     (search.node_projection_marker_weights, "projection_weights")):
        np.testing.assert_allclose(got.to_numpy(), ref[key], rtol=0.0, atol=1e-6, err_msg=key)


# ---------------------------------------------------------------------------
# predictor tiles
# ---------------------------------------------------------------------------


@pytest.mark.parametrize("nodes,graded,dt", [
    ((4, 4, 4), False, 1.0e-2),
    ((9, 17, 33), True, 1.0e-2),    # one past a tile along j and k
    ((13, 8, 70), True, 2.0e-1),    # departure points several cells away
    ((50, 65, 96), False, 1.0e-3),  # one plane a block, more than a wave
    ((57, 45, 40), True, 1.0e-2),   # two planes a block, the last block with one
    ((67, 123, 130), False, 1.0e-2),  # six planes a block, the last block with one
])
@pytest.mark.parametrize("rk2", [False, True])
def test_predictor_matches_the_oracle(nodes, graded, dt, rk2):
    """Random velocities and masked cells; the tile's arithmetic rounds as the
    oracle's (quotients by a corrected reciprocal), so the bound is half a
    unit in the last place of the result, 2^-24."""
    from easyfsi_b200.fluid import CartesianFluidSolver, FluidDomainSpec

    grid = _grid(nodes, graded)
    fl = CartesianFluidSolver(FluidDomainSpec((0, 0, 0), grid.bounds_max_m, None, 1000.0, 1.0e-2, 1.0e-3,
                                              cartesian_grid=grid))
    ofl = orc.OracleFluid(grid, rho=1000.0, mu=1.0e-2)
    rng = np.random.default_rng(nodes[2])
    obs = (rng.random(nodes) < 0.05).astype(np.int32)
    vel = (0.3 * rng.normal(size=nodes + (3,))).astype(np.float32)
    fl.obstacle.from_numpy(obs)
    fl.velocity.from_numpy(vel)
    ofl.obstacle[...] = obs
    ofl.velocity[...] = vel
    fl.predict(dt, advection_scheme="rk2" if rk2 else "euler")
    ofl.predict(dt, rk2=rk2)
    assert _rel(fl.velocity.to_numpy(), ofl.velocity) <= 2.0**-24


# ---------------------------------------------------------------------------
# tensor-core convolution and weight gradient
# ---------------------------------------------------------------------------


def _volume(shape, ch, gen):
    return torch.randn(shape + (ch,), generator=gen, device="cuda").to(torch.bfloat16)


def _shifted(x, t):
    """x[v + off(t)], zeros outside the volume (float64)."""
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    i, j, k = t // 9, (t // 3) % 3, t % 3
    return p[i : i + x.shape[0], j : j + x.shape[1], k : k + x.shape[2]]


CONV_SHAPES = [
    (16, 16, (1, 1, 1)), (16, 16, (2, 1, 62)), (16, 32, (3, 5, 63)), (48, 16, (17, 9, 65)), (16, 48, (5, 33, 130)),
    (64, 64, (4, 4, 4)), (112, 48, (3, 9, 34)), (48, 112, (2, 7, 16)), (176, 16, (3, 3, 64)), (64, 256, (2, 3, 5)),
    (80, 32, (20, 18, 32)), (48, 112, (16, 18, 32)),  # the last one: the last channel split has fewer
]


@pytest.mark.parametrize("cin,cout,shape", CONV_SHAPES)
def test_convolution_boxes(cin, cout, shape):
    """Every box rule: lines split along z, several MMA tiles per plane, plane
    rings, channel splits, single lines.  FP32 sums of 27 cin products against
    float64 on the same BF16 values."""
    from easyfsi_b200 import _native

    gen = torch.Generator(device="cuda")
    gen.manual_seed(cin * 1000 + cout)
    x = _volume(shape, cin, gen)
    w = (torch.randn((cout, 27, cin), generator=gen, device="cuda") / math.sqrt(27 * cin)).to(torch.bfloat16)
    b = torch.randn(cout, generator=gen, device="cuda")
    yf = torch.full(shape + (cout,), float("nan"), dtype=torch.float32, device="cuda")
    yb = torch.zeros(shape + (cout,), dtype=torch.bfloat16, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    _native.call("efsi_conv3d_bf16", *shape, cin, cout, x.data_ptr(), w.data_ptr(), b.data_ptr(), 1, yb.data_ptr(),
                 yf.data_ptr(), err.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    xd, wd = x.double(), w.double()
    ref = torch.relu(sum(_shifted(xd, t) @ wd[:, t].T for t in range(27)) + b.double())
    assert _rel(yf.cpu().numpy(), ref.cpu().numpy()) <= 1e-5
    assert torch.equal(yb, yf.to(torch.bfloat16))


def _weight_gradient(x, g, start):
    from easyfsi_b200 import _native

    dw = start.clone()
    _native.call("efsi_conv3d_wgrad", *x.shape[:3], x.shape[3], g.shape[3], x.data_ptr(), g.data_ptr(), dw.data_ptr(),
                 torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return dw


def _weight_gradient_reference(x, g, start):
    xd, gd = x.double(), g.double().reshape(-1, g.shape[3])
    return torch.stack([gd.T @ _shifted(xd, t).reshape(-1, x.shape[3]) for t in range(27)], dim=1) + start.double()


@pytest.mark.parametrize("cin,cout,shape", [c for c in CONV_SHAPES if c[0] * c[1] <= 7168] + [
    (448, 16, (2, 2, 9)), (16, 448, (3, 4, 17)), (16, 16, (40, 33, 31))])
def test_weight_gradient_boxes(cin, cout, shape):
    """Boxes of a plane, several M blocks and channel splits; FP32 sums over
    the voxels against float64, added to what is there."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(cin * 1000 + cout + 1)
    x, g = _volume(shape, cin, gen), _volume(shape, cout, gen)
    start = torch.randn((cout, 27, cin), generator=gen, device="cuda")
    dw = _weight_gradient(x, g, start)
    assert _rel(dw.cpu().numpy(), _weight_gradient_reference(x, g, start).cpu().numpy()) <= 1e-5


@pytest.mark.parametrize("x_off,g_off", [(1, 0), (0, 3), (4, 8), (8, 5)])  # elements past a 16-byte boundary
def test_weight_gradient_of_operands_at_any_element(x_off, g_off):
    """Operands that do not start on a 16-byte boundary: the same gradient, to
    the same bound as the aligned ones."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(10 * x_off + g_off)
    shape, cin, cout = (3, 9, 34), 48, 32

    def at(t, off):
        buf = torch.empty(t.numel() + 16, dtype=t.dtype, device="cuda")
        view = buf[off : off + t.numel()].view(t.shape)
        view.copy_(t)
        return view

    x, g = at(_volume(shape, cin, gen), x_off), at(_volume(shape, cout, gen), g_off)
    assert x.data_ptr() % 16 == 2 * x_off % 16 and g.data_ptr() % 16 == 2 * g_off % 16
    start = torch.randn((cout, 27, cin), generator=gen, device="cuda")
    dw = _weight_gradient(x, g, start)
    assert _rel(dw.cpu().numpy(), _weight_gradient_reference(x, g, start).cpu().numpy()) <= 1e-5


@pytest.mark.parametrize("shape", [(2, 3, 5), (3, 9, 130)])  # one box a plane, and lines split along z
@pytest.mark.parametrize("where", ["x", "dy"])
def test_weight_gradient_with_values_that_are_not_finite(shape, where):
    """Infinities and a NaN on faces, a corner and a line's inside: each reaches
    the taps that pair it with a voxel of the volume, and no other (in dy, zeros
    outside the volume too: infinity times zero)."""
    cin, cout = 16, 32
    gen = torch.Generator(device="cuda")
    gen.manual_seed(shape[2])
    x, g = _volume(shape, cin, gen), _volume(shape, cout, gen)
    bad = x if where == "x" else g
    n = shape[2]
    for (i, j, k), ch, value in (((0, 0, 0), 0, math.inf), ((shape[0] - 1, shape[1] - 1, n - 1), 1, -math.inf),
                                 ((0, 1, n // 2), 2, math.inf), ((1, 0, n - 1), 3, math.nan), ((1, 2, 0), 4, math.inf),
                                 ((1, 1, 1), 5, math.inf), ((1, 1, 2), 5, -math.inf)):
        bad[i, j, k, ch] = value
    dw = _weight_gradient(x, g, torch.zeros((cout, 27, cin), device="cuda")).double().cpu()
    ref = _weight_gradient_reference(x, g, torch.zeros((cout, 27, cin), device="cuda")).cpu()
    assert torch.equal(torch.isnan(dw), torch.isnan(ref))
    assert torch.equal(torch.isinf(dw), torch.isinf(ref)) and torch.equal(dw[torch.isinf(dw)], ref[torch.isinf(ref)])
    fin = torch.isfinite(ref)
    assert not fin.all() and _rel(dw[fin].numpy(), ref[fin].numpy()) <= 1e-5


# ---------------------------------------------------------------------------
# single-CTA tail of the V-cycle
# ---------------------------------------------------------------------------


@pytest.mark.parametrize("nodes,outlet,solid", [
    ((7, 6, 9), 0, 0.03),      # two levels, 60 cells: two warps at the coarsest
    ((8, 8, 8), 1, 0.03),      # 64 + 8 cells, one warp
    ((20, 17, 23), 0, 0.03),   # 1080 cells: more than one a thread, odd extents
    ((33, 17, 31), 1, 0.03),   # 2448 + 360 + 60 cells: the first does not fit beside the others
    ((16, 16, 16), 0, 0.15),   # the coarsest levels are obstacles throughout
    ((16, 16, 16), 1, 0.6),    # all coarse levels are
    ((20, 17, 23), 1, 0.0),
])
def test_vcycle_tail_matches_the_oracle(nodes, outlet, solid):
    """The tail's rows round as the oracle's (quotients by a corrected
    reciprocal), so the V-cycle agrees to f64 rounding of the level-0 sweeps,
    1e-13 as in the general V-cycle test."""
    from easyfsi_b200.fluid import CartesianFluidSolver, FluidDomainSpec

    grid = _grid(nodes, min(nodes) > 12)
    fl = CartesianFluidSolver(FluidDomainSpec((0, 0, 0), grid.bounds_max_m, None, 1000.0, 1.0e-3, 1.0e-3,
                                              cartesian_grid=grid))
    ofl = orc.OracleFluid(grid, rho=1000.0, mu=1.0e-3)
    rng = np.random.default_rng(nodes[0])
    obs = (rng.random(nodes) < solid).astype(np.int32)
    fl.obstacle.from_numpy(obs)
    ofl.obstacle[...] = obs
    r = rng.normal(size=nodes) * (obs == 0)
    fl.cg_r.from_numpy(r)
    fl._apply_fv_multigrid_preconditioner(fl.cg_r, pressure_outlet_zmin=bool(outlet))
    assert _rel(fl.cg_z.to_numpy(), ofl.vcycle(r, outlet)) <= 1e-13


# ---------------------------------------------------------------------------
# column-marching kernels of the finest level
# ---------------------------------------------------------------------------

# odd nx (a last plane without its pair), ny % 8 != 0 and odd (partial tiles,
# patches whose second row lies outside), nz on both sides of a 64-cell tile
COLUMN_NODES = [(13, 9, 48), (5, 8, 64), (21, 19, 80), (8, 15, 144)]


def _column_pair(nodes, rows, monkeypatch):
    """The same problem with the column kernels and without them; with `rows`,
    Dirichlet velocity rows weigh faces."""
    from easyfsi_b200.fluid import CartesianFluidSolver, FluidDomainSpec

    grid = _grid(nodes, True)
    rng = np.random.default_rng(nodes[2])
    obs = (rng.random(nodes) < 0.03).astype(np.int32)
    act, weight = (rng.random(nodes) < 0.05).astype(np.int32), rng.random(nodes).astype(np.float32)
    out = []
    for off in (False, True):
        with monkeypatch.context() as m:
            if off:
                m.setenv("EFSI_NO_COLUMN", "1")
            else:
                m.delenv("EFSI_NO_COLUMN", raising=False)
            fl = CartesianFluidSolver(FluidDomainSpec((0, 0, 0), grid.bounds_max_m, None, 1000.0, 1.0e-3, 1.0e-3,
                                                      cartesian_grid=grid))
            fl.obstacle.from_numpy(obs)
            if rows:
                fl.velocity_dirichlet_boundary_active.from_numpy(act)
                fl.velocity_dirichlet_boundary_projection_weight.from_numpy(weight)
            fl._refresh_structure()
        out.append(fl)
    ofl = orc.OracleFluid(grid, rho=1000.0, mu=1.0e-3)
    ofl.obstacle[...] = obs
    return rng, obs, out, ofl


@pytest.mark.parametrize("nodes", COLUMN_NODES)
@pytest.mark.parametrize("rows", [False, True])
@pytest.mark.parametrize("outlet", [0, 1])
def test_column_vcycle_rows(nodes, rows, outlet, monkeypatch):
    """A V-cycle without sums: bit for bit that of the other kernels, and the
    oracle's (which takes no Dirichlet rows) to 1e-13 as in the general test."""
    rng, obs, pair, ofl = _column_pair(nodes, rows, monkeypatch)
    r = rng.normal(size=nodes) * (obs == 0)
    z = []
    for fl in pair:
        fl.cg_r.from_numpy(r)
        fl._apply_fv_multigrid_preconditioner(fl.cg_r, pressure_outlet_zmin=bool(outlet))
        z.append(fl.cg_z.to_numpy())
    np.testing.assert_array_equal(z[0], z[1])
    if not rows:
        assert _rel(z[0], ofl.vcycle(r, outlet)) <= 1e-13


@pytest.mark.parametrize("nodes", COLUMN_NODES)
@pytest.mark.parametrize("precond", ["fv_multigrid", "fv_multigrid_mixed"])
@pytest.mark.parametrize("rows,outlet", [(False, 0), (False, 1), (True, 0), (True, 1)])
def test_column_iterations(nodes, precond, rows, outlet, monkeypatch):
    """Three CG iterations (a fresh direction, two with the last one added, the
    dots in the last sweep): the rows are the same and only the order of the
    f64 sums differs, 1e-11 of the pressure."""
    rng, _, pair, ofl = _column_pair(nodes, rows, monkeypatch)
    div = rng.normal(size=nodes).astype(np.float32)
    p = []
    for fl in pair:
        fl.divergence.from_numpy(div)
        fl.pressure.tensor.zero_()
        fl._solve_pressure_poisson_fv_cg(iterations=3, rhs_scale=1.0e6, pressure_outlet_zmin=bool(outlet),
                                         tolerance=1e-14, preconditioner=precond)
        assert fl.last_cg_iterations == 3
        p.append(fl.pressure.to_numpy())
    assert _rel(p[0], p[1]) <= 1e-11
    if precond == "fv_multigrid" and not rows and not outlet:
        ofl.divergence[...] = div
        ofl.prepare_rhs(1.0e6)
        ofl.pcg_solve(outlet=0, max_iters=3, tol=1e-14, precond=1, remove_mean=True)
        assert _rel(p[0], ofl.pressure) <= 1e-11


# ---------------------------------------------------------------------------
# particle binning
# ---------------------------------------------------------------------------


@pytest.mark.parametrize("nodes", [(8, 8, 8), (80, 84, 76), (84, 84, 84)])
def test_substep_over_many_tiles_matches_the_oracle(nodes):
    """Tile counts on both sides of one scan block's 8192 entries, particles in
    the first, middle and last tiles: the exchange with the grid changes every
    particle's velocity, so one that a wrong offset leaves out of either transfer
    keeps its own.  f32 sums by atomics in another order, 1e-5 as in the general
    test; the report counts every particle."""
    from easyfsi_b200.neo_hookean_mpm import NeoHookeanMpmState

    rng = np.random.default_rng(nodes[1])
    lo, hi = 3.0 / np.asarray(nodes), 1.0 - 3.0 / np.asarray(nodes)
    x = np.concatenate([lo + 0.02 * rng.random((40, 3)), 0.4 + 0.04 * rng.random((400, 3)),
                        hi - 0.02 * rng.random((40, 3))]).astype(np.float32)
    n = len(x)
    v = (0.01 * rng.normal(size=(n, 3))).astype(np.float32)
    vol, mass = np.full(n, 1e-6, np.float32), np.full(n, 1e-3, np.float32)
    so = NeoHookeanMpmState(particle_capacity=n, bounds_min_m=(0, 0, 0), bounds_max_m=(1, 1, 1), grid_nodes=nodes)
    so.load_particles(positions_m=x, volumes_m3=vol, masses_kg=mass, region_ids=np.full(n, 1, np.int32))
    so.v.tensor[:n] = torch.as_tensor(v, device=so.device)
    ref = orc.OracleSolid(capacity=n, grid_nodes=nodes)
    ref.load(x=x, volume=vol, mass=mass, region=np.full(n, 1, np.int32))
    ref.v[:n] = v
    rep = so.step(dt_s=1.0e-4, mu_pa=1.0e4, lambda_pa=1.0e4, primary_region_id=1, secondary_region_id=2)
    ref.step(dt=1.0e-4, mu=1.0e4, lam=1.0e4, primary=1, secondary=2)
    assert np.linalg.norm(ref.v[:n] - v, axis=1).min() > 1e-4  # every particle met the grid
    for got, want in ((so.v, ref.v), (so.x, ref.x), (so.C, ref.C)):
        assert _rel(got.to_numpy()[:n], want[:n]) <= 1e-5
    assert rep.transfer_relative_error < 2e-5


# ---------------------------------------------------------------------------
# marker exchange
# ---------------------------------------------------------------------------


def _exchange(x, v, normal, area, marker_x, marker_f, radius):
    """Force on the particles, the markers after the feedback, and both reports."""
    from easyfsi_b200.hibm_mpm import HibmMpmSurfaceMarkers

    m = len(marker_x)
    mk = HibmMpmSurfaceMarkers(marker_capacity=m)
    mk.load_markers(positions_m=np.zeros((m, 3)).tolist(), velocities_mps=np.zeros_like(marker_x).tolist(),
                    normals=[(0.0, 0.0, 1.0)] * m, areas_m2=[1.0] * m, region_ids=[1] * m)
    mk.x_gamma_m.from_numpy(marker_x)  # (loading refuses what is not finite)
    mk.F_gamma_n.from_numpy(marker_f)
    xt, vt, nt, at = (torch.from_numpy(q).cuda() for q in (x, v, normal, area))
    force = torch.zeros_like(xt)
    scatter = mk.scatter_marker_forces_to_mpm_particles(force, xt, particle_count=len(x), support_radius_m=radius)
    feedback = mk.update_surface_feedback_from_mpm_surface_particles(xt, vt, nt, at, particle_count=len(x),
                                                                     support_radius_m=radius, dt_s=1.0e-3)
    state = [f.to_numpy() for f in (mk.x_gamma_m, mk.v_gamma_mps, mk.n_gamma, mk.A_gamma_m2)]
    return force.cpu().numpy(), state, scatter, feedback


@pytest.mark.parametrize("count,radius", [(500, 0.02), (3000, 0.3)])  # more bins than particles, and fewer
def test_marker_exchange_ignores_particles_that_are_not_finite(count, radius):
    """Particles with NaN or infinite positions among others: markers, reports
    and forces are those of the finite particles alone.  The feedback sums the
    same values in the same order; the forces are f32 atomic sums of at most 60
    contributions, 60 x 2^-24 of the sum of their sizes."""
    rng = np.random.default_rng(count)
    x = rng.random((count, 3)).astype(np.float32)
    v, normal = (rng.normal(size=(count, 3)).astype(np.float32) for _ in range(2))
    area = rng.random(count).astype(np.float32)
    marker_x = (x[:60] + 0.3 * radius * rng.uniform(-1.0, 1.0, (60, 3))).astype(np.float32)
    marker_f = rng.normal(size=(60, 3))
    bad = np.concatenate([[0, count - 1], rng.choice(np.arange(100, count - 1), 20, replace=False)])
    x[bad, np.arange(len(bad)) % 3] = np.resize([np.nan, np.inf, -np.inf], len(bad))
    good = np.setdiff1d(np.arange(count), bad)
    force, state, scatter, feedback = _exchange(x, v, normal, area, marker_x, marker_f, radius)
    ref_force, ref_state, ref_scatter, ref_feedback = _exchange(x[good], v[good], normal[good], area[good], marker_x,
                                                                marker_f, radius)
    assert scatter.active_marker_count >= 40
    for got, ref in zip(state, ref_state):
        np.testing.assert_array_equal(got, ref)
    assert feedback == ref_feedback
    assert (scatter.active_marker_count, scatter.invalid_marker_count, scatter.active_particle_count) == (
        ref_scatter.active_marker_count, ref_scatter.invalid_marker_count, ref_scatter.active_particle_count)
    assert not force[bad].any()
    np.testing.assert_allclose(force[good], ref_force, rtol=0.0, atol=60 * 2.0**-24 * np.abs(marker_f).sum(0).max())


def test_marker_exchange_with_markers_that_are_not_finite():
    """Markers with a NaN or infinite position, or force, count as invalid and
    leave the others' exchange as it is; a marker whose force alone is not finite
    still moves with its particles."""
    rng = np.random.default_rng(3)
    x = rng.random((800, 3)).astype(np.float32)
    v, normal = (rng.normal(size=(800, 3)).astype(np.float32) for _ in range(2))
    area = rng.random(800).astype(np.float32)
    marker_x, marker_f = x[:40].copy(), rng.normal(size=(40, 3))
    bad_x, bad_f = np.array([0, 9, 39]), np.array([4, 17])
    want = _exchange(x, v, normal, area, marker_x, np.where(np.isin(np.arange(40), bad_x)[:, None], 0.0, marker_f), 0.1)
    marker_x[bad_x, [0, 1, 2]] = [np.nan, np.inf, -np.inf]
    marker_f[bad_f, [0, 2]] = [np.nan, np.inf]
    force, state, scatter, feedback = _exchange(x, v, normal, area, marker_x, marker_f, 0.1)
    assert (scatter.active_marker_count, scatter.invalid_marker_count) == (35, 5)
    assert (feedback.updated_marker_count, feedback.invalid_marker_count) == (37, 3)
    assert np.isfinite(force).all() and math.isfinite(scatter.action_reaction_residual_n)
    good = np.setdiff1d(np.arange(40), bad_x)
    for got, ref in zip(state, want[1]):
        np.testing.assert_array_equal(got[good], ref[good])


def test_marker_exchange_with_a_radius_whose_reciprocal_overflows():
    """A support radius of 1e-39 reaches the particle at the marker itself, with
    weight one."""
    origin = np.zeros((1, 3), np.float32)
    force, state, scatter, feedback = _exchange(origin, np.ones((1, 3), np.float32), np.ones((1, 3), np.float32),
                                                np.ones(1, np.float32), origin, np.array([[1.0, -2.0, 3.0]]), 1.0e-39)
    assert scatter.active_marker_count == 1 and feedback.updated_marker_count == 1
    np.testing.assert_array_equal(force, [[1.0, -2.0, 3.0]])
    np.testing.assert_array_equal(state[1], [[1.0, 1.0, 1.0]])


# ---------------------------------------------------------------------------
# projection reports
# ---------------------------------------------------------------------------


@pytest.mark.parametrize("nodes", [(5, 4, 7), (12, 9, 33), (40, 50, 60)])
def test_dirichlet_row_report_sums(nodes):
    """Row count, sum and maximum of |dv| against float64 sums of the same f32
    values; the square root rounds to f32, so 1e-6."""
    from easyfsi_b200.fluid import CartesianFluidSolver, FluidDomainSpec

    grid = _grid(nodes, False)
    fl = CartesianFluidSolver(FluidDomainSpec((0, 0, 0), grid.bounds_max_m, None, 1000.0, 1.0e-3, 1.0e-3,
                                              cartesian_grid=grid))
    rng = np.random.default_rng(nodes[0])
    obs = (rng.random(nodes) < 0.1).astype(np.int32)
    act = (rng.random(nodes) < 0.3).astype(np.int32)
    vel, val = (rng.normal(size=nodes + (3,)).astype(np.float32) for _ in range(2))
    fl.obstacle.from_numpy(obs)
    fl.velocity_dirichlet_boundary_active.from_numpy(act)
    fl.velocity_dirichlet_boundary_value_mps.from_numpy(val)
    fl.velocity_dirichlet_boundary_projection_weight.from_numpy(np.ones(nodes, np.float32))
    fl.velocity.from_numpy(vel)
    rep = fl.apply_velocity_dirichlet_boundary_rows()
    rows = (act != 0) & (obs == 0)
    d = np.linalg.norm((val - vel).astype(np.float64)[rows], axis=1)
    h = [1.0 / m for m in nodes]
    impulse = 1000.0 * h[0] * h[1] * h[2] * (val - vel).astype(np.float64)[rows].sum(0)
    assert rep.active_cells == rows.sum()
    assert rep.max_delta_mps == pytest.approx(d.max(), rel=1e-6)
    assert rep.mean_delta_mps == pytest.approx(d.mean(), rel=1e-6)
    np.testing.assert_allclose(rep.momentum_delta_n_s, impulse, rtol=0.0,
                               atol=1e-6 * 1000.0 * h[0] * h[1] * h[2] * d.sum())
    np.testing.assert_array_equal(fl.velocity.to_numpy()[rows], val[rows])


@pytest.mark.parametrize("nodes", [(4, 5, 6), (17, 9, 33), (40, 50, 60)])  # one block, some, more than a grid's turn
@pytest.mark.parametrize("outlet", [0, 1])
@pytest.mark.parametrize("value", [0.0, math.nan, math.inf])
def test_final_divergence_report_slots(nodes, outlet, value):
    """All nine categories against numpy: counts and maxima exact, sums of
    squares to the order of f64 sums.  A value that is not finite stays in the
    slots of its cell's categories."""
    from ctypes import c_double

    from easyfsi_b200 import _native
    from easyfsi_b200.fluid import CartesianFluidSolver, FluidDomainSpec

    grid = _grid(nodes, False)
    fl = CartesianFluidSolver(FluidDomainSpec((0, 0, 0), grid.bounds_max_m, None, 1000.0, 1.0e-3, 1.0e-3,
                                              cartesian_grid=grid))
    rng = np.random.default_rng(nodes[0])
    fluid = rng.random(nodes) > 0.3
    act, reach = (rng.random(nodes) < 0.5).astype(np.int32), (rng.random(nodes) < 0.8).astype(np.int32)
    div, src = (rng.normal(size=nodes).astype(np.float32) for _ in range(2))
    iface = rng.normal(size=nodes)
    cell = tuple(np.argwhere(fluid)[len(np.argwhere(fluid)) // 2])
    if value != 0.0:
        div[cell] = value
    fl.obstacle.from_numpy((~fluid).astype(np.int32))
    fl._refresh_structure()
    gdiv, gsrc, gact, greach, giface = (torch.from_numpy(q).cuda() for q in (div, src, act, reach, iface))
    out = (c_double * 54)()
    _native.call("efsi_divergence_final_report", fl._plan, gdiv.data_ptr(), giface.data_ptr(), gsrc.data_ptr(),
                 gact.data_ptr(), greach.data_ptr(), outlet, out, torch.cuda.current_stream().cuda_stream)
    raw = np.abs(div.astype(np.float64) + iface)
    res = np.abs(div.astype(np.float64) + iface - src)
    va = act != 0

    def ahead(m, axis):  # the next cell's value, False behind the last
        return np.concatenate([np.delete(m, 0, axis), np.zeros_like(np.take(m, [0], axis))], axis)

    def behind(m, axis):
        return np.concatenate([np.zeros_like(np.take(m, [0], axis)), np.delete(m, -1, axis)], axis)

    near, corr = va.copy(), np.zeros(nodes, bool)
    for axis in range(3):
        near |= ahead(va, axis)
        corr |= (behind(fluid, axis) & ~va) | (ahead(fluid, axis) & ~ahead(va, axis))
    if outlet:
        corr[:, :, 0] |= ~va[:, :, 0]
    inside = np.zeros(nodes, bool)
    inside[1:-1, 1:-1, 1:-1] = True
    on = fluid & (reach != 0)
    sets = [on, on & inside, on & near, on & ~near, on & corr, on & ~corr, on & inside & corr, on & inside & ~corr,
            fluid & (reach == 0)]
    for q, cells in enumerate(sets):
        for e, v in enumerate((raw[cells], res[cells])):
            got = out[3 * (2 * q + e) : 3 * (2 * q + e) + 3]
            assert got[2] == cells.sum()
            np.testing.assert_allclose(got[:2], [v.max(initial=0.0), (v * v).sum()], rtol=1e-12, equal_nan=True)
