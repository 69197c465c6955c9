"""Performance cases: the work a program of this framework has it do.

Every case is one pass through the public entry points that a coupled
fluid-structure program calls: the whole coupled step, the pressure projection
with its options, the predictor, the MPM substep, the marker exchange, the
immersed-boundary node search with its boundary rows, the membrane step, and
the learned preconditioner's network in both directions.  ``listed`` names a
few of each over the range from the smallest test scene to the largest
workload of the benchmark; ``draw`` gives more of the same ranges.

Inputs are made from the seed alone; the large fields are made on the GPU.
``exact`` restates the paths whose results are computed numbers in 64 bits
with plain torch.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from easyfsi_b200.fluid import CartesianFluidSolver, FluidDomainSpec
from easyfsi_b200.geometry import UvSphereResolution, make_plate_mesh, make_uv_sphere
from easyfsi_b200.grid import CartesianGrid
from easyfsi_b200.hibm_mpm import HibmMpmIbBoundaryConditions, HibmMpmIbNodeSearch, HibmMpmSurfaceMarkers
from easyfsi_b200.hyperelastic import lame_parameters
from easyfsi_b200.learned import UNetPreconditioner
from easyfsi_b200.mooney_shell_mpm import TriMooneyShellMpmState
from easyfsi_b200.neo_hookean_mpm import NeoHookeanMpmState
from easyfsi_b200.scenarios import Body, CoupledScene, ScenarioConfig, graded_axis_widths, markers, particles

REGION = 101
DENSITY = 1000.0
VISCOSITY = 1.0e-3


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # the smallest coupled scene of the test suite: a graded 12 x 12 x 16
        # box, all launch latency
        _step("step_tiny", 12, 12, 16, True, 12, 12, 12, (0.22, 0.2, 0.25), 5.0e4, 5.0e-4, 8),
        # the uniform 64^3 sphere scene, the usual size of a first coupled run
        _step("step_uniform64", 64, 64, 64, False, 64, 64, 64, (0.15, 0.15, 0.15), 1.0e5, 1.0e-4, 32),
        # the graded 128 x 128 x 256 ellipsoid scene of the benchmark
        _step("step_graded128x128x256", 128, 128, 256, True, 116, 116, 232, (0.12, 0.08, 0.2), 5.0e4, 5.0e-5, 64),
        # an odd-sized graded domain with an outlet and velocity-Dirichlet rows
        # around the body, reports on: a projection of a sharp-interface run
        dict(name="project_outlet_rows_75x61x143", kind="project", nx=75, ny=61, nz=143, graded=True, outlet=True,
             rows=True, precond="fv_multigrid", tol=1.0e-10, report=True),
        # a closed graded projection with the FP32 V-cycle
        dict(name="project_mixed_96x160x192", kind="project", nx=96, ny=160, nz=192, graded=True, outlet=False,
             rows=False, precond="fv_multigrid_mixed", tol=1.0e-8, report=False),
        # the predictor alone on the largest fluid grid of the workloads
        dict(name="predict_rk2_256", kind="predict", nx=256, ny=256, nz=256, graded=True, scheme="rk2"),
        # one MPM substep of half a million particles (two-sphere workload's count)
        dict(name="mpm_step_500k", kind="mpm", n=196, radius=0.126, report=False),
        # marker forces out to the particles and the surface feedback back, at
        # the benchmark scene's counts
        dict(name="marker_exchange_8k", kind="markers", n=116, radius=0.123, bands=64, report=False),
        # node search, boundary targets and reconstructed velocity rows of a
        # sharp-interface step on a graded 96 x 96 x 128 grid
        dict(name="ib_rows_96x96x128", kind="ib", nx=96, ny=96, nz=128, graded=True, bands=48),
        # the membrane step on the 20,000-triangle plate
        dict(name="shell_step_20k", kind="shell", nu=100, nv=100, nodes=36),
        # the learned preconditioner's network: applied to a residual field,
        # and the gradients of a batch of four crops as in its training
        dict(name="unet_forward_64x72x128", kind="unet_forward", nx=64, ny=72, nz=128),
        dict(name="unet_gradients_4x32", kind="unet_train", crop=32, batch=4),
    ]


def draw(rng):
    kind = rng.choice(("step", "project", "project", "predict", "mpm", "markers", "ib", "shell", "unet_forward",
                       "unet_train"))
    if kind == "step":
        nx, ny, nz = (_log_int(rng, 12, 112) for _ in range(3))
        m = _log_int(rng, 12, 112)
        r = rng.uniform(0.12, 0.22)
        c = _step("", nx, ny, nz, rng.random() < 0.5, m, m, m, (r, r * rng.uniform(0.8, 1.0), r), 1.0e5, 1.0e-4,
                  rng.randrange(8, 49))
        del c["name"]
        return c
    if kind == "project":
        outlet = rng.random() < 0.5
        return dict(kind="project", nx=_log_int(rng, 12, 144), ny=_log_int(rng, 12, 144), nz=_log_int(rng, 12, 200),
                    graded=rng.random() < 0.6, outlet=outlet, rows=rng.random() < 0.4,
                    precond=rng.choice(("fv_multigrid", "fv_multigrid", "jacobi")), tol=1.0e-10,
                    report=rng.random() < 0.5)
    if kind == "predict":
        return dict(kind="predict", nx=_log_int(rng, 12, 250), ny=_log_int(rng, 12, 250), nz=_log_int(rng, 12, 250),
                    graded=rng.random() < 0.5, scheme=rng.choice(("euler", "rk2")))
    if kind == "mpm":
        return dict(kind="mpm", n=_log_int(rng, 12, 190), radius=round(rng.uniform(0.1, 0.13), 4),
                    report=rng.random() < 0.5)
    if kind == "markers":
        return dict(kind="markers", n=_log_int(rng, 16, 116), radius=round(rng.uniform(0.1, 0.123), 4),
                    bands=_log_int(rng, 8, 64), report=rng.random() < 0.5)
    if kind == "ib":
        return dict(kind="ib", nx=_log_int(rng, 16, 96), ny=_log_int(rng, 16, 96), nz=_log_int(rng, 16, 128),
                    graded=rng.random() < 0.5, bands=_log_int(rng, 8, 48))
    if kind == "shell":
        return dict(kind="shell", nu=_log_int(rng, 8, 100), nv=_log_int(rng, 8, 100), nodes=rng.randrange(12, 37))
    if kind == "unet_forward":
        return dict(kind="unet_forward", nx=_log_int(rng, 8, 72), ny=_log_int(rng, 8, 72), nz=_log_int(rng, 8, 112))
    return dict(kind="unet_train", crop=rng.randrange(12, 33), batch=rng.randrange(1, 5))


def _step(name, nx, ny, nz, graded, mx, my, mz, axes, youngs, dt, bands):
    return dict(name=name, kind="step", nx=nx, ny=ny, nz=nz, graded=graded, mx=mx, my=my, mz=mz, ax=axes[0],
                ay=axes[1], az=axes[2], youngs=youngs, dt=dt, bands=bands)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _grid(c):
    nodes = (c["nx"], c["ny"], c["nz"])
    if not c["graded"]:
        return CartesianGrid.uniform(bounds_min_m=(0.0, 0.0, 0.0), bounds_max_m=(1.0, 1.0, 1.0), grid_nodes=nodes)
    return CartesianGrid(bounds_min_m=(0.0, 0.0, 0.0), cell_widths_x_m=graded_axis_widths(nodes[0], 0.0, 1.0, 0.3, 0.7),
                         cell_widths_y_m=graded_axis_widths(nodes[1], 0.0, 1.0, 0.3, 0.7),
                         cell_widths_z_m=graded_axis_widths(nodes[2], 0.0, 1.0, 0.2, 0.8))


def _fluid(c, dt):
    grid = _grid(c)
    return CartesianFluidSolver(FluidDomainSpec(bounds_min_m=(0.0, 0.0, 0.0), bounds_max_m=grid.bounds_max_m,
                                                grid_nodes=None, density_kgm3=DENSITY, viscosity_pa_s=VISCOSITY,
                                                dt_s=dt, cartesian_grid=grid))


def _wave_field(points, gen, amplitude, modes=6):
    """Random smooth vector field at the broadcastable coordinates `points`:
    a few Fourier modes per component, scaled to the amplitude."""
    shape = torch.broadcast_shapes(*(p.shape for p in points))
    out = torch.empty(shape + (3,), dtype=torch.float32, device="cuda")
    k = (torch.randint(-4, 5, (3, modes, 3), generator=gen, device="cuda") * math.pi).tolist()
    ph = (torch.rand((3, modes), generator=gen, device="cuda") * 2 * math.pi).tolist()
    for d in range(3):
        acc = torch.zeros(shape, dtype=torch.float32, device="cuda")
        for m in range(modes):
            acc += torch.cos(k[d][m][0] * points[0] + k[d][m][1] * points[1] + k[d][m][2] * points[2] + ph[d][m])
        out[..., d] = acc * (amplitude / modes)
    return out


def _centres(fluid):
    return (fluid.cell_center_x_m.tensor[:, None, None], fluid.cell_center_y_m.tensor[None, :, None],
            fluid.cell_center_z_m.tensor[None, None, :])


def _scenario(c, seed):
    return ScenarioConfig(name="case", grid_nodes=(c["nx"], c["ny"], c["nz"]), graded=c["graded"],
                          refine_box=((0.3, 0.3, 0.2), (0.7, 0.7, 0.8)), mpm_nodes=(c["mx"], c["my"], c["mz"]),
                          bodies=(Body((0.5, 0.5, 0.5), (c["ax"], c["ay"], c["az"]), c["youngs"], REGION),),
                          dt_s=c["dt"], steps=1, velocity_seed=seed, particle_seed=seed + 1,
                          marker_resolution=(c["bands"], 2 * c["bands"]))


def _ball_config(n, radius, seed, bands=8):
    return ScenarioConfig(name="case", grid_nodes=(n, n, n), graded=False, refine_box=None, mpm_nodes=(n, n, n),
                          bodies=(Body((0.5, 0.5, 0.5), (radius, radius, radius), 1.0e5, REGION),), dt_s=1.0e-4,
                          steps=1, velocity_seed=seed, particle_seed=seed + 1, marker_resolution=(bands, 2 * bands))


def _solid(cfg):
    part = particles(cfg)
    solid = NeoHookeanMpmState(particle_capacity=part["x"].shape[0], bounds_min_m=(0.0, 0.0, 0.0),
                               bounds_max_m=(1.0, 1.0, 1.0), grid_nodes=cfg.mpm_nodes)
    solid.load_particles(positions_m=part["x"], volumes_m3=part["volume"], masses_kg=part["mass"],
                         region_ids=part["region"], normals=part["normal"], areas_m2=part["area"])
    return solid


def _surface(cfg):
    mk = markers(cfg)
    out = HibmMpmSurfaceMarkers(marker_capacity=mk["x"].shape[0])
    out.load_markers(positions_m=mk["x"].tolist(), velocities_mps=np.zeros_like(mk["x"]).tolist(),
                     normals=mk["normal"].tolist(), areas_m2=mk["area"].tolist(), region_ids=mk["region"].tolist())
    return out


def _points(field):
    return field[:, 0], field[:, 1], field[:, 2]


# ---------------------------------------------------------------------------
# prepare / run per kind
# ---------------------------------------------------------------------------


def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, int(seed)), case=case)


def run(state):
    return _RUN[state["case"]["kind"]](state)


def _prepare_step(c, seed):
    cfg = _scenario(c, seed)
    scene = CoupledScene(cfg, initial_velocity=np.zeros(cfg.grid_nodes + (3,), np.float32), project_initial=False)
    fl = scene.fluid
    fl.velocity.from_torch(_wave_field(_centres(fl), _generator(seed), cfg.amplitude_mps))
    fl.project(iterations=400, pressure_solver="fv_cg", cg_tolerance=1.0e-8, cg_preconditioner="fv_multigrid",
               read_report=False)
    fl.clear_pressure()
    return {"scene": scene}


def _run_step(s):
    scene = s["scene"]
    scene.step()
    fl, so, mk = scene.fluid, scene.solid, scene.markers
    return {"velocity": fl.velocity.tensor, "pressure": fl.pressure.tensor, "x": so.x.tensor, "F": so.F.tensor,
            "force": so.external_force_n.tensor, "marker_x": mk.x_gamma_m.tensor}


def _prepare_project(c, seed):
    fl = _fluid(c, 1.0e-3)
    gen = _generator(seed)
    pts = _centres(fl)
    r = torch.sqrt(sum((p - 0.5) ** 2 for p in pts))
    solid = r < 0.15
    fl.obstacle.from_torch(solid.to(torch.int32))
    if c["rows"]:
        shell = (r >= 0.15) & (r < 0.19)
        value = 0.05 * torch.randn(shell.shape + (3,), generator=gen, device="cuda")
        weight = torch.rand(shell.shape, generator=gen, device="cuda") * 0.8 + 0.1
        fl.velocity_dirichlet_boundary_active.from_torch(shell.to(torch.int32))
        fl.velocity_dirichlet_boundary_value_mps.from_torch(value * shell[..., None])
        fl.velocity_dirichlet_boundary_projection_weight.from_torch(weight * shell)
    return {"fluid": fl, "velocity": _wave_field(pts, gen, 0.1)}


def _run_project(s):
    c, fl = s["case"], s["fluid"]
    fl.velocity.tensor.copy_(s["velocity"])
    fl.project(iterations=4000, pressure_outlet_zmin=c["outlet"], dt_s=1.0e-3, reset_pressure=True,
               pressure_solver="fv_cg", cg_tolerance=c["tol"], cg_preconditioner=c["precond"],
               read_report=c["report"])
    return {"velocity": fl.velocity.tensor, "pressure": fl.pressure.tensor}


def _prepare_predict(c, seed):
    fl = _fluid(c, 1.0e-3)
    pts = _centres(fl)
    fl.obstacle.from_torch((torch.sqrt(sum((p - 0.5) ** 2 for p in pts)) < 0.15).to(torch.int32))
    fl.velocity.from_torch(_wave_field(pts, _generator(seed), 0.5))
    return {"fluid": fl}


def _run_predict(s):
    fl = s["fluid"]
    fl.predict(1.0e-3, advection_scheme=s["case"]["scheme"])
    return fl.velocity.tensor


def _prepare_mpm(c, seed):
    gen = _generator(seed)
    solid = _solid(_ball_config(c["n"], c["radius"], seed))
    x = _points(solid.x.tensor)
    solid.v.from_torch(_wave_field(x, gen, 0.05))
    jitter = 0.01 * torch.randn(solid.F.tensor.shape, generator=gen, device="cuda")
    solid.F.tensor.add_(jitter)
    solid.external_force_n.from_torch(_wave_field(x, gen, 1.0) * solid.mass_kg.tensor[:, None])
    mu, lam = lame_parameters(1.0e5, 0.45)
    return {"solid": solid, "mu": mu, "lam": lam, "dt": min(1.0e-4, 2.0e-3 / c["n"])}


def _run_mpm(s):
    so = s["solid"]
    so.step(dt_s=s["dt"], mu_pa=s["mu"], lambda_pa=s["lam"], primary_region_id=REGION, secondary_region_id=REGION + 1,
            velocity_damping=0.999, read_report=s["case"]["report"])
    return {"x": so.x.tensor, "v": so.v.tensor, "C": so.C.tensor, "F": so.F.tensor,
            "area": so.area_weight_m2.tensor}


def _prepare_markers(c, seed):
    gen = _generator(seed)
    cfg = _ball_config(c["n"], c["radius"], seed, c["bands"])
    solid, mk = _solid(cfg), _surface(cfg)
    solid.v.from_torch(_wave_field(_points(solid.x.tensor), gen, 0.05))
    mk.F_gamma_n.from_torch(torch.randn(mk.F_gamma_n.tensor.shape, generator=gen, device="cuda",
                                        dtype=torch.float64) * 1.0e-3)
    keep = tuple(f.tensor.clone() for f in (mk.x_gamma_m, mk.n_gamma, mk.A_gamma_m2))
    return {"solid": solid, "markers": mk, "radius": 1.5 / c["n"], "keep": keep}


def _run_markers(s):
    so, mk, n, report = s["solid"], s["markers"], s["solid"].particle_count, s["case"]["report"]
    for f, t in zip((mk.x_gamma_m, mk.n_gamma, mk.A_gamma_m2), s["keep"]):
        f.from_torch(t)
    mk.clear_mpm_external_forces(so.external_force_n, particle_count=n, read_report=report)
    mk.scatter_marker_forces_to_mpm_particles(so.external_force_n, so.x, particle_count=n, support_radius_m=s["radius"],
                                              read_report=report)
    mk.update_surface_feedback_from_mpm_surface_particles(so.x, so.v, so.surface_normal, so.area_weight_m2,
                                                          particle_count=n, support_radius_m=s["radius"], dt_s=1.0e-4,
                                                          read_report=report)
    return {"force": so.external_force_n.tensor, "x": mk.x_gamma_m.tensor, "v": mk.v_gamma_mps.tensor,
            "n": mk.n_gamma.tensor, "area": mk.A_gamma_m2.tensor}


def _prepare_ib(c, seed):
    gen = _generator(seed)
    fl = _fluid(c, 1.0e-3)
    mesh = make_uv_sphere(UvSphereResolution(c["bands"], 2 * c["bands"]), 0.18)
    shift = (torch.rand(3, generator=gen, device="cuda") * 0.04 - 0.02).cpu().numpy() + 0.5
    n = mesh.vertices / 0.18
    speed = (0.05 * torch.randn(mesh.vertices.shape, generator=gen, device="cuda")).cpu().numpy()
    mk = HibmMpmSurfaceMarkers(marker_capacity=mesh.vertex_count, projection_triangle_capacity=mesh.face_count)
    mk.load_markers(positions_m=(mesh.vertices + shift).tolist(), velocities_mps=speed.tolist(), normals=n.tolist(),
                    areas_m2=[1.0e-4] * mesh.vertex_count, region_ids=[REGION] * mesh.vertex_count)
    mk.set_projection_triangles(mesh.faces.tolist())
    g = fl.grid
    search = HibmMpmIbNodeSearch(grid_nodes=g.grid_nodes, bounds_min_m=g.bounds_min_m, bounds_max_m=g.bounds_max_m,
                                 marker_capacity=mk.marker_capacity)
    rows = HibmMpmIbBoundaryConditions(grid_nodes=g.grid_nodes, marker_capacity=mk.marker_capacity)
    fl.velocity.from_torch(_wave_field(_centres(fl), gen, 0.1))
    radius = 2.0 * min(min(g._widths(a)) for a in range(3))
    grad = torch.zeros(mk.marker_capacity, dtype=torch.float32, device="cuda")
    return {"fluid": fl, "markers": mk, "search": search, "rows": rows, "radius": radius, "grad": grad}


def _run_ib(s):
    fl, mk, search, rows = s["fluid"], s["markers"], s["search"], s["rows"]
    axes = dict(cell_center_x_m=fl.cell_center_x_m, cell_center_y_m=fl.cell_center_y_m,
                cell_center_z_m=fl.cell_center_z_m)
    fl.clear_velocity_dirichlet_boundary_rows()
    search.reset_node_anchor_cells()
    search.search_and_classify_grid_fields(mk, search_radius_m=s["radius"], interior_probe_distance_m=s["radius"],
                                           classify_far_internal_nodes=True, **axes)
    rows.build_from_search_device_fields(search, mk, marker_pressure_neumann_gradient_pa_per_m_field=s["grad"])
    rows.assemble_velocity_dirichlet_reconstructed_boundary_rows(
        fl.velocity_dirichlet_boundary_active, fl.velocity_dirichlet_boundary_value_mps,
        fl.velocity_dirichlet_boundary_projection_weight, fl.obstacle, fl.velocity, search,
        cell_face_x_m=fl.cell_face_x_m, cell_face_y_m=fl.cell_face_y_m, cell_face_z_m=fl.cell_face_z_m,
        grid_nodes=fl.grid.grid_nodes, **axes)
    return {"kind": search.node_kind_code.tensor, "nearest": search.nearest_marker.tensor,
            "distance": search.node_signed_distance_m.tensor, "point": search.node_boundary_point_m.tensor,
            "probe": search.node_interior_fluid_point_m.tensor,
            "active": fl.velocity_dirichlet_boundary_active.tensor,
            "value": fl.velocity_dirichlet_boundary_value_mps.tensor,
            "weight": fl.velocity_dirichlet_boundary_projection_weight.tensor}


def _prepare_shell(c, seed):
    gen = _generator(seed)
    mesh, region = make_plate_mesh(c["nu"], c["nv"], seed=seed)
    st = TriMooneyShellMpmState(mesh, thickness_m=2.0e-3, density_kgm3=1000.0, c1_pa=1.0e5, c2_pa=2.0e4,
                                grid_nodes=(c["nodes"],) * 3, face_region_id=region, primary_region_id=1,
                                secondary_region_id=2, fixed_region_id=3)
    # a stretched, moving membrane (at rest its strains are below f32)
    stretch = torch.tensor([1.05, 1.05, 1.0], device="cuda")
    st.x.tensor.mul_(stretch)
    st.v.from_torch(_wave_field(_points(st.x.tensor), gen, 0.02))
    return {"shell": st}


def _run_shell(s):
    st = s["shell"]
    st.step(dt_s=1.0e-5, pressure_pa=5.0, velocity_damping=0.999, read_report=False)
    return {"x": st.x.tensor, "v": st.v.tensor, "force": st.internal_force_n.tensor, "normal": st.surface_normal.tensor}


def _network(gen):
    net = UNetPreconditioner(seed=0)
    p = np.zeros(net.param_count, np.float32)
    for layer in net.layer_layout():
        w0, b0, nw = layer["weight_offset"], layer["bias_offset"], layer["cout"] * 27 * layer["cin"]
        scale = math.sqrt(2.0 / (27 * layer["cin"]))
        p[w0 : w0 + nw] = (torch.randn(nw, generator=gen, device="cuda") * scale).cpu().numpy()
        p[b0 : b0 + layer["cout"]] = (0.05 * torch.randn(layer["cout"], generator=gen, device="cuda")).cpu().numpy()
    net.set_parameters(p)
    return net, p


def _encoded(shape, gen):
    """The network's input encoding: a unit-RMS residual, the fluid mask and
    the log cell widths, the other channels zero."""
    x = torch.zeros(shape + (16,), dtype=torch.float32, device="cuda")
    mask = (torch.rand(shape, generator=gen, device="cuda") < 0.95).float()
    x[..., 0] = torch.randn(shape, generator=gen, device="cuda") * mask
    x[..., 1] = mask
    for a in range(3):
        width = torch.linspace(-1.0, 1.0, shape[a], device="cuda").abs() * 2.0
        x[..., 2 + a] = width.reshape([-1 if b == a else 1 for b in range(3)])
    return x.to(torch.bfloat16).contiguous(), mask


def _prepare_unet_forward(c, seed):
    gen = _generator(seed)
    net, p = _network(gen)
    x, _ = _encoded((c["nx"], c["ny"], c["nz"]), gen)
    return {"net": net, "params": p, "x": x}


def _run_unet_forward(s):
    return s["net"].forward(s["x"])


def _prepare_unet_train(c, seed):
    gen = _generator(seed)
    net, p = _network(gen)
    crops = []
    for _ in range(c["batch"]):
        x, mask = _encoded((c["crop"],) * 3, gen)
        crops.append((x, torch.randn(mask.shape, generator=gen, device="cuda"), mask))
    return {"net": net, "params": p, "crops": crops}


def _run_unet_train(s):
    net = s["net"]
    net.zero_grad()
    losses = [net.accumulate_gradient(x, t, m) for x, t, m in s["crops"]]
    return {"loss": np.asarray(losses), "grad": net.gradients()}


_PREPARE = {"step": _prepare_step, "project": _prepare_project, "predict": _prepare_predict, "mpm": _prepare_mpm,
            "markers": _prepare_markers, "ib": _prepare_ib, "shell": _prepare_shell,
            "unet_forward": _prepare_unet_forward, "unet_train": _prepare_unet_train}
_RUN = {"step": _run_step, "project": _run_project, "predict": _run_predict, "mpm": _run_mpm,
        "markers": _run_markers, "ib": _run_ib, "shell": _run_shell, "unet_forward": _run_unet_forward,
        "unet_train": _run_unet_train}


# ---------------------------------------------------------------------------
# work and tolerance
# ---------------------------------------------------------------------------


def _ball_particles(n, ax, ay, az):
    return 8.0 * 4.0 / 3.0 * math.pi * ax * ay * az * n


def work(case):
    c, kind = case, case["kind"]
    if kind in ("step", "project"):
        n = c["nx"] * c["ny"] * c["nz"]
        # per iteration of the preconditioned CG: the iterate, the residual
        # and the direction read and written, the preconditioned residual
        # written and read, the stencil structure (one byte) read; 32
        # iterations; the velocity read and written.  Operator and smoother:
        # about 20 operations a row, four sweeps, a residual and the operator.
        sweeps = 1 if c.get("precond") == "jacobi" else 6 * 8 / 7
        bytes_ = n * (32 * (8 * 8 + 1) + 24)
        flops = n * 32 * 20.0 * (sweeps + 1)
        if kind == "step":
            p = _ball_particles(c["mx"] * c["my"] * c["mz"], c["ax"], c["ay"], c["az"])
            bytes_ += 216 * p
            flops += 2500 * p
        return {"bytes": bytes_, "flops": flops}
    if kind == "predict":
        n = c["nx"] * c["ny"] * c["nz"]
        return {"bytes": 25.0 * n, "flops": (300.0 if c["scheme"] == "rk2" else 200.0) * n}
    if kind in ("mpm", "markers"):
        p = _ball_particles(c["n"] ** 3, c["radius"], c["radius"], c["radius"])
        if kind == "mpm":
            # particle state read and written; mass, momentum, force of the
            # touched nodes (about one in eight particles) written and read
            return {"bytes": 216.0 * p + 56.0 * p / 8, "flops": 2500.0 * p}
        m = 2.0 * c["bands"] ** 2
        return {"bytes": 64.0 * p + 88.0 * m, "flops": m * 216 * 60.0}
    if kind == "ib":
        n = c["nx"] * c["ny"] * c["nz"]
        return {"bytes": 100.0 * n, "flops": 200.0 * n}
    if kind == "shell":
        v, f, g = (c["nu"] + 1) * (c["nv"] + 1), 2 * c["nu"] * c["nv"], c["nodes"] ** 3
        return {"bytes": 120.0 * v + 16.0 * f + 40.0 * g, "flops": 600.0 * f + 400.0 * v + 20.0 * g}
    layers = ((0, 16, 16), (0, 16, 16), (1, 16, 32), (1, 32, 32), (2, 32, 48), (2, 48, 48), (3, 48, 64), (3, 64, 64),
              (2, 112, 48), (2, 48, 48), (1, 80, 32), (1, 32, 32), (0, 48, 16), (0, 16, 16), (0, 16, 16))
    n = c["nx"] * c["ny"] * c["nz"] if kind == "unet_forward" else c["crop"] ** 3 * c["batch"]
    flops = sum(2.0 * 27 * ci * co * n / 8**lv for lv, ci, co in layers)
    if kind == "unet_forward":
        return {"bytes": 96.0 * n, "flops": flops}
    return {"bytes": 40.0 * n + 2.8e6, "flops": 3.0 * flops}


def tolerance(case):
    return dict(_TOLERANCE[case["kind"]])


_TOLERANCE = {
    # the CG stops at 1e-8; f32 velocities, f32 sums in any order
    "step": {"rel": 1e-5, "max": 1e-2},
    "project": {"rel": 1e-5, "max": 1e-3},
    "predict": {"rel": 1e-6, "max": 1e-4},
    # the affine velocity is 1e-5 off 64 bits (f32 grid coordinates)
    "mpm": {"rel": 5e-5, "max": 5e-3},
    "markers": {"rel": 1e-5, "max": 1e-3},
    # the nearest of equally near triangles is a tie
    "ib": {"rel": 1e-5, "max": 1e-3, "differ": 1e-4},
    "shell": {"rel": 1e-4, "max": 1e-2},
    "unet_forward": {"rel": 1e-2, "max": 0.3},
    "unet_train": {"rel": 2e-2, "max": 0.5},
}


# ---------------------------------------------------------------------------
# 64-bit restatements in plain torch
# ---------------------------------------------------------------------------


def exact(case, seed):
    fn = _EXACT.get(case["kind"])
    return None if fn is None else fn(case, int(seed))


def _axis(t, a):
    return t.double().reshape([-1 if b == a else 1 for b in range(3)])


def _shifted(t, axis, step):
    """t at index + step along axis, the edge value where there is none."""
    n = t.shape[axis]
    idx = (torch.arange(n, device=t.device) + step).clamp(0, n - 1)
    return t.index_select(axis, idx)


def _edge(shape, axis, side):
    m = torch.zeros(shape[axis], dtype=torch.bool, device="cuda")
    m[0 if side < 0 else -1] = True
    return m.reshape([-1 if b == axis else 1 for b in range(3)])


class _Box:
    """Widths, centre distances, open faces and the operator of one domain."""

    def __init__(self, fl, outlet, face_weight):
        self.fluid = fl.obstacle.tensor == 0
        shape = self.fluid.shape
        self.w = [_axis(getattr(fl, f"cell_width_{a}_m").tensor, i) for i, a in enumerate("xyz")]
        self.vol = self.w[0] * self.w[1] * self.w[2]
        self.cd, self.lower, self.upper, self.k_lo, self.k_hi = [], [], [], [], []
        for a, name in enumerate("xyz"):
            cd = _axis(getattr(fl, f"center_distance_{name}_m").tensor, a)
            cd_lo = cd.narrow(a, 0, shape[a])
            cd_hi = cd.narrow(a, 1, shape[a]) if cd.shape[a] > shape[a] else _shifted(cd, a, 1)
            lo = _shifted(self.fluid, a, -1) & ~_edge(shape, a, -1) & self.fluid
            hi = _shifted(self.fluid, a, 1) & ~_edge(shape, a, 1) & self.fluid
            self.cd.append(cd_lo)
            self.lower.append(lo)
            self.upper.append(hi)
            self.k_lo.append(lo * face_weight / (self.w[a] * cd_lo))
            self.k_hi.append(hi * _shifted(face_weight, a, 1) / (self.w[a] * cd_hi))
        den = sum(self.k_lo) + sum(self.k_hi)
        self.outlet = outlet
        if outlet:
            den = den + _edge(shape, 2, -1) * self.fluid * (2.0 / self.w[2] ** 2)
        self.den = den

    def apply(self, p):
        out = self.den * p
        for a in range(3):
            out = out - self.k_lo[a] * _shifted(p, a, -1) - self.k_hi[a] * _shifted(p, a, 1)
        return out

    def mean(self, f):
        return (f * self.vol * self.fluid).sum() / (self.vol * self.fluid).sum()

    def solve(self, b, closed):
        """CG on the volume-weighted (symmetric) system with the diagonal."""
        act = self.den > 0
        if closed:
            b = (b - self.mean(b)) * self.fluid
        v = self.vol
        inv = torch.where(act, 1.0 / torch.where(act, self.den, 1.0), 0.0)
        x = torch.zeros_like(b)
        r = b * act
        z = r * inv
        d = z.clone()
        rz = (r * z * v).sum()
        stop = 1e-13 * math.sqrt(float((r * r * v).sum()))
        for it in range(20000):
            q = self.apply(d) * act
            alpha = rz / (d * q * v).sum()
            x += alpha * d
            r -= alpha * q
            if it % 50 == 49 and math.sqrt(float((r * r * v).sum())) <= stop:
                break
            z = r * inv
            new = (r * z * v).sum()
            d = z + (new / rz) * d
            rz = new
        if closed:
            x = (x - self.mean(x)) * self.fluid
        return x


def _exact_project(c, seed):
    s = _prepare_project(c, seed)
    fl, rows = s["fluid"], c["rows"]
    u = s["velocity"].double()
    shape = u.shape[:3]
    active = fl.velocity_dirichlet_boundary_active.tensor != 0
    weight = torch.where(active, fl.velocity_dirichlet_boundary_projection_weight.tensor.double().clamp(0, 1), 1.0)
    value = fl.velocity_dirichlet_boundary_value_mps.tensor.double()
    box = _Box(fl, c["outlet"], weight)
    fixed = (active & box.fluid)[..., None]

    def no_flow():
        for a in range(3):
            if a < 2 or not c["outlet"]:
                u[..., a] = torch.where(_edge(shape, a, -1), 0.0, u[..., a])

    def boundary():
        if rows:
            u[:] = torch.where(fixed, value, u)
        if c["outlet"]:
            back = _edge(shape, 2, -1) & box.fluid & (u[..., 2] > 0)
            u[..., 2] = torch.where(back, 0.0, u[..., 2])
            no_flow()

    boundary()
    div = torch.zeros(shape, dtype=torch.float64, device="cuda")
    for a in range(3):
        lo = u[..., a] * box.lower[a]
        if a == 2 and c["outlet"]:
            lo = torch.where(_edge(shape, 2, -1) & box.fluid, u[..., 2], lo)
        div += (_shifted(u[..., a], a, 1) * box.upper[a] - lo) / box.w[a]
    dt = 1.0e-3
    p = box.solve(-(DENSITY / dt) * div * box.fluid, not c["outlet"])
    for a in range(3):
        g = (p - _shifted(p, a, -1)) / box.cd[a] * box.lower[a]
        if a == 2 and c["outlet"]:
            g = torch.where(_edge(shape, 2, -1) & box.fluid, 2.0 * p / box.w[2], g)
        u[..., a] -= weight * (dt / DENSITY) * g
    u *= box.fluid[..., None]
    boundary()
    if not c["outlet"]:
        no_flow()
    return {"velocity": u, "pressure": p}


def _exact_predict(c, seed):
    s = _prepare_predict(c, seed)
    fl = s["fluid"]
    u = fl.velocity.tensor.double()
    n = u.shape[:3]
    box = _Box(fl, False, torch.ones(n, dtype=torch.float64, device="cuda"))
    centres = [getattr(fl, f"cell_center_{a}_m").tensor.double() for a in "xyz"]
    flat = u.reshape(-1, 3)
    wet = box.fluid.reshape(-1)

    def sample(pos):
        i0, t = [], []
        for a in range(3):
            x = centres[a]
            q = pos[a].clamp(x[0], x[-1])
            lo = (torch.searchsorted(x, q.contiguous(), right=True) - 1).clamp(0, n[a] - 2)
            i0.append(lo)
            t.append((q - x[lo]) / (x[lo + 1] - x[lo]))
        num = torch.zeros(pos[0].shape + (3,), dtype=torch.float64, device="cuda")
        den = torch.zeros(pos[0].shape, dtype=torch.float64, device="cuda")
        for o in range(8):
            b = (o >> 2, (o >> 1) & 1, o & 1)
            w = torch.ones_like(den)
            for a in range(3):
                w = w * (t[a] if b[a] else 1.0 - t[a])
            at = ((i0[0] + b[0]) * n[1] + i0[1] + b[1]) * n[2] + i0[2] + b[2]
            w = w * wet[at]
            num += w[..., None] * flat[at]
            den += w
        ok = den > 1e-12
        return torch.where(ok[..., None], num / torch.where(ok, den, 1.0)[..., None], u_part)

    dt, nu = 1.0e-3, VISCOSITY / DENSITY
    out = torch.empty_like(u)
    chunk = max(1, 4_000_000 // (n[1] * n[2]))
    for i in range(0, n[0], chunk):
        u_part = u[i : i + chunk]
        base = [centres[0][i : i + chunk, None, None], centres[1][None, :, None], centres[2][None, None, :]]
        tr = u_part
        if c["scheme"] == "rk2":
            tr = sample([base[a] - 0.5 * dt * u_part[..., a] for a in range(3)])
        out[i : i + chunk] = sample([base[a] - dt * tr[..., a] for a in range(3)])
    lap = torch.zeros_like(u)
    for a in range(3):
        cd_hi = _shifted(box.cd[a], a, 1)
        back = (u - _shifted(u, a, -1)) / box.cd[a][..., None] * box.lower[a][..., None]
        fwd = (_shifted(u, a, 1) - u) / cd_hi[..., None] * box.upper[a][..., None]
        lap += (fwd - back) / box.w[a][..., None]
    return (out + dt * nu * lap) * box.fluid[..., None]


def _exact_mpm(c, seed):
    s = _prepare_mpm(c, seed)
    so, dt, mu, lam = s["solid"], s["dt"], s["mu"], s["lam"]
    n = c["n"]
    h = 1.0 / n
    x, v, C, F = (f.tensor.double() for f in (so.x, so.v, so.C, so.F))
    mass, vol, fe = so.mass_kg.tensor.double(), so.volume_m3.tensor.double(), so.external_force_n.tensor.double()
    X = x / h
    base = torch.floor(X - 0.5)
    fx = X - base
    w = torch.stack([0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1.0) ** 2, 0.5 * (fx - 0.5) ** 2], dim=0)
    base = base.long()
    J = torch.linalg.det(F)
    Fit = torch.linalg.inv(F).transpose(1, 2)
    P = mu * (F - Fit) + lam * torch.log(J)[:, None, None] * Fit
    aff = -dt * vol[:, None, None] * (P @ F.transpose(1, 2)) * (4.0 / h**2) + mass[:, None, None] * C
    node = torch.zeros((n**3, 7), dtype=torch.float64, device="cuda")
    offsets = [(a, b, d) for a in range(3) for b in range(3) for d in range(3)]

    def stencil(o):
        wt = w[o[0], :, 0] * w[o[1], :, 1] * w[o[2], :, 2]
        d = (torch.tensor(o, device="cuda", dtype=torch.float64) - fx) * h
        at = ((base[:, 0] + o[0]) * n + base[:, 1] + o[1]) * n + base[:, 2] + o[2]
        return wt, d, at

    for o in offsets:
        wt, d, at = stencil(o)
        mom = mass[:, None] * v + torch.einsum("pij,pj->pi", aff, d)
        node.index_add_(0, at, wt[:, None] * torch.cat([mass[:, None], mom, fe], dim=1))
    m = node[:, 0].clamp_min(1e-300)
    gv = torch.where((node[:, 0] > 1e-20)[:, None], (node[:, 1:4] + dt * node[:, 4:7]) / m[:, None], 0.0) * 0.999
    nv, nC = torch.zeros_like(v), torch.zeros_like(C)
    for o in offsets:
        wt, d, at = stencil(o)
        g = wt[:, None] * gv[at]
        nv += g
        nC += g[:, :, None] * (4.0 / h**2 * d)[:, None, :]
    x2 = x + dt * nv
    F2 = F + dt * nC @ F
    ra, rn = so.rest_area_weight_m2.tensor.double(), so.rest_surface_normal.tensor.double()
    J2 = torch.linalg.det(F2)
    av = torch.einsum("pij,pj->pi", torch.linalg.inv(F2).transpose(1, 2) * J2[:, None, None], rn)
    return {"x": x2, "v": nv, "C": nC, "F": F2, "area": torch.where(ra > 0, ra * av.norm(dim=1), ra)}


def _exact_markers(c, seed):
    s = _prepare_markers(c, seed)
    so, mk, R = s["solid"], s["markers"], s["radius"]
    xp, vp = so.x.tensor.double(), so.v.tensor.double()
    npart, ap = so.surface_normal.tensor.double(), so.area_weight_m2.tensor.double()
    skin = (npart.norm(dim=1) > 1e-12) & (ap > 0)
    fext = torch.zeros_like(xp)
    xm, Fm = mk.x_gamma_m.tensor.double(), mk.F_gamma_n.tensor
    v2, n2, a2 = torch.zeros_like(xm), mk.n_gamma.tensor.double().clone(), mk.A_gamma_m2.tensor.double().clone()
    x2 = xm.clone()
    step = max(1, 20_000_000 // xp.shape[0])
    for i in range(0, xm.shape[0], step):
        q = slice(i, i + step)
        w = torch.ones((xm[q].shape[0], xp.shape[0]), dtype=torch.float64, device="cuda")
        for a in range(3):
            w *= (1.0 - (xm[q, a, None] - xp[None, :, a]).abs() / R).clamp_min(0.0)
        ws = w.sum(dim=1)
        ok = ws > 1e-12
        fext += (w / ws.clamp_min(1e-300)[:, None] * ok[:, None]).T @ Fm[q]
        vel = w @ vp / ws.clamp_min(1e-300)[:, None]
        v2[q] = torch.where(ok[:, None], vel, v2[q])
        x2[q] = torch.where(ok[:, None], xm[q] + 1.0e-4 * vel, xm[q])
        wg = w * skin[None, :]
        gs, nn = wg.sum(dim=1), wg @ npart
        good = ok & (gs > 1e-12) & (nn.norm(dim=1) > 1e-12)
        n2[q] = torch.where(good[:, None], nn / nn.norm(dim=1).clamp_min(1e-300)[:, None], n2[q])
        a2[q] = torch.where(good, wg @ ap / gs.clamp_min(1e-300), a2[q])
    return {"force": fext, "x": x2, "v": v2, "n": n2, "area": a2}


def _unet64(params, layout, x):
    """The network in 64 bits: x (nx, ny, nz, 16) -> (nx, ny, nz, 16)."""
    import torch.nn.functional as nnf

    def conv(h, l):
        q = layout[l]
        nw = q["cout"] * 27 * q["cin"]
        w = params[q["weight_offset"] : q["weight_offset"] + nw].reshape(q["cout"], 3, 3, 3, q["cin"])
        b = params[q["bias_offset"] : q["bias_offset"] + q["cout"]]
        shape = h.shape[2:]
        pad = nnf.pad(h, (1, 1, 1, 1, 1, 1))
        y = b.reshape(1, -1, 1, 1, 1)
        for t in range(27):
            i, j, k = t // 9, (t // 3) % 3, t % 3
            part = pad[:, :, i : i + shape[0], j : j + shape[1], k : k + shape[2]]
            y = y + torch.einsum("oc,bcijk->boijk", w[:, i, j, k, :], part)
        return torch.relu(y) if q["relu"] else y

    def pool(h):
        return nnf.avg_pool3d(h, 2, ceil_mode=True, count_include_pad=False)

    def up(h, shape):
        for a in range(3):
            h = h.index_select(2 + a, torch.arange(shape[a], device=h.device) // 2)
        return h

    h = x.permute(3, 0, 1, 2)[None]
    skips = []
    for lv in range(4):
        h = conv(conv(h if lv == 0 else pool(h), 2 * lv), 2 * lv + 1)
        skips.append(h)
    for q in range(3):
        lv = 2 - q
        h = torch.cat([up(h, skips[lv].shape[2:]), skips[lv]], dim=1)
        h = conv(conv(h, 8 + 2 * q), 9 + 2 * q)
    return conv(h, 14)[0].permute(1, 2, 3, 0)


def _exact_unet_forward(c, seed):
    s = _prepare_unet_forward(c, seed)
    params = torch.as_tensor(s["params"], device="cuda").double()
    with torch.no_grad():
        return _unet64(params, s["net"].layer_layout(), s["x"].double())


def _exact_unet_train(c, seed):
    s = _prepare_unet_train(c, seed)
    params = torch.as_tensor(s["params"], device="cuda").double().requires_grad_(True)
    losses = []
    for x, target, mask in s["crops"]:
        out = _unet64(params, s["net"].layer_layout(), x.double())[..., 0]
        loss = ((mask.double() * (out - target.double())) ** 2).mean()
        loss.backward()
        losses.append(float(loss))
    return {"loss": np.asarray(losses), "grad": params.grad.cpu().numpy()}


_EXACT = {"project": _exact_project, "predict": _exact_predict, "mpm": _exact_mpm, "markers": _exact_markers,
          "unet_forward": _exact_unet_forward, "unet_train": _exact_unet_train}
