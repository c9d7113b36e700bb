"""Performance cases of the joint LM path: what a user of the library has it do, over the range of sizes,
options and entry points in which it is used.

A case is a dict of plain values. ``kind`` names the entry point:

* ``solve``       -- a kept ``Problem`` handle (its device state and symbolic analysis are there), one call
                     per pass: set the start state, ``solve`` some LM iterations, read the state back;
* ``batch``       -- the same with several uneven problems in one handle;
* ``cold``        -- the whole call on new host data: handle, upload, analysis, ``solve``, state, close;
* ``incremental`` -- ``run_incremental_scene``: frames appended one at a time, some iterations each;
* ``serve``       -- a kept ``Server``: a burst of requests submitted, drained and polled;
* ``ldlt``        -- a kept ``LdltSolver`` (the factor-only interface): new values factorized, one solve.

``scene`` is one of the generators of ``sdf_slam_b200.scenes`` (room, floorplan, office); the other values are
its sizes and the problem's and solver's options.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch


def _package():
    """The package (directory sdf-slam_b200, imported as sdf_slam_b200)."""
    if "sdf_slam_b200" not in sys.modules:
        root = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sdf-slam_b200")
        spec = importlib.util.spec_from_file_location("sdf_slam_b200", os.path.join(root, "__init__.py"),
                                                      submodule_search_locations=[root])
        module = importlib.util.module_from_spec(spec)
        sys.modules["sdf_slam_b200"] = module
        spec.loader.exec_module(module)
    return sys.modules["sdf_slam_b200"]


P = _package()
import sdf_slam_b200.scenes as scenes  # noqa: E402

# Defaults of what a case does not say: the library's own (dense state, no Huber loss, smooth gradients, fixed
# damping, FP64).
_DEFAULTS = dict(active=False, huber=0.0, gradient="smooth", lm="fixed", precision="fp64", refine_tolerance=1e-13)


def listed():
    room = dict(scene="room", grid=40, frames=10, beams=180)
    floor = dict(scene="floorplan", grid=100, frames=76, beams=360)
    office = dict(scene="office", grid=200, frames=910, beams=180)
    return [
        # the smallest workload: a ten-pose room; an iteration is launches and dependent small fronts
        dict(name="room-10", kind="solve", iterations=10, **room),
        # a ragged small problem under the options that change the path: active-region state, Huber loss, exact
        # patch gradients, trust region with steps taken back
        dict(name="room-23-options", kind="solve", iterations=8, scene="room", grid=57, frames=23, beams=131,
             active=True, huber=0.5, gradient="exact", lm="trust"),
        # the ordinary batch solve: one floor of a building
        dict(name="floorplan-76", kind="solve", iterations=10, **floor),
        # the same in mixed precision at the default refinement tolerance
        dict(name="floorplan-76-mixed", kind="solve", iterations=10, precision="mixed", **floor),
        # the largest: three laps through an office, the workload of the benchmark
        dict(name="office-910", kind="solve", iterations=5, **office),
        dict(name="office-910-mixed", kind="solve", iterations=5, precision="mixed", refine_tolerance=1e-6, **office),
        # a middle size between floor plan and office, with many poses that see the same walls
        dict(name="room-331", kind="solve", iterations=5, scene="room", grid=143, frames=331, beams=180),
        # many independent uneven problems solved together (half of them with an active-region state)
        dict(name="batch-32", kind="batch", iterations=5, instances=32, grid=150, frames=200, beams=360),
        # a program that solves one problem and ends: host arrays in, state out
        dict(name="cold-floorplan-76", kind="cold", iterations=10, **floor),
        # a robot adding scans one by one
        dict(name="incremental-24", kind="incremental", iterations=5, scene="room", grid=60, frames=24, beams=180),
        # a burst of mixed-size requests at the server
        dict(name="serve-12", kind="serve", iterations=10, instances=12, grid=120, frames=120, beams=180),
        # the factor-only interface on a floor plan's damped normal matrix
        dict(name="ldlt-floorplan-76", kind="ldlt", **floor),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_scene(rng):
    scene = rng.choice(["room", "room", "floorplan", "office"])
    if scene == "room":
        return dict(scene=scene, grid=_log_int(rng, 40, 200), frames=_log_int(rng, 10, 400), beams=rng.randint(90, 180))
    if scene == "floorplan":
        return dict(scene=scene, grid=rng.randint(70, 140), frames=_log_int(rng, 30, 200), beams=rng.randint(180, 360))
    return dict(scene=scene, grid=rng.randint(150, 200), frames=_log_int(rng, 300, 910), beams=rng.randint(90, 180))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "batch", "cold", "incremental", "serve", "ldlt"])
    case = dict(kind=kind)
    if kind in ("solve", "cold"):
        case.update(_draw_scene(rng), iterations=rng.randint(2, 5), active=rng.random() < 0.25,
                    huber=rng.choice([0.0, 0.0, 0.5]), gradient=rng.choice(["smooth", "smooth", "meters", "exact"]),
                    lm=rng.choice(["fixed", "fixed", "factor", "reject", "trust"]))
        if rng.random() < 0.3:
            case.update(precision="mixed", refine_tolerance=rng.choice([1e-13, 1e-6]))
    elif kind == "batch":
        case.update(instances=_log_int(rng, 2, 32), grid=rng.randint(50, 150), frames=rng.randint(20, 200),
                    beams=rng.randint(90, 360), iterations=rng.randint(2, 5))
        if rng.random() < 0.3:
            case.update(precision="mixed", refine_tolerance=1e-6)
    elif kind == "incremental":
        case.update(scene="room", grid=rng.randint(40, 70), frames=rng.randint(6, 24), beams=rng.randint(90, 180),
                    iterations=rng.randint(2, 5))
    elif kind == "serve":
        case.update(instances=rng.randint(2, 12), grid=rng.randint(50, 120), frames=rng.randint(20, 120),
                    beams=rng.randint(90, 180), iterations=rng.randint(5, 10))
    else:
        case.update(scene="floorplan", grid=rng.randint(60, 100), frames=rng.randint(20, 76), beams=rng.randint(180, 360))
    return case


# ------------------------------------------------------------------ inputs --

def _scene(case, seed):
    if case["scene"] == "room":
        g = case["grid"]
        return scenes.room_scene(seed=seed, grid=g, frames=case["frames"], beams=case["beams"],
                                 max_range=min(30.0, 0.1 * g + 4))
    build = scenes.floorplan_scene if case["scene"] == "floorplan" else scenes.office_scene
    return build(seed=seed, grid=case["grid"], frames=case["frames"], beams=case["beams"])


def _members(case, seed):
    """The scenes of a batch or a burst: sizes log-uniform up to the case's, the first at them. The sizes
    are the case's (they belong to its plan), the worlds the seed's."""
    sizes = np.random.default_rng([case["instances"], case["grid"], case["frames"]])
    out = []
    for i in range(case["instances"]):
        u, v, w = (sizes.uniform() if i else 1.0 for _ in range(3))
        out.append(dict(case, scene="room", grid=int(round(40 * (case["grid"] / 40) ** u)),
                        frames=int(round(10 * (case["frames"] / 10) ** v)),
                        beams=int(round(90 + w * (case["beams"] - 90))),
                        active=case["kind"] == "batch" and i % 2 == 1))
    return [(c, _scene(c, seed * 64 + i)) for i, c in enumerate(out)]


def _problem_options(case):
    c = {**_DEFAULTS, **case}
    return P.ProblemOptions(active_region=c["active"], huber_delta=c["huber"], smooth_gradient=c["gradient"] != "exact",
                            smooth_gradient_step=0.1 if c["gradient"] == "meters" else 0.0)


def _solver_options(case):
    c = {**_DEFAULTS, **case}
    return P.SolverOptions(max_iterations=c["iterations"], step_tolerance=1e-9, precision=c["precision"],
                           refine_tolerance=c["refine_tolerance"], lambda_factor=2.0 if c["lm"] in ("factor", "reject") else 1.0,
                           reject_worse_steps=c["lm"] == "reject", trust_region=c["lm"] == "trust",
                           marquardt_scaling=c["lm"] == "factor")


def _specs(case, scene):
    """The scene's problem as flat arrays (built on the host): what a caller with its own Problem holds."""
    o = _problem_options(case)
    with P.Problem.from_scene(scene, o) as problem:
        return problem.specs(min_corner=scene.min_corner, max_corner=scene.max_corner, huber_delta=o.huber_delta,
                             smooth_gradient=o.smooth_gradient, smooth_gradient_step=o.smooth_gradient_step)


def _all_specs(case, seed):
    if case["kind"] in ("batch", "serve"):
        return [_specs(c, s) for c, s in _members(case, seed)]
    return [_specs(case, _scene(case, seed))]


def _dissect(w0, h0, w, h, out):
    """Nested dissection of a block of grid nodes (nodes of a nine-point stencil), separators last."""
    if w * h <= 16:
        out.extend((x, y) for y in range(h0, h0 + h) for x in range(w0, w0 + w))
    elif w >= h:
        m = w // 2
        _dissect(w0, h0, m, h, out)
        _dissect(w0 + m + 1, h0, w - m - 1, h, out)
        out.extend((w0 + m, y) for y in range(h0, h0 + h))
    else:
        m = h // 2
        _dissect(w0, h0, w, m, out)
        _dissect(w0, h0 + m + 1, w, h - m - 1, out)
        out.extend((x, h0 + m) for x in range(w0, w0 + w))


def _normal_matrix(case, seed):
    """The damped normal matrix of a floor plan whose map holds the distance to the nearest wall point."""
    specs = _all_specs(case, seed)[0]
    ref = _Reference(specs)
    xy, _ = ref.world(ref.poses)
    xy = xy[specs.pt_expected == 0.0]  # the scan points
    h, w = np.divmod(np.arange(specs.nx * specs.ny), specs.nx)
    nodes = torch.as_tensor(np.stack([specs.min_corner[0] + w * ref.dx, specs.min_corner[1] + h * ref.dy], 1), device=ref.device)
    ref.map = torch.cat([torch.cdist(block, xy).amin(1) for block in nodes.split(1024)]).clamp(max=1.0)
    A, rhs, _ = ref.normal()
    A.diagonal().add_(1.0)
    # 24 bits of every value: the order in which the sums were taken does not reach the inputs
    A, rhs = A.float().double(), rhs.float().double()
    return specs, A, rhs


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "batch"):
        options = _solver_options(case)
        if kind == "solve":
            scene = _scene(case, seed)
            problem = P.Problem.from_scene(scene, _problem_options(case))
        else:
            problem = P.Problem.batch(_all_specs(case, seed))
        start = [problem.state(i) for i in range(problem.count)]
        problem.cost()
        return dict(kind=kind, problem=problem, options=options, start=start)
    if kind == "cold":
        return dict(kind=kind, specs=_all_specs(case, seed)[0], options=_solver_options(case))
    if kind == "incremental":
        return dict(kind=kind, scene=_scene(case, seed), options=_problem_options(case), iterations=case["iterations"])
    if kind == "serve":
        return dict(kind=kind, specs=_all_specs(case, seed), options=_solver_options(case), server=P.Server(8 << 30, 64))
    specs, A, rhs = _normal_matrix(case, seed)
    n = A.shape[0]
    cols, rows = torch.nonzero(A, as_tuple=True)  # A is symmetric: its rows are its columns
    outer = torch.searchsorted(cols, torch.arange(n + 1, device=A.device)).to(torch.int32).cpu().numpy()
    order = []
    _dissect(0, 0, specs.nx, specs.ny, order)
    perm = [y * specs.nx + x for x, y in order] + list(range(specs.nx * specs.ny, n))
    solver = P.LdltSolver(n, outer, rows.to(torch.int32).cpu().numpy(), perm)
    return dict(kind=kind, solver=solver, values=A[cols, rows].cpu().numpy(), rhs=rhs.cpu().numpy())


def _answer(result, state):
    return dict(map=state[0], poses=state[1], cost=np.array(result.cost_history), iterations=result.iterations)


def run(state):
    kind = state["kind"]
    if kind in ("solve", "batch"):
        problem = state["problem"]
        for i, (m, p) in enumerate(state["start"]):
            problem.set_state(m, p, i)
        results = P.solve(problem, state["options"])
        if kind == "solve":
            return _answer(results, problem.state())
        states = [problem.state(i) for i in range(problem.count)]
        return dict(map=np.concatenate([m for m, _ in states]), poses=np.concatenate([p for _, p in states]),
                    cost=np.array([r.cost_history for r in results]))
    if kind == "cold":
        with P.Problem.from_specs(state["specs"]) as problem:
            result = P.solve(problem, state["options"])
            return _answer(result, problem.state())
    if kind == "incremental":
        r = P.run_incremental_scene(state["scene"], state["options"], solver=P.SolverOptions(step_tolerance=1e-9),
                                    iterations_per_increment=state["iterations"])
        return _answer(r.result, (r.map_values, r.poses))
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(s, state["options"]) for s in state["specs"]]
        server.drain()
        done = [server.poll(i, s.nx * s.ny, len(s.poses)) for i, s in zip(ids, state["specs"])]
        return dict(map=np.concatenate([m for _, m, _ in done]), poses=np.concatenate([p for _, _, p in done]),
                    cost=np.array([r.final_cost for r, _, _ in done]))
    state["solver"].factorize(state["values"])
    return state["solver"].solve(state["rhs"])


# -------------------------------------------------------------------- work --

def work(case):
    """Bytes: the specs and the start state in, the state out, and per iteration the specs again (they do not
    fit on the chip at the larger sizes). Flops: per iteration 70 for each point row's products, the
    elimination of the grid (nested dissection of a g x g grid, 10 g^3, and the square of every node's coupled
    pose columns) and of the dense pose block (a third of its cube)."""
    specs = _all_specs(case, 0)
    iterations = case.get("iterations", 1)
    bytes_, flops = 0.0, 0.0
    for s in specs:
        ref = _Reference(s)
        poses = 3.0 * (ref.frames - 1)
        coupled = ref.couplings() * 3.0
        per = 10.0 * (s.nx * s.ny) ** 1.5 + float((coupled ** 2).sum()) + poses ** 3 / 3
        state = 8.0 * (s.nx * s.ny + 3 * ref.frames)
        if case["kind"] == "ldlt":
            # the values of the full matrix (grid stencil and couplings, both triangles), the two vectors
            bytes_ += 8.0 * (9.0 * s.nx * s.ny + 2 * float(coupled.sum()) + 2 * (s.nx * s.ny + poses))
            flops += per
            continue
        # frames appended one by one: step t has t frames of F, so sums over t of t/F and of (t/F)^3 (or ^2)
        F = ref.frames
        rows, cubes = (F / 2.0, F / 4.0) if case["kind"] == "incremental" else (1.0, 1.0)
        bytes_ += 2 * state + iterations * rows * (36.0 * len(s.pt_frame) + 36.0 * len(s.eik_sqrtw))
        flops += iterations * (rows * 70.0 * len(s.pt_frame) + cubes * per)
    return dict(bytes=bytes_, flops=flops)


# ------------------------------------------------------------------- exact --

class _Reference:
    """The LM iteration of one problem in plain FP64 torch: residuals and Jacobian rows, a dense normal
    matrix, a dense Cholesky solve, and the damping rules."""

    def __init__(self, s):
        self.device = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a, d=torch.float64: torch.as_tensor(np.ascontiguousarray(a), device=self.device).to(d)  # noqa: E731
        self.s, self.nx, self.ny = s, s.nx, s.ny
        self.min = s.min_corner
        self.dx = (s.max_corner[0] - s.min_corner[0]) / (s.nx - 1)
        self.dy = (s.max_corner[1] - s.min_corner[1]) / (s.ny - 1)
        self.frame, self.xy = t(s.pt_frame, torch.int64), t(s.pt_xy)
        self.expected, self.sw = t(s.pt_expected), t(s.pt_sqrtw)
        self.eik_node = t(s.eik_wh[:, 1].astype(np.int64) * s.nx + s.eik_wh[:, 0], torch.int64)
        self.eik_n, self.eik_sw = t(s.eik_n), t(s.eik_sqrtw)
        self.odom, self.meas, self.odom_sw = t(s.odom_ij, torch.int64), t(s.odom_meas), t(s.odom_sqrtw)
        self.column = t(s.node_to_active, torch.int64)
        self.frames = len(s.poses)
        self.active = int((s.node_to_active >= 0).sum())
        self.n = self.active + 3 * (self.frames - 1)
        self.map, self.poses = t(s.map_values), np.array(s.poses, np.float64).reshape(-1, 3)

    def world(self, poses):
        cs = torch.as_tensor(np.stack([np.cos(poses[:, 2]), np.sin(poses[:, 2])], 1), device=self.device)
        p = torch.as_tensor(poses, device=self.device)[self.frame]
        c, s = cs[self.frame, 0], cs[self.frame, 1]
        x, y = self.xy[:, 0], self.xy[:, 1]
        world = torch.stack([(c * x + (-s) * y) + p[:, 0], (s * x + c * y) + p[:, 1]], 1)
        return world, torch.stack([(-s) * x - c * y, c * x - s * y], 1)

    def _cells(self, xy, clamp=False):
        fx, fy = (xy[:, 0] - self.min[0]) / self.dx, (xy[:, 1] - self.min[1]) / self.dy
        inside = (fx >= 0) & (fy >= 0) & (fx <= self.nx - 1) & (fy <= self.ny - 1)
        w = fx.clamp(0, self.nx - 2).long()
        h = fy.clamp(0, self.ny - 2).long()
        a, b = fx - w, fy - h
        if not clamp:
            a, b = torch.where(inside, a, 0.0), torch.where(inside, b, 0.0)
        weights = torch.stack([(1 - a) * (1 - b), a * (1 - b), (1 - a) * b, a * b], 1)
        node = h * self.nx + w
        return inside, w, h, torch.stack([node, node + 1, node + self.nx, node + self.nx + 1], 1), weights

    def couplings(self):
        """Frames (other than the fixed one) that each node's rows couple it with, at the start."""
        inside, _, _, nodes, _ = self._cells(self.world(self.poses)[0])
        keep = inside & (self.frame > 0)
        pairs = torch.unique((self.frame[keep, None] * (self.nx * self.ny) + nodes[keep]).flatten())
        return torch.bincount(pairs % (self.nx * self.ny), minlength=self.nx * self.ny).double()

    def _gradient(self, xy, w, h, nodes, weights):
        s, m = self.s, self.map
        if s.smooth_gradient and s.smooth_gradient_step > 0:
            st, out = s.smooth_gradient_step, []
            for axis in (0, 1):
                v = []
                for sign in (st, -st):
                    at = xy.clone()
                    at[:, axis] += sign
                    _, _, _, nd, wt = self._cells(at, clamp=True)
                    v.append((wt * m[nd]).sum(1))
                out.append((v[0] - v[1]) / (2 * st))
            return torch.stack(out, 1)
        if s.smooth_gradient:
            g = torch.zeros(len(w), 2, device=self.device, dtype=torch.float64)
            for q in range(4):
                ww, hh = w + (q & 1), h + (q >> 1)
                wl, wh = (ww - 1).clamp(min=0), (ww + 1).clamp(max=self.nx - 1)
                hl, hh2 = (hh - 1).clamp(min=0), (hh + 1).clamp(max=self.ny - 1)
                g[:, 0] += weights[:, q] * (m[hh * self.nx + wh] - m[hh * self.nx + wl]) / ((wh - wl).double() * self.dx)
                g[:, 1] += weights[:, q] * (m[hh2 * self.nx + ww] - m[hl * self.nx + ww]) / ((hh2 - hl).double() * self.dy)
            return g
        d = m[nodes]
        a, b = weights[:, 1] + weights[:, 3], weights[:, 2] + weights[:, 3]
        return torch.stack([((1 - b) * (d[:, 1] - d[:, 0]) + b * (d[:, 3] - d[:, 2])) / self.dx,
                            ((1 - a) * (d[:, 2] - d[:, 0]) + a * (d[:, 3] - d[:, 1])) / self.dy], 1)

    def _eikonal(self):
        k = self.eik_node
        gx, gy = (self.map[k + 1] - self.map[k]) / self.dx, (self.map[k + self.nx] - self.map[k]) / self.dy
        return self.eik_sw * (1 - (self.eik_n[:, 0] * gx + self.eik_n[:, 1] * gy))

    def _odometry(self):
        p = torch.as_tensor(self.poses, device=self.device)
        pi, pj = p[self.odom[:, 0]], p[self.odom[:, 1]]
        c, s = torch.cos(pi[:, 2]), torch.sin(pi[:, 2])
        d = pj - pi
        wrap = d[:, 2] - self.meas[:, 2]
        r = torch.stack([c * d[:, 0] + s * d[:, 1] - self.meas[:, 0], -s * d[:, 0] + c * d[:, 1] - self.meas[:, 1],
                         torch.atan2(torch.sin(wrap), torch.cos(wrap))], 1)
        z, one = torch.zeros_like(c), torch.ones_like(c)
        ji = torch.stack([-c, -s, -s * d[:, 0] + c * d[:, 1], s, -c, -c * d[:, 0] - s * d[:, 1], z, z, -one], 1)
        jj = torch.stack([c, s, z, -s, c, z, z, z, one], 1)
        k = self.odom_sw[:, None]
        return k * r, (k * ji).view(-1, 3, 3), (k * jj).view(-1, 3, 3)

    def _pose_columns(self, frame):
        return torch.where(frame[:, None] > 0, self.active + 3 * (frame[:, None] - 1) + torch.arange(3, device=self.device), -1)

    def cost(self):
        inside, _, _, nodes, weights = self._cells(self.world(self.poses)[0])
        r = self.sw * (torch.where(inside, (weights * self.map[nodes]).sum(1), 0.0) - self.expected)
        terms, delta = r * r, self.s.huber_delta
        if delta > 0:
            terms = torch.where(r.abs() > delta, delta * (2 * r.abs() - delta), terms)
        return float(terms.sum() + self._eikonal().square().sum() + self._odometry()[0].square().sum())

    def normal(self):
        """(J^T J as a dense matrix, -J^T r, the diagonal of J^T J)."""
        n = self.n
        A = torch.zeros(n + 1, n + 1, device=self.device, dtype=torch.float64)  # the last one takes constant columns
        g = torch.zeros(n + 1, device=self.device, dtype=torch.float64)
        flat = A.view(-1)

        def add(columns, J, r):
            columns = torch.where(columns < 0, n, columns)
            for c, j, e in zip(columns.split(1 << 18), J.split(1 << 18), r.split(1 << 18)):
                flat.index_add_(0, (c[:, :, None] * (n + 1) + c[:, None, :]).flatten(), (j[:, :, None] * j[:, None, :]).flatten())
                g.index_add_(0, c.flatten(), (j * e[:, None]).flatten())

        xy, turn = self.world(self.poses)
        inside, w, h, nodes, weights = self._cells(xy)
        grad = self._gradient(xy, w, h, nodes, weights)
        r = self.sw * (torch.where(inside, (weights * self.map[nodes]).sum(1), 0.0) - self.expected)
        hw = torch.ones_like(r)
        if self.s.huber_delta > 0:
            hw = torch.where(r.abs() > self.s.huber_delta, self.s.huber_delta / r.abs(), hw).sqrt()
        J = torch.cat([weights, grad, (grad * turn).sum(1, keepdim=True)], 1) * (hw * self.sw)[:, None]
        columns = torch.cat([self.column[nodes], self._pose_columns(self.frame)], 1)
        add(columns[inside], J[inside], (hw * r)[inside])
        k, e = self.eik_node, self.eik_n / torch.tensor([self.dx, self.dy], device=self.device, dtype=torch.float64)
        add(self.column[torch.stack([k, k + 1, k + self.nx], 1)],
            self.eik_sw[:, None] * torch.stack([e[:, 0] + e[:, 1], -e[:, 0], -e[:, 1]], 1), self._eikonal())
        r, ji, jj = self._odometry()
        columns = torch.cat([self._pose_columns(self.odom[:, 0]), self._pose_columns(self.odom[:, 1])], 1)
        for q in range(3):
            add(columns, torch.cat([ji[:, q], jj[:, q]], 1), r[:, q])
        A = A[:n, :n]
        return A, -g[:n], A.diagonal().clone()

    def solve(self, o):
        cost = self.cost()
        history, lam, nu, done = [cost], o.lambda_init, 2.0, 0
        while done < o.max_iterations:
            A, rhs, diagonal = self.normal()
            A.diagonal().add_(lam * diagonal.clamp(min=1e-12) if o.marquardt_scaling else lam)
            step = torch.cholesky_solve(rhs[:, None], torch.linalg.cholesky(A))[:, 0]
            del A
            before = self.map, self.poses
            self.map = torch.where(self.column >= 0, self.map + step[self.column.clamp(min=0)], self.map)
            self.poses = self.poses.copy()
            self.poses[1:] += step[self.active:].view(-1, 3).cpu().numpy()
            self.poses[1:, 2] = np.arctan2(np.sin(self.poses[1:, 2]), np.cos(self.poses[1:, 2]))
            done, new, keep = done + 1, self.cost(), True
            if float(step.norm()) < o.step_tolerance:
                history.append(new)
                break
            if o.trust_region:
                predicted = float((step * (lam * step + rhs)).sum())
                rho = (cost - new) / predicted if predicted > 0 else -1.0
                keep = rho > 0
                lam, nu = (max(lam * max(1 / 3, 1 - (2 * rho - 1) ** 3), 1e-7), 2.0) if keep else (lam * nu, nu * 2)
            elif new < cost:
                lam /= o.lambda_factor
            else:
                lam, keep = lam * o.lambda_factor, not o.reject_worse_steps
            if keep:
                cost = new
            else:
                self.map, self.poses = before
            history.append(cost)
        return dict(map=self.map.cpu().numpy(), poses=self.poses, cost=np.array(history), iterations=done)


def exact(case, seed):
    kind = case["kind"]
    if kind == "incremental":
        return None  # a rebuilt problem per step: its normals and rows have no short restatement here
    if kind == "ldlt":
        _, A, rhs = _normal_matrix(case, seed)
        return torch.cholesky_solve(rhs[:, None], torch.linalg.cholesky(A))[:, 0].cpu().numpy()
    done = [_Reference(s).solve(_solver_options(case)) for s in _all_specs(case, seed)]
    if kind in ("solve", "cold"):
        return done[0]
    cost = [d["cost"] if kind == "batch" else d["cost"][-1] for d in done]
    return dict(map=np.concatenate([d["map"] for d in done]), poses=np.concatenate([d["poses"] for d in done]), cost=np.array(cost))
