"""The work that programs give this framework, as cases that can be timed.

A case names what is done (`kind`) and its sizes:

  solve     a study that stays on the device gets another load vector: resolve, solve, displacements
  study     a part from its description to its results: mesh, model, study, solve, stress recovery
  recovery  the stress field of a solved study
  batch     resident small studies of uneven size solved together
  product   the system operator on vectors of the caller's device memory, with their energies
  serve     a burst of requests of mixed kind and size through the serving loop
  system    a raw CSR system under the default (Jacobi) preconditioner

Parts are structured boxes of hexes split into six ten-node tetrahedra each: the steel cantilever
(bar), the thin plate under pressure (plate) and the two-material printed block (block).
"""
import math

import numpy as np
import torch

import solidfem_b200 as sf
from solidfem_b200 import workloads

PRECISIONS = {"double": sf.Precision.DOUBLE, "single_storage": sf.Precision.SINGLE_STORAGE,
              "single": sf.Precision.SINGLE, "mixed": sf.Precision.MIXED}

# Shape of each part: box edge lengths (mm), the axis whose low face is clamped and the axis whose
# high face is loaded.
PARTS = {"bar": ((100.0, 10.0, 10.0), 0, 0), "plate": ((100.0, 100.0, 0.8), 0, 2), "block": ((60.0, 60.0, 60.0), 2, 2)}
MATERIALS = {"bar": (210000.0, 0.30), "plate": (2000.0, 0.35)}
SHELL, CORE, SHELL_DEPTH = (2400.0, 0.36), (800.0, 0.30), 2.0
TRACTION = {"bar": (0.0, 0.0, -10.0), "plate": (0.0, 0.0, -0.01), "block": (0.5, 0.0, 0.0)}

EXACT_DOFS = 16000      # dense 64-bit solves up to this many unknowns
EXACT_TETS = 150000     # matrix-free 64-bit products up to this many elements


def part(kind, shape, nx, ny, nz, **more):
    return dict(kind=kind, shape=shape, nx=nx, ny=ny, nz=nz, **more)


def listed():
    return [
        # The reference's steel cantilever, another load on a resident study, the plain FP64 method:
        # a design loop's smallest call, all launches and latency.
        part("solve", "bar", 20, 4, 4, precision="double", tolerance=1e-10, name="bar_solve"),
        # The same part from its description to its stresses with the default multigrid options:
        # what a user of one small part waits for.
        part("study", "bar", 20, 4, 4, precision="single_storage", tolerance=1e-9, name="bar_study"),
        # The 217,800-unknown thin plate, mixed precision: an ordinary resident solve.
        part("solve", "plate", 60, 60, 2, precision="mixed", tolerance=1e-8, name="plate_solve"),
        # The 603,000-unknown plate of the headline benchmark, mixed and plain FP64.
        part("solve", "plate", 100, 100, 2, precision="mixed", tolerance=1e-8, name="gate_solve"),
        part("solve", "plate", 100, 100, 2, precision="double", tolerance=1e-8, name="gate_solve_fp64"),
        # That plate end to end from its description, mesh to nodal stresses.
        part("study", "plate", 100, 100, 2, precision="mixed", tolerance=1e-8, name="gate_study"),
        # The stress field of that plate once more, after a new load (a load sweep's second half).
        part("recovery", "plate", 100, 100, 2, precision="mixed", tolerance=1e-8, name="gate_recovery"),
        # The printed block's 5.3 million unknowns: the largest resident solve.
        part("solve", "block", 60, 60, 60, precision="mixed", tolerance=1e-8, name="block_solve"),
        # Sixteen small cantilevers of uneven length solved as one batch.
        part("batch", "bar", 20, 4, 4, count=16, precision="mixed", tolerance=1e-8, name="batch_solve"),
        # The gate plate's operator on the most vectors one call takes (a serving loop's energies).
        part("product", "plate", 100, 100, 2, count=8, name="product_8"),
        # A burst of the serving stream's mixed requests, 10k to 600k unknowns.
        dict(kind="serve", count=24, stream=0, low=10000, high=600000, precision="mixed", tolerance=1e-8, name="serve_burst"),
        # A caller's own symmetric matrix with the default options: 45^3 cells, Jacobi.
        dict(kind="system", nx=45, ny=45, nz=45, tolerance=1e-9, name="jacobi_system"),
    ]


def _log(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def _plate(rng, low, high, most_layers=3):
    layers = rng.randint(2, most_layers)
    n = math.sqrt(_log(rng, low, high) / (6.0 * 2.0 * (2 * layers + 1)) * 1.5)
    return max(8, round(n * rng.uniform(0.8, 1.25))), max(8, round(n)), layers


def draw(rng):
    kind = rng.choice(("solve", "solve", "solve", "study", "recovery", "batch", "product", "product", "serve", "system"))
    precision = rng.choice(("mixed", "mixed", "double", "single_storage", "single"))
    if kind == "solve":
        shape = rng.choice(("bar", "plate", "block"))
        if shape == "bar":
            ny, nz = rng.randint(2, 9), rng.randint(2, 9)
            return part(kind, shape, rng.randint(12, 60), ny, nz, precision=precision, tolerance=rng.choice((1e-8, 1e-9, 1e-10)))
        if shape == "plate":
            nx, ny, nz = _plate(rng, 20e3, 600e3)
            return part(kind, shape, nx, ny, nz, precision=rng.choice(("mixed", "double")), tolerance=1e-8)
        n = _log(rng, 8, 40)
        return part(kind, shape, round(n), max(4, round(n * rng.uniform(0.75, 1.0))), max(4, round(n * rng.uniform(0.75, 1.0))),
                    precision=precision, tolerance=1e-8)
    if kind in ("study", "recovery"):
        if rng.random() < 0.5:
            return part(kind, "bar", rng.randint(12, 60), rng.randint(2, 9), rng.randint(2, 9), precision=precision, tolerance=1e-9)
        nx, ny, nz = _plate(rng, 20e3, 400e3)
        return part(kind, "plate", nx, ny, nz, precision="mixed", tolerance=1e-8)
    if kind == "batch":
        return part(kind, "bar", rng.randint(16, 24), rng.choice((3, 4)), 4, count=rng.randint(2, 24),
                    precision=rng.choice(("mixed", "double")), tolerance=rng.choice((1e-8, 1e-9)))
    if kind == "product":
        if rng.random() < 0.4:
            return part(kind, "bar", rng.randint(12, 60), rng.randint(2, 9), rng.randint(2, 9), count=rng.randint(1, 8))
        nx, ny, nz = _plate(rng, 40e3, 600e3)
        return part(kind, "plate", nx, ny, nz, count=rng.randint(1, 8))
    if kind == "serve":
        return dict(kind=kind, count=rng.randint(4, 24), stream=rng.randint(1, 999), low=10000,
                    high=rng.choice((100000, 600000)), precision="mixed", tolerance=1e-8)
    n = _log(rng, 12, 45)
    return dict(kind="system", nx=round(n), ny=max(2, round(n * rng.uniform(0.7, 1.0))), nz=max(2, round(n * rng.uniform(0.7, 1.0))),
                tolerance=rng.choice((1e-8, 1e-9, 1e-10)))


# ------------------------------------------------------------------ what a program has in hand


def _dims(case):
    return (case["nx"], case["ny"], case["nz"])


def _options(case, batchable=False):
    return sf.StudyOptions(pcg=sf.PcgOptions(tolerance=case["tolerance"]), batchable=batchable,
                           preconditioner=sf.MultigridOptions(precision=PRECISIONS[case["precision"]]))


def _traction(case, rng):
    """The part's load with its size and direction varied a little: another load case."""
    t = np.array(TRACTION[case["shape"]])
    return tuple(t * rng.uniform(0.5, 1.5) + 0.05 * np.abs(t).max() * rng.uniform(-1.0, 1.0, 3))


def _mesh(case):
    return sf.box_tet_mesh((0.0, 0.0, 0.0), PARTS[case["shape"]][0], _dims(case), device=0)


def _model(case, mesh, traction, material=None):
    size, clamp, load = PARTS[case["shape"]]
    nodes = mesh.nodes()
    if case["shape"] == "block":
        material = sf.ShellCore(sf.Material(*SHELL), sf.Material(*CORE), (0.0, 0.0, 0.0), size, SHELL_DEPTH)
    model = sf.Model(mesh, material or sf.Material(*MATERIALS[case["shape"]]))
    model.fix_nodes(np.flatnonzero(np.abs(nodes[:, clamp]) < 1e-9))
    faces = mesh.boundary_face_array()
    on_end = np.all(np.abs(nodes[faces["nodes"][:, :3], load] - size[load]) < 1e-9, axis=1)
    model.add_face_tractions(faces[on_end], traction)
    return model


def _load_vector(free_dofs, rng):
    """A load vector over the free unknowns: a body force of any direction with a random part per node."""
    g = rng.standard_normal(3)
    nodes = free_dofs // 3
    return ((g + 0.25 * rng.standard_normal((nodes, 3))) * (10.0 / nodes)).ravel()


def _requests(case):
    return workloads.serving_stream(count=case["count"], seed=case["stream"], dof_range=(case["low"], case["high"]))


def _conduction(case, rng):
    """Finite volumes on a grid of cells with random conductivities, as scalar CSR (columns
    ascending): the seven-point operator plus a leak of every cell to its surroundings."""
    nx, ny, nz = _dims(case)
    n = nx * ny * nz
    k = np.exp(0.5 * rng.standard_normal((nz, ny, nx)))
    at = np.arange(n).reshape(nz, ny, nx)
    diag = np.full((nz, ny, nx), 0.02)
    rows, cols, vals = [], [], []
    for axis in range(3):
        low = [slice(None)] * 3
        high = [slice(None)] * 3
        low[axis], high[axis] = slice(0, -1), slice(1, None)
        a, b = tuple(low), tuple(high)
        g = 2.0 * k[a] * k[b] / (k[a] + k[b])
        np.add.at(diag, a, g)
        np.add.at(diag, b, g)
        for p, q in ((a, b), (b, a)):
            rows.append(at[p].ravel())
            cols.append(at[q].ravel())
            vals.append(-g.ravel())
    rows.append(at.ravel())
    cols.append(at.ravel())
    vals.append(diag.ravel())
    rows, cols, vals = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    order = np.lexsort((cols, rows))
    starts = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return starts.astype(np.uint64), cols[order].astype(np.uint32), vals[order], rng.standard_normal(n)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    state = {"kind": kind, "case": case}
    if kind == "system":
        state["csr"] = _conduction(case, rng)
        return state
    if kind == "serve":
        state["server"] = sf.Server()
        state["requests"] = []
        for r in _requests(case):
            r.force *= rng.uniform(0.5, 1.5)
            r.youngs_modulus *= rng.uniform(0.9, 1.1)
            mesh, model = workloads.build_model(r, device=0)
            state["requests"].append((model, mesh.node_count()))
        return state
    if kind == "study":
        state["traction"] = _traction(case, rng)
        return state
    if kind == "batch":
        state["studies"] = []
        for i in range(case["count"]):
            one = dict(case, nx=case["nx"] + i % 4)
            material = sf.Material(210000.0 * rng.uniform(0.3, 1.0), rng.uniform(0.28, 0.33))
            state["studies"].append(sf.StaticStudy.new(_model(one, _mesh(one), _traction(one, rng), material), _options(one, True)))
        return state
    if kind == "product":
        study = sf.StaticStudy.new(_model(case, _mesh(case), _traction(case, rng)))
        n = study.report()["free_dofs"]
        x = torch.from_numpy(rng.standard_normal((case["count"], n))).cuda()
        state.update(study=study, x=x, y=torch.empty_like(x), energy=torch.empty(case["count"], dtype=torch.float64, device="cuda"),
                     stream=torch.cuda.ExternalStream(study.stream()))
        return state
    study = sf.StaticStudy.new(_model(case, _mesh(case), _traction(case, rng)), _options(case))
    state["study"] = study
    if kind == "recovery":
        study.solve()
    else:
        state["load"] = _load_vector(study.report()["free_dofs"], rng)
    return state


# ------------------------------------------------------------------ one pass


def _fields(solution):
    return {"displacements": solution.displacements, "point_stress": solution.point_stresses["stress"],
            "point_von_mises": solution.point_stresses["von_mises"], "nodal_stress": solution.nodal_stress,
            "nodal_von_mises": solution.nodal_von_mises}


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "solve":
        study = state["study"]
        study.resolve(state["load"])
        study.solve()
        return study.displacements()
    if kind == "study":
        study = sf.StaticStudy.new(_model(case, _mesh(case), state["traction"]), _options(case))
        study.solve()
        return _fields(study.solution())
    if kind == "recovery":
        return _fields(state["study"].solution())
    if kind == "batch":
        sf.solve_batch(state["studies"])
        return [study.displacements() for study in state["studies"]]
    if kind == "product":
        state["study"].energy_products(state["x"].data_ptr(), state["y"].data_ptr(), state["energy"].data_ptr(), case["count"])
        state["stream"].synchronize()  # the energies are read next; calls that overlap share their scratch
        return {"y": state["y"], "energy": state["energy"]}
    if kind == "serve":
        server, options = state["server"], _options(case)
        ids = [(server.submit(model, options), nodes) for model, nodes in state["requests"]]
        out = []
        for rid, nodes in ids:
            server.wait(rid)
            out.append(server.take(rid, nodes))
        return out
    system = sf.System(*state["csr"], sf.StudyOptions(pcg=sf.PcgOptions(tolerance=case["tolerance"])))
    system.solve()
    return system.estimate()


# ------------------------------------------------------------------ what a pass cannot do without


def _counts(case):
    """(nodes, tets, 3x3 blocks of the system) of a box, clamped face included."""
    nx, ny, nz = _dims(case)
    vertices = (nx + 1) * (ny + 1) * (nz + 1)
    nodes = (2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1)
    return nodes, 6 * nx * ny * nz, 25 * nodes, vertices


def _solve_bytes(nodes, blocks, iterations, precision):
    """Each iteration reads the FP64 system once and the fine operator at every smoother and residual
    pass of the cycle (six), in the cycle's storage; coarser levels add about a third."""
    stored = 76 if precision == "double" else 40
    return iterations * (76 * blocks + 6 * 1.33 * stored * blocks + 12 * 24 * nodes)


def _iterations(case):
    return {"bar": 62, "plate": 3.8 * max(case.get("nx", 0), case.get("ny", 0)), "block": 45}[case.get("shape", "bar")]


def work(case):
    kind = case["kind"]
    if kind == "system":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 12.0 * 7 * n + 24 * n, "flops": 2.0 * 7 * n * 100}
    if kind == "serve":
        nodes = sum(r.target_dofs for r in _requests(case)) / 3.0
        b = _solve_bytes(nodes, 25 * nodes, 100, case["precision"])
        return {"bytes": b, "flops": b / 3}
    nodes, tets, blocks, vertices = _counts(case)
    if kind == "product":
        return {"bytes": 76.0 * blocks + case["count"] * 48.0 * nodes, "flops": case["count"] * 18.0 * blocks}
    fields = 72.0 * nodes + 56.0 * 4 * tets + 24.0 * nodes
    if kind == "recovery":
        return {"bytes": fields + 24.0 * nodes + 40.0 * tets, "flops": 4.0 * tets * 400}
    solve = case.get("count", 1) * (_solve_bytes(nodes, blocks, _iterations(case), case["precision"]) + 48 * nodes)
    if kind == "study":
        return {"bytes": solve + fields + 72.0 * blocks, "flops": solve / 3 + 17200.0 * tets}
    return {"bytes": solve, "flops": solve / 3}


# ------------------------------------------------------------------ the same in 64 bits

_EDGES = ((0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3))
_ORDERS = ((0, 1, 2), (1, 2, 0), (2, 0, 1), (0, 2, 1), (2, 1, 0), (1, 0, 2))
_NEAR, _FAR = 0.5854101966249685, 0.1381966011250105  # the four-point rule's barycentric coordinates


def _box(case):
    """Nodes and ten-node tets of a box: vertices with x fastest, six tets around each cell's
    diagonal, midside nodes numbered by their edge's corner pair."""
    dims, size = _dims(case), PARTS[case["shape"]][0]
    axes = [np.array([s * (i / d) if i < d else s for i in range(d + 1)]) for s, d in zip(size, dims)]
    z, y, x = np.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    vertices = np.stack([x.ravel(), y.ravel(), z.ravel()], axis=1)
    step = (1, dims[0] + 1, (dims[0] + 1) * (dims[1] + 1))
    k, j, i = np.meshgrid(np.arange(dims[2]), np.arange(dims[1]), np.arange(dims[0]), indexing="ij")
    base = (i * step[0] + j * step[1] + k * step[2]).ravel()
    tets = np.empty((len(base), 6, 4), dtype=np.int64)
    for o, order in enumerate(_ORDERS):
        corner = [base]
        for a in order:
            corner.append(corner[-1] + step[a])
        if o >= 3:
            corner[1], corner[2] = corner[2], corner[1]
        tets[:, o] = np.stack(corner, axis=1)
    tets = tets.reshape(-1, 4)
    ends = np.sort(np.stack([tets[:, list(e)] for e in _EDGES], axis=1), axis=2)
    key = ends[..., 0] * len(vertices) + ends[..., 1]
    unique, number = np.unique(key, return_inverse=True)
    mid = 0.5 * (vertices[unique // len(vertices)] + vertices[unique % len(vertices)])
    tets = np.concatenate([tets, len(vertices) + number.reshape(key.shape)], axis=1)
    return np.concatenate([vertices, mid]), tets


def _elasticity(youngs, poisson):
    lam, mu = youngs * poisson / ((1 + poisson) * (1 - 2 * poisson)), youngs / (2 * (1 + poisson))
    d = torch.zeros(6, 6, dtype=torch.float64, device="cuda")
    d[:3, :3] = lam
    d[range(3), range(3)] = lam + 2 * mu
    d[range(3, 6), range(3, 6)] = mu
    return d


def _strain_operators(nodes, tets):
    """B (4 points x tets x 6 x 30), strains in the order xx yy zz xy yz zx, and each tet's volume."""
    p = torch.from_numpy(nodes).cuda()[torch.from_numpy(tets[:, :4]).cuda()]
    jac = p[:, 1:] - p[:, :1]
    grad = torch.linalg.inv(jac).transpose(1, 2)                    # tets x 3 corners x 3 axes
    grad = torch.cat([-grad.sum(1, keepdim=True), grad], dim=1)
    volume = torch.linalg.det(jac) / 6.0
    out = []
    for q in range(4):
        bary = [_NEAR if c == q else _FAR for c in range(4)]
        shape = [(4 * bary[c] - 1) * grad[:, c] for c in range(4)]
        shape += [4 * (bary[a] * grad[:, b] + bary[b] * grad[:, a]) for a, b in _EDGES]
        g = torch.stack(shape, dim=1)
        b = torch.zeros(len(tets), 6, 10, 3, dtype=torch.float64, device="cuda")
        for a in range(3):
            b[:, a, :, a] = g[:, :, a]
        for row, (u, v) in enumerate(((0, 1), (1, 2), (2, 0))):
            b[:, 3 + row, :, u], b[:, 3 + row, :, v] = g[:, :, v], g[:, :, u]
        out.append(b.reshape(len(tets), 6, 30))
    return out, volume


def _free_nodes(case, nodes):
    return np.flatnonzero(~(np.abs(nodes[:, PARTS[case["shape"]][1]]) < 1e-9))


def _element_stiffness(case, nodes, tets):
    operators, volume = _strain_operators(nodes, tets)
    d = _elasticity(*MATERIALS[case["shape"]])
    return operators, d, sum(torch.einsum("tsi,sr,trj->tij", b, d, b) * (volume / 4.0)[:, None, None] for b in operators)


def _end_load(case, nodes, tets, traction):
    """The consistent load of a uniform traction: a third of each loaded face's share at its midsides."""
    size, _, axis = PARTS[case["shape"]]
    load = np.zeros_like(nodes)
    on = np.abs(nodes[:, axis] - size[axis]) < 1e-9
    for face, mids in (((1, 2, 3), (5, 9, 8)), ((0, 3, 2), (7, 9, 6)), ((0, 1, 3), (4, 8, 7)), ((0, 2, 1), (6, 5, 4))):
        hit = tets[on[tets[:, list(face)]].all(axis=1)]
        a, b, c = (nodes[hit[:, k]] for k in face)
        area = 0.5 * np.linalg.norm(np.cross(b - a, c - a), axis=1)
        for m in mids:
            np.add.at(load, hit[:, m], area[:, None] / 3.0 * np.asarray(traction))
    return load


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "system":
        starts, cols, vals, rhs = _conduction(case, rng)
        n = len(rhs)
        a = torch.sparse_csr_tensor(torch.from_numpy(starts.astype(np.int64)), torch.from_numpy(cols.astype(np.int64)),
                                    torch.from_numpy(vals), size=(n, n)).cuda()
        b = torch.from_numpy(rhs).cuda()
        scale = a.to_sparse_coo().coalesce()
        diagonal = torch.zeros_like(b)
        i, v = scale.indices(), scale.values()
        diagonal[i[0][i[0] == i[1]]] = v[i[0] == i[1]]
        x = torch.zeros_like(b)
        for _ in range(3):  # conjugate gradient, refined from the true residual
            r = b - a @ x
            dx, z = torch.zeros_like(b), r / diagonal
            p, rz = z.clone(), r @ z
            for _ in range(600):
                ap = a @ p
                alpha = rz / (p @ ap)
                dx, r = dx + alpha * p, r - alpha * ap
                if float(r.norm()) <= 1e-13 * float(b.norm()):
                    break
                z = r / diagonal
                rz, old = r @ z, rz
                p = z + (rz / old) * p
            x = x + dx
        return x.cpu()
    if kind not in ("solve", "study", "product") or case["shape"] == "block":
        return None
    count, tet_count, _, _ = _counts(case)
    if tet_count > EXACT_TETS or (kind != "product" and 3 * count > EXACT_DOFS):
        return None
    traction = _traction(case, rng)
    nodes, tets = _box(case)
    free = _free_nodes(case, nodes)
    operators, d, ke = _element_stiffness(case, nodes, tets)
    dof = torch.from_numpy((3 * tets[:, :, None] + np.arange(3)).reshape(len(tets), 30)).cuda()
    unknown = torch.from_numpy((3 * free[:, None] + np.arange(3)).ravel()).cuda()
    if kind == "product":
        x = torch.from_numpy(rng.standard_normal((case["count"], 3 * len(free)))).cuda()
        full = torch.zeros(case["count"], 3 * len(nodes), dtype=torch.float64, device="cuda")
        full[:, unknown] = x
        y = torch.zeros_like(full)
        for k in range(case["count"]):
            y[k].index_add_(0, dof.ravel(), torch.bmm(ke, full[k][dof][:, :, None]).ravel())
        y = y[:, unknown]
        return {"y": y, "energy": (x * y).sum(1)}
    n = 3 * len(nodes)
    stiffness = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    stiffness.index_add_(0, (dof[:, :, None] * n + dof[:, None, :]).ravel(), ke.ravel())
    stiffness = stiffness.view(n, n)[unknown][:, unknown]
    if kind == "solve":
        load = torch.from_numpy(_load_vector(3 * len(free), rng)).cuda()
    else:
        load = torch.from_numpy(_end_load(case, nodes, tets, traction)).cuda().ravel()[unknown]
    factor = torch.linalg.cholesky(stiffness)
    u = torch.cholesky_solve(load[:, None], factor)
    u = u + torch.cholesky_solve(load[:, None] - stiffness @ u, factor)
    full = torch.zeros(n, dtype=torch.float64, device="cuda")
    full[unknown] = u[:, 0]
    displacements = full.view(-1, 3)
    if kind == "solve":
        return displacements
    stress = torch.stack([torch.einsum("sr,trj,tj->ts", d, b, full[dof]) for b in operators], dim=1).reshape(-1, 6)
    s = stress.T
    von_mises = torch.sqrt(0.5 * ((s[0] - s[1]) ** 2 + (s[1] - s[2]) ** 2 + (s[2] - s[0]) ** 2) +
                           3.0 * (s[3] ** 2 + s[4] ** 2 + s[5] ** 2))
    return {"displacements": displacements, "point_stress": stress, "point_von_mises": von_mises,
            "nodal_stress": None, "nodal_von_mises": None}
