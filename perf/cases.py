"""Performance cases of the solve path.

Every case is one call sequence a program makes to solve A x = b with this
framework: the complete solve from host arrays (`solve`), the complete solve
on device arrays (`Handle.from_device`, `solve_device`, `close`), solves on a
hierarchy that is kept (`solve_device`), batched solves on a kept hierarchy
(`solve_batch_device`) and requests to the solve server (`Server.submit`,
`wait`).  The matrices are the ones of the benchmark and the tests: 5-, 7- and
27-point Poisson operators, a 2-D anisotropic finite-volume operator with a
random coefficient field, and random geometric graph Laplacians with unordered
vertices; the settings are those of the benchmark (two aggregation sweeps,
l1-Jacobi 4/4, 16 coarse sweeps, relative tolerance 1e-8).

A case is a dict:
  call       "solve" | "complete" | "handle" | "batch" | "serve"
  matrix     "poisson5" | "poisson7" | "poisson27" | "fv2d" | "rgg"
  nx, ny, nz grid ("rgg": nx is the number of vertices, ny = nz = 1)
  precision  "fp64" | "mixed"
  storage    coarse-level storage of the mixed cycle: "fp32" | "bf16" | "fp16"
  cycle      0 V, 1 H, 2 W, 3 K
  hierarchies, composite   bootstrap's max_hrc and solver_type
  nrhs       right-hand sides ("batch": solved together, "serve": requests)
"""
import torch

import bootcmatchg_b200 as bc

_OFFSETS = [(x, y, z) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)]
_STORAGE = {"fp32": bc.STORE_FP32, "bf16": bc.STORE_BF16, "fp16": bc.STORE_FP16}


def _case(call, matrix, nx, ny=1, nz=1, precision="fp64", storage="fp32", cycle=0,
          hierarchies=1, composite=0, nrhs=1, **name):
    return dict(name, call=call, matrix=matrix, nx=nx, ny=ny, nz=nz, precision=precision,
                storage=storage, cycle=cycle, hierarchies=hierarchies, composite=composite,
                nrhs=nrhs)


def listed():
    return [
        # The smallest useful problem through the one-call interface: a
        # program that solves many small systems, each with its own matrix.
        _case("solve", "poisson7", 32, 32, 32, name="solve_host_7pt_32"),
        # A small 2-D problem with odd sides solved again and again on a kept
        # hierarchy (a time stepper's inner solve): launches and latency.
        _case("handle", "poisson5", 97, 61, name="handle_5pt_97x61"),
        # The benchmark's main workload: setup and solve on device arrays.
        _case("complete", "poisson27", 128, 128, 128, "mixed", name="complete_27pt_128_mixed"),
        # The same matrix kept, plain FP64 throughout.
        _case("handle", "poisson27", 128, 128, 128, name="handle_27pt_128_fp64"),
        # A ragged grid from host arrays with both copies inside the call.
        _case("solve", "poisson27", 101, 90, 77, "mixed", name="solve_host_27pt_ragged"),
        # Anisotropic diffusion with a random coefficient: three bootstrapped
        # hierarchies, BF16 coarse storage; the largest case.
        _case("complete", "fv2d", 2048, 2048, 1, "mixed", "bf16", hierarchies=3,
              name="complete_fv2d_2048_boot3"),
        # Many right-hand sides on one hierarchy, full and odd batch widths.
        _case("batch", "poisson7", 96, 96, 96, "mixed", nrhs=32, name="batch_7pt_96_x32_mixed"),
        _case("batch", "poisson7", 49, 50, 51, nrhs=5, name="batch_7pt_49x50x51_x5"),
        # Unordered graphs: no stencil to exploit; one complete solve in FP64
        # and a kept hierarchy in mixed precision.
        _case("complete", "rgg", 300001, name="complete_rgg_300k_fp64"),
        _case("handle", "rgg", 1000000, precision="mixed", name="handle_rgg_1m_mixed"),
        # The W-cycle, which lives on its coarse levels, with FP16 storage and
        # the symmetrized composite of two hierarchies.
        _case("handle", "poisson27", 64, 63, 61, "mixed", "fp16", cycle=2, hierarchies=2,
              composite=1, name="handle_27pt_64_wcycle_sym2"),
        # A served stream: twelve requests over three matrices that the
        # server keeps, solved together where they meet in the queue.
        _case("serve", "poisson7", 41, 40, 37, "mixed", nrhs=12, name="serve_12_requests"),
    ]


def draw(rng):
    def size(lo, hi):
        return lo * (hi / lo) ** rng.random()

    def sides(n, dims):
        out = []
        for d in range(dims):
            left = n ** (1.0 / (dims - d))
            s = max(4, int(left * rng.uniform(0.8, 1.25))) if d < dims - 1 else max(4, int(left))
            out.append(s)
            n = max(1.0, n / s)
        return out + [1] * (3 - dims)

    call = rng.choice(["solve", "complete", "complete", "handle", "handle", "batch", "serve"])
    matrix = rng.choice(["poisson5", "poisson7", "poisson27", "fv2d", "rgg"])
    precision = rng.choice(["fp64", "mixed"])
    storage = rng.choice(["fp32", "bf16", "fp16"]) if precision == "mixed" else "fp32"
    cycle, hierarchies, composite, nrhs = 0, 1, 0, 1
    n = size(2e3, {"poisson27": 1.5e6, "rgg": 8e5}.get(matrix, 1.2e6))
    if call == "batch":
        nrhs = rng.randint(2, 32)
        n = size(2e3, 4e6 / nrhs)
    elif call == "serve":
        nrhs = rng.randint(3, 16)
        n = size(2e3, 1.5e5)
    else:
        cycle = rng.choice([0, 0, 0, 1, 2, 3])
        if cycle or rng.random() < 0.25:
            n = min(n, 2e5)
            hierarchies, composite = rng.randint(1, 3), rng.randint(0, 2)
    dims = 1 if matrix == "rgg" else 2 if matrix in ("poisson5", "fv2d") else 3
    nx, ny, nz = (int(n), 1, 1) if dims == 1 else sides(n, dims)
    return _case(call, matrix, nx, ny, nz, precision, storage, cycle, hierarchies, composite,
                 nrhs)


# ---- inputs -----------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _grid_csr(nx, ny, nz, offsets, value):
    """CSR of a grid operator: value(k, nb, inside) gives the entries of
    offset k of every row (nb: the neighbour's index)."""
    dev = _device()
    n = nx * ny * nz
    r = torch.arange(n, device=dev)
    x, y, z = r % nx, (r // nx) % ny, r // (nx * ny)
    cols, vals, keep = [], [], []
    for k, (dx, dy, dz) in enumerate(offsets):
        inside = ((x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny)
                  & (z + dz >= 0) & (z + dz < nz))
        nb = r + dx + nx * (dy + ny * dz)
        cols.append(nb.to(torch.int32))
        vals.append(value(k, nb.clamp(0, n - 1), inside))
        keep.append(inside)
    keep = torch.stack(keep, 1)
    row = torch.zeros(n + 1, dtype=torch.int32, device=dev)
    row[1:] = keep.sum(1).cumsum(0)
    return row, torch.stack(cols, 1)[keep], torch.stack(vals, 1)[keep]


def _poisson(points, nx, ny, nz):
    offs = [o for o in _OFFSETS if points == 27 or sum(map(abs, o)) <= 1]
    if points == 5:
        offs, nz = [o for o in offs if o[2] == 0], 1
    diag = {5: 4.0, 7: 6.0, 27: 26.0}[points]
    n = nx * ny * nz

    def value(k, nb, inside):
        v = diag if offs[k] == (0, 0, 0) else -1.0
        return torch.full((n,), v, dtype=torch.float64, device=_device())

    return _grid_csr(nx, ny, nz, offs, value)


def _fv2d(nx, ny, gen):
    """Cell-centred -div(K grad u), K = exp(2 g), g normal smoothed over
    3 x 3 cells, faces in y weakened by 1e-3, Dirichlet boundary."""
    g = torch.randn(1, 1, ny, nx, dtype=torch.float64, device=_device(), generator=gen)
    g = torch.nn.functional.pad(g, (1, 1, 1, 1), mode="replicate")
    K = torch.exp(2 * torch.nn.functional.avg_pool2d(g, 3, 1)).reshape(-1)
    offs = [(0, -1, 0), (-1, 0, 0), (0, 0, 0), (1, 0, 0), (0, 1, 0)]
    n = nx * ny
    r = torch.arange(n, device=_device())
    face = []
    for dx, dy, _ in offs:
        inside = ((r % nx + dx >= 0) & (r % nx + dx < nx) & (r // nx + dy >= 0)
                  & (r // nx + dy < ny))
        Kn = K[(r + dx + nx * dy).clamp(0, n - 1)]
        face.append((1e-3 if dy else 1.0) * torch.where(inside, 2 * K * Kn / (K + Kn), 2 * K))

    def value(k, nb, inside):
        return face[0] + face[1] + face[3] + face[4] if k == 2 else -face[k]

    return _grid_csr(nx, ny, 1, offs, value)


def _rgg(n, seed, gen):
    """Graph Laplacian + 1e-3 I of n random points in the unit cube joined
    within a radius that gives mean degree 12, weights U[0.5, 2]; the
    vertices keep their random order."""
    dev = _device()
    radius = (12.0 / (n * 4.0 / 3.0 * 3.14159265358979)) ** (1.0 / 3.0)
    p = torch.rand(n, 3, dtype=torch.float64, device=dev, generator=gen)
    g = max(1, int(1.0 / radius))
    c3 = (p * g).long().clamp(max=g - 1)
    cell = (c3[:, 2] * g + c3[:, 1]) * g + c3[:, 0]
    order = torch.argsort(cell, stable=True)
    count = torch.bincount(cell, minlength=g ** 3)
    start = torch.cumsum(count, 0) - count
    ids, keys = torch.arange(n, device=dev), []
    for dx, dy, dz in _OFFSETS:
        q = c3 + torch.tensor([dx, dy, dz], device=dev)
        i = ids[((q >= 0) & (q < g)).all(1)]
        q = q[i]
        nb = (q[:, 2] * g + q[:, 1]) * g + q[:, 0]
        m = count[nb]
        src = torch.repeat_interleave(i, m)
        first = torch.repeat_interleave(start[nb] - (torch.cumsum(m, 0) - m), m)
        dst = order[first + torch.arange(src.numel(), device=dev)]
        near = (((p[src] - p[dst]) ** 2).sum(1) < radius * radius) | (src == dst)
        keys.append(src[near] * n + dst[near])
    keys = torch.sort(torch.cat(keys)).values
    i, j = keys // n, keys % n
    lo, hi = torch.minimum(i, j), torch.maximum(i, j)
    mix = (lo * 2654435761 + hi * 40503 + int(seed) * 97) & 0x7FFFFFFF
    mix = ((mix ^ (mix >> 15)) * 739982445) & 0x7FFFFFFF
    w = 0.5 + 1.5 * (mix ^ (mix >> 12)).double() / float(0x80000000)
    w = torch.where(i == j, torch.zeros_like(w), w)
    row = torch.zeros(n + 1, dtype=torch.int32, device=dev)
    row[1:] = torch.bincount(i, minlength=n).cumsum(0)
    deg = torch.segment_reduce(w, "sum", offsets=row.long())
    val = torch.where(i == j, deg[i] + 1e-3, -w)
    return row, j.to(torch.int32), val


def _matrix(kind, nx, ny, nz, seed):
    if kind == "rgg":
        return _rgg(nx, seed, _generator(seed))
    if kind == "fv2d":
        return _fv2d(nx, ny, _generator(seed))
    return _poisson(int(kind[len("poisson"):]), nx, ny, nz)


def _served(case):
    """The three matrices of a served stream: the case's own and two smaller."""
    out = []
    for shrink in (1, 2, 3):
        d = [max(4, s - 3 * (shrink - 1)) if s > 1 else 1
             for s in (case["nx"], case["ny"], case["nz"])]
        if case["matrix"] == "rgg":
            d = [max(64, case["nx"] // shrink), 1, 1]
        out.append(d)
    return out


def _inputs(case, seed):
    """[(row, col, val, B)]: one system, or the three of a served stream; B
    is n x nrhs (of each system), its columns contiguous."""
    kind = case["matrix"]
    grids = _served(case) if case["call"] == "serve" else [
        (case["nx"], case["ny"], case["nz"])]
    gen = _generator(seed + 1000003)
    out = []
    for k, (nx, ny, nz) in enumerate(grids):
        row, col, val = _matrix(kind, nx, ny, nz, seed + k)
        m = len(range(k, case["nrhs"], len(grids)))
        B = torch.randn(m, row.numel() - 1, dtype=torch.float64, device=_device(), generator=gen)
        out.append((row, col, val, B.t()))
    return out


def _params(case):
    p = bc.Params.default()
    p.solver_type, p.max_hrc, p.conv_ratio = case["composite"], case["hierarchies"], 0.5
    p.aggrsweeps, p.aggrtype, p.max_levels, p.cycle_type = 2, 0, 20, case["cycle"]
    p.relax_type, p.coarse_solver = 4, 4
    p.prerelax_sweeps, p.postrelax_sweeps, p.relaxnumber_coarse = 4, 4, 16
    p.itnlim, p.rtol = 1000, 1e-8
    return p


def _ext(case, stream=0):
    mixed = case["precision"] == "mixed"
    return bc.Extensions(precision=bc.PREC_MIXED if mixed else bc.PREC_FP64,
                         coarse_storage=_STORAGE[case["storage"]],
                         replace_every=10 if mixed else 0, stream=stream)


def _handle(s):
    row, col, val, _ = s["system"]
    return bc.Handle.from_device(row.numel() - 1, col.numel(), row.data_ptr(), col.data_ptr(),
                                 val.data_ptr(), s["params"], s["ext"])


def _host(system):
    row, col, val, B = system
    A = bc.CsrMatrix(row.numel() - 1, row.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy())
    return A, [B[:, j].contiguous().cpu().numpy() for j in range(B.shape[1])]


def prepare(case, seed):
    systems = _inputs(case, seed)
    s = {"case": case, "params": _params(case)}
    if case["call"] == "solve":
        s["A"], (s["b"],) = _host(systems[0])
        s["ext"] = _ext(case)
    elif case["call"] == "serve":
        s["systems"] = [_host(t) for t in systems]
        s["server"] = bc.Server(s["params"], _ext(case), slots=4)
    else:
        s["stream"] = torch.cuda.Stream()
        s["system"] = systems[0]
        s["ext"] = _ext(case, s["stream"].cuda_stream)
        torch.cuda.synchronize()
        if case["call"] != "complete":
            s["handle"] = _handle(s)
    return s


def run(s):
    call = s["case"]["call"]
    if call == "solve":
        x, _ = bc.solve(s["A"], s["params"], s["b"], s["ext"])
        return x
    if call == "serve":
        n = s["case"]["nrhs"]
        tickets = []
        for i in range(n):
            A, b = s["systems"][i % 3]
            tickets.append(s["server"].submit(A, b[i // 3], key=1 + i % 3))
        return [s["server"].wait(t)[0] for t in tickets]
    B = s["system"][3]
    with torch.cuda.stream(s["stream"]):
        x = torch.zeros(B.shape[1], B.shape[0], dtype=torch.float64, device=B.device)
    if call == "complete":
        with _handle(s) as h:
            h.solve_device(B.data_ptr(), x.data_ptr())
    elif call == "handle":
        s["handle"].solve_device(B.data_ptr(), x.data_ptr())
    else:
        s["handle"].solve_batch_device(B.shape[1], B.data_ptr(), B.shape[0], x.data_ptr(),
                                       B.shape[0])
    return x


# ---- what a pass cannot do without, and what it must give -----------------------

_POINTS = {"poisson5": 5, "poisson7": 7, "poisson27": 27, "fv2d": 5, "rgg": 13}


def work(case):
    """Each system read once (CSR and right-hand sides), each solution
    written once; a multiply-add per entry and right-hand side."""
    grids = _served(case) if case["call"] == "serve" else [
        (case["nx"], case["ny"], case["nz"])]
    nbytes = flops = 0
    for k, (nx, ny, nz) in enumerate(grids):
        n = nx * ny * nz
        m = len(range(k, case["nrhs"], len(grids)))
        nnz = _POINTS[case["matrix"]] * n
        nbytes += 12 * nnz + 4 * (n + 1) + 16 * n * m
        flops += 2 * nnz * m
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    return {"rel": 1e-6}


def exact(case, seed):
    """x = A^-1 b in FP64: Jacobi-preconditioned CG on the true residual,
    restarted until it no longer falls."""
    out = []
    systems = _inputs(case, seed)
    for row, col, val, B in systems:
        n = row.numel() - 1
        A = torch.sparse_csr_tensor(row, col, val, (n, n))
        i = torch.repeat_interleave(torch.arange(n, device=row.device),
                                    (row[1:] - row[:-1]).long())
        dinv = torch.zeros(n, dtype=torch.float64, device=row.device)
        dinv[i[col == i]] = 1.0 / val[col == i]
        dinv = dinv[:, None]
        B = B.contiguous()
        bnorm = B.norm(dim=0)
        X = torch.zeros_like(B)
        for _ in range(3):
            R = B - A @ X
            start = R.norm(dim=0)
            D, Z = torch.zeros_like(B), dinv * R
            P, rz = Z.clone(), (R * Z).sum(0)
            for it in range(20000):
                Q = A @ P
                alpha = rz / (P * Q).sum(0).clamp(min=1e-300)
                D += alpha * P
                R -= alpha * Q
                Z = dinv * R
                new = (R * Z).sum(0)
                P = Z + (new / rz.clamp(min=1e-300)) * P
                rz = new
                if it % 50 == 49 and bool((R.norm(dim=0) <= 1e-10 * start).all()):
                    break
            X += D
            if bool(((B - A @ X).norm(dim=0) <= 1e-14 * bnorm).all()):
                break
        out.append(X)
    if case["call"] == "serve":
        return [out[i % 3][:, i // 3].cpu().numpy() for i in range(case["nrhs"])]
    X = out[0].t().contiguous()
    return X[0].cpu().numpy() if case["call"] == "solve" else X
