"""The work this library is used for, as cases that can be timed.

Each case is one call (or the short sequence of calls) that a user's program
makes through cel_v3_b200.celgpu, on seeded synthetic systems of the sizes of
the library's workloads.  Right-hand sides are manufactured, b = A x_true with
x_true ~ U[0, 1), so that the 64-bit answer of a solve is known.

Kinds:
  spmv       y = A x on a stored matrix (CSR or JAD)
  pcg        Jacobi-PCG on device vectors (FP64, or FP32 with FP64 updates)
  gmres      restarted GMRES(m) with Jacobi on device vectors
  batched    many independent systems of uneven size in one call
  multirhs   many right-hand sides of one matrix in one call
  gradient   adjoint solve and the gradients of a diffusion solve
  elm        the ELM assembly API on host arrays: assemble, solve, collect

Matrices: "poisson" (7-point, constant coefficients), "diffusion" (7-point,
one coefficient exp(sigma N(0,1)) per cell face), "band" (unstructured SPD:
`degree` random neighbours per row within +-`width` rows).
"""
import numpy as np
import torch

from cel_v3_b200 import celgpu, synth

F64 = torch.float64
PRECISION = {"fp64": celgpu.PREC_FP64, "fp32_ir": celgpu.PREC_FP32_IR, "fp32_ru": celgpu.PREC_FP32_RU}


def listed():
    return [
        # the building block inside a user's own iteration on a small system:
        # one call's latency
        {"name": "spmv_csr_32", "kind": "spmv", "fmt": "csr", "matrix": "poisson", "nx": 32, "ny": 32, "nz": 32},
        # the SpMV bandwidth sweep's largest size
        {"name": "spmv_csr_256", "kind": "spmv", "fmt": "csr", "matrix": "poisson", "nx": 256, "ny": 256, "nz": 256},
        # jagged diagonals, variable coefficients, sides that fill no tile
        {"name": "spmv_jad_ragged", "kind": "spmv", "fmt": "jad", "matrix": "diffusion", "sigma": 1.0,
         "nx": 131, "ny": 127, "nz": 113},
        # the small plain solve: many launches of little work
        {"name": "pcg_poisson_32", "kind": "pcg", "matrix": "poisson", "nx": 32, "ny": 32, "nz": 32,
         "precision": "fp64", "eps_rel": 1e-8},
        # the large plain solve, the headline workload
        {"name": "pcg_poisson_256", "kind": "pcg", "matrix": "poisson", "nx": 256, "ny": 256, "nz": 256,
         "precision": "fp64", "eps_rel": 1e-8},
        # the precision workload: FP32 sweeps, FP64 updates, tight tolerance
        {"name": "pcg_diffusion_256_fp32_ru", "kind": "pcg", "matrix": "diffusion", "sigma": 1.0,
         "nx": 256, "ny": 256, "nz": 256, "precision": "fp32_ru", "eps_rel": 1e-10},
        # a matrix without grid structure, int32 columns, rows of many lengths
        {"name": "pcg_band_200k", "kind": "pcg", "matrix": "band", "n": 200003, "degree": 9, "width": 3000,
         "precision": "fp64", "eps_rel": 1e-8},
        # GMRES(30) on the middle size of the sweep
        {"name": "gmres30_poisson_128", "kind": "gmres", "matrix": "poisson", "nx": 128, "ny": 128, "nz": 128,
         "restart": 30, "eps_rel": 1e-8},
        # the batching workload: 64 systems, sides 16..96
        {"name": "batched_64", "kind": "batched", "count": 64, "lo": 16, "hi": 96, "sides": 4, "sigma": 0.5,
         "precision": "fp64", "eps_rel": 1e-8},
        # the batching workload's shared matrix: 32 right-hand sides
        {"name": "multirhs_128_k32", "kind": "multirhs", "matrix": "poisson", "nx": 128, "ny": 128, "nz": 128,
         "k": 32, "precision": "fp64", "eps_rel": 1e-8},
        # the differentiation workload, one instance
        {"name": "gradient_128", "kind": "gradient", "sigma": 1.0, "nx": 128, "ny": 128, "nz": 128, "eps_rel": 1e-10},
        # a program that links the ELM interface: host rows in, host solution out
        {"name": "elm_pcg_ragged", "kind": "elm", "matrix": "diffusion", "sigma": 0.5, "nx": 61, "ny": 57, "nz": 45,
         "eps_rel": 1e-8},
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], uniform over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _grid(rng, lo, hi):
    side = _log_int(rng, lo, hi)
    return {k: max(lo, min(hi, int(round(side * rng.uniform(0.8, 1.2))))) for k in ("nx", "ny", "nz")}


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "pcg", "pcg", "pcg", "gmres", "batched", "multirhs", "gradient", "elm"])
    if kind == "spmv":
        c = {"kind": kind, "fmt": rng.choice(["csr", "jad"]), "matrix": rng.choice(["poisson", "diffusion"])}
        c.update(_grid(rng, 16, 256))
    elif kind == "pcg":
        c = {"kind": kind, "matrix": rng.choice(["poisson", "diffusion", "band"]),
             "precision": rng.choice(["fp64", "fp32_ru"]), "eps_rel": rng.choice([1e-8, 1e-10])}
        if c["matrix"] == "band":
            c.update(n=_log_int(rng, 3000, 400000), degree=rng.randint(4, 12), width=_log_int(rng, 300, 3000))
        else:
            c.update(_grid(rng, 16, 200))
    elif kind == "gmres":
        c = {"kind": kind, "matrix": rng.choice(["poisson", "diffusion"]), "restart": rng.randint(10, 30),
             "eps_rel": 1e-6}
        c.update(_grid(rng, 16, 64))
    elif kind == "batched":
        lo = rng.randint(8, 24)
        c = {"kind": kind, "count": _log_int(rng, 4, 64), "lo": lo, "hi": lo + rng.randint(8, 64),
             "sides": rng.randint(0, 1 << 20), "sigma": 0.5,
             "precision": rng.choice(["fp64", "fp32_ir", "fp32_ru"]), "eps_rel": 1e-8}
    elif kind == "multirhs":
        c = {"kind": kind, "matrix": rng.choice(["poisson", "diffusion"]), "k": rng.randint(2, 32),
             "precision": rng.choice(["fp64", "fp32_ir", "fp32_ru"]), "eps_rel": 1e-8}
        c.update(_grid(rng, 16, 100))
    elif kind == "gradient":
        c = {"kind": kind, "eps_rel": 1e-10}
        c.update(_grid(rng, 12, 128))
    else:
        c = {"kind": kind, "matrix": rng.choice(["poisson", "diffusion"]), "eps_rel": 1e-8}
        c.update(_grid(rng, 12, 64))
    if (c.get("matrix") == "diffusion" or kind == "gradient") and "sigma" not in c:
        c["sigma"] = rng.choice([0.5, 1.0])
    return c


# ---- inputs ------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 1)
    return g


def _faces(gen, nx, ny, nz, sigma):
    m = sum(synth.face_counts(nx, ny, nz))
    return torch.exp(sigma * torch.randn(m, generator=gen, dtype=F64, device="cuda"))


def _band(gen, n, degree, width):
    """Rows linked to `degree` random neighbours within +-width, symmetrised;
    diagonal = sum of the row's couplings + 0.01.  Returns int32 row pointers
    and columns and FP64 values on the device."""
    i = torch.arange(n, device="cuda").repeat_interleave(degree)
    off = torch.randint(1, width + 1, (n * degree,), generator=gen, device="cuda")
    j = i + off
    keep = j < n
    edge = torch.unique(i[keep] * n + j[keep])
    a, b = edge // n, edge % n
    u = 0.5 + torch.rand(edge.numel(), generator=gen, dtype=F64, device="cuda")
    diag = torch.arange(n, device="cuda")
    rows, cols = torch.cat([a, b, diag]), torch.cat([b, a, diag])
    vals = torch.cat([-u, -u, torch.zeros(n, dtype=F64, device="cuda")])
    order = torch.argsort(rows * n + cols)
    rows, cols, vals = rows[order], cols[order], vals[order]
    lens = torch.bincount(rows, minlength=n)
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(lens, 0)
    slot = torch.arange(rows.numel(), device="cuda") - rp[rows]
    wide = torch.zeros(n, int(lens.max()), dtype=F64, device="cuda")
    wide[rows, slot] = vals
    vals[rows == cols] = 0.01 - wide.sum(1)
    return rp.to(torch.int32), cols.to(torch.int32), vals


def _csr(case, gen):
    """Row pointers, columns and values on the device, and the number of rows."""
    if case["matrix"] == "band":
        return _band(gen, case["n"], case["degree"], case["width"])
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["matrix"] == "poisson":
        k = torch.ones(sum(synth.face_counts(nx, ny, nz)), dtype=F64, device="cuda")
    else:
        k = _faces(gen, nx, ny, nz, case["sigma"])
    return synth.diffusion7_device(nx, ny, nz, k)


def _handle():
    return celgpu.Handle(0, torch.cuda.current_stream().cuda_stream)


def _matrix(h, csr):
    rp, ci, v = csr
    return h.matrix_from_csr_device(rp.numel() - 1, ci.numel(), rp.data_ptr(), ci.data_ptr(), v.data_ptr())


def _rhs(h, m, x):
    b = torch.empty_like(x)
    h.spmv(m, x.data_ptr(), b.data_ptr())
    return b


def _uniform(gen, *shape):
    return torch.rand(*shape, generator=gen, dtype=F64, device="cuda")


def _batch_sides(case):
    return [int(s) for s in np.random.default_rng(case["sides"]).integers(case["lo"], case["hi"] + 1, case["count"])]


def _params(case, **kw):
    p = {"eps_rel": case["eps_rel"], "iter_max": 5000, "x0_mode": celgpu.X0_ZERO,
         "precision": PRECISION[case.get("precision", "fp64")]}
    if case.get("precision") == "fp32_ru":
        p["inner_eps_rel"] = 1e-2
    p.update(kw)
    return celgpu.params(**p)


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    s = {"case": dict(case)}
    if kind == "elm":
        csr = _csr(case, gen)
        n = csr[0].numel() - 1
        x = _uniform(gen, n)
        h = _handle()
        m = _matrix(h, csr)
        b = _rhs(h, m, x)
        torch.cuda.synchronize()
        m.destroy()
        s.update(h=h, n=n, rp=csr[0].cpu().numpy() + 1, ci=csr[1].cpu().numpy() + 1, v=csr[2].cpu().numpy(),
                 b=b.cpu().numpy(), p=_params(case))
        return s
    h = s["h"] = _handle()
    if kind == "batched":
        sides = _batch_sides(case)
        total = sum(q ** 3 for q in sides)
        xt, b = _uniform(gen, total), torch.empty(total, dtype=F64, device="cuda")
        mats, at = [], 0
        for q in sides:
            m = _matrix(h, synth.diffusion7_device(q, q, q, _faces(gen, q, q, q, case["sigma"])))
            h.spmv(m, xt.data_ptr() + 8 * at, b.data_ptr() + 8 * at)
            mats.append(m.jacobi())
            at += q ** 3
        x = torch.empty_like(b)
        starts = np.cumsum([0] + [q ** 3 for q in sides[:-1]])
        s.update(mats=mats, b=b, x=x, p=_params(case), b_at=[b.data_ptr() + 8 * int(a) for a in starts],
                 x_at=[x.data_ptr() + 8 * int(a) for a in starts])
        return s
    if kind == "gradient":
        case = dict(case, matrix="diffusion")
    csr = _csr(case, gen)
    n = csr[0].numel() - 1
    m = s["m"] = _matrix(h, csr)
    if kind == "spmv":
        if case["fmt"] == "jad":
            m.to_jad()
        s.update(x=_uniform(gen, n), y=torch.empty(n, dtype=F64, device="cuda"),
                 fmt=celgpu.FMT_JAD if case["fmt"] == "jad" else celgpu.FMT_CSR)
        return s
    m.jacobi()
    if case.get("precision", "fp64") != "fp64":
        m.make_fp32()
    if kind == "multirhs":
        k = case["k"]
        xt = _uniform(gen, n, k)
        b = torch.empty(n, k, dtype=F64, device="cuda")
        for c in range(k):
            b[:, c] = _rhs(h, m, xt[:, c].contiguous())
        s.update(b=b, x=torch.empty_like(b), p=_params(case))
        return s
    xt = _uniform(gen, n)
    if kind == "gradient":
        # x of the forward solve is in hand; g = dL/dx = A lambda_true
        s.update(x=_uniform(gen, n), g=_rhs(h, m, xt), lam=torch.empty_like(xt), p=_params(case),
                 gv=torch.empty(csr[1].numel(), dtype=F64, device="cuda"),
                 gk=[torch.empty(q, dtype=F64, device="cuda")
                     for q in synth.face_counts(case["nx"], case["ny"], case["nz"])])
        return s
    s.update(b=_rhs(h, m, xt), x=torch.empty_like(xt), p=_params(case))
    if kind == "gmres":
        s["p"] = _params(case, restart=case["restart"], iter_max=2000)
    return s


# ---- one pass ------------------------------------------------------------------

def run(s):
    kind, h = s["case"]["kind"], s["h"]
    if kind == "spmv":
        h.spmv(s["m"], s["x"].data_ptr(), s["y"].data_ptr(), fmt=s["fmt"])
        return s["y"]
    if kind == "elm":
        h.elm_init(s["n"])
        h.elm_set_solver(celgpu.SOLVER_PCG, s["p"])
        h.elm_insert_rows(1, s["rp"], s["ci"], s["v"])
        h.elm_matrix_completed()
        _, niter, _ = h.elm_doit(s["b"])
        x = h.elm_collect_solution(s["n"])
        h.elm_destroy()
        return {"x": x, "iterations": niter}
    if kind == "batched":
        info = h.pcg_batched(s["mats"], s["b_at"], s["x_at"], p=s["p"])
        return {"x": s["x"], "iterations": np.array([i.iter_done for i in info])}
    if kind == "multirhs":
        info = h.pcg_multirhs(s["m"], s["case"]["k"], s["b"].data_ptr(), s["x"].data_ptr(), p=s["p"])
        return {"x": s["x"], "iterations": np.array([i.iter_done for i in info])}
    if kind == "gradient":
        c = s["case"]
        info = h.pcg_adjoint(s["m"], s["x"].data_ptr(), s["g"].data_ptr(), s["lam"].data_ptr(), s["gv"].data_ptr(),
                             p=s["p"])
        h.diffusion7_face_grad(c["nx"], c["ny"], c["nz"], s["lam"].data_ptr(), s["x"].data_ptr(),
                               *[g.data_ptr() for g in s["gk"]])
        return {"lam": s["lam"], "gv": s["gv"], "gk": s["gk"], "iterations": info.iter_done}
    if kind == "gmres":
        info = h.gmres_jacobi(s["m"], s["b"].data_ptr(), s["x"].data_ptr(), p=s["p"])
        return {"x": s["x"], "iterations": info.arnoldi_steps}
    info = h.pcg_jacobi(s["m"], s["b"].data_ptr(), s["x"].data_ptr(), p=s["p"])
    return {"x": s["x"], "iterations": info.iter_done}


# ---- what a pass cannot do without ----------------------------------------------

def _shape(case):
    """Rows and stored entries."""
    if case.get("matrix") == "band":
        n = case["n"]
        return n, n + 2 * n * case["degree"]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    return n, 7 * n - 2 * (nx * ny + ny * nz + nx * nz)


def work(case):
    """The call's inputs and outputs moved once (a matrix as CSR: 12 bytes an
    entry and 4 a row) and, for a solve, the operations of one iteration: how
    many iterations a system takes is not known beforehand."""
    kind = case["kind"]
    if kind == "batched":
        shapes = [_shape({"nx": q, "ny": q, "nz": q}) for q in _batch_sides(case)]
        n, nnz = sum(s[0] for s in shapes), sum(s[1] for s in shapes)
    else:
        n, nnz = _shape(case)
    k = case.get("k", 1)
    moved = 12 * nnz + 4 * n + 16 * n * k
    if kind == "gradient":
        moved += 8 * n + 8 * nnz + 8 * sum(synth.face_counts(case["nx"], case["ny"], case["nz"]))
    flops = (2 * nnz + (0 if kind == "spmv" else 12 * n)) * k
    return {"bytes": moved, "flops": flops}


# ---- the 64-bit answer -------------------------------------------------------------

def exact(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "batched":
        # the solutions are drawn first, as in prepare()
        return {"x": _uniform(gen, sum(q ** 3 for q in _batch_sides(case))), "iterations": None}
    if kind == "gradient":
        case = dict(case, matrix="diffusion")
    rp, ci, v = _csr(case, gen)
    n = rp.numel() - 1
    if kind == "spmv":
        x = _uniform(gen, n)
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), (rp[1:] - rp[:-1]).long())
        return torch.zeros(n, dtype=F64, device="cuda").index_add_(0, rows, v * x[ci.long()])
    if kind == "multirhs":
        return {"x": _uniform(gen, n, case["k"]), "iterations": None}
    x = _uniform(gen, n)
    if kind == "gradient":
        lam, x = x, _uniform(gen, n)
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), (rp[1:] - rp[:-1]).long())
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        gk = []
        for axis, ghost in ((2, (1, 1)), (1, (0, 0, 1, 1)), (0, (0, 0, 0, 0, 1, 1))):
            l, u = (torch.nn.functional.pad(t.reshape(nz, ny, nx), ghost) for t in (lam, x))
            gk.append((-torch.diff(l, dim=axis) * torch.diff(u, dim=axis)).reshape(-1))
        return {"lam": lam, "gv": -lam[rows] * x[ci.long()], "gk": gk, "iterations": None}
    return {"x": x.cpu().numpy() if kind == "elm" else x, "iterations": None}
