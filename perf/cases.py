"""Performance cases of ttgpu: the calls a user's program makes, over the range of sizes it makes them at.

A case is a dict of plain values.  ``prepare`` makes what the program holds before the call (device
operands or device-resident TT handles), ``run`` is one call through the public entry points (the C ABI
of include/ttgpu.h and its Python binding), ``work`` the bytes and operations the call cannot do without,
``exact`` the same outputs from plain torch / numpy in 64 bits.

Kinds
  matvec        one local matvec bfun3 on device operands, FP64 or mixed (BF16 tensor cores)
  phi           one interface update compute_next_Phi, 'lr' or 'rl', normalised as the sweeps call it
  local_solve   one local GMRES solve (the MEX gateway solve3d_2), FP64 or mixed
  round         TT rounding of a sum of Gaussian TTs, handle in, cores out
  amen          a whole AMEn solve of a d-dimensional diffusion problem, its solution as a full tensor
  batch         a grouped batch of independent AMEn solves, every solution as a full tensor
  grad_xAx      value and gradient of <x, A x> with respect to every core
  grad_sampled  value and gradient of sum_s (X[idx_s] - y_s)^2 with respect to every core

TT results have a gauge: singular vectors are defined up to their sign, and the cores of an AMEn solution
up to rotations of nearly converged directions.  Rounded tensors are therefore returned with the signs
fixed core by core, and AMEn solutions contracted to the full tensor, both on the GPU.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tt-toolbox_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ttgpu  # noqa: E402

F64 = torch.float64
PREC = {"fp64": ttgpu.TTG_FP64, "mixed": ttgpu.TTG_MIXED}


# --------------------------------------------------------------------------- the cases

def listed():
    return [
        # Local matvec of a small solve (d=8, n=32 Laplacian, ranks capped at 20): launch latency.
        dict(name="matvec_f64_r20_n32", kind="matvec", r1=20, n=32, r2=20, ra=2, precision="fp64"),
        # Local matvec of the largest solves in FP64, with uneven ranks as truncation leaves them.
        dict(name="matvec_f64_r187_n64", kind="matvec", r1=187, n=64, r2=203, ra=3, precision="fp64"),
        # Local matvec on the BF16 tensor cores at the largest rank a solve is given.
        dict(name="matvec_mixed_r512_n64", kind="matvec", r1=512, n=64, r2=512, ra=3,
             precision="mixed"),
        # Interface update of the d=10, n=64 diffusion solve at its usual ranks.
        dict(name="phi_lr_r61_n64", kind="phi", dir="lr", r1=61, n=64, r2=67, ra=3),
        # Local solve of the same problem, FP64, the reference's GMRES defaults (40 x 2).
        dict(name="solve_f64_r64_n64", kind="local_solve", r1=64, n=64, r2=64, precision="fp64"),
        # Local solve in mixed precision, uneven ranks.
        dict(name="solve_mixed_r97_n64", kind="local_solve", r1=97, n=64, r2=83, precision="mixed"),
        # Rounding after a short sum with a repeated term: ranks drop from 54 to 36.
        dict(name="round_d7_n11_r54", kind="round", d=7, n=11, r=18, terms=2, repeat=1),
        # The rounding workload of the benchmark: d=20, n=16, four rank-64 terms, ranks 256.
        dict(name="round_d20_n16_r256", kind="round", d=20, n=16, r=64, terms=4, repeat=0),
        # Whole AMEn solve, anisotropic diffusion with reaction (operator rank 3), FP64, tol 1e-10.
        dict(name="amen_f64_d4_n40", kind="amen", d=4, n=40, rhs_rank=4, precision="fp64"),
        # Grouped batch of small uneven systems in mixed precision.
        dict(name="batch_mixed_12", kind="batch", precision="mixed",
             systems="3x32r20,4x16r24,5x8r16,3x16r16,6x8r32,4x8r20,3x31r33,5x9r24,4x13r40,3x64r18,"
                     "4x16r64,6x7r16"),
        # Gradient of the energy <x, A x>, d=12, n=32, rank 64: the differentiation workload.
        dict(name="grad_xAx_d12_n32_r64", kind="grad_xAx", d=12, n=32, r=64),
        # Gradient of the sampled loss at a million entries, same tensor.
        dict(name="grad_sampled_1M_r64", kind="grad_sampled", d=12, n=32, r=64, samples=1000000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "phi", "local_solve", "round", "round", "amen", "batch",
                       "grad_xAx", "grad_sampled"])
    if kind == "matvec":
        p = rng.choice(["fp64", "mixed"])
        top = 200 if p == "fp64" else 500
        return dict(kind=kind, r1=_log(rng, 4, top), n=_log(rng, 6, 64), r2=_log(rng, 4, top),
                    ra=rng.choice([2, 3, 5]) if top == 200 else rng.choice([2, 3]), precision=p)
    if kind == "phi":
        return dict(kind=kind, dir=rng.choice(["lr", "rl"]), r1=_log(rng, 4, 200),
                    n=_log(rng, 6, 64), r2=_log(rng, 4, 200), ra=rng.choice([2, 3, 5]))
    if kind == "local_solve":
        return dict(kind=kind, r1=_log(rng, 8, 120), n=_log(rng, 8, 64), r2=_log(rng, 8, 120),
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "round":
        return dict(kind=kind, d=rng.randint(3, 16), n=_log(rng, 4, 32), r=_log(rng, 4, 56),
                    terms=rng.randint(1, 4), repeat=rng.choice([0, 1]))
    if kind == "amen":
        d = rng.randint(3, 6)
        top = {3: 64, 4: 40, 5: 17, 6: 11}[d]
        return dict(kind=kind, d=d, n=_log(rng, max(6, top // 4), top), rhs_rank=rng.randint(1, 4),
                    precision=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "batch":
        sys_ = []
        for _ in range(rng.randint(2, 12)):
            d = rng.randint(3, 6)
            sys_.append("%dx%dr%d" % (d, _log(rng, 6, {3: 64, 4: 17, 5: 9, 6: 8}[d]),
                                      rng.randint(16, 64)))
        return dict(kind=kind, precision=rng.choice(["fp64", "mixed"]), systems=",".join(sys_))
    if kind == "grad_xAx":
        return dict(kind=kind, d=rng.randint(3, 12), n=_log(rng, 6, 32), r=_log(rng, 4, 64))
    return dict(kind=kind, d=rng.randint(3, 12), n=_log(rng, 6, 32), r=_log(rng, 4, 64),
                samples=_log(rng, 2000, 800000))


# --------------------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=F64)


def _lap(n):
    return (n + 1) ** 2 * (2.0 * np.eye(n) - np.eye(n, k=1) - np.eye(n, k=-1))


def _mass(n):
    return (4.0 * np.eye(n) + np.eye(n, k=1) + np.eye(n, k=-1)) / 6.0


def _flat(a):
    """Column-major flat copy of a numpy or torch array."""
    if isinstance(a, torch.Tensor):
        return a.permute(*range(a.dim() - 1, -1, -1)).contiguous().reshape(-1)
    return np.ascontiguousarray(a.ravel(order="F"))


def _inner_operator(n, ra):
    """Inner operator core [ra, n, n, ra]: the Kronecker-sum core (2), with a reaction term (3), or a
    sum of two such operators (5)."""
    c = np.zeros((ra, n, n, ra))
    c[0, :, :, 0] = c[1, :, :, 1] = np.eye(n)
    c[1, :, :, 0] = _lap(n)
    if ra >= 3:
        c[2, :, :, 2] = _mass(n)
    if ra == 5:
        c[3, :, :, 3] = c[4, :, :, 4] = _mass(n)
        c[4, :, :, 3] = _lap(n)
    return c


def _operator(coef, n, reaction):
    """TT-matrix cores of sum_k coef_k L_k, plus (n + 1)^2 M x .. x M when `reaction`."""
    d, R = len(coef), 3 if reaction else 2
    cores = []
    for k in range(d):
        c = np.zeros((R, n, n, R))
        c[0, :, :, 0] = c[1, :, :, 1] = np.eye(n)
        c[1, :, :, 0] = coef[k] * _lap(n)
        if reaction:
            c[2, :, :, 2] = _mass(n) * ((n + 1) ** 2 if k == 0 else 1.0)
        if k == 0:
            c = c[1:2] + (c[2:3] if reaction else 0.0)
        if k == d - 1:
            last = c[:, :, :, 0:1].copy()
            if reaction:
                last[2] = c[2, :, :, 2:3]
            c = last
        cores.append(c)
    return cores


def _right_orth(n, d, r, rng):
    """Right-orthogonal random TT cores of rank r."""
    rr, cores = [1] + [r] * (d - 1) + [1], [None] * d
    for k in range(d - 1, -1, -1):
        q = np.linalg.qr(rng.standard_normal((n * rr[k + 1], rr[k])))[0].T
        rr[k] = q.shape[0]
        cores[k] = q.reshape((rr[k], n, rr[k + 1]), order="F")
    return cores


def _system(d, n, rhs_rank, reaction, rng):
    """One diffusion system: host TTs (A, y, x0, z0) and what the exact solution needs."""
    coef = rng.uniform(0.5, 2.0, size=d)
    rr = [1] + [rhs_rank] * (d - 1) + [1]
    if rhs_rank == 1:
        y = [1.0 + 0.2 * rng.standard_normal((1, n, 1)) for _ in range(d)]
    else:
        y = [rng.standard_normal((rr[k], n, rr[k + 1])) for k in range(d)]
    x0 = [rng.standard_normal((1 if k == 0 else 2, n, 1 if k == d - 1 else 2)) for k in range(d)]
    A = ttgpu.TTMatrix.from_cores(_operator(coef, n, reaction))
    return dict(A=A, y=ttgpu.TensorTrain.from_cores(y), x0=ttgpu.TensorTrain.from_cores(x0),
                z0=ttgpu.TensorTrain.from_cores(_right_orth(n, d, 4, rng)), coef=coef, ycores=y)


def _round_cores(case, g):
    """Cores of sum_i t_i (+ 0.5 t_0 when `repeat`): Gaussian TTs of rank r, entries N(0, 1/(r n))."""
    d, n, r, terms, rep = (case[k] for k in ("d", "n", "r", "terms", "repeat"))
    T = terms + rep
    cores = []
    for k in range(d):
        r1, r2 = (1 if k == 0 else r), (1 if k == d - 1 else r)
        t = [_randn(g, r1, n, r2) / math.sqrt(r1 * n) for _ in range(terms)]
        if rep:
            t.append(0.5 * t[0] if k == 0 else t[0])
        if k == 0:
            c = torch.cat(t, 2) if d > 1 else sum(t)
        elif k == d - 1:
            c = torch.cat(t, 0)
        else:
            c = torch.zeros(T * r, n, T * r, device="cuda", dtype=F64)
            for i in range(T):
                c[i * r:(i + 1) * r, :, i * r:(i + 1) * r] = t[i]
        cores.append(c)
    return cores


def _tt(cores):
    """Host TensorTrain of torch cores."""
    n = [int(c.shape[1]) for c in cores]
    r = [int(cores[0].shape[0])] + [int(c.shape[2]) for c in cores]
    return ttgpu.TensorTrain(n, r, torch.cat([_flat(c) for c in cores]).cpu().numpy())


def _gauss_tt(d, n, r, g):
    cores = []
    for k in range(d):
        r1, r2 = (1 if k == 0 else r), (1 if k == d - 1 else r)
        cores.append(_randn(g, r1, n, r2) / math.sqrt(r1 * n))
    return cores


def _sym(g, r):
    """Symmetric positive definite interface block, eigenvalues log-uniform in [10, 3000]."""
    q = torch.linalg.qr(_randn(g, r, r))[0]
    lam = torch.exp(torch.rand(r, generator=g, device="cuda", dtype=F64) * math.log(300.0)) * 10.0
    return (q * lam) @ q.T


def _kron_sum(P1, L, P2, x):
    return (torch.einsum("ia,ajk->ijk", P1, x) + torch.einsum("jm,imk->ijk", L, x)
            + torch.einsum("kb,ijb->ijk", P2, x))


def _kron_sum_solve(P1, L, P2, b):
    (l1, q1), (l2, q2), (l3, q3) = (torch.linalg.eigh(M) for M in (P1, L, P2))
    t = torch.einsum("ai,ajk->ijk", q1, b)
    t = torch.einsum("bj,ibk->ijk", q2, t)
    t = torch.einsum("ck,ijc->ijk", q3, t)
    t = t / (l1[:, None, None] + l2[None, :, None] + l3[None, None, :])
    t = torch.einsum("ia,ajk->ijk", q1, t)
    t = torch.einsum("jb,ibk->ijk", q2, t)
    return torch.einsum("kc,ijc->ijk", q3, t)


def _inputs(case, seed):
    """The operands of a kernel-level case, as torch arrays with their mathematical shapes."""
    g, kind = _gen(seed), case["kind"]
    r1, n, r2 = case["r1"], case["n"], case["r2"]
    if kind == "local_solve":
        # One local system of a diffusion solve: (P1 + L + P2) as interfaces and operator core, the
        # right-hand side of a Gaussian solution, and the previous sweep's solution near it.
        P1, P2, L = _sym(g, r1), _sym(g, r2), torch.from_numpy(_lap(n)).cuda()
        L = L * (3000.0 / (4.0 * (n + 1) ** 2))
        x = _randn(g, r1, n, r2)
        rhs = _kron_sum(P1, L, P2, x)
        prev = x + 1e-2 * _randn(g, r1, n, r2)
        e1, e2 = (torch.eye(r, device="cuda", dtype=F64) for r in (r1, r2))
        A = torch.zeros(2, n, n, 2, device="cuda", dtype=F64)
        A[0, :, :, 0] = A[1, :, :, 1] = torch.eye(n, device="cuda", dtype=F64)
        A[1, :, :, 0] = L
        return dict(Phi1=torch.stack([P1, e1], 2), A=A, Phi2=torch.stack([e2, P2], 1), rhs=rhs,
                    prev=prev, blocks=(P1, L, P2))
    ra = case["ra"]
    A = torch.from_numpy(_inner_operator(n, ra)).cuda() / (n + 1) ** 2
    x = _randn(g, r1, n, r2) / math.sqrt(r1 * n)
    if kind == "matvec":
        return dict(Phi1=_randn(g, r1, r1, ra) / r1, A=A, Phi2=_randn(g, r2, ra, r2) / r2, x=x)
    if case["dir"] == "lr":
        return dict(Phi=_randn(g, r1, r1, ra) / r1, A=A, x=x, y=x)
    return dict(Phi=_randn(g, r2, ra, r2) / r2, A=A, x=x, y=x)


def _samples(case, seed):
    """x cores, multi-indices [S, d] and the values of a hidden rank-8 TT at them plus noise."""
    g = _gen(seed)
    d, n, r, S = case["d"], case["n"], case["r"], case["samples"]
    x = _gauss_tt(d, n, r, g)
    idx = torch.randint(0, n, (S, d), generator=g, device="cuda", dtype=torch.int32)
    hidden = _gauss_tt(d, n, min(8, r), g)
    v = torch.ones(S, 1, device="cuda", dtype=F64)
    for k in range(d):
        v = _step(v, hidden[k], idx[:, k])
    return x, idx, v[:, 0] + 1e-3 * _randn(g, S)


def _step(v, core, col):
    """Rows v[s] times core[:, col[s], :], by the values of the index."""
    out = torch.empty(v.shape[0], core.shape[2], device="cuda", dtype=F64)
    for j in range(core.shape[1]):
        at = (col == j).nonzero()[:, 0]
        out[at] = v[at] @ core[:, j, :]
    return out


def _parse(systems):
    out = []
    for t in systems.split(","):
        d, rest = t.split("x")
        n, r = rest.split("r")
        out.append((int(d), int(n), int(r)))
    return out


def _energy_operator(d, n):
    return ttgpu.TTMatrix.from_cores(_operator([1.0] * d, n, True))


def prepare(case, seed):
    kind = case["kind"]
    ctx = ttgpu.default_context()
    s = dict(case=case, ctx=ctx, kind=kind)
    if kind in ("matvec", "phi", "local_solve"):
        ops = _inputs(case, seed)
        s.update({k: _flat(v) for k, v in ops.items() if isinstance(v, torch.Tensor)})
        r1, n, r2 = case["r1"], case["n"], case["r2"]
        size = r1 * n * r2
        if kind == "phi":
            r = r2 if case["dir"] == "lr" else r1
            size = r * r * case["ra"]
        s["out"] = torch.empty(size, device="cuda", dtype=F64)
    elif kind == "round":
        t = _tt(_round_cores(case, _gen(seed)))
        s["x"] = ttgpu.DeviceTT.upload(ctx, t)
        s["host"] = torch.empty(t.core.size, dtype=F64, pin_memory=True)
    elif kind == "amen":
        sy = _system(case["d"], case["n"], case["rhs_rank"], True, np.random.default_rng(seed))
        s.update({k: ttgpu.DeviceTT.upload(ctx, sy[k]) for k in ("A", "y", "x0", "z0")})
    elif kind == "batch":
        rng = np.random.default_rng(seed)
        sys_ = [_system(d, n, 1, False, rng) for d, n, _ in _parse(case["systems"])]
        for k in ("A", "y", "x0", "z0"):
            s[k] = [ttgpu.DeviceTT.upload(ctx, sy[k]) for sy in sys_]
        s["per"] = [dict(rmax=r) for _, _, r in _parse(case["systems"])]
    elif kind == "grad_xAx":
        x = _gauss_tt(case["d"], case["n"], case["r"], _gen(seed))
        s["x"] = ttgpu.DeviceTT.upload(ctx, _tt(x))
        s["A"] = ttgpu.DeviceTT.upload(ctx, _energy_operator(case["d"], case["n"]))
        s["grad"] = torch.empty(sum(c.numel() for c in x), device="cuda", dtype=F64)
    else:
        x, idx, y = _samples(case, seed)
        s["x"] = ttgpu.DeviceTT.upload(ctx, _tt(x))
        s["idx"] = idx.T.contiguous()  # column-major [S, d]
        s["yv"] = y.contiguous()
        s["grad"] = torch.empty(sum(c.numel() for c in x), device="cuda", dtype=F64)
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------------- one call

def _check(code):
    if code:
        raise ttgpu.TTGError(code, ttgpu.lib().ttg_last_error().decode(errors="replace"))


def _full(t):
    """Full tensor of a solution handle, last index fastest, on the GPU."""
    host = t.download()
    t.free()
    core, pos, v = torch.from_numpy(host.core).cuda(), 0, None
    for k in range(host.d):
        r1, n, r2 = int(host.r[k]), int(host.n[k]), int(host.r[k + 1])
        c = core[pos:pos + r1 * n * r2].view(r2, n, r1).permute(2, 1, 0).reshape(r1, n * r2)
        pos += r1 * n * r2
        v = c.reshape(n, r2) if v is None else (v @ c).reshape(-1, r2)
    return v.reshape(-1)


def _signs(cores):
    """Fix the signs of a rounded TT (cores as [r2, n, r1] views): every row of an inner core's right
    unfolding gets a positive weighted sum, its sign moves to the core on its left."""
    for k in range(len(cores) - 1, 0, -1):
        c = cores[k]
        w = torch.linspace(1.0, 2.0, c.shape[0] * c.shape[1], device="cuda", dtype=F64)
        sg = torch.sign(w @ c.reshape(-1, c.shape[2]))
        cores[k] = c * sg
        cores[k - 1] = cores[k - 1] * sg[:, None, None]
    return [c.reshape(-1) for c in cores]


def run(s):
    L, ctx, case, kind = ttgpu.lib(), s["ctx"], s["case"], s["kind"]
    if kind == "matvec":
        ra = case["ra"]
        _check(L.ttg_local_matvec(ctx.h, case["r1"], case["n"], case["r2"], ra, ra,
                                  s["Phi1"].data_ptr(), s["A"].data_ptr(), s["Phi2"].data_ptr(),
                                  s["x"].data_ptr(), s["out"].data_ptr(), PREC[case["precision"]]))
        return s["out"]
    if kind == "phi":
        nrm, ra = ctypes.c_double(0.0), case["ra"]
        _check(L.ttg_next_phi(ctx.h, 0 if case["dir"] == "lr" else 1, case["r1"], case["n"],
                              case["r2"], case["r1"], case["r2"], ra, ra, s["Phi"].data_ptr(),
                              s["x"].data_ptr(), s["A"].data_ptr(), s["y"].data_ptr(),
                              s["out"].data_ptr(), ctypes.byref(nrm)))
        return {"Phi": s["out"], "norm": nrm.value}
    if kind == "local_solve":
        it = ctypes.c_int64(0)
        _check(L.ttg_local_solve(ctx.h, case["r1"], case["n"], case["r2"], 2, 2,
                                 s["Phi1"].data_ptr(), s["A"].data_ptr(), s["Phi2"].data_ptr(),
                                 s["rhs"].data_ptr(), 1e-11, 1, s["prev"].data_ptr(), 0, 40, 2,
                                 s["out"].data_ptr(), PREC[case["precision"]], ctypes.byref(it)))
        return s["out"]
    if kind == "round":
        t = ttgpu.round(s["x"], 1e-8)
        n, _, r, numel = t.shape()
        _check(L.ttg_tt_download(t.h, ctypes.cast(s["host"].data_ptr(),
                                                  ctypes.POINTER(ctypes.c_double))))
        t.free()
        core, cores, pos = s["host"][:numel].cuda(), [], 0
        for k in range(len(n)):
            r1, nk, r2 = int(r[k]), int(n[k]), int(r[k + 1])
            cores.append(core[pos:pos + r1 * nk * r2].view(r2, nk, r1))
            pos += r1 * nk * r2
        return _signs(cores)
    if kind == "amen":
        x = ttgpu.amen_solve2(s["A"], s["y"], 1e-10, x0=s["x0"], z0=s["z0"], rmax=128,
                              precision=case["precision"])
        return _full(x)
    if kind == "batch":
        xs = ttgpu.amen_solve2_batch(s["A"], s["y"], 1e-10, x0s=s["x0"], z0s=s["z0"], grouped=True,
                                     per_system=s["per"], precision=case["precision"], nswp=20)
        return [_full(x) for x in xs]
    val = ctypes.c_double(0.0)
    if kind == "grad_xAx":
        _check(L.ttg_grad_xAx(s["x"].h, s["A"].h, s["grad"].data_ptr(), ctypes.byref(val)))
    else:
        _check(L.ttg_grad_sampled(s["x"].h, case["samples"], s["idx"].data_ptr(),
                                  s["yv"].data_ptr(), s["grad"].data_ptr(), ctypes.byref(val)))
    return {"grad": s["grad"], "value": val.value}


# --------------------------------------------------------------------------- least work

def _mv(r1, n, r2, ra):
    """Bytes and flops of one local contraction (three products) with operator ranks ra."""
    flops = 2.0 * n * r1 * r2 * (r1 * ra + ra * ra * n + r2 * ra)
    return 8.0 * (r1 * r1 * ra + ra * n * n * ra + r2 * ra * r2 + 2 * r1 * n * r2), flops


def _ranks(d, n, r):
    return [int(min(r, n ** min(k, d - k))) for k in range(d + 1)]


def work(case):
    kind = case["kind"]
    if kind == "matvec":
        b, f = _mv(case["r1"], case["n"], case["r2"], case["ra"])
        return {"bytes": b, "flops": f}
    if kind == "phi":
        r1, n, r2, ra = case["r1"], case["n"], case["r2"], case["ra"]
        return {"bytes": 8.0 * (r1 * r1 * ra + ra * n * n * ra + r2 * ra * r2 + r1 * n * r2),
                "flops": _mv(r1, n, r2, ra)[1]}
    if kind == "local_solve":  # one restart cycle: 40 matvecs, the basis read once a step
        N = case["r1"] * case["n"] * case["r2"]
        b, f = _mv(case["r1"], case["n"], case["r2"], 2)
        return {"bytes": b + 8.0 * N * 40, "flops": 40 * f + 2.0 * 2 * N * 40 * 20}
    d, n = case.get("d"), case.get("n")
    if kind == "round":  # QR sweep, then an SVD of every core, each followed by one product
        R = [1] + [case["r"] * (case["terms"] + case["repeat"])] * (d - 1) + [1]
        q = [1] + [case["r"] * case["terms"]] * (d - 1) + [1]
        q = [int(min(q[k], n ** min(k, d - k))) for k in range(d + 1)]
        fl = 0.0
        for k in range(d - 1):
            fl += 4.0 * q[k] * n * R[k + 1] * min(R[k + 1], q[k] * n) + 2.0 * q[k + 1] * R[k + 1] * n * R[k + 2]
            fl += 22.0 * q[k + 1] ** 3 + 4.0 * q[k + 1] ** 2 * n * q[k + 2] + 2.0 * q[k] * n * q[k + 1] ** 2
        size = sum(R[k] * n * R[k + 1] for k in range(d)) + sum(q[k] * n * q[k + 1] for k in range(d))
        return {"bytes": 8.0 * size, "flops": fl}
    if kind in ("amen", "batch"):  # two sweeps of 40-step local solves at the rank of the solution
        one = [(d, n, 64)] if kind == "amen" else _parse(case["systems"])
        by = fl = 0.0
        for dd, nn, r in one:
            rk = _ranks(dd, nn, min(r, 12))
            fl += 2 * 40 * sum(_mv(rk[k], nn, rk[k + 1], 2)[1] for k in range(dd))
            by += 8.0 * (nn ** dd + dd * 9 * nn * nn)
        return {"bytes": by, "flops": fl}
    rk = [1] + [case["r"]] * (d - 1) + [1]
    size = sum(rk[k] * n * rk[k + 1] for k in range(d))
    if kind == "grad_xAx":  # a sweep of interfaces from either side, two matvecs a core
        return {"bytes": 8.0 * (2 * size + d * 9 * n * n),
                "flops": 4 * sum(_mv(rk[k], n, rk[k + 1], 3)[1] for k in range(d))}
    S = case["samples"]
    return {"bytes": 8.0 * 2 * size + 4.0 * S * d + 8.0 * S,
            "flops": 6.0 * S * sum(rk[k] * rk[k + 1] for k in range(d))}


# --------------------------------------------------------------------------- exact results

def _diffusion_solution(d, n, coef, ycores, reaction):
    """The full solution: L and M are both diagonal in the sine basis."""
    j = torch.arange(1, n + 1, device="cuda", dtype=F64)
    Q = math.sqrt(2.0 / (n + 1)) * torch.sin(math.pi * j[:, None] * j[None, :] / (n + 1))
    co = torch.cos(math.pi * j / (n + 1))
    lam = (n + 1) ** 2 * 2.0 * (1.0 - co)
    mu = (4.0 + 2.0 * co) / 6.0
    full = None
    for c in ycores:
        t = torch.from_numpy(np.ascontiguousarray(c)).cuda()
        full = t.reshape(n, -1) if full is None else torch.einsum("pa,ajb->pjb", full, t).reshape(
            -1, t.shape[2])
    full = full.reshape((n,) * d)
    for k in range(d):
        full = torch.movedim(torch.tensordot(Q, torch.movedim(full, k, 0), dims=1), 0, k)
    den, prod = torch.zeros((n,) * d, device="cuda", dtype=F64), float((n + 1) ** 2)
    for k in range(d):
        shape = [1] * d
        shape[k] = n
        den = den + coef[k] * lam.reshape(shape)
        prod = prod * mu.reshape(shape)
    full = full / (den + (prod if reaction else 0.0))
    for k in range(d):
        full = torch.movedim(torch.tensordot(Q, torch.movedim(full, k, 0), dims=1), 0, k)
    return full.reshape(-1)


def _exact_round(cores):
    d = len(cores)
    cores = [c.cpu() for c in cores]
    for k in range(d - 1):
        r1, n, r2 = cores[k].shape
        q, rr = torch.linalg.qr(cores[k].reshape(r1 * n, r2))
        cores[k] = q.reshape(r1, n, -1)
        cores[k + 1] = torch.einsum("ab,bjc->ajc", rr, cores[k + 1])
    nrm = float(torch.linalg.norm(cores[-1]))
    cores[-1] = cores[-1] / nrm
    for k in range(d - 1, 0, -1):
        r1, n, r2 = cores[k].shape
        u, sv, vt = torch.linalg.svd(cores[k].reshape(r1, n * r2), full_matrices=False)
        tail = torch.flip(torch.cumsum(torch.flip(sv * sv, [0]), 0), [0])
        keep = int((tail >= (1e-8 / math.sqrt(d - 1)) ** 2 * tail[0]).sum())
        cores[k] = vt[:keep].reshape(keep, n, r2)
        cores[k - 1] = torch.einsum("ajb,bc->ajc", cores[k - 1], u[:, :keep] * sv[:keep])
    cores[0] = cores[0] / torch.linalg.norm(cores[0])
    scale = nrm ** (1.0 / d)
    return _signs([(c * scale).permute(2, 1, 0).contiguous().cuda() for c in cores])


def _exact_energy(x, A):
    """Value and gradient of <x, A x> by interfaces in 64 bits; x, A lists of cores."""
    d = len(x)
    one = torch.ones(1, 1, 1, device="cuda", dtype=F64)
    left, right = [one], [None] * d + [one]
    for k in range(d):
        t = torch.einsum("apb,ajc->jcpb", left[k], x[k])
        t = torch.einsum("jcpb,pjmq->cbmq", t, A[k])
        left.append(torch.einsum("cbmq,bme->cqe", t, x[k]))
    for k in range(d - 1, -1, -1):
        t = torch.einsum("bme,cqe->bmcq", x[k], right[k + 1])
        t = torch.einsum("bmcq,pjmq->bcpj", t, A[k])
        right[k] = torch.einsum("bcpj,ajc->apb", t, x[k])
    grad = []
    for k in range(d):
        # derivative through the row copy, then through the column copy
        t = torch.einsum("apb,bme->apme", left[k], x[k])
        t = torch.einsum("apme,pjmq->ajqe", t, A[k])
        g = torch.einsum("ajqe,cqe->ajc", t, right[k + 1])
        t = torch.einsum("apb,ajc->bpjc", left[k], x[k])
        t = torch.einsum("bpjc,pjmq->bmqc", t, A[k])
        g = g + torch.einsum("bmqc,cqe->bme", t, right[k + 1])
        grad.append(_flat(g))
    return {"grad": torch.cat(grad), "value": float(left[d].reshape(-1)[0])}


def _exact_sampled(x, idx, y):
    d, S = len(x), idx.shape[0]
    left = [torch.ones(S, 1, device="cuda", dtype=F64)]
    for k in range(d):
        left.append(_step(left[k], x[k], idx[:, k]))
    e = left[d][:, 0] - y
    right = (2.0 * e)[:, None]
    grad = [None] * d
    for k in range(d - 1, -1, -1):
        r1, n, r2 = x[k].shape
        g = torch.zeros(r1, n, r2, device="cuda", dtype=F64)
        nxt = torch.empty(S, r1, device="cuda", dtype=F64)
        for j in range(n):
            at = (idx[:, k] == j).nonzero()[:, 0]
            g[:, j, :] = left[k][at].T @ right[at]
            nxt[at] = right[at] @ x[k][:, j, :].T
        grad[k] = _flat(g)
        right = nxt
    return {"grad": torch.cat(grad), "value": float((e * e).sum())}


def exact(case, seed):
    kind = case["kind"]
    if kind == "matvec":
        o = _inputs(case, seed)
        t = torch.einsum("amb,bqk->amqk", o["x"], o["Phi2"])
        t = torch.einsum("pjmq,amqk->apjk", o["A"], t)
        return _flat(torch.einsum("iap,apjk->ijk", o["Phi1"], t))
    if kind == "phi":
        o = _inputs(case, seed)
        if case["dir"] == "lr":
            t = torch.einsum("abp,ajc->bpjc", o["Phi"], o["x"])
            t = torch.einsum("bpjc,pjmq->bmqc", t, o["A"])
            r = torch.einsum("bmqc,bme->ceq", t, o["y"])
        else:
            t = torch.einsum("bme,eqc->bmqc", o["y"], o["Phi"])
            t = torch.einsum("bmqc,pjmq->bpjc", t, o["A"])
            r = torch.einsum("bpjc,ajc->bpa", t, o["x"])
        nrm = float(torch.linalg.norm(r))
        return {"Phi": _flat(r / nrm), "norm": nrm}
    if kind == "local_solve":
        o = _inputs(case, seed)
        return _flat(_kron_sum_solve(*o["blocks"], o["rhs"]))
    if kind == "round":
        return _exact_round(_round_cores(case, _gen(seed)))
    if kind == "amen":
        sy = _system(case["d"], case["n"], case["rhs_rank"], True, np.random.default_rng(seed))
        return _diffusion_solution(case["d"], case["n"], sy["coef"], sy["ycores"], True)
    if kind == "batch":
        rng, out = np.random.default_rng(seed), []
        for d, n, _ in _parse(case["systems"]):
            sy = _system(d, n, 1, False, rng)
            out.append(_diffusion_solution(d, n, sy["coef"], sy["ycores"], False))
        return out
    if kind == "grad_xAx":
        x = _gauss_tt(case["d"], case["n"], case["r"], _gen(seed))
        A = [torch.from_numpy(c).cuda() for c in _operator([1.0] * case["d"], case["n"], True)]
        return _exact_energy(x, A)
    x, idx, y = _samples(case, seed)
    return _exact_sampled(x, idx, y)
