"""What a program that uses this library has it do, as measurable cases.

A case names one call sequence of the multigrid hot path through the C ABI
(include/gmg.h), with its sizes; listed() gives twelve of them, draw() others of
the same ranges.  The sizes are those of the benchmark configurations (fine
lattices of 16^4 and 32^4, nbasis 24 to 40, 1 to 32 right-hand sides) and of
the tests, down to the 256-site lattices of the coarse levels.

  stencil         coarse Dirac operator M / Mdag, 1 to 32 RHS, each compute type
  transfer        the K-cycle's restriction (project) and prolongation (promote)
  ortho           block orthonormalisation of a fresh set of test vectors
  wilson          fine Wilson-clover M
  wilson_mr       the smoother's step: M with the minimal-residual products
  coarsen_wilson  Galerkin coarse operator from the Wilson-clover operator
  coarsen_coarse  Galerkin coarse operator from a coarse operator
  mg_solve        the mixed-precision multigrid solve of D x = b

Fields are torch CUDA tensors in the library's layouts.  exact() restates each
result in 64 bits with plain torch.
"""
import ctypes
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "grid-mg-bench_b200"))
import gmg  # noqa: E402

PREC = {"f64": 0, "f32": 1, "bf16": 2, "f16": 3}
OPS = {"M": 0, "Mdag": 1}


# ------------------------------------------------------------------ the cases
def _lat(p, d):
    return {p + "x": d[0], p + "y": d[1], p + "z": d[2], p + "t": d[3]}


def _dims(case, p=""):
    return tuple(case[p + k] for k in "xyzt")


def _vol(d):
    return d[0] * d[1] * d[2] * d[3]


def listed():
    L32, L16, L8, L4, b4, b2 = ((n,) * 4 for n in (32, 16, 8, 4, 4, 2))
    return [
        # one application of the coarsest operator inside a single-RHS Krylov solve: latency
        dict(name="stencil_f64_1rhs", kind="stencil", op="M", compute="f64", nbasis=24, nrhs=1, **_lat("", L4)),
        # an adjoint apply on an uneven lattice with a batch that some RHS have left
        dict(name="stencil_f32_ragged", kind="stencil", op="Mdag", compute="f32", nbasis=40, nrhs=5,
             **_lat("", (6, 4, 5, 7))),
        # the multi-RHS coarse operator in full precision and as the preconditioner uses it
        dict(name="stencil_f64_32rhs", kind="stencil", op="M", compute="f64", nbasis=32, nrhs=32, **_lat("", L8)),
        dict(name="stencil_bf16_32rhs", kind="stencil", op="M", compute="bf16", nbasis=32, nrhs=32, **_lat("", L8)),
        # restriction and prolongation of an FP64 cycle, and of the preconditioner's 32-RHS batch
        dict(name="transfer_f64", kind="transfer", compute="f64", nbasis=24, nrhs=12, **_lat("", L16), **_lat("b", b4)),
        dict(name="transfer_bf16", kind="transfer", compute="bf16", nbasis=32, nrhs=32, **_lat("", L32),
             **_lat("b", b4)),
        # setup: the test vectors of a level made into a block basis
        dict(name="ortho", kind="ortho", nbasis=32, **_lat("", L32), **_lat("b", b4)),
        # the fine operator of an unpreconditioned single-RHS solve
        dict(name="wilson_f64_1rhs", kind="wilson", prec="f64", nrhs=1, **_lat("", L32)),
        # one step of the fine smoother on the whole batch
        dict(name="wilson_mr_bf16_24rhs", kind="wilson_mr", prec="bf16", nrhs=24, **_lat("", L32)),
        # setup: coarse operators of both levels
        dict(name="coarsen_wilson", kind="coarsen_wilson", nbasis=40, **_lat("", L32), **_lat("b", b4)),
        dict(name="coarsen_coarse", kind="coarsen_coarse", dof=40, nbasis=40, **_lat("", L8), **_lat("b", b2)),
        # the whole solve of a batch
        dict(name="mg_solve", kind="mg_solve", prec="bf16", nrhs=24, nvec0=12, nvec1=16, **_lat("", L16)),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stencil", "stencil", "transfer", "transfer", "wilson", "wilson_mr", "ortho", "coarsen_wilson",
                       "coarsen_coarse", "mg_solve"])
    nbasis = 2 * rng.randint(4, 20)
    if kind == "stencil":
        return dict(kind=kind, op=rng.choice(["M", "Mdag"]), compute=rng.choice(["f64", "f32", "bf16", "f16"]),
                    nbasis=nbasis, nrhs=_log_int(rng, 1, 32), **_lat("", [rng.randint(3, 8) for _ in range(4)]))
    if kind in ("wilson", "wilson_mr"):
        prec = rng.choice(["f64", "f32"] if kind == "wilson" else ["f32", "bf16"])
        return dict(kind=kind, prec=prec, nrhs=_log_int(rng, 1, 24), **_lat("", [rng.randint(8, 24) for _ in range(4)]))
    if kind in ("transfer", "ortho"):
        b = [rng.choice([2, 3, 4]) for _ in range(4)]
        more = dict(compute=rng.choice(["f64", "f32", "bf16"]), nrhs=_log_int(rng, 1, 32)) if kind == "transfer" else {}
        return dict(kind=kind, nbasis=nbasis, **more, **_lat("", [x * rng.randint(2, 6) for x in b]), **_lat("b", b))
    if kind == "coarsen_wilson":
        b = [rng.choice([2, 4]) for _ in range(4)]
        return dict(kind=kind, nbasis=nbasis, **_lat("", [x * 2 * rng.randint(1, 3) for x in b]), **_lat("b", b))
    if kind == "coarsen_coarse":
        return dict(kind=kind, dof=2 * rng.randint(8, 20), nbasis=nbasis,
                    **_lat("", [4 * rng.randint(1, 2) for _ in range(4)]), **_lat("b", (2,) * 4))
    return dict(kind=kind, prec=rng.choice(["bf16", "f32"]), nrhs=rng.randint(2, 24), nvec0=rng.randint(8, 12),
                nvec1=rng.randint(8, 16), **_lat("", [8 * rng.randint(1, 2) for _ in range(4)]))


# ------------------------------------------------------------------ inputs
def _gen(seed, stream):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + stream)
    return g


def _gauss(shape, seed, stream, dtype=torch.complex128):
    """Unit Gaussian complex numbers (E|z|^2 = 1)."""
    z = torch.randn(tuple(shape) + (2,), generator=_gen(seed, stream), device="cuda", dtype=torch.float64)
    return torch.view_as_complex(z.mul_(0.5 ** 0.5)).to(dtype)


def _gauge(dims, seed, eps=0.3):
    """U = exp(i eps H), H traceless Hermitian with unit-variance Gaussian entries: [V][4][3][3]."""
    a = _gauss((_vol(dims) * 4, 3, 3), seed, 1)
    h = (a + a.mH) / math.sqrt(2.0)
    h = h - torch.diagonal(h, dim1=-2, dim2=-1).sum(-1)[:, None, None] / 3 * torch.eye(3, device="cuda", dtype=torch.float64)
    a = h * (1j * eps / 32)
    u = torch.eye(3, device="cuda", dtype=a.dtype) + a
    term = a
    for k in range(2, 13):
        term = term @ a / k
        u = u + term
    for _ in range(5):
        u = u @ u
    return u.reshape(_vol(dims), 4, 3, 3).contiguous()


def _blocked(f, dims, b):
    """[V][...] in lattice order -> [Vc][bv][...], block sites in lattice order."""
    c = [n // k for n, k in zip(dims, b)]
    v = f.reshape(c[3], b[3], c[2], b[2], c[1], b[1], c[0], b[0], -1).permute(0, 2, 4, 6, 1, 3, 5, 7, 8)
    return v.reshape(_vol(c), _vol(b), *f.shape[1:])


def _unblocked(f, dims, b):
    c = [n // k for n, k in zip(dims, b)]
    v = f.reshape(c[3], c[2], c[1], c[0], b[3], b[2], b[1], b[0], -1).permute(0, 4, 1, 5, 2, 6, 3, 7, 8)
    return v.reshape(_vol(dims), *f.shape[2:])


def _orthonormal(B, dims, b):
    """Block Gram-Schmidt of basis vectors [N][V][dof], as one Cholesky factorisation per block."""
    out = torch.empty_like(B)
    N, dof = B.shape[0], B.shape[2]
    V = _blocked(B.permute(1, 0, 2), dims, b).permute(0, 2, 1, 3).reshape(-1, N, _vol(b) * dof)
    W = torch.linalg.solve_triangular(torch.linalg.cholesky(V @ V.mH), V, upper=False)
    del V
    out.copy_(_unblocked(W.reshape(W.shape[0], N, _vol(b), dof).permute(0, 2, 1, 3), dims, b).permute(1, 0, 2))
    return out


def _doubled(N, V, dof, seed, stream):
    """N / 2 Gaussian vectors, chirally doubled: [N][V][dof]."""
    h = _gauss((N // 2, V, dof), seed, stream)
    B = torch.zeros((N, V, dof), dtype=torch.complex128, device="cuda")
    B[: N // 2, :, : dof // 2] = h[:, :, : dof // 2]
    B[N // 2:, :, dof // 2:] = h[:, :, dof // 2:]
    return B


def _nbr(dims, p):
    """Neighbour of every site for stencil point p (p < 4: +dir p, p < 8: -dir p - 4, 8: the site)."""
    s = torch.arange(_vol(dims), device="cuda").reshape(dims[3], dims[2], dims[1], dims[0])
    return (s if p == 8 else torch.roll(s, -1 if p < 4 else 1, 3 - p % 4)).reshape(-1)


def _signs(N):
    """-1 where the two indices lie in different chiral halves."""
    k = torch.arange(N, device="cuda") // (N // 2)
    return 1.0 - 2.0 * ((k[:, None] + k[None, :]) % 2).double()


def _links(dims, N, seed, stream):
    """Coarse links [9][V][N][N] with the gamma5-hermitian structure of a Galerkin operator."""
    A = _gauss((9, _vol(dims), N, N), seed, stream) / math.sqrt(9.0 * N)
    S = _signs(N)
    for d in range(4):
        A[d] = S * A[4 + d][_nbr(dims, d)].mH
    A[8] = 0.5 * (A[8] + S * A[8].mH)
    return A


def _inputs(case, seed):
    """The tensors of a case, from the seed alone."""
    kind, d = case["kind"], _dims(case)
    V = _vol(d)
    if kind == "stencil":
        N, R = case["nbasis"], case["nrhs"]
        dt = torch.complex128 if case["compute"] == "f64" else torch.complex64
        return dict(links=_links(d, N, seed, 2), x=_gauss((V, R, N), seed, 3, dt))
    if kind == "transfer":
        dt = torch.complex128 if case["compute"] == "f64" else torch.complex64
        B = _orthonormal(_doubled(case["nbasis"], V, 12, seed, 4), d, _dims(case, "b"))
        return dict(basis=B, x=_gauss((V, case["nrhs"], 12), seed, 5, dt))
    if kind == "ortho":
        return dict(basis=_doubled(case["nbasis"], V, 12, seed, 6))
    if kind in ("wilson", "wilson_mr"):
        x = _gauss((V, case["nrhs"], 12), seed, 7, torch.complex128 if case["prec"] == "f64" else torch.complex64)
        return dict(gauge=_gauge(d, seed), x=torch.view_as_real(x).to(torch.bfloat16) if case["prec"] == "bf16" else x)
    if kind == "coarsen_wilson":
        return dict(gauge=_gauge(d, seed),
                    basis=_orthonormal(_doubled(case["nbasis"], V, 12, seed, 8), d, _dims(case, "b")))
    if kind == "coarsen_coarse":
        return dict(links=_links(d, case["dof"], seed, 9),
                    basis=_orthonormal(_doubled(case["nbasis"], V, case["dof"], seed, 10), d, _dims(case, "b")))
    # the right-hand sides of a solve whose solution is known
    U, x = _gauge(d, seed), _gauss((V, case["nrhs"], 12), seed, 11)
    return dict(gauge=U, x=x, b=_wilson(d, U, MASS["mg_solve"], x))


# the configurations' masses (clover coefficient 1, antiperiodic in time)
MASS = {"wilson": -0.3, "wilson_mr": -0.35, "coarsen_wilson": -0.3, "mg_solve": -0.35}


# ------------------------------------------------------------------ the calls
def _abi(fn, *args):
    st = getattr(gmg.lib(), fn)(*args)
    if st != 0:
        raise gmg.GmgError(st, gmg.lib().gmg_last_error().decode())


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _wilson_handle(case, d, U):
    w = gmg.WilsonClover(d, MASS[case["kind"]], 1.0, antiperiodic=True)
    w.set_gauge(U)
    return w


def prepare(case, seed):
    kind, d = case["kind"], _dims(case)
    i, s = _inputs(case, seed), gmg._stream()
    V = _vol(d)
    if kind == "stencil":
        cm = gmg.CoarsenedMatrix(d, case["nbasis"])
        cm.set_links(i["links"])
        cm.prepare(case["compute"])
        x, out = i["x"], torch.zeros_like(i["x"])
        call = [("gmg_coarse_apply", cm._h, OPS[case["op"]], 8, PREC[case["compute"]],
                 PREC["f64" if case["compute"] == "f64" else "f32"], case["nrhs"], _p(x), _p(out), None, 0, s)]
        return dict(calls=call, out=out, keep=(cm, x))
    if kind in ("wilson", "wilson_mr"):
        w = _wilson_handle(case, d, i["gauge"])
        x, out = i["x"], torch.zeros_like(i["x"])
        if kind == "wilson":
            call = ("gmg_wilson_apply", w._h, OPS["M"], 0, 0, PREC[case["prec"]], case["nrhs"], _p(x), _p(out), s)
            return dict(calls=[call], out=out, keep=(w, x))
        dots = torch.zeros((2, case["nrhs"]), dtype=torch.complex128, device="cuda")
        call = ("gmg_wilson_apply_mr", w._h, PREC[case["prec"]], case["nrhs"], _p(x), _p(out), _p(dots[0]), _p(dots[1]),
                s)
        return dict(calls=[call], out=[out, dots], keep=(w, x))
    if kind == "mg_solve":
        w = _wilson_handle(case, d, i["gauge"])
        mg = gmg.MultiGrid(w, case["nrhs"], prec=case["prec"], nlevels=3,
                           block=(tuple(4 if n == 16 else 2 for n in d), (2,) * 4),
                           nvec=(case["nvec0"], case["nvec1"]), smoother_iters=8)
        mg.setup()
        return dict(mg=mg, b=i["b"], out=torch.zeros_like(i["b"]), keep=w)
    N, c = case["nbasis"], [n // k for n, k in zip(d, _dims(case, "b"))]
    ag = gmg.Aggregation(d, c, case.get("dof", 12), N)
    if kind == "ortho":
        out = torch.zeros_like(i["basis"])
        calls = [("gmg_agg_set_basis", ag._h, _p(i["basis"]), 1, s), ("gmg_agg_orthonormalise", ag._h, 1, s),
                 ("gmg_agg_get_basis", ag._h, _p(out), 1, s)]
        return dict(calls=calls, out=out, keep=(ag, i["basis"]))
    ag.set_basis(i["basis"])
    if kind == "transfer":
        x, back = i["x"], torch.zeros_like(i["x"])
        y = torch.zeros((_vol(c), case["nrhs"], N), dtype=x.dtype, device="cuda")
        cp, vp = PREC[case["compute"]], PREC["f64" if case["compute"] == "f64" else "f32"]
        calls = [("gmg_agg_project", ag._h, cp, vp, case["nrhs"], _p(x), _p(y), s),
                 ("gmg_agg_promote", ag._h, cp, vp, case["nrhs"], _p(y), _p(back), s)]
        return dict(calls=calls, out=[y, back], keep=(ag, x))
    # the new coarse operator, and its links as a program reads them
    cm, links = gmg.CoarsenedMatrix(c, N), torch.zeros((9, _vol(c), N, N), dtype=torch.complex128, device="cuda")
    if kind == "coarsen_wilson":
        fine, call = _wilson_handle(case, d, i["gauge"]), "gmg_coarsen_wilson"
    else:
        fine, call = gmg.CoarsenedMatrix(d, case["dof"]), "gmg_coarsen_coarse"
        fine.set_links(i["links"])
    return dict(calls=[(call, cm._h, ag._h, fine._h, s), ("gmg_coarse_get_links", cm._h, _p(links), 1, s)], out=links,
                keep=(cm, ag, fine))


def run(state):
    if "mg" in state:  # from a zero initial guess, to where the solution itself is converged
        state["out"].zero_()
        state["mg"].solve(state["b"], state["out"], tol=1e-12, maxiter=400)
    else:
        for call in state["calls"]:
            _abi(*call)
    return state["out"]


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Bytes: every input read once, every output written once, at the stored precision (a BF16 / F16
    coarse link counts 4 bytes, its vectors 8).  Flops: 8 per complex multiply-add."""
    kind, d = case["kind"], _dims(case)
    V, R, N = _vol(d), case.get("nrhs", 1), case.get("nbasis", 0)
    if kind == "stencil":
        cb = 16 if case["compute"] == "f64" else 8
        lb = {"f64": 16, "f32": 8}.get(case["compute"], 4)
        return dict(bytes=V * (9 * N * N * lb + 2 * R * N * cb), flops=8.0 * 9 * V * N * N * R)
    if kind in ("wilson", "wilson_mr"):
        cb = {"f64": 16, "f32": 8, "bf16": 4}[case["prec"]]
        return dict(bytes=V * (24 * R * cb + 108 * max(cb, 8)), flops=1824.0 * V * R)
    if kind == "mg_solve":  # one K-cycle's smoothing and operator products, some 25 times
        return dict(bytes=25 * 10 * V * R * 24 * 4, flops=25 * 10 * 1824.0 * V * R)
    Vc, dof = V // _vol(_dims(case, "b")), case.get("dof", 12)
    if kind == "transfer":
        cb = 16 if case["compute"] == "f64" else 8
        return dict(bytes=2 * cb * (N * V * dof + V * R * dof + Vc * R * N), flops=16.0 * V * dof * N * R)
    if kind == "ortho":
        return dict(bytes=2 * 16 * N * V * dof, flops=8.0 * V * dof * N * N)
    # four backward hops on one face of each block and the self term without the hops between blocks
    face = sum(1.0 / b for b in _dims(case, "b"))
    hop, diag = (2 * 72 + 24 + 24, 504) if kind == "coarsen_wilson" else (8.0 * dof * dof, 8.0 * dof * dof)
    fine = 16 * (108 if kind == "coarsen_wilson" else 9 * dof * dof)
    return dict(bytes=V * (fine + 16 * N * dof) + 16 * 9 * Vc * N * N,
                flops=V * N * (face * hop + (8 - 2 * face) * hop + diag) + (1 + face) * 8.0 * V * dof * N * N)


# ------------------------------------------------------------------ the results in 64 bits
def _gammas():
    g = torch.zeros((4, 4, 4), dtype=torch.complex128)
    for mu, e in enumerate([(1j, 1j, -1j, -1j), (-1, 1, 1, -1), (1j, -1j, -1j, 1j), (1, 1, 1, 1)]):
        for a, (b, v) in enumerate(zip((3, 2, 1, 0) if mu < 2 else (2, 3, 0, 1), e)):
            g[mu, a, b] = v
    return g.cuda()


def _hop(dims, U, p, x):
    """-1/2 (1 -+ gamma) U x(neighbour), antiperiodic in time; x [V][R][12]."""
    mu, n = p % 4, _nbr(dims, p)
    t = torch.arange(_vol(dims), device="cuda") // _vol((dims[0], dims[1], dims[2], 1))
    edge = (t == (dims[3] - 1 if p < 4 else 0)) if mu == 3 else torch.zeros_like(t, dtype=torch.bool)
    L = U[:, mu] if p < 4 else U[n, mu].mH
    L = L * torch.where(edge, 0.5, -0.5)[:, None, None]
    P = torch.eye(4, device="cuda") + (-1 if p < 4 else 1) * _gammas()[mu]
    y = (x[n].reshape(x.shape[0], -1, 3) @ L.mT).reshape(-1, x.shape[1], 4, 3)
    return torch.einsum("ab,srbc->srac", P, y).reshape(x.shape)


def _diag(dims, U, mass, x, csw=1.0):
    """(4 + m + clover) x."""
    G, V = _gammas(), _vol(dims)
    Cl = torch.zeros((V, 4, 3, 4, 3), dtype=torch.complex128, device="cuda")
    u = lambda mu, s: U[s, mu]  # noqa: E731
    for mu in range(4):
        for nu in range(mu + 1, 4):
            s = _nbr(dims, 8)
            pm, pn, mm, mn = _nbr(dims, mu), _nbr(dims, nu), _nbr(dims, 4 + mu), _nbr(dims, 4 + nu)
            Q = u(mu, s) @ u(nu, pm) @ u(mu, pn).mH @ u(nu, s).mH
            Q = Q + u(nu, s) @ u(mu, pn[mm]).mH @ u(nu, mm).mH @ u(mu, mm)
            Q = Q + u(mu, mm).mH @ u(nu, mn[mm]).mH @ u(mu, mn[mm]) @ u(nu, mn)
            Q = Q + u(nu, mn).mH @ u(mu, mn) @ u(nu, pm[mn]) @ u(mu, s).mH
            sig = 0.5j * (G[mu] @ G[nu] - G[nu] @ G[mu])
            Cl += torch.einsum("ab,scd->sacbd", -0.5 * csw * sig, (Q - Q.mH) / 8j)
    Cl = Cl.reshape(V, 12, 12) + (4 + mass) * torch.eye(12, device="cuda", dtype=torch.float64)
    return x @ Cl.mT


def _wilson(dims, U, mass, x):
    y = _diag(dims, U, mass, x)
    for p in range(8):
        y += _hop(dims, U, p, x)
    return y


def _galerkin(case, basis, hop, self_term):
    """Links of the coarse operator: hop(p, x) the fine hop, self_term(x) its site-diagonal part."""
    d, b, N = _dims(case), _dims(case, "b"), case["nbasis"]
    V, c = _vol(d), [n // k for n, k in zip(_dims(case), _dims(case, "b"))]
    phi = basis.permute(1, 0, 2).contiguous()
    panel = _blocked(phi, d, b).permute(0, 2, 1, 3).reshape(_vol(c), N, -1).conj()

    def project(w):
        return panel @ _blocked(w, d, b).permute(0, 1, 3, 2).reshape(_vol(c), -1, N)

    s = torch.arange(V, device="cuda")
    at, even = [], 0
    for k in range(4):
        at.append(s % d[k])
        even = even + at[k] // b[k]
        s = s // d[k]
    A = torch.zeros((9, _vol(c), N, N), dtype=torch.complex128, device="cuda")
    w = self_term(phi)
    for p in range(8):
        n = _nbr(d, p)
        h = hop(p, phi)
        if p >= 4:
            A[p] = project(h * (at[p - 4] % b[p - 4] == 0)[:, None, None])
        w += h * ((even[n] - even) % 2 == 0)[:, None, None]
        del h
    A[8] = project(w)
    for k in range(4):
        A[k] = _signs(N) * A[4 + k][_nbr(c, k)].mH
    return A


def exact(case, seed):
    kind, d = case["kind"], _dims(case)
    i = _inputs(case, seed)
    if kind == "stencil":
        x = i["x"].to(torch.complex128)
        g5 = torch.ones(case["nbasis"], device="cuda", dtype=torch.float64)
        g5[case["nbasis"] // 2:] = -1
        if case["op"] == "Mdag":
            x = x * g5
        y = torch.zeros_like(x)
        for p in range(9):
            y += x[_nbr(d, p)] @ i["links"][p].mT
        return y * g5 if case["op"] == "Mdag" else y
    if kind == "transfer":
        N, b = case["nbasis"], _dims(case, "b")
        panel = _blocked(i["basis"].permute(1, 0, 2), d, b).permute(0, 2, 1, 3)
        panel = panel.reshape(panel.shape[0], N, -1)
        f = _blocked(i["x"].to(torch.complex128), d, b).permute(0, 2, 1, 3)
        y = f.reshape(f.shape[0], f.shape[1], -1) @ panel.mH
        back = (y @ panel).reshape(f.shape).permute(0, 2, 1, 3)
        return [y, _unblocked(back, d, b)]
    if kind == "ortho":
        return _orthonormal(i["basis"], d, _dims(case, "b"))
    if kind in ("wilson", "wilson_mr"):
        x = (torch.view_as_complex(i["x"].double()) if case["prec"] == "bf16" else i["x"]).to(torch.complex128)
        y = _wilson(d, i["gauge"], MASS[kind], x)
        if kind == "wilson":
            return y
        dots = torch.stack([(y.conj() * x).sum((0, 2)), (y.conj() * y).sum((0, 2)).real + 0j])
        return [torch.view_as_real(y) if case["prec"] == "bf16" else y, dots]
    if kind == "coarsen_wilson":
        U, m = i["gauge"], MASS[kind]
        return _galerkin(case, i["basis"], lambda p, x: _hop(d, U, p, x), lambda x: _diag(d, U, m, x))
    if kind == "coarsen_coarse":
        A = i["links"]
        return _galerkin(case, i["basis"], lambda p, x: x[_nbr(d, p)] @ A[p].mT, lambda x: x @ A[8].mT)
    return i["x"]
