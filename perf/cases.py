"""The work a user of mpsgb has it do, as cases that can be timed and compared.

A case names a `call` (the entry point a driver or a user's program goes through), the bond
dimensions on the left and right (`Dl`, `Dr`), the MPO, the storage type and the arithmetic:

  apply     y = H x with a prepared operator (Galerkin errors, expectation values)
  solve     operator built from its environments, then the Lanczos ground state (a local
            update of DMRG, DMRG2, VUMPS or IDMRG up to the gauge step)
  evolve    operator built from its environments, then exp(-i dt H) x (a TDVP local step)
  transfer  one environment step to the left and one to the right
  orth      positive QR and LQ of a site tensor (the gauge step of one-site algorithms)
  update    solve followed by the truncated factorisation of the two-site tensor
  timestep  a whole TDVP time step of a finite chain

`sym` = "u1" runs the charge-conserving forms on a Heisenberg chain or a J1-J2 cylinder; the
dense cases use an XXZ interaction that is a sum of decaying exponentials (`nexp` of them:
MPO width 2 + 3 nexp; decay 0 is the nearest-neighbour chain) or the transverse-field Ising
chain, on environments of a random canonical state.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpskit.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import mpsgb  # noqa: E402
from mpsgb import u1 as mu1  # noqa: E402

D_PHYS = 2
QP = mpsgb.operators.SPIN_HALF_CHARGES
KINDS = {"C": mpsgb._lib.GB_HEFF_C, "AC": mpsgb._lib.GB_HEFF_AC, "AC2": mpsgb._lib.GB_HEFF_AC2}
XKIND = {"C": "bond", "AC": "mps", "AC2": "ac2"}


def listed():
    return [
        # the bond operator of a tiny edge bond: nothing but latency and launches
        _dense("bond_apply_D23", "apply", "C", 23, 23, "tfim", 0, "c128", "fp64"),
        # two-site DMRG of a Heisenberg chain at D = 64, the plain default precision
        _dense("ac2_solve_D64_c128", "solve", "AC2", 64, 64, "xxz", 1, "c128", "fp64", krylov=20),
        # VUMPS of an XXZ chain at D = 256, plain and split (the precision sweep users run)
        _dense("ac_solve_D256_c128", "solve", "AC", 256, 256, "xxz", 1, "c128", "fp64", krylov=30),
        _dense("ac_solve_D256_c128_tf32x3", "solve", "AC", 256, 256, "xxz", 1, "c128", "tf32x3",
               krylov=30),
        # the local step of one-site TDVP
        _dense("ac_evolve_D128_c128", "evolve", "AC", 128, 128, "xxz", 1, "c128", "fp64",
               krylov=30),
        # environment recursions, ragged bonds
        _dense("transfer_D450x515_f64", "transfer", "", 450, 515, "xxz", 1, "f64", "fp64"),
        # gauge of a uniform state (the QR and LQ that VUMPS repeats)
        _dense("orth_D256_c128", "orth", "", 256, 256, "", 0, "c128", "fp64"),
        # long-range dense Hamiltonian on the tensor cores, odd bonds
        _dense("ac2_solve_D509_f64_bf16x3", "solve", "AC2", 509, 509, "xxz", 4, "f64", "bf16x3",
               krylov=12),
        # a whole time step of a small chain
        _chain("timestep_L12_D32_c128", 12, 32),
        # the plain-precision leg of a symmetric run
        _u1("ac2_solve_u1_D512_f64", "solve", "chain", 512, "fp64", 12),
        # two-site DMRG of the U(1) Heisenberg chain, D = 1024 over ~20 sectors
        _u1("update_u1_D1024_bf16x3", "update", "chain", 1024, "bf16x3", 12),
        # the J1-J2 width-6 cylinder at D = 2048
        _u1("ac2_solve_u1_j1j2_D2048_bf16x3", "solve", "cylinder", 2048, "bf16x3", 12),
    ]


def _dense(name, call, op, Dl, Dr, model, nexp, dtype, prec, krylov=0):
    return {"name": name, "call": call, "op": op, "Dl": Dl, "Dr": Dr, "model": model,
            "nexp": nexp, "dtype": dtype, "prec": prec, "krylov": krylov, "sym": ""}


def _u1(name, call, model, D, prec, krylov):
    return {"name": name, "call": call, "op": "AC2", "Dl": D, "Dr": D, "model": model, "nexp": 0,
            "dtype": "f64", "prec": prec, "krylov": krylov, "sym": "u1"}


def _chain(name, L, D):
    return {"name": name, "call": "timestep", "op": "", "Dl": D, "Dr": D, "model": "xxz",
            "nexp": 1, "dtype": "c128", "prec": "fp64", "krylov": 30, "sym": "", "L": L}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    call = rng.choice(["apply", "apply", "solve", "solve", "evolve", "transfer", "orth", "u1",
                       "u1", "timestep"])
    dtype = rng.choice(["c128", "f64"])
    prec = rng.choice(["fp64", "fp64", "bf16x3", "tf32x3"])
    if call == "timestep":
        c = _chain("", rng.randint(8, 14), _log(rng, 8, 40))
    elif call == "u1":
        model = rng.choice(["chain", "chain", "cylinder"])
        D = _log(rng, 256, 2048) if model == "cylinder" else _log(rng, 256, 1024)
        split = rng.choice(["bf16x3", "tf32x3"])
        prec = rng.choice(["fp64", split]) if model == "chain" and D <= 512 else split
        c = _u1("", rng.choice(["solve", "update"]) if D <= 1024 else "solve", model, D, prec,
                rng.randint(4, 12))
    else:
        nexp = rng.choice([1, 1, 2, 4])
        model = rng.choice(["tfim", "xxz", "xxz"])
        if call == "orth":
            Dl = _log(rng, 32, 512)
            Dr = min(512, max(17, int(Dl * rng.uniform(0.55, 1.8))))
            c = _dense("", call, "", Dl, Dr, "", 0, dtype, "fp64")
        elif call == "transfer":
            Dl = _log(rng, 32, 512)
            Dr = min(515, max(17, int(Dl * rng.uniform(0.55, 1.8))))
            c = _dense("", call, "", Dl, Dr, model, nexp, dtype, prec)
        else:
            op = rng.choice(["C", "AC", "AC2"])
            top = {"C": 512, "AC": 320, "AC2": 256 if dtype == "f64" else 160}[op]
            if prec != "fp64":
                top = 512
            Dl = _log(rng, 16, top)
            Dr = Dl if op == "C" else min(top, max(9, int(Dl * rng.uniform(0.55, 1.8))))
            if call == "evolve":
                dtype = "c128"
            c = _dense("", call, op, Dl, Dr, model, nexp, dtype, prec,
                       krylov={"apply": 0, "solve": rng.randint(4, 30), "evolve": 30}[call])
    c.pop("name")
    return c


# ---------------------------------------------------------------- inputs

def _np_dtype(case):
    return np.complex128 if case["dtype"] == "c128" else np.float64


def _rng(seed, tag):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, tag])


def _normal(rng, shape, dtype):
    a = rng.standard_normal(shape)
    if np.dtype(dtype).kind == "c":
        a = a + 1j * rng.standard_normal(shape)
    return a.astype(dtype)


def _width(case):
    return 3 if case["model"] == "tfim" else 2 + 3 * case["nexp"]


def _mpo(case, rng):
    """Bulk MPO tensor W[wl, s, s', wr], channel 0 "not started", the last "finished"."""
    w = _width(case)
    sp = np.array([[0, 1], [0, 0]], dtype=np.float64)
    sz = np.diag([0.5, -0.5])
    eye = np.eye(2)
    W = np.zeros((w, 2, 2, w))
    W[0, :, :, 0] = W[-1, :, :, -1] = eye
    if case["model"] == "tfim":
        W[0, :, :, 1] = -2 * sz
        W[1, :, :, 2] = 2 * sz
        W[0, :, :, 2] = -rng.uniform(0.1, 2.0) * (sp + sp.T)
    else:
        for k in range(case["nexp"]):
            lam = 0.0 if case["nexp"] == 1 else (k + 1.0) / (case["nexp"] + 1.0)
            amp = 1.0 / (k + 1.0)
            for j, (a, b, g) in enumerate(((sp, sp.T, 0.5), (sp.T, sp, 0.5),
                                           (sz, sz, rng.uniform(0.8, 1.6)))):
                c = 1 + 3 * k + j
                W[0, :, :, c] = amp * g * a
                W[c, :, :, c] = lam * eye
                W[c, :, :, -1] = b
    return W.astype(_np_dtype(case))


def _site(rng, Dl, Dr, dtype):
    """A left-isometric site tensor A[l, s, r] (Dr <= 2 Dl) on the GPU."""
    a = torch.from_numpy(_normal(rng, (Dl * D_PHYS, Dr), dtype)).cuda()
    return torch.linalg.qr(a)[0].reshape(Dl, D_PHYS, Dr)


def _step_left(G, A, W):
    """GL'[a, w', a'] = GL[b, w, b'] A[b', s', a'] W[w, s, s', w'] conj(A[b, s, a])."""
    b, w, k = G.shape
    n = A.shape[2]
    T = torch.matmul(G.reshape(b * w, k), A.reshape(k, -1)).reshape(b, w, D_PHYS, n)
    T = torch.tensordot(T, W, dims=([1, 2], [0, 2]))           # (b, a', s, w')
    T = T.permute(0, 2, 3, 1).reshape(b * D_PHYS, -1)          # (b s, w' a')
    return torch.matmul(A.reshape(b * D_PHYS, n).conj().T, T).reshape(n, W.shape[3], n)


def _environment(rng, D, W, dtype, right):
    """GL[a, w, a'] (or GR[b', w, b]) of a random canonical state with bonds 1, 2, 4, ..., D,
    as Fortran-ordered host memory."""
    Wt = torch.from_numpy(np.ascontiguousarray(W.transpose(3, 1, 2, 0) if right else W)).cuda()
    G = torch.zeros(1, W.shape[0], 1, dtype=Wt.dtype, device="cuda")
    G[0, -1 if right else 0, 0] = 1
    d = 1
    while d < D:
        n = min(D, d * D_PHYS)
        G = _step_left(G, _site(rng, d, n, dtype), Wt)
        d = n
    if right:                                                  # bra leg last
        G = G.permute(2, 1, 0)
    return G


def _host(G):
    """Fortran-ordered numpy array of a GPU tensor, without a transposing copy on the host."""
    return G.permute(*reversed(range(G.ndim))).contiguous().cpu().numpy().T


def _xshape(case):
    Dl, Dr = case["Dl"], case["Dr"]
    return {"C": (Dl, Dr), "AC": (Dl, D_PHYS, Dr), "AC2": (Dl, D_PHYS, Dr, D_PHYS)}[case["op"]]


def _dense_inputs(case, seed):
    dt = _np_dtype(case)
    W = _mpo(case, _rng(seed, 1))
    GL = _environment(_rng(seed, 2), case["Dl"], W, dt, False)
    GR = _environment(_rng(seed, 3), case["Dr"], W, dt, True)
    x = _normal(_rng(seed, 4), _xshape(case), dt)
    return W, GL, GR, x / np.linalg.norm(x)


def _transfer_inputs(case, seed):
    dt = _np_dtype(case)
    W = _mpo(case, _rng(seed, 1))
    GL = _environment(_rng(seed, 2), case["Dl"], W, dt, False)
    GR = _environment(_rng(seed, 3), case["Dr"], W, dt, True)
    A = _normal(_rng(seed, 4), (case["Dl"], D_PHYS, case["Dr"]), dt)
    return W, GL, GR, A / math.sqrt(2.0 * case["Dl"])


@functools.lru_cache(maxsize=None)
def _context(gauge):
    """One context per way of working; a user's program keeps it."""
    ctx = mpsgb.Context(0)
    if gauge:
        ctx.set_svd_method(gauge)
    return ctx


@functools.lru_cache(maxsize=None)
def _u1_model(model, D):
    """(H, sites) of the symmetric models: long enough for the central bond to hold D states."""
    if model == "cylinder":
        return mpsgb.j1j2_cylinder(4, 6, u1=True), 24
    L = 2 * math.ceil(math.log2(D)) + 6
    return mpsgb.heisenberg_XXX(L, dtype=np.float64, u1=True), L


def prepare(case, seed):
    call = case["call"]
    if call == "timestep":
        return _prepare_timestep(case, seed)
    if case["sym"] == "u1":
        return _prepare_u1(case, seed)
    ctx = _context("")
    dev = lambda kind, a: mpsgb.DeviceTensor.from_numpy(ctx, kind, a)
    if call == "orth":
        a = _normal(_rng(seed, 1), (case["Dl"], D_PHYS, case["Dr"]), _np_dtype(case))
        return {"case": case, "A": dev("mps", a)}
    backend = mpsgb.GB300Backend(case["prec"])
    if call == "transfer":
        W, GL, GR, A = _transfer_inputs(case, seed)
        return {"case": case, "W": dev("mpo", W), "GL": dev("gl", _host(GL)),
                "GR": dev("gr", _host(GR)), "A": dev("mps", A), "backend": backend}
    W, GL, GR, x = _dense_inputs(case, seed)
    s = {"case": case, "ctx": ctx, "W": dev("mpo", W), "GL": dev("gl", _host(GL)),
         "GR": dev("gr", _host(GR)), "x": dev(XKIND[case["op"]], x), "backend": backend}
    if call == "apply":
        s["op"] = _operator(s)
    return s


def _operator(s):
    op, W = s["case"]["op"], s["W"]
    W1, W2 = {"C": (None, None), "AC": (W, None), "AC2": (W, s.get("W2", W))}[op]
    return mpsgb.DerivativeOperator(s["ctx"], KINDS[op], s["GL"], W1, W2, s["GR"], s["backend"])


def _prepare_u1(case, seed):
    """The two sites left and right of the central bond, with the environments that a sweep
    with this precision has there."""
    ctx = _context("gram" if case["call"] == "update" else "")
    D = case["Dl"]
    H, L = _u1_model(case["model"], D)
    mid = L // 2 - 1
    backend = mpsgb.GB300Backend(case["prec"])
    qb = mu1.bond_charges(L, D)
    rng = _rng(seed, 1)
    W = H.device(ctx, np.float64)

    def site(ql, qr):
        mask = mu1.block_mask(ql, QP, qr)
        a = np.zeros(mask.shape)
        a[mask] = rng.standard_normal(int(mask.sum()))
        t = mpsgb.DeviceTensor.from_numpy(ctx, "mps", a)
        t.charges = mu1.mps_charges(ql, QP, qr)
        return t

    one = np.ones((1, 1, 1))
    GL = mpsgb.DeviceTensor.from_numpy(ctx, "gl", one)
    GR = mpsgb.DeviceTensor.from_numpy(ctx, "gr", one)
    ql, qr = qb[0], qb[L]                                       # the gauge may shrink a sector
    for i in range(mid):
        A, _ = mpsgb.left_orth(site(ql, qb[i + 1]))
        GL = mpsgb.transfer_left(GL, W[i], A, backend=backend)
        ql = A.charges[2]
    for i in range(L - 1, mid + 1, -1):
        _, A = mpsgb.right_orth(site(qb[i], qr))
        GR = mpsgb.transfer_right(GR, W[i], A, backend=backend)
        qr = A.charges[0]
    mask = mu1.block_mask(ql, QP, QP, qr)                       # (l, s1, s2, r)
    x = np.zeros(mask.shape)
    x[mask] = rng.standard_normal(int(mask.sum()))
    x = mpsgb.DeviceTensor.from_numpy(ctx, "ac2", x.transpose(0, 1, 3, 2))
    x.charges = tuple(np.asarray(q, np.int32) for q in (ql, QP, qr, QP))
    x.normalize_()
    return {"case": case, "ctx": ctx, "W": W[mid], "W2": W[mid + 1], "GL": GL, "GR": GR, "x": x,
            "backend": backend}


def _prepare_timestep(case, seed):
    ctx = _context("")
    L, D = case["L"], case["Dl"]
    rng = _rng(seed, 1)
    Jz = rng.uniform(0.8, 1.6)
    H = mpsgb.xxz(L, 1.0, Jz, 0.0)
    bonds = [min(D, 2 ** min(i, L - i)) for i in range(L + 1)]
    As = [_normal(rng, (bonds[i], D_PHYS, bonds[i + 1]), np.complex128) for i in range(L)]
    psi = mpsgb.FiniteMPS.from_tensors(As, ctx)
    return {"case": case, "psi": psi, "H": H, "alg": mpsgb.TDVP()}


# ---------------------------------------------------------------- one pass

def run(s):
    case = s["case"]
    call = case["call"]
    if call == "apply":
        return s["op"](s["x"]).numpy()
    if call == "transfer":
        a = mpsgb.transfer_left(s["GL"], s["W"], s["A"], backend=s["backend"])
        b = mpsgb.transfer_right(s["GR"], s["W"], s["A"], backend=s["backend"])
        return a.numpy(), b.numpy()
    if call == "orth":
        al, c = mpsgb.left_orth(s["A"])
        c2, ar = mpsgb.right_orth(s["A"])
        return al.numpy(), c.numpy(), c2.numpy(), ar.numpy()
    if call == "evolve":
        y = mpsgb.integrate(_operator(s), s["x"], 0.0, 0.05, mpsgb.Lanczos(case["krylov"], 100, 1e-10))
        return y.numpy()
    if call == "timestep":
        p = s["psi"]
        psi = mpsgb.FiniteMPS(list(p.AL), list(p.AR), list(p.C), p.center)
        psi, _ = mpsgb.timestep(psi, s["H"], 0.0, 0.05, s["alg"])
        return [psi.ac_tensor.numpy()] + [a.numpy() for a in psi.AR[1:]]
    # the budget of a local update: one Lanczos pass of at most `krylov` vectors, checked
    # after every vector
    solver = mpsgb.Lanczos(case["krylov"], 1, 1e-12, True)
    lam, x, _ = mpsgb.fixedpoint(_operator(s), s["x"], "SR", solver)
    if call == "solve":
        return lam, x.numpy()
    al, S, ar, eps = mpsgb.svd_trunc(x, case["Dl"], 0.0)
    return lam, eps, al.numpy(), S.numpy(), ar.numpy()


# ---------------------------------------------------------------- what a pass cannot do without

def _apply_flops(case):
    """2 (8 when complex) flops per multiply-add of x . GR and GL . (.) over the MPO channels."""
    Dl, Dr, w = case["Dl"], case["Dr"], _width(case)
    p = {"C": 1, "AC": 2, "AC2": 4}[case["op"]]
    mac = p * Dl * Dr * Dr * w + p * Dl * Dl * Dr * w
    return (8.0 if case["dtype"] == "c128" else 2.0) * mac


def _u1_work(case):
    """The same over charge blocks: bonds of `n_q` states in sector q couple q to q, q +- 2."""
    H, L = _u1_model(case["model"], case["Dl"])
    mid = L // 2 - 1
    qb = mu1.bond_charges(L, case["Dl"])
    n = lambda q: dict(zip(*(v.tolist() for v in np.unique(np.asarray(q), return_counts=True))))
    nl, nr = n(qb[mid]), n(qb[mid + 2])
    phys = [a + b for a in QP.tolist() for b in QP.tolist()]
    ent = [(q, q + p) for q in nl for p in phys if q + p in nr]
    shift = [-2, 0, 2]                                          # charge carried by a channel
    wl, wr = H[mid].shape[0], H[mid + 1].shape[3]
    mac = sum(nl[a] * nr[b] * (wr / 3.0 * sum(nr.get(b + t, 0) for t in shift) +
                               wl / 3.0 * sum(nl.get(a + t, 0) for t in shift)) for a, b in ent)
    env = (sum(nl[a] * nl.get(a + t, 0) for a in nl for t in shift) * wl / 3.0 +
           sum(nr[a] * nr.get(a + t, 0) for a in nr for t in shift) * wr / 3.0)
    return 2.0 * mac, 8.0 * env, 8.0 * sum(nl[a] * nr[b] for a, b in ent)


def work(case):
    e = 16 if case["dtype"] == "c128" else 8
    f = 4.0 if case["dtype"] == "c128" else 1.0
    Dl, Dr, call = case["Dl"], case["Dr"], case["call"]
    if call == "orth":
        k1, k2 = min(2 * Dl, Dr), min(Dl, 2 * Dr)
        flops = f * (4.0 * 2 * Dl * Dr * k1 + 4.0 * Dl * 2 * Dr * k2)
        return {"bytes": e * (2 * Dl * Dr + 2 * Dl * k1 + k1 * Dr + k2 * 2 * Dr + Dl * k2),
                "flops": flops}
    if call == "transfer":
        w = _width(case)
        return {"bytes": e * (2 * w * (Dl * Dl + Dr * Dr) + 2 * Dl * Dr),
                "flops": f * 2.0 * w * 2 * 2 * (Dl * Dl * Dr + Dl * Dr * Dr)}
    if call == "timestep":
        L = case["L"]
        b = [min(Dl, 2 ** min(i, L - i)) for i in range(L + 1)]
        nmat = 10                                               # applications per local step
        mac = sum(2 * 5 * (2 * b[i] * b[i + 1] ** 2 + 2 * b[i] ** 2 * b[i + 1]) +
                  2 * 5 * 2 * b[i] ** 3 for i in range(L))
        return {"bytes": 2 * e * sum(2 * b[i] * b[i + 1] for i in range(L)),
                "flops": 8.0 * nmat * mac}
    n = max(1, case["krylov"]) if call != "evolve" else 10
    if case["sym"] == "u1":
        fl, env, x = _u1_work(case)
        out = x if call == "solve" else 8.0 * (4 * Dl * Dl + Dl * Dl) / 4
        return {"bytes": env + x + out, "flops": n * fl}
    w, nx = _width(case), int(np.prod(_xshape(case)))
    return {"bytes": e * (w * (Dl * Dl + Dr * Dr) + 2 * nx), "flops": n * _apply_flops(case)}


# ---------------------------------------------------------------- the same in 64 bits

def _full_apply(case, W, GL, GR):
    """x -> H x by plain contractions of every channel (torch, 64 bits)."""
    w, Dl, Dr = W.shape[0], case["Dl"], case["Dr"]
    Wt = torch.from_numpy(W).cuda()
    R = GR.reshape(Dr, w * Dr).contiguous()                     # (r', w r)
    G = GL.reshape(Dl, w * Dl)                                  # (l, w l')
    op = case["op"]

    def apply(x):
        T = torch.matmul(x.reshape(-1, Dr), R)
        if op == "C":
            T = T.reshape(Dl, w, Dr)                            # (l', w, r)
        elif op == "AC":
            T = T.reshape(Dl, D_PHYS, w, Dr)                    # (l', t, w', r)
            T = torch.tensordot(T, Wt, dims=([1, 2], [2, 3]))   # (l', r, w, s)
            T = T.permute(0, 2, 3, 1)                           # (l', w, s, r)
        else:
            T = T.reshape(Dl, D_PHYS, D_PHYS, w, Dr)            # (l', t1, t2, w', r)
            T = torch.tensordot(T, Wt, dims=([2, 3], [2, 3]))   # (l', t1, r, m, s2)
            T = torch.tensordot(T, Wt, dims=([1, 3], [2, 3]))   # (l', r, s2, w, s1)
            T = T.permute(0, 3, 4, 2, 1)                        # (l', w, s1, s2, r)
        T = T.transpose(0, 1).reshape(w * Dl, -1)               # (w l', ...)
        return torch.matmul(G, T).reshape(x.shape)

    return apply


def _lanczos(apply, x, steps):
    """Orthonormal Krylov vectors (rows) and the projected matrix after `steps` applications."""
    V = [x.reshape(-1) / torch.linalg.vector_norm(x)]
    T = np.zeros((steps, steps))
    for j in range(steps):
        u = apply(V[j].reshape(x.shape)).reshape(-1)
        B = torch.stack(V)
        T[j, j] = float(torch.vdot(V[j], u).real)
        for _ in range(2):
            u = u - torch.matmul(B.conj() @ u, B)
        if j + 1 < steps:
            b = float(torch.linalg.vector_norm(u))
            T[j, j + 1] = T[j + 1, j] = b
            V.append(u / b)
    return torch.stack(V), T


def _pos_qr(a):
    q, r = np.linalg.qr(a)
    ph = np.diagonal(r) / np.abs(np.diagonal(r))
    return q * ph, np.conj(ph)[:, None] * r


def exact(case, seed):
    call, dt = case["call"], _np_dtype(case)
    if case["sym"] == "u1" or call == "timestep":
        return None
    if call == "orth":
        Dl, Dr = case["Dl"], case["Dr"]
        a = _normal(_rng(seed, 1), (Dl, D_PHYS, Dr), dt)
        q, r = _pos_qr(a.reshape(Dl * D_PHYS, Dr, order="F"))
        p, l = _pos_qr(a.reshape(Dl, D_PHYS * Dr, order="F").conj().T)
        return (q.reshape(Dl, D_PHYS, -1, order="F"), r, l.conj().T,
                p.conj().T.reshape(-1, D_PHYS, Dr, order="F"))
    if call == "transfer":
        W, GL, GR, A = _transfer_inputs(case, seed)
        At, Wt = torch.from_numpy(A).cuda(), torch.from_numpy(W).cuda()
        left = _step_left(GL, At, Wt)
        mirror = Wt.permute(3, 1, 2, 0).contiguous()
        right = _step_left(GR.permute(2, 1, 0).contiguous(), At.permute(2, 1, 0).contiguous(),
                           mirror).permute(2, 1, 0)
        return left.cpu().numpy(), right.cpu().numpy()
    W, GL, GR, x = _dense_inputs(case, seed)
    apply = _full_apply(case, W, GL, GR)
    # operators take x in the order (l, s1, r, s2); contractions here in (l, s1, s2, r)
    xt = torch.from_numpy(np.ascontiguousarray(x.transpose(0, 1, 3, 2) if x.ndim == 4 else x)).cuda()
    back = lambda y: (y.permute(0, 1, 3, 2) if y.ndim == 4 else y).contiguous().cpu().numpy()
    if call == "apply":
        return back(apply(xt))
    if call == "solve":
        _, T = _lanczos(apply, xt, min(case["krylov"], x.size))
        return float(np.linalg.eigvalsh(T)[0]), None             # the vector has no fixed sign
    for _ in range(2):                                           # evolve: two half steps
        V, T = _lanczos(apply, xt, min(case["krylov"], x.size))
        d, U = np.linalg.eigh(T)
        c = U @ (np.exp(-0.025j * d) * U[0]) * float(torch.linalg.vector_norm(xt))
        xt = (torch.from_numpy(c).cuda() @ V).reshape(xt.shape)
    return back(xt)
