"""The timed cases of the engine: the calls a Wannier90 library user makes, at the sizes
they make them.

Kinds of case:

* ``solve``        wann_main on device buffers (``w90_wannierise_device``), a fixed number
                   of iterations; ``tensor`` selects the tcgen05 path or the FP64 default;
* ``host``         the same through the reference-named call on NumPy arrays
                   (``w90_wannierise``: upload, solve, download);
* ``project``      the Loewdin start of an isolated group (``w90_project_overlap_device``);
* ``disentangle``  dis_main + setup_m_loc on device buffers (``w90_disentangle_device``);
* ``batch``        many uneven problems in one call (``w90_wannierise_batch_device``).

Inputs are seeded tight-binding models: W smooth bands out of a few more orbitals (so that
Omega_I > 0), each k in its own random gauge as eigenvectors come, projections onto the
orbitals rotated by a small random unitary per k.  The gauge noise and the iteration counts
keep the minimisation in the range where its result follows its input (rounding at the level
of the tensor path's products stays below 1e-9 in M and U), so that two builds can be compared.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from wannier90_gb300 import library as w90
from wannier90_gb300 import synth

CELL = 5.0    # lattice constant, Angstrom
NOISE = 0.4   # gauge noise of the projections (norm of the rotation's generator)


def listed():
    return [
        # a regression-test sized cell (GaAs, 2x2x2, four sp3 orbitals): latency only
        dict(name="solve_w4_k8", kind="solve", lattice="fcc", n1=2, n2=2, n3=2, num_wann=4, iters=20, tensor=False),
        # the suite's small workload, default options
        dict(name="solve_w8_k64", kind="solve", lattice="sc", n1=4, n2=4, n3=4, num_wann=8, iters=20, tensor=False),
        # an odd band count on an uneven mesh (several b-shells), tensor path
        dict(name="solve_w13_k80_tensor", kind="solve", lattice="sc", n1=5, n2=4, n3=4, num_wann=13, iters=10,
             tensor=True),
        # an ordinary production cell on the default FP64 path
        dict(name="solve_w24_k216", kind="solve", lattice="sc", n1=6, n2=6, n3=6, num_wann=24, iters=10,
             tensor=False),
        # the headline workload's shape: fcc 10x10x10, 32 bands
        dict(name="solve_w32_k1000_tensor", kind="solve", lattice="fcc", n1=10, n2=10, n3=10, num_wann=32, iters=4,
             tensor=True),
        # a wider cell between two tile widths
        dict(name="solve_w48_k216_tensor", kind="solve", lattice="sc", n1=6, n2=6, n3=6, num_wann=48, iters=6,
             tensor=True),
        # the precision workload's shape: a supercell with 128 orbitals on 8x8x8
        dict(name="solve_w128_k512_tensor", kind="solve", lattice="sc", n1=8, n2=8, n3=8, num_wann=128, iters=4,
             tensor=True),
        # a DFT code calling the library with host arrays
        dict(name="host_w20_k125_tensor", kind="host", lattice="sc", n1=5, n2=5, n3=5, num_wann=20, iters=8,
             tensor=True),
        # the projection before the headline solve
        dict(name="project_w32_k1000", kind="project", lattice="fcc", n1=10, n2=10, n3=10, num_wann=32),
        # silicon-like disentanglement: 12 bands to 8 on 4x4x4
        dict(name="disentangle_b12_w8_k64", kind="disentangle", lattice="sc", n1=4, n2=4, n3=4, num_bands=12,
             num_wann=8, iters=40),
        # the entangled workload's shape: fcc 8x8x8, 48 bands to 32
        dict(name="disentangle_b48_w32_k512", kind="disentangle", lattice="fcc", n1=8, n2=8, n3=8, num_bands=48,
             num_wann=32, iters=10),
        # uneven problems in one batched call (num_wann 4..64, meshes 3^3..6^3)
        dict(name="batch_24", kind="batch", problems=24, shapes=7, iters=6),
    ]


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "host", "project", "disentangle", "batch"])
    if kind == "batch":
        return dict(kind=kind, problems=rng.randint(4, 24), shapes=rng.randint(0, 10 ** 6), iters=rng.randint(4, 6))
    lattice = rng.choice(["sc", "fcc"])
    mesh = rng.randint(2 if lattice == "fcc" else 3, 8)
    case = dict(kind=kind, lattice=lattice, n1=mesh, n2=mesh, n3=mesh)
    if lattice == "sc":
        case["n3"] = max(3, mesh - rng.randint(0, 1))
    kpts = case["n1"] * case["n2"] * case["n3"]
    if kind == "disentangle":
        bands = _log_int(rng, 6, 48)
        return dict(case, num_bands=bands, num_wann=max(3, (2 * bands) // 3), iters=rng.randint(5, 20))
    if kind == "project":
        return dict(case, num_wann=_log_int(rng, 4, 40))
    width = _log_int(rng, 4, 100 if kpts <= 216 else 64)
    tensor = rng.random() < 0.6 or width > 40
    return dict(case, num_wann=width, iters=rng.randint(3, 8 if kpts <= 216 else 4), tensor=bool(tensor))


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# ---- inputs ---------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, *shape):
    return torch.complex(torch.randn(*shape, generator=g, dtype=torch.float64, device="cuda"),
                         torch.randn(*shape, generator=g, dtype=torch.float64, device="cuda"))


def _rotations(g, K, n, size):
    """exp(X_k), X_k random anti-Hermitian with a norm of about `size`."""
    X = _randn(g, K, n, n)
    return torch.matrix_exp(size / math.sqrt(8.0 * n) * (X - X.mH))


def _mesh(case):
    """Lattice, k-points, neighbour lists and b-vectors (their order fixes the overlaps' layout)."""
    A = synth.lattice(case["lattice"], CELL)
    kp = synth.mp_kpoints(case["n1"], case["n2"], case["n3"])
    _, nnlist, _, bk = synth.kmesh_tables(A, kp)
    return A, kp, nnlist, bk


def _smooth(g, kp, rows, cols, size):
    """sum_R F_R exp(2 pi i k.R) over the home cell and its six neighbours."""
    R = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1], [-1, 0, 0], [0, -1, 0], [0, 0, -1]], dtype=np.float64)
    ph = torch.from_numpy(np.exp(2j * math.pi * (kp @ R.T))).cuda()
    return torch.einsum("kr,rij->kij", ph, _randn(g, len(R), rows, cols)) * size


def _overlaps(C, tau, nnlist, bk):
    """M[k, b] = C(k)^H exp(-i b.tau) C(k+b)."""
    nn = torch.from_numpy(nnlist).cuda()
    phase = torch.exp(-1j * torch.einsum("kbi,ai->kba", torch.from_numpy(bk).cuda(), tau))
    M = torch.empty(nn.shape + (C.shape[2],) * 2, dtype=torch.complex128, device="cuda")
    for b in range(nn.shape[1]):
        M[:, b] = C.mH @ (phase[:, b, :, None] * C[nn[:, b]])
    return M


def _isolated(case, seed):
    """M[k, b, m, n], A[k, m, n] of num_wann smooth bands out of num_wann + num_wann / 4 + 1 orbitals."""
    A, kp, nnlist, bk = _mesh(case)
    g = _generator(seed)
    W = case["num_wann"]
    extra = W // 4 + 1
    tau = torch.rand(W + extra, 3, generator=g, dtype=torch.float64, device="cuda") @ torch.from_numpy(A).cuda()
    F = _smooth(g, kp, extra, W, 0.03 / math.sqrt(extra))
    T = torch.cat([torch.eye(W, dtype=torch.complex128, device="cuda").expand(len(kp), W, W), F], 1)
    L = torch.linalg.cholesky(T.mH @ T)
    C = torch.linalg.solve_triangular(L, T.mH, upper=False).mH @ _rotations(g, len(kp), W, 3.0)
    M = _overlaps(C, tau, nnlist, bk)
    proj = C[:, :W].mH @ _rotations(g, len(kp), W, NOISE)
    return dict(lattice=A, kpoints=kp, nnlist=nnlist, bk=bk, M=M, A=proj)


def _entangled(case, seed):
    """M[k, b, m, n], A[k, m, n], energies E[k, m] and windows of num_bands bands of which
    the num_wann lower orbitals are wanted and the others lie above and mix in."""
    A, kp, nnlist, bk = _mesh(case)
    g = _generator(seed)
    nb, W = case["num_bands"], case["num_wann"]
    H = _smooth(g, kp, nb, nb, 0.5 / math.sqrt(nb))
    H = H + H.mH
    E, C = np.linalg.eigh((H + torch.diag(torch.arange(nb, device="cuda") * (8.0 / nb) + 2.0 *
                                          (torch.arange(nb, device="cuda") >= W))).cpu().numpy())
    C = torch.from_numpy(C).cuda()
    tau = torch.rand(nb, 3, generator=g, dtype=torch.float64, device="cuda") @ torch.from_numpy(A).cuda()
    M = _overlaps(C, tau, nnlist, bk)
    proj = C[:, :W].mH @ _rotations(g, len(kp), W, NOISE)
    return dict(lattice=A, kpoints=kp, nnlist=nnlist, bk=bk, M=M, A=proj, E=E, windows=synth.entangled_windows(E, W))


def _projected(p):
    """U0 = polar factor of A, M0 = U0^H M U0': what an earlier projection call left."""
    U = _polar(p["A"])
    return _rotate(p["M"], U, torch.from_numpy(p["nnlist"]).cuda()), U


def _polar(A):
    L, V = np.linalg.eigh((A.mH @ A).cpu().numpy())
    V = torch.from_numpy(V).cuda()
    return A @ ((V / torch.from_numpy(np.sqrt(L)).cuda()[:, None, :]) @ V.mH)


def _rotate(M, U, nn):
    out = torch.empty(M.shape[:2] + (U.shape[2],) * 2, dtype=M.dtype, device=M.device)
    for b in range(M.shape[1]):
        out[:, b] = U.mH @ M[:, b] @ U[nn[:, b]]
    return out


def _flat(X):
    """The library's layout: the last index pair column-major, k slowest."""
    return X.transpose(-1, -2).contiguous()


# ---- the calls ------------------------------------------------------------------------

def _options(case):
    o = dict(iprint=0, conv_window=-1)
    if "iters" in case:
        o["num_iter"] = case["iters"]
    if case.get("tensor"):
        o["gpu_tensor"] = 1
    return o


def _handle(p, W, **options):
    return w90.setup(kpoints=p["kpoints"], unit_cell_cart=p["lattice"], num_wann=W, **options)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, case=case, stream=torch.cuda.Stream())
    if kind == "batch":
        s["jobs"] = []
        for i, c in enumerate(_batch_shapes(case)):
            p = _isolated(c, 1000 * seed + i)
            M, U = _projected(p)
            m0, u0 = _flat(M), _flat(U)
            s["jobs"].append(dict(m0=m0, u0=u0, m=torch.empty_like(m0), u=torch.empty_like(u0), W=c["num_wann"],
                                  h=_handle(p, c["num_wann"], **_options(c))))
        for j in s["jobs"]:
            w90.w90_set_stream(j["h"], s["stream"].cuda_stream)
    elif kind == "disentangle":
        p = _entangled(case, seed)
        w = p["windows"]
        h = _handle(p, case["num_wann"], num_bands=case["num_bands"], iprint=0, dis_num_iter=case["iters"],
                    dis_conv_tol=0.0, dis_mix_ratio=0.5, dis_win_min=w["win_min"], dis_win_max=w["win_max"],
                    dis_froz_max=w["froz_max"])
        K, W = len(p["kpoints"]), case["num_wann"]
        s.update(h=h, m0=_flat(p["M"]), a0=_flat(p["A"]), eig=torch.from_numpy(p["E"].copy()).cuda())
        s.update(m=torch.empty_like(s["m0"]), a=torch.empty_like(s["a0"]),
                 u=torch.zeros(K, W, W, dtype=torch.complex128, device="cuda"))
        w90.w90_set_stream(h, s["stream"].cuda_stream)
    else:
        p = _isolated(case, seed)
        W = case["num_wann"]
        h = _handle(p, W, **_options(case))
        M, U = (p["M"], p["A"]) if kind == "project" else _projected(p)
        s.update(h=h, W=W, m0=_flat(M), u0=_flat(U))
        if kind == "host":
            # the library's Fortran-ordered arrays: (W, W, B, K) and (W, W, K)
            s["m0"], s["u0"] = s["m0"].cpu().numpy().T, s["u0"].cpu().numpy().T
            s["m"], s["u"] = s["m0"].copy(order="F"), s["u0"].copy(order="F")
            w90.w90_set_m_local(h, s["m"])
            w90.w90_set_u_matrix(h, s["u"])
            w90.w90_set_u_opt(h, s["u"].copy(order="F"))
        else:
            s["m"], s["u"] = torch.empty_like(s["m0"]), torch.empty_like(s["u0"])
            w90.w90_set_stream(h, s["stream"].cuda_stream)
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "batch":
        with torch.cuda.stream(s["stream"]):
            for j in s["jobs"]:
                j["m"].copy_(j["m0"])
                j["u"].copy_(j["u0"])
        # the groups of a batch run on streams of their own
        s["stream"].synchronize()
        rc = w90.w90_wannierise_batch_device([j["h"] for j in s["jobs"]], [j["m"].data_ptr() for j in s["jobs"]],
                                             [j["u"].data_ptr() for j in s["jobs"]])
        for j, r in zip(s["jobs"], rc):
            w90.check(j["h"], r, "batch")
        return {"u": torch.cat([j["u"].flatten() for j in s["jobs"]]),
                "m": torch.cat([j["m"].flatten() for j in s["jobs"]]),
                "centres": np.concatenate([w90.w90_get_centres(j["h"], j["W"]).T.ravel() for j in s["jobs"]]),
                "omega": np.array([w90.w90_get_omega(j["h"])[3] for j in s["jobs"]])}
    h = s["h"]
    if kind == "host":
        np.copyto(s["m"], s["m0"])
        np.copyto(s["u"], s["u0"])
        w90.check(h, w90.w90_wannierise(h), "wannierise")
        return _result(s)
    if kind == "disentangle":
        with torch.cuda.stream(s["stream"]):
            s["m"].copy_(s["m0"])
            s["a"].copy_(s["a0"])
        w90.check(h, w90.w90_disentangle_device(h, s["m"].data_ptr(), s["a"].data_ptr(), s["u"].data_ptr(),
                                                s["eig"].data_ptr()), "disentangle")
        W = s["case"]["num_wann"]
        # the columns of u_opt carry eigenvectors' free phases; u_opt u, the rotation from
        # bands to Wannier functions, and the rotated overlaps do not
        return {"m": s["m"][:, :, :W, :W], "v": s["u"] @ s["a"],
                "omega": w90.w90_get_dis_log(h, s["case"]["iters"])[:, 1:3]}
    with torch.cuda.stream(s["stream"]):
        s["m"].copy_(s["m0"])
        s["u"].copy_(s["u0"])
    if kind == "project":
        w90.check(h, w90.w90_project_overlap_device(h, s["m"].data_ptr(), s["u"].data_ptr()), "project")
        return {"m": s["m"], "u": s["u"]}
    w90.check(h, w90.w90_wannierise_device(h, s["m"].data_ptr(), s["u"].data_ptr()), "wannierise")
    return _result(s)


def _result(s):
    h, W = s["h"], s["W"]
    return {"m": s["m"], "u": s["u"], "centres": w90.w90_get_centres(h, W), "spreads": w90.w90_get_spreads(h, W),
            "omega": w90.w90_get_omega(h), "trace": w90.w90_get_log(h, s["case"]["iters"] + 1)[:, 3].copy()}


def _batch_shapes(case):
    """num_wann from {4, 8, ..., 64} and meshes from {3^3, 4^3, 6^3}, the tensor path from
    the width on where it is the faster one."""
    rng = np.random.default_rng(case["shapes"])
    out = []
    for _ in range(case["problems"]):
        n, W = int(rng.choice([3, 4, 6])), 4 * int(rng.integers(1, 17))
        out.append(dict(kind="solve", lattice="sc", n1=n, n2=n, n3=n, num_wann=W, iters=case["iters"], tensor=W >= 8))
    return out


# ---- what a pass cannot do without ----------------------------------------------------

def work(case):
    if case["kind"] == "batch":
        parts = [work(c) for c in _batch_shapes(case)]
        return {k: float(sum(p[k] for p in parts)) for k in ("bytes", "flops")}
    K = case["n1"] * case["n2"] * case["n3"]
    B = 8 if case["lattice"] == "fcc" else 6
    W = case["num_wann"]
    if case["kind"] == "disentangle":
        nb = case["num_bands"]
        # per iteration C_b = M_w U', the upper triangle of sum_b w_b C_b C_b^H, one eigensolve
        flops = case["iters"] * K * (B * (8.0 * nb * nb * W + 4.0 * nb * nb * W) + 8.0 * (nb - W // 2) ** 3)
        return {"bytes": 16.0 * K * (B * (nb * nb + W * W) + 2 * nb * W + W * W), "flops": flops}
    state = 2 * 16.0 * K * W * W * (B + 1)
    if case["kind"] == "project":
        return {"bytes": state, "flops": K * W ** 3 * (16.0 * B + 24.0)}
    # per iteration two updates (trial and optimal step): M <- dU^H M dU', exp and U dU
    return {"bytes": state, "flops": case["iters"] * 2.0 * K * W ** 3 * (16.0 * B + 40.0)}


# ---- the same results in plain 64-bit torch --------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        parts = []
        for i, c in enumerate(_batch_shapes(case)):
            p = _isolated(c, 1000 * seed + i)
            parts.append(_minimise(p, *_projected(p), c["iters"]))
        return {"u": torch.cat([r["U"].flatten() for r in parts]), "m": torch.cat([r["M"].flatten() for r in parts]),
                "centres": np.concatenate([r["centres"].ravel() for r in parts]),
                "omega": np.array([r["omega"][3] for r in parts])}
    if kind == "disentangle":
        return _disentangled(case, _entangled(case, seed))
    p = _isolated(case, seed)
    M, U = _projected(p)
    if kind == "project":
        return {"m": _flat(M), "u": _flat(U)}
    r = _minimise(p, M, U, case["iters"])
    if kind == "host":
        r["M"], r["U"] = r["M"].cpu().numpy().T, r["U"].cpu().numpy().T
    return {"m": r["M"], "u": r["U"], "centres": r["centres"].T, "spreads": r["spreads"], "omega": r["omega"],
            "trace": r["trace"]}


def _weights(bk):
    """w_b with sum_b w_b b b^T = 1, one weight per shell."""
    d = np.linalg.norm(bk[0], axis=1)
    shells = np.unique(np.round(d, 6))
    member = np.abs(d[:, None] - shells[None, :]) < 1e-5
    outer = np.einsum("bi,bj,bs->ijs", bk[0], bk[0], member.astype(float)).reshape(9, -1)
    return member @ np.linalg.lstsq(outer, np.eye(3).ravel(), rcond=None)[0]


def _minimise(p, M, U, iters):
    """Marzari-Vanderbilt minimisation: conjugate gradients (restart after 5 steps), a trial
    step and the parabola through it."""
    bk = torch.from_numpy(p["bk"]).cuda()
    wb = torch.from_numpy(_weights(p["bk"])).cuda()
    nn = torch.from_numpy(p["nnlist"]).cuda()
    K, B, W = M.shape[:3]
    total = 4.0 * float(wb.sum())

    def spread(M):
        d = torch.diagonal(M, dim1=2, dim2=3)
        ln, a = torch.angle(d), d.real ** 2 + d.imag ** 2
        r = -torch.einsum("b,kbi,kbn->ni", wb, bk, ln) / K
        r2 = torch.einsum("b,kbn->n", wb, 1.0 - a + ln ** 2) / K
        norm = torch.stack([torch.linalg.vector_norm(M[:, b], dim=(1, 2)) ** 2 for b in range(B)], 1)
        om_i = float((wb * (W - norm)).sum()) / K
        om_od = float((wb * (norm - a.sum(2))).sum()) / K
        q = ln + torch.einsum("kbi,ni->kbn", bk, r)
        om_d = float(torch.einsum("b,kbn->", wb, q ** 2)) / K
        return dict(om=(om_i, om_d, om_od), r=r, s=r2 - (r ** 2).sum(1), d=d, q=q)

    def gradient(M, o):
        G = torch.zeros_like(U)
        for b in range(B):
            d = o["d"][:, b]
            alpha = wb[b] * (0.5 * d.conj() + 0.5j * o["q"][:, b] / d)
            G += M[:, b] * alpha[:, None, :]
        return (G - G.mH) * (4.0 / K)

    def step(M, U, D, size):
        dU = torch.matrix_exp(D * size)
        return _rotate(M, dU, nn), U @ dU

    inner = lambda X, Y: float((X.conj() * Y).real.sum())  # noqa: E731
    o = spread(M)
    om_i = o["om"][0]
    tot = lambda o: om_i + o["om"][1] + o["om"][2]  # noqa: E731
    trace, D, g0, ncg = [tot(o)], torch.zeros_like(U), 0.0, 0
    for it in range(iters):
        G = gradient(M, o)
        g1 = inner(G, G)
        if it == 0 or ncg >= 5 or g0 <= 2.220446049250313e-16 or g1 / g0 > 3.0:
            beta, ncg = 0.0, 0
        else:
            beta, ncg = g1 / g0, ncg + 1
        g0 = g1
        D = G + beta * D
        slope = -inner(G, D) / total
        if slope > 0.0 and ncg > 0:
            D, ncg = G, 0
            slope = -g1 / total
        elif slope > 0.0:
            D, slope = -D, -slope
        Mt, Ut = step(M, U, D, 2.0 / total)
        t = spread(Mt)
        fac = 1.0 / (tot(t) - tot(o))
        eqb = fac * slope
        eqa = 1.0 - 2.0 * eqb
        alpha = -2.0 * eqb / eqa if eqa != 0.0 else 2.0
        if abs(eqa / (fac * tot(o))) > 2.220446049250313e-16 and slope * alpha <= 0.0:
            M, U = step(M, U, D, alpha / total)
            o = spread(M)
        else:
            M, U, o = Mt, Ut, t
        trace.append(tot(o))
    return dict(M=_flat(M), U=_flat(U), centres=o["r"].cpu().numpy(), spreads=o["s"].cpu().numpy(),
                omega=np.array([om_i, o["om"][1], o["om"][2], tot(o)]), trace=np.array(trace))


def _disentangled(case, p):
    """Souza-Marzari-Vanderbilt disentanglement in the bands' own indices; states outside
    the window or frozen are pushed below every eigenvalue instead of being cut out."""
    nb, W, w = case["num_bands"], case["num_wann"], p["windows"]
    E, K, B = p["E"], len(p["kpoints"]), p["nnlist"].shape[1]
    wb = _weights(p["bk"])
    nn = torch.from_numpy(p["nnlist"]).cuda()
    win = (E >= w["win_min"]) & (E <= w["win_max"])
    frozen = win & (E <= w["froz_max"])
    free = torch.from_numpy((win & ~frozen).astype(float)).cuda()
    nf = frozen.sum(1)
    inside = torch.from_numpy(win.astype(float)).cuda()
    M = p["M"] * inside[:, None, :, None] * inside[nn][:, :, None, :]
    A = p["A"] * inside[:, :, None]
    # per column: taken from the frozen states first, from the eigenvectors after them
    picks = torch.zeros(K, nb, W, dtype=torch.complex128, device="cuda")
    for k in range(K):
        for c, i in enumerate(np.nonzero(frozen[k])[0]):
            picks[k, i, c] = 1.0
    column = torch.arange(W, device="cuda")[None, :] >= torch.from_numpy(nf).cuda()[:, None]

    def leading(Z):
        """U: the frozen states, then the W - nf leading eigenvectors on the free states."""
        Z = Z * free[:, :, None] * free[:, None, :] - 1e3 * torch.diag_embed(1.0 - free)
        ev, V = np.linalg.eigh(Z.cpu().numpy())
        ev, V = torch.from_numpy(ev).cuda(), torch.from_numpy(V).cuda()
        # the last W - nf eigenvectors, in ascending order, go to columns nf .. W - 1
        return torch.where(column[:, None, :], V[:, :, nb - W:], picks), (ev[:, nb - W:] * column).sum(1)

    def zmatrix(U):
        Z = torch.zeros(K, nb, nb, dtype=torch.complex128, device="cuda")
        for b in range(B):
            C = M[:, b] @ U[nn[:, b]]
            Z += wb[b] * (C @ C.mH)
        return Z

    U = _polar(A)
    U = leading(U @ U.mH)[0]
    Z = zmatrix(U)
    Zin, trace = Z, []
    for it in range(case["iters"]):
        if it > 0:
            Zin = 0.5 * Z + 0.5 * Zin
        kept = (torch.diagonal(Z, dim1=1, dim2=2).real * torch.from_numpy(frozen).cuda()).sum(1)
        U, taken = leading(Zin)
        Z = zmatrix(U)
        before = W * wb.sum() - kept - taken
        after = W * wb.sum() - torch.einsum("kij,kil,klj->k", U.conj(), Z, U).real
        trace.append([float(before.sum()) / K, float(after.sum()) / K])
    V = U @ _polar(U.mH @ A)
    rows = torch.from_numpy(win.argmax(1)).cuda()[:, None] + torch.arange(nb, device="cuda")[None, :]
    shifted = torch.where((rows < nb)[:, :, None], torch.gather(V, 1, rows.clamp(max=nb - 1)[:, :, None].expand(K, nb, W)),
                          torch.zeros_like(V))
    return {"m": _flat(_rotate(M, V, nn)), "v": _flat(shifted), "omega": np.array(trace)}
