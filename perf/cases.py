"""The work that programs have this framework do, as cases that can be timed.

A case is a dict of plain values.  `kind` names the call:

  ladder    one pass of the (q, omega) loop as a program runs it: stage the
            vertex of every omega of the block, run the block qw0 .. qw0 +
            points - 1, fetch the accumulators into pinned host arrays;
  tangent   the same with forward-mode tangents (couplings U and J and the
            hopping scale t) and their accumulators;
  ingest    the full program of a run with a non-local interaction: the
            two-particle Green's function of the vertex file ingested, the
            ladder with V(q), and the post-loop self-energy and densities;
  point     one (q, omega) point through bse_point;
  inverse   inverse_matrix of one dense complex matrix.

The models are tight-binding bands on a cubic k mesh with Kanamori
couplings, a causal local self-energy, an impurity Green's function with a
semicircular bath and the local susceptibility (chi0_loc^-1 + Gamma)^-1 whose
irreducible vertex Gamma carries a small frequency-dependent part: the
orders of magnitude and the conditioning that the ladder meets.
"""
import math

import numpy as np
import torch

from adga_b200 import Ladder
from adga_b200.ladder import generate_q_vol, inverse_matrix

DIRECTIONS = ("U", "J", "t")


def _ladder_case(name, ndim, nk, nq, iwf, iwb, beta, U, J, precision, qw0, points, kind="ladder",
                 directions=0, big_box=False, do_chi=True, do_eom=True):
    return dict(name=name, kind=kind, ndim=ndim, nk=nk, nq=nq, iwf=iwf, iwb=iwb, beta=beta, U=U, J=J,
                precision=precision, qw0=qw0, points=points, directions=directions, big_box=big_box,
                do_chi=do_chi, do_eom=do_eom)


def listed():
    return [
        # smallest call: one point of a single-orbital model, launch and host latency (BSE 40 x 40)
        _ladder_case("point_1orb_fp64", 1, 10, 5, 20, 10, 10.0, 2.0, 0.0, "fp64", 1 + 10 * 125 + 37, 1, "point"),
        # one point of the t2g model in FP64, as a loop of the caller's own asks for it (BSE 1080 x 1080)
        _ladder_case("point_t2g_fp64", 3, 20, 10, 60, 10, 10.0, 5.0, 0.75, "fp64", 1 + 10 * 1000 + 421, 1, "point"),
        # drop-in inverse of a dense matrix of odd order
        dict(name="inverse_357", kind="inverse", n=357),
        # whole grid of the single-orbital model in FP64: 21 bosonic frequencies x 125 q
        _ladder_case("grid_1orb_fp64", 1, 10, 5, 20, 10, 10.0, 2.0, 0.0, "fp64", 1, 21 * 125),
        # single-orbital member of a parameter sweep, all 11 frequencies, mixed (BSE 160 x 160)
        _ladder_case("grid_1orb_mixed", 1, 12, 6, 80, 5, 20.0, 3.0, 0.0, "mixed", 1, 11 * 216),
        # one frequency of the two-orbital model, mixed (BSE 320 x 320)
        _ladder_case("slice_2orb_mixed", 2, 16, 8, 40, 5, 20.0, 4.0, 0.6, "mixed", 1 + 5 * 512, 512),
        # one rank's ragged block of it in FP64, across a frequency boundary
        _ladder_case("block_2orb_fp64", 2, 16, 8, 40, 5, 20.0, 4.0, 0.6, "fp64", 1 + 5 * 512 + 333, 389),
        # two-orbital block with the derivatives in U, J and t, mixed
        _ladder_case("tangent_2orb_mixed", 2, 16, 8, 40, 5, 20.0, 4.0, 0.6, "mixed", 1 + 5 * 512, 256, "tangent", 3),
        # t2g model with V(q) from the vertex file to the densities, mixed (BSE 486 x 486)
        _ladder_case("ingest_t2g_vq_mixed", 3, 12, 6, 27, 3, 10.0, 4.0, 0.6, "mixed", 1 + 3 * 216, 216, "ingest"),
        # one frequency of the SrVO3-like t2g model, mixed (1000 points, BSE 1080 x 1080)
        _ladder_case("slice_t2g_mixed", 3, 20, 10, 60, 10, 10.0, 5.0, 0.75, "mixed", 1 + 10 * 1000, 1000),
        # a rank's block of it in FP64, the default precision
        _ladder_case("block_t2g_fp64", 3, 20, 10, 60, 10, 10.0, 5.0, 0.75, "fp64", 1 + 9 * 1000 + 700, 250),
        # five-orbital member of the sweep, one frequency, mixed (BSE 1000 x 1000, 25 right-hand sides)
        _ladder_case("slice_5orb_mixed", 5, 12, 6, 20, 5, 10.0, 3.0, 0.45, "mixed", 1 + 4 * 216, 216),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.12:
        return dict(kind="inverse", n=_log_int(rng, 24, 720))
    while True:
        kind = rng.choice(["ladder", "ladder", "ladder", "ladder", "tangent", "ingest", "point"])
        ndim = rng.choice([1, 2, 2, 3, 3, 3, 5] if kind != "tangent" else [1, 2, 3])
        nq = rng.randint(3, 8)
        nk = nq * rng.choice([1, 2])
        iwf = _log_int(rng, 8, {1: 160, 2: 90, 3: 60, 5: 22}[ndim])
        iwb = rng.randint(1, 6)
        total = nq ** 3 * (2 * iwb + 1)
        big = {"point": 1, "tangent": 256}.get(kind, nq ** 3 * 2)
        points = 1 if kind == "point" else min(total, _log_int(rng, 8, max(9, big)))
        qw0 = 1 + rng.randint(0, total - points)
        U = rng.uniform(2.0, 4.0)
        c = _ladder_case("", ndim, nk, nq, iwf, iwb, rng.choice([8.0, 10.0, 15.0, 20.0]), U,
                         0.0 if ndim == 1 else U * rng.uniform(0.1, 0.18), rng.choice(["fp64", "mixed"]), qw0,
                         points, kind, rng.randint(1, 3) if kind == "tangent" else 0,
                         kind == "ladder" and rng.random() < 0.15,
                         *(rng.choice([(True, True), (True, True), (True, False), (False, True)])
                           if kind == "ladder" else (True, True)))
        del c["name"]
        limit = 1.5e12 if c["precision"] == "fp64" else 5e12
        if work(c)["flops"] * (1 + c["directions"]) <= limit:
            return c


# ---- inputs ------------------------------------------------------------------


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _bands(ndim, n, t):
    """H(k) of the model, (n^3, ndim, ndim), k in the order of the mesh files (kz fastest)."""
    ax = 2 * np.pi * np.arange(n) / n
    kx, ky, kz = (a.ravel() for a in np.meshgrid(ax, ax, ax, indexing="ij"))
    c = [np.cos(kx), np.cos(ky), np.cos(kz)]
    H = np.zeros((n ** 3, ndim, ndim), dtype=complex)
    for a in range(ndim):
        if ndim == 3:      # t2g: each band disperses in its own plane
            p, q, r = [(0, 1, 2), (0, 2, 1), (1, 2, 0)][a]
            H[:, a, a] = -2 * t * (c[p] + c[q]) - 0.23 * t * c[r] - 1.2 * t * c[p] * c[q]
        elif ndim == 2:    # e_g: planar and axial band
            w = [(1, 1, 0.5), (0.5, 0.5, 1)][a]
            H[:, a, a] = -2 * t * sum(x * y for x, y in zip(w, c))
        else:
            H[:, a, a] = -2 * t * (1 + 0.15 * a) * sum(c) + 0.05 * a
        for b in range(a):
            v = 0.1 * t * (np.sin(kx) * np.sin(ky) + 0.7j * (a - b) * np.sin(kz) * c[0])
            H[:, a, b], H[:, b, a] = v, v.conj()
    return H


def _kanamori(ndim, U, V, J):
    """u({k,i},{j,l}) = U_ijkl and u~({k,i},{j,l}) = U_ijlk."""
    Um = np.zeros((ndim,) * 4)
    for i in range(ndim):
        for j in range(ndim):
            Um[i, i, j, j] = U if i == j else J
            if i != j:
                Um[i, j, i, j], Um[i, j, j, i] = V, J
    nd2 = ndim * ndim
    u = Um.transpose(0, 2, 3, 1).reshape(nd2, nd2)        # [i, k, l, j]
    ut = Um.transpose(0, 3, 2, 1).reshape(nd2, nd2)       # U_ijlk as [i, k, l, j]
    return u.astype(complex), ut.astype(complex)


def _chemical_potential(H, iw, sig, beta, filling):
    e = np.linalg.eigvalsh(H[:: max(1, len(H) // 400)])
    lo, hi = -8.0, 8.0
    for _ in range(24):
        mu = 0.5 * (lo + hi)
        n = 2 * (1 / (1j * iw + mu - e[:, :, None] - sig)).real.sum(-1).mean() / beta + 0.5
        lo, hi = (lo, mu) if n > filling else (mu, hi)
    return mu


def _inputs(case, seed):
    """Everything a ladder is built from, as numpy arrays (frequency index n + iwmax holds nu_n)."""
    rng = np.random.default_rng(seed)
    nd, iwf, iwb, beta = case["ndim"], case["iwf"], case["iwb"], case["beta"]
    nd2, iwmax = nd * nd, 4 * (iwf + iwb)
    U, J = case["U"] * rng.uniform(0.95, 1.05), case["J"] * rng.uniform(0.95, 1.05)
    t = {1: 0.25, 2: 0.3, 3: 0.26, 5: 0.2}[nd] * rng.uniform(0.95, 1.05)
    filling = {1: 0.5, 2: 0.25, 3: 1 / 6, 5: 0.4}[nd]
    iw = np.pi * (2 * np.arange(-iwmax, iwmax) + 1) / beta
    H = _bands(nd, case["nk"], t)
    s = 0.5 * U * filling * (1 - filling) / (1j * iw + 0.5j * np.sign(iw))
    mu = _chemical_potential(H, iw[iwmax:], s[iwmax:], beta, filling)
    bath = 0.5 * (1j * iw - 1j * np.sign(iw) * np.sqrt(iw ** 2 + 1))
    g = 1 / (1j * iw + mu - bath - s)
    u, ut = _kanamori(nd, U, U - 2 * J, J)
    P = dict(iwmax=iwmax, iw=iw, H=H, mu=float(mu), siw=np.repeat(s[:, None], nd, 1),
             giw=np.repeat(g[:, None], nd, 1), u=u, ut=ut,
             n_dmft=np.full(nd, 2 * g[iwmax:].real.sum() / beta + 0.5, dtype=complex), vertex={}, dvertex={})
    q1 = case["qw0"] - 1
    for w in range(q1 // case["nq"] ** 3 - iwb, (q1 + case["points"] - 1) // case["nq"] ** 3 - iwb + 1):
        c0 = _chi0_loc(torch.as_tensor(P["giw"]), iwmax, iwf, w, beta).reshape(-1).to(_dev())
        chi, dchi = [], {d: [] for d in DIRECTIONS[:2]}
        for ch, V in enumerate((2 * u - ut, -ut)):
            R = rng.uniform(-1, 1, (2 * iwf, 2 * iwf)) + 1j * rng.uniform(-1, 1, (2 * iwf, 2 * iwf))
            W = torch.as_tensor(1 + 0.005 * (R + R.conj().T)).to(_dev()) / beta ** 2
            x = torch.linalg.inv(torch.diag(1 / c0) + torch.kron(W, torch.as_tensor(V).to(_dev())))
            chi.append(x)
            for d, cpl in zip(DIRECTIONS[:case["directions"]], ((1.0, 1.0, 0.0), (0.0, -2.0, 1.0))):
                du, dut = _kanamori(nd, *cpl)
                dV = torch.as_tensor((2 * du - dut, -dut)[ch]).to(_dev())
                dchi[d].append(-x @ torch.kron(W, dV) @ x)
        P["vertex"][w] = chi
        P["dvertex"][w] = dchi
    for d, cpl in zip(DIRECTIONS, ((1.0, 1.0, 0.0), (0.0, -2.0, 1.0))):
        P["d" + d] = _kanamori(nd, *cpl)
    P["dHt"] = H / t
    if case["kind"] == "ingest":      # V(q): nearest-neighbour density-density interaction, read per q
        q = _q_points(case)
        ck = sum(np.cos(2 * np.pi * (q // m % case["nk"]) / case["nk"]) for m in (1, case["nk"], case["nk"] ** 2))
        vq = np.zeros((nd, nd, nd, nd, len(q)), dtype=complex)
        for i in range(nd):
            for j in range(nd):
                vq[i, j, i, j] = 0.1 * U * ck / (1 + abs(i - j))
        P["vq"] = vq
    return P


def _q_points(case):
    """0-based k index of every q point."""
    a = np.arange(case["nq"]) * (case["nk"] // case["nq"])
    return (a[:, None, None] * case["nk"] ** 2 + a[None, :, None] * case["nk"] + a[None, None, :]).ravel()


def _host(x):
    """A matrix as a program keeps it for the upload: complex128, Fortran order, pinned."""
    x = x.T.contiguous().cpu()
    return (x.pin_memory() if torch.cuda.is_available() else x).numpy().T


def _pinned(shape):
    x = torch.zeros(tuple(reversed(shape)), dtype=torch.complex128, pin_memory=torch.cuda.is_available())
    return x.numpy().transpose()


def prepare(case, seed):
    if case["kind"] == "inverse":
        rng = np.random.default_rng(seed)
        n = case["n"]
        M = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / math.sqrt(2 * n)
        return dict(case=case, M=np.asfortranarray(M + np.diag(1.5 + rng.uniform(0, 1, n))))
    P = _inputs(case, seed)
    nd, n = case["ndim"], case["points"]
    lad = Ladder(ndim=nd, nk=(case["nk"],) * 3, nq=(case["nq"],) * 3, iwmax=P["iwmax"],
                 iwfmax_small=case["iwf"], iwbmax_small=case["iwb"], beta=case["beta"], mu=P["mu"],
                 iw_data=P["iw"], hk=P["H"].transpose(1, 2, 0), siw=P["siw"], giw=P["giw"],
                 dc=np.zeros((2, nd), dtype=complex), u=P["u"], u_tilde=P["ut"], n_dmft=P["n_dmft"],
                 q_data=generate_q_vol((case["nk"],) * 3, (case["nq"],) * 3), do_chi=case["do_chi"],
                 do_eom=case["do_eom"], bubble_big_box=case["big_box"])
    s = dict(case=case, lad=lad, last=case["qw0"] + n - 1)
    if case["kind"] == "ingest":
        # the vertex file's array g4(ndim, ndim, 2W, ndim, ndim, 2W), connected part, before the beta factor
        F, s["g4"] = 2 * case["iwf"], {}
        for w, chi in P["vertex"].items():
            bub = torch.diag(_chi0_loc(torch.as_tensor(P["giw"]), P["iwmax"], case["iwf"], w, case["beta"]).reshape(-1))
            s["g4"][w] = [np.asfortranarray(((x.cpu() - bub) / case["beta"]).reshape(F, nd, nd, F, nd, nd)
                                            .permute(1, 2, 0, 5, 4, 3).numpy()) for x in chi]
        lad.set_vq(P["vq"])
    else:
        s["vertex"] = {w: [_host(x) for x in chi] for w, chi in P["vertex"].items()}
    if case["kind"] == "point":
        for w, chi in s["vertex"].items():
            lad.set_vertex(w, *chi)
        return s
    for d, name in enumerate(DIRECTIONS[:case["directions"]]):
        if name == "t":
            lad.set_tangent(P["dHt"].transpose(1, 2, 0), None, None, direction=d)
            continue
        lad.set_tangent(None, *P["d" + name], direction=d)
        for w, dchi in P["dvertex"].items():
            lad.set_vertex_tangent(w, *(_host(x) for x in dchi[name]), direction=d)
    s["out"] = {k: _pinned(shape) for k, shape in lad.output_shapes(n).items()}
    return s


def run(state):
    c = state["case"]
    if c["kind"] == "inverse":
        return inverse_matrix(state["M"])[:2]
    lad = state["lad"]
    if c["kind"] == "point":
        q, nqp = c["qw0"] - 1, c["nq"] ** 3
        return lad.bse_point(q % nqp + 1, q // nqp - c["iwb"], c["precision"])
    lad.reset_outputs()
    if c["kind"] == "ingest":
        for w, g4 in state["g4"].items():
            lad.set_vertex_g4(w, *g4)
    else:
        for w, chi in state["vertex"].items():
            lad.set_vertex(w, *chi)
    if c["kind"] == "tangent":
        status, _ = lad.ladder_run_tangent(c["qw0"], state["last"], c["precision"])
        out = dict(lad.get_outputs(state["out"]), status=status)
        out["tangents"] = [lad.get_tangent_outputs(d) for d in range(c["directions"])]
        return out
    status, _ = lad.ladder_run(c["qw0"], state["last"], c["precision"])
    out = dict(lad.get_outputs(state["out"]), status=status)
    if c["kind"] == "ingest":
        out["post"] = lad.post_loop()
    return out


def work(case):
    """Bytes: every input once (vertices, H(k), local quantities), every output once.  Flops: the bubble as a
    transform, the BSE matrices, one LU of each with ndim^2 right-hand sides, the sums and the EOM."""
    if case["kind"] == "inverse":
        return {"bytes": 32.0 * case["n"] ** 2, "flops": 8.0 * case["n"] ** 3}
    nd2, iwf, n, nkp, nqp = case["ndim"] ** 2, case["iwf"], case["points"], case["nk"] ** 3, case["nq"] ** 3
    N = 2 * iwf * nd2
    q1 = case["qw0"] - 1
    nw = (q1 + n - 1) // nqp - q1 // nqp + 1
    lu = 8 / 3 * N ** 3 + 8 * nd2 * N ** 2
    build = 8 * nd2 * N ** 2
    sums = 4 * 8 * nd2 ** 2 * N
    fft = 5 * math.log2(nkp + 1)
    mesh = nw * 2 * iwf * (nkp * nd2 * (8 * nd2 + fft) + nqp * nd2 ** 2 * fft)
    eom = nw * iwf * nkp * nd2 * (8 * nd2 + fft)
    if case["kind"] == "point":
        nkp_work = 8 * nkp * nd2 ** 2 * 2 * iwf
        return {"bytes": 16.0 * (2 * N * N + nkp * nd2 + 3 * nd2 * N), "flops": 2.0 * (lu + build + sums) + nkp_work}
    out = 16.0 * (3 * nd2 ** 2 * n + nd2 * 2 * iwf * nkp)
    nt = case["directions"]
    tangent = nt * n * 2 * (3 * 8 * nd2 * N ** 2 + sums)
    return {"bytes": 16.0 * (2 * N * N * nw + nkp * nd2) * (1 + nt) + out * (1 + nt),
            "flops": n * 2.0 * (lu + build + sums) + (mesh + eom) * (1 + nt) + tangent}


# ---- the same outputs in plain torch, 64 bits ------------------------------------


def _chi0_loc(giw, iwmax, iwf, w, beta):
    """chi0_loc({i,j}, nu) = -beta g_i(nu) g_j(nu - omega), (2 iwf, ndim^2)."""
    n = torch.arange(-iwf, iwf, device=giw.device) + iwmax
    return (-beta * giw[n][:, :, None] * giw[n - w][:, None, :]).reshape(2 * iwf, -1)


def _lattice_g(case, P, H, lo, hi, sig=None):
    """G(k, nu_n), n = lo .. hi - 1: (hi - lo, nkp, ndim, ndim); sig: a self-energy matrix instead of siw."""
    nd, dev = case["ndim"], H.device
    n = torch.arange(lo, hi, device=dev) + P["iwmax"]
    eye = torch.eye(nd, dtype=H.dtype, device=dev)
    s = torch.diag_embed(torch.as_tensor(P["siw"]).to(dev)[n])[:, None] if sig is None else sig
    z = 1j * torch.as_tensor(P["iw"]).to(dev)[n] + P["mu"]
    return torch.linalg.inv(z[:, None, None, None] * eye - H[None] - s)


def _ladder(case, P, H, u, ut, vertex):
    """Accumulators of the block in the framework's shapes, and what `point` returns of its last point."""
    nd, iwf, iwb, beta, nk = case["ndim"], case["iwf"], case["iwb"], case["beta"], case["nk"]
    dev, nd2, nqp, nkp, npts = H.device, case["ndim"] ** 2, case["nq"] ** 3, case["nk"] ** 3, case["points"]
    N, F, nw = nd2 * 2 * iwf, 2 * iwf, 2 * iwb + 1
    lo, hi = (-P["iwmax"] + iwb, P["iwmax"] - iwb) if case["big_box"] and case["do_chi"] else (-iwf, iwf)
    giw, nd_mat = torch.as_tensor(P["giw"]).to(dev), torch.as_tensor(P["n_dmft"]).to(dev)
    qk = torch.as_tensor(_q_points(case)).to(dev)
    vq = None
    if "vq" in P:                                                 # v({i,k},{l,j}) = V_ijkl
        vq = torch.as_tensor(P["vq"]).to(dev).permute(4, 0, 2, 3, 1).reshape(nqp, nd2, nd2)
    z = lambda *s: torch.zeros(s, dtype=torch.complex128, device=dev)  # noqa: E731
    eye, eyeN = torch.eye(nd2, dtype=H.dtype, device=dev), torch.eye(N, dtype=H.dtype, device=dev)
    G = _lattice_g(case, P, H, lo - iwb, hi + iwb)
    mesh = lambda x: x.reshape(x.shape[0], nk, nk, nk, *x.shape[2:])  # noqa: E731
    Gf = torch.fft.fftn(mesh(G), dim=(1, 2, 3))
    chi_d, chi_m, bub_nl, last = [], [], [], None
    bub_loc, loc_d, loc_m = [z(nd2, nd2)] * nw, [z(nd2, nd2)] * nw, [z(nd2, nd2)] * nw
    sig, sdmft, shf = z(iwf, nkp, nd, nd), z(iwf, nd, nd), z(nkp, nd, nd)
    sdmft_static = z(nd)
    first = case["qw0"] - 1
    for w in sorted(vertex):
        a, b = max(first, (w + iwb) * nqp), min(first + npts, (w + iwb + 1) * nqp)
        iq = torch.arange(a, b, device=dev) - (w + iwb) * nqp
        starts = a == (w + iwb) * nqp
        # chi0^q(nu) = -(beta / nkp) sum_k G_il(k, nu) G_k'j(k - q, nu - omega)
        c0q, bubble = [], z(len(iq), nd2, nd2)
        step = max(1, int(5e8 / (nkp * nd2 ** 2 * 16)))
        for n0 in range(lo, hi, step):
            n = torch.arange(n0, min(hi, n0 + step), device=dev) - (lo - iwb)
            B = torch.fft.ifftn(mesh(G[n - w]), dim=(1, 2, 3))    # 1/nkp of the transform at -p
            x = torch.einsum("nxyzil,nxyzkj->nijlkxyz", Gf[n], B)
            x = torch.fft.ifftn(x, dim=(5, 6, 7)).reshape(len(n), nd2, nd2, nkp)[..., qk[iq]]
            x = -beta * x.permute(3, 0, 1, 2)
            bubble = bubble + x.sum(1)
            k0, k1 = max(0, -iwf - n0), min(len(n), iwf - n0)
            if k1 > k0:
                c0q.append(x[:, k0:k1])
        c0q = torch.cat(c0q, 1)                                  # (q, nu, nd2, nd2)
        c0w = _chi0_loc(giw, P["iwmax"], iwf, w, beta)
        nall = torch.arange(lo, hi, device=dev) + P["iwmax"]
        bl = torch.diag((-beta * giw[nall][:, :, None] * giw[nall - w][:, None, :]).reshape(-1, nd2).sum(0)) / beta ** 2
        Fs = []
        for x in vertex[w]:
            Fs.append(0.5 * (x + x.T) / c0w.reshape(1, -1) - eyeN)
        gam = [f.reshape(F, nd2, N).sum(0) for f in Fs]
        opg = [x + eye.repeat(1, F) for x in gam]
        sum_chi = lambda x, c: torch.einsum("...anb,...nbc->...ac", x.reshape(*x.shape[:-1], F, nd2), c) / beta ** 2  # noqa: E731
        if starts and case["do_chi"]:
            bub_loc[w + iwb] = bl
            loc_d[w + iwb], loc_m[w + iwb] = (sum_chi(x, torch.diag_embed(c0w)) for x in gam)
        if case["do_eom"] and w == 0 and starts:
            for i in range(nd):
                e = torch.zeros(nd, dtype=H.dtype, device=dev)
                e[i] = 1
                t = sum((2 * u[i * nd + i, j * nd + j] - u[i * nd + j, i * nd + j]) * nd_mat[j] for j in range(nd))
                sdmft_static = sdmft_static + t * e
        if case["do_eom"] and starts:
            m = (-(u @ gam[0]) / beta).reshape(nd, nd, F, nd, nd)[:, :, iwf:]       # [i, k, nu, l, k]
            gk = giw[torch.arange(0, iwf, device=dev) + P["iwmax"] - w]
            sdmft = sdmft + torch.einsum("iknlk,nk->nil", m, gk)
        if case["do_eom"] and w == 0 and vq is not None:
            dg = torch.arange(nd, device=dev)
            if starts:
                t = 2 * vq[0].reshape(nd, nd, nd, nd)[dg[:, None], dg[:, None], dg[None], dg[None]] @ nd_mat
                shf = shf + torch.diag(t)
            nf = sum(_lattice_g(case, P, H, n, n + 1)[0].real for n in range(P["iwmax"])) * 2 / beta
            nf = (nf + 0.5 * torch.eye(nd, device=dev)).to(H.dtype)
            vm = z(nkp, nd2, nd2).index_copy(0, qk[iq], vq[iq]).reshape(1, nkp, nd, nd, nd, nd)   # [q, i, k, l, j]
            cv = torch.einsum("nxyziklj,nxyzjk->nxyzil", torch.fft.fftn(mesh(vm), dim=(1, 2, 3)),
                              torch.fft.fftn(mesh(nf[None]), dim=(1, 2, 3)))
            shf = shf - torch.fft.ifftn(cv, dim=(1, 2, 3)).reshape(nkp, nd, nd) / nqp
        mt = []
        step = max(1, int(2e9 / (N * N * 16)))
        for p0 in range(0, len(iq), step):
            c = c0q[p0:p0 + step]
            sw = c / c0w[None, :, None, :] - eye
            eta, gq = [], None
            for ch in range(2):
                rect = torch.einsum("qnab,nbN->qnaN", sw, Fs[ch].reshape(F, nd2, N))
                gq = rect.sum(1) if ch == 0 else gq
                A = eyeN - rect.reshape(-1, N, N)
                if vq is not None and ch == 0:
                    sm = 2 / beta ** 2 * (c @ vq[iq[p0:p0 + step]][:, None])
                    A = A - torch.einsum("qnab,bN->qnaN", sm, opg[0]).reshape(-1, N, N)
                X = torch.linalg.solve(A.transpose(1, 2), opg[ch].T.expand(len(c), N, nd2)).transpose(1, 2)
                eta.append(X - opg[ch])
            cnl = c - torch.diag_embed(c0w)
            chi_d.append(sum_chi(gam[0], cnl) + sum_chi(eta[0], c))
            chi_m.append(sum_chi(gam[1], cnl) + sum_chi(eta[1], c))
            uw = u - 0.5 * ut if vq is None else vq[iq[p0:p0 + step]] + u - 0.5 * ut
            m = -(uw @ eta[0]) + 1.5 * (ut @ eta[1]) + u @ gq
            if vq is not None:
                m = m - vq[iq[p0:p0 + step]] @ gam[0]
            mt.append(m[:, :, N // 2:] / (beta * nqp))
            last = [x[-1] for x in (*eta, gq)]
        bub_nl.append(bubble / beta ** 2 - bl)
        if case["do_eom"]:
            # Sigma_il(k, nu) += sum_q m_ij,lk'(q, nu) G_jk'(k - q, nu - omega)
            mt = torch.cat(mt).reshape(len(iq), nd, nd, iwf, nd, nd)
            parts = []
            step = max(1, int(5e8 / (nkp * nd2 ** 2 * 16)))
            for n0 in range(0, iwf, step):
                x = mt[:, :, :, n0:n0 + step].permute(3, 0, 1, 2, 4, 5)
                x = z(x.shape[0], nkp, nd, nd, nd, nd).index_copy(1, qk[iq], x.contiguous())
                n = torch.arange(n0, n0 + x.shape[0], device=dev) - w - (lo - iwb)
                x = torch.einsum("nxyzijlk,nxyzjk->nxyzil", torch.fft.fftn(mesh(x), dim=(1, 2, 3)), Gf[n])
                parts.append(torch.fft.ifftn(x, dim=(1, 2, 3)).reshape(-1, nkp, nd, nd))
            sig = sig + torch.cat(parts)
    # nu >= 0 computed; Sigma(-nu-1) = Sigma(nu)^dagger
    full = lambda x: torch.cat([x.transpose(-1, -2).conj().flip(0), x])  # noqa: E731
    sdmft = full(sdmft) + torch.diag(sdmft_static)
    stack = lambda xs: torch.stack(xs, -1)  # noqa: E731
    zero = z(nd2, nd2, npts)
    perq = lambda x: torch.cat(x).permute(1, 2, 0) if case["do_chi"] else zero  # noqa: E731
    out = dict(chi_qw_dens=perq(chi_d), chi_qw_magn=perq(chi_m), bubble_nl=perq(bub_nl), bubble_loc=stack(bub_loc),
               chi_loc_dens=stack(loc_d), chi_loc_magn=stack(loc_m), sigma_nl=full(sig).permute(2, 3, 0, 1),
               sigma_dmft=sdmft.permute(1, 2, 0), sigma_hf=shf.permute(1, 2, 0))
    return out, last


def _post(case, P, H, sigma_nl):
    nd, iwf, iwmax, beta = case["ndim"], case["iwf"], P["iwmax"], case["beta"]
    siw = torch.diag_embed(torch.as_tensor(P["siw"]).to(H.device)[iwmax - iwf:iwmax + iwf])
    s = sigma_nl.permute(2, 3, 0, 1) + siw[:, None]
    gl, nk = [], 0
    for n in range(iwmax):
        g = _lattice_g(case, P, H, n, n + 1, s[n + iwf] if n < iwf else None)[0]
        gl.append(g.mean(0))
        nk = nk + g.real
    gl = torch.stack(gl)
    gl = torch.cat([gl.transpose(1, 2).conj().flip(0), gl])
    nk = (2 * nk / beta + 0.5 * torch.eye(nd, device=H.device)).to(H.dtype)
    return dict(sigma_loc=s.mean(1).permute(1, 2, 0), gloc=gl, n_dga_k=nk,
                n_dga=nk.diagonal(dim1=1, dim2=2).mean(0))


def _numpy(x):
    return {k: v.cpu().numpy() for k, v in x.items()}


def exact(case, seed):
    if case["kind"] == "inverse":
        return np.linalg.inv(prepare(case, seed)["M"]), None
    P = _inputs(case, seed)
    H, u, ut = (torch.as_tensor(P[k]).to(_dev()) for k in ("H", "u", "ut"))
    if case["kind"] != "tangent":
        out, point = _ladder(case, P, H, u, ut, P["vertex"])
        if case["kind"] == "point":
            return [x.cpu().numpy() for x in point] + [None]
        out = dict(_numpy(out), status=None)
        if case["kind"] == "ingest":
            out["post"] = _numpy(_post(case, P, H, torch.as_tensor(out["sigma_nl"]).to(_dev())))
        return out
    out, tangents = None, []
    fw = torch.autograd.forward_ad
    for d in DIRECTIONS[:case["directions"]]:
        with fw.dual_level():
            args, zero = [H, u, ut], torch.zeros_like
            tan = [torch.as_tensor(P["dHt"]).to(_dev()), zero(u), zero(u)] if d == "t" else \
                [zero(H)] + [torch.as_tensor(x).to(_dev()) for x in P["d" + d]]
            dual = [fw.make_dual(x, t) for x, t in zip(args, tan)]
            vertex = P["vertex"] if d == "t" else {
                w: [fw.make_dual(x, t) for x, t in zip(chi, P["dvertex"][w][d])] for w, chi in P["vertex"].items()}
            y, _ = _ladder(case, P, *dual, vertex)
            parts = {k: fw.unpack_dual(v) for k, v in y.items()}
            if out is None:
                out = dict(_numpy({k: v.primal.detach() for k, v in parts.items()}), status=None)
            tangents.append(_numpy({k: zero(v.primal) if v.tangent is None else v.tangent for k, v in parts.items()}))
    out["tangents"] = tangents
    return out
