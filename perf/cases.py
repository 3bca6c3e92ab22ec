"""The work this framework is measured on, through its public entry points.

Each case is one thing a user's program does on a GPU: transform fields
between collocation values and coefficients, evaluate fields at points,
evaluate a system's residual, take a Newton step or a whole solve, solve a
dense system with the mixed-precision LU, take the gradient of an observable.
Sizes are those of the framework's own workloads (the isolated star, the
binary's resolution on a spherical space, the toy problem) and of its tests.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

# basis codes of the transform descriptors (include/kadath_gb300.h)
CHEB, CHEB_EVEN, CHEB_ODD, COSSIN, COS_EVEN, SIN_ODD = 1, 2, 3, 4, 6, 10
KINDS = ("nucleus", "shell", "compact")


def listed():
    return [
        # the smallest call: one field of one domain to coefficients (an
        # initial-data reader, a diagnostic); latency decides
        {"name": "coef_one_field", "kind": "transform", "dir": "coef", "nr": 13, "nt": 9, "np": 4, "domains": 1,
         "batch": 1},
        # a block of tangent fields over the isolated star's six domains
        {"name": "coef_star_block", "kind": "transform", "dir": "coef", "nr": 13, "nt": 9, "np": 4, "domains": 6,
         "batch": 430},
        # the way back at a ragged higher resolution, larger than L2
        {"name": "coef_i_fine_block", "kind": "transform", "dir": "coef_i", "nr": 21, "nt": 11, "np": 14,
         "domains": 5, "batch": 600},
        # an exporter asking for a thousand points of one field from the host
        {"name": "points_host_1k", "kind": "points", "host": True, "points": 1000, "fields": 1, "nr": 13, "nt": 9,
         "np": 4},
        # an exporter filling a Cartesian grid with the star's five fields
        {"name": "points_device_1m", "kind": "points", "host": False, "points": 1000003, "fields": 5, "nr": 13,
         "nt": 9, "np": 4},
        # sec_member of the isolated star (line searches, convergence checks)
        {"name": "residual_star", "kind": "residual", "system": "star", "nr": 13, "nt": 9, "np": 4},
        # a complete solve of a small problem: launch latency and host work
        {"name": "solve_toy", "kind": "solve", "system": "toy", "nr": 9, "nt": 5, "np": 4},
        # a complete mixed-precision solve of the isolated star: first step
        # (tangents, pivoting) and later ones, as an initial-data run does
        {"name": "solve_star", "kind": "solve", "system": "star", "nr": 13, "nt": 9, "np": 4},
        # one do_newton with the default FP64 LU, shift in index notation
        {"name": "step_star_fp64", "kind": "step", "system": "star_vector", "lu": "fp64", "nr": 11, "nt": 7, "np": 4},
        # one mixed step at the binary's resolution (twelve domains)
        {"name": "step_large_mixed", "kind": "step", "system": "star_large", "lu": "mixed", "nr": 11, "nt": 9,
         "np": 8},
        # the dense solver by itself on a caller's matrix of a ragged size
        {"name": "lu_mixed_6001", "kind": "lu", "n": 6001},
        # the backward direction: gradient of the ADM mass at a converged star
        {"name": "adjoint_star", "kind": "adjoint", "system": "star", "nr": 11, "nt": 7, "np": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["transform", "transform", "points", "residual", "solve", "step", "lu", "adjoint"])
    if kind == "transform":
        c = {"kind": kind, "dir": rng.choice(["coef", "coef_i"]), "nr": rng.choice([5, 9, 11, 13, 15, 17, 21, 25]),
             "nt": rng.choice([5, 7, 9, 11, 13]), "np": rng.choice([4, 6, 8, 12, 14]),
             "domains": rng.randint(1, 12)}
        points = c["nr"] * c["nt"] * c["np"] * c["domains"]
        return {**c, "batch": _log(rng, 1, max(1, min(1000, 9000000 // points)))}
    if kind == "points":
        return {"kind": kind, "host": rng.random() < 0.5, "points": _log(rng, 100, 1000000),
                "fields": rng.randint(1, 5), "nr": rng.choice([9, 11, 13, 17]), "nt": rng.choice([5, 7, 9, 11]),
                "np": rng.choice([4, 6, 8])}
    if kind == "lu":
        return {"kind": kind, "n": _log(rng, 600, 14000)}
    nr, nt = rng.choice([(9, 5), (9, 7), (11, 5), (11, 7), (13, 5), (13, 7)])
    if kind == "residual":
        return {"kind": kind, "system": rng.choice(["toy", "star", "star_vector"]), "nr": nr + rng.choice([0, 2, 4]),
                "nt": nt, "np": rng.choice([4, 6, 8])}
    if kind == "solve":
        return {"kind": kind, "system": rng.choice(["toy", "star", "star_vector"]), "nr": nr, "nt": nt, "np": 4}
    if kind == "step":
        lu = rng.choice(["fp64", "mixed"])
        return {"kind": kind, "system": rng.choice(["toy", "star", "star_vector"]), "lu": lu,
                "nr": nr if lu == "mixed" else min(nr, 11), "nt": nt, "np": 4}
    return {"kind": kind, "system": rng.choice(["toy", "star"]), "nr": nr, "nt": nt, "np": 4}


# ------------------------------------------------------------- transforms --
def _domain_kinds(n):
    """nucleus, shells, compactified exterior; a single domain is a shell."""
    return ["shell"] if n == 1 else ["nucleus"] + ["shell"] * (n - 2) + ["compact"]


def _m_even(np_):
    return [(k // 2) % 2 == 0 for k in range(np_ + 2)]


def _phi_basis(phi, np_):
    cols = [np.cos((k // 2) * phi) if k % 2 == 0 else np.sin((k // 2) * phi) for k in range(np_ + 2)]
    return np.stack(cols, -1)


def _theta_basis(th, nt, even):
    j = np.arange(nt)
    return np.cos(2 * j * th[..., None]) if even else np.sin((2 * j + 1) * th[..., None])


def _radial_basis(x, nr, kind, even):
    a = np.arccos(np.clip(x, -1.0, 1.0))[..., None]
    i = np.arange(nr)
    return np.cos((i if kind != "nucleus" else (2 * i if even else 2 * i + 1)) * a)


def _grid(nr, nt, np_, kind):
    i = np.arange(nr) / (nr - 1)
    x = np.sin(0.5 * math.pi * i) if kind == "nucleus" else -np.cos(math.pi * i)
    return x, 0.5 * math.pi * np.arange(nt) / (nt - 1), 2 * math.pi * np.arange(np_) / np_


def _random_coefs(rng, batch, nr, nt, np_, kind):
    """Decaying coefficients of smooth fields in the standard bases; the
    entries whose basis function vanishes on the grid are zero."""
    c = rng.standard_normal((batch, nr, nt, np_ + 2))
    c *= (0.6 ** np.arange(nr))[:, None, None] * (0.5 ** np.arange(nt))[:, None]
    c *= 0.4 ** (np.arange(np_ + 2) // 2)
    c[..., 1] = 0.0
    c[..., np_ + 1] = 0.0
    for k, even in enumerate(_m_even(np_)):
        if not even:
            c[:, :, nt - 1, k] = 0.0
            if kind == "nucleus":
                c[:, nr - 1, :, k] = 0.0
    return c


def _synthesis(c, nr, nt, np_, kind):
    """Values of the series at the collocation points, in 64 bits."""
    x, th, ph = _grid(nr, nt, np_, kind)
    t = np.empty(c.shape[:1] + (nr, nt, np_ + 2))
    for k, even in enumerate(_m_even(np_)):
        t[..., k] = np.einsum("xi,bij,tj->bxt", _radial_basis(x, nr, kind, even), c[..., k],
                              _theta_basis(th, nt, even), optimize=True)
    return t @ _phi_basis(ph, np_).T


def _transform_data(case, seed):
    """(coefficients, values) of every domain; fields beyond the 16th are the
    first ones with factors of their own, so that the host makes few."""
    nr, nt, np_ = case["nr"], case["nt"], case["np"]
    rng = np.random.default_rng([seed, nr, nt, np_])
    made = min(16, case["batch"])
    out = []
    for kind in _domain_kinds(case["domains"]):
        c = _random_coefs(rng, made, nr, nt, np_, kind)
        v = _synthesis(c, nr, nt, np_, kind)
        f = torch.tensor(rng.uniform(0.5, 1.5, case["batch"]))
        at = torch.arange(case["batch"]) % made
        if torch.cuda.is_available():
            f, at = f.cuda(), at.cuda()
        out.append(tuple(torch.tensor(a, device=f.device)[at] * f[:, None, None, None] for a in (c, v)))
    return out


def _prepare_transform(case, seed):
    from kadath_frontera_gb300 import default_context
    from kadath_frontera_gb300._lib import TransformDesc
    nr, nt, np_ = case["nr"], case["nt"], case["np"]
    forward = case["dir"] == "coef"
    kinds = _domain_kinds(case["domains"])
    descs = (TransformDesc * len(kinds))()
    keep, outs = [], []
    for d, kind, (c, v) in zip(descs, kinds, _transform_data(case, seed)):
        even = _m_even(np_)
        t = (C.c_int * (np_ + 2))(*[COS_EVEN if e else SIN_ODD for e in even])
        row = [CHEB if kind != "nucleus" else (CHEB_EVEN if e else CHEB_ODD) for e in even]
        r = (C.c_int * (nt * (np_ + 2)))(*(row * nt))
        src = (v if forward else c).contiguous()
        dst = torch.zeros_like(c if forward else v)
        d.nbr_points[:] = (nr, nt, np_)
        d.nbr_coefs[:] = (nr, nt, np_ + 2)
        d.base_r, d.base_t, d.base_p = C.cast(r, C.POINTER(C.c_int)), C.cast(t, C.POINTER(C.c_int)), COSSIN
        d.batch, d.in_, d.out = case["batch"], src.data_ptr(), dst.data_ptr()
        keep += [t, r, src]
        outs.append(dst)
    ctx = default_context()
    call = ctx.lib.kd_coef_many if forward else ctx.lib.kd_coef_i_many
    return {"kind": "transform", "ctx": ctx, "call": call, "n": len(kinds), "descs": descs, "keep": keep,
            "outs": outs}


# ----------------------------------------------------------------- points --
STAR_BOUNDS = (8.0, 12.0, 16.0, 24.0, 32.0)


def _points_data(case, seed):
    rng = np.random.default_rng([seed, case["points"], 7])
    nd = len(STAR_BOUNDS) + 1
    coefs = [[_random_coefs(rng, 1, case["nr"], case["nt"], case["np"], kind)[0] for kind in _domain_kinds(nd)]
             for _ in range(case["fields"])]
    return coefs, rng.uniform(-25.0, 25.0, (case["points"], 3))


def _prepare_points(case, seed):
    from kadath_frontera_gb300.kadath import CHEB_TYPE, Scalar, Space_spheric
    res = (case["nr"], case["nt"], case["np"])
    coefs, xyz = _points_data(case, seed)
    space = Space_spheric(CHEB_TYPE, (0, 0, 0), res, STAR_BOUNDS)
    fields = []
    for per in coefs:
        f = Scalar(space)
        for d, kind in enumerate(_domain_kinds(len(per))):
            f.set_domain(d, _synthesis(per[d][None], *res, kind)[0])
        fields.append(f.std_base())
    state = {"kind": "points", "host": case["host"], "space": space, "fields": fields, "xyz": xyz}
    if not case["host"]:
        state["xyz"] = torch.tensor(xyz, device="cuda:0")
        state["out"] = torch.zeros((case["fields"], case["points"]), dtype=torch.float64, device="cuda:0")
    return state


def _exact_points(case, seed):
    coefs, xyz = _points_data(case, seed)
    dev = "cuda:0" if torch.cuda.is_available() else "cpu"
    nt, np_, nr = case["nt"], case["np"], case["nr"]
    r = np.sqrt((xyz ** 2).sum(1))
    th = np.arccos(np.clip(xyz[:, 2] / r, -1, 1))
    ph = np.arctan2(xyz[:, 1], xyz[:, 0])
    edges = np.concatenate([[0.0], STAR_BOUNDS, [np.inf]])
    out = torch.empty((case["fields"], case["points"]), dtype=torch.float64, device=dev)
    for d, kind in enumerate(_domain_kinds(len(edges) - 1)):
        lo, hi = edges[d], edges[d + 1]
        every = np.nonzero((r >= lo) & (r < hi))[0]
        for at in np.array_split(every, max(1, len(every) // 65536)):
            if kind == "nucleus":
                x = r[at] / hi
            elif kind == "shell":
                x = (r[at] - 0.5 * (lo + hi)) / (0.5 * (hi - lo))
            else:
                x = 1.0 - 2.0 * lo / r[at]
            where = torch.tensor(at, device=dev)
            phi = torch.tensor(_phi_basis(ph[at], np_), device=dev)
            theta = {e: torch.tensor(_theta_basis(th[at], nt, e), device=dev) for e in (True, False)}
            rad = {e: torch.tensor(_radial_basis(x, nr, kind, e), device=dev) for e in (True, False)}
            for f in range(case["fields"]):
                c = torch.tensor(coefs[f][d], device=dev)
                v = 0.0
                for k, e in enumerate(_m_even(np_)):
                    v = v + phi[:, k] * ((rad[e] @ c[:, :, k]) * theta[e]).sum(1)
                out[f, where] = v
    return out if not case["host"] else out.cpu().numpy()


# ---------------------------------------------------------------- systems --
def _workload(case, seed):
    from kadath_frontera_gb300 import workloads
    rng = np.random.default_rng([seed, case["nr"], case["nt"], case["np"]])
    res = (case["nr"], case["nt"], case["np"])
    if case["system"] == "toy":
        # the toy's density profile with an amplitude and a width of its own
        amp, width = rng.uniform(0.03, 0.06), rng.uniform(0.2, 0.3)
        x, _, _ = _grid(*res, "nucleus")
        s, _, _ = _grid(*res, "shell")
        shape = np.ones(res)
        rho = [amp * np.exp(-x ** 2 / width)[:, None, None] * shape,
               amp * np.exp(-(1.5 + 0.5 * s) ** 2 / width)[:, None, None] * shape]
        far = np.zeros(res)
        far[:-1] = (amp * np.exp(-(4.0 / (1.0 - s[:-1])) ** 2 / width))[:, None, None]
        return workloads.toy(res=res, rho_values=rho + [far])
    rho_c = float(rng.uniform(8e-4, 2e-3))
    if case["system"] == "star_large":
        return workloads.star(res, workloads.LARGE_BOUNDS, rho_c=rho_c, matter_domains=4)
    return {"star": workloads.star, "star_vector": workloads.star_vector}[case["system"]](res=res, rho_c=rho_c)


def _perturb(wl, seed):
    """An iterate on its way: smooth bumps in the scalars, a rotating shift."""
    rng = np.random.default_rng([seed, 11])
    sp = wl.space
    for name, f in wl.unknowns:
        a, w = rng.uniform(0.02, 0.2), rng.uniform(3.0, 9.0)
        for d in range(sp.get_nbr_domains()):
            r, x, y = sp.get_radius(d), sp.get_cart(d, 1), sp.get_cart(d, 2)
            fin = np.isfinite(r)
            q = np.zeros_like(r)
            q[fin] = 1.0 / (1.0 + (r[fin] / w) ** 2)
            v = np.zeros_like(r)
            if name.startswith("b"):
                sign, arm = {"x": (-1.0, y), "y": (1.0, x), "z": (0.0, x)}[name[-1]]
                v[fin] = sign * 0.1 * a * arm[fin] * q[fin] ** 2
            else:
                v[:] = 1.0 + a * q
            f.set_domain(d, v)


def _prepare_system(case, seed):
    from kadath_frontera_gb300.kadath import KD_LU_FP64, KD_LU_TF32_IR
    wl = _workload(case, seed)
    state = {"kind": case["kind"], "wl": wl, "lu": KD_LU_FP64 if case.get("lu") == "fp64" else KD_LU_TF32_IR}
    if case["kind"] == "residual":
        _perturb(wl, seed)
    if case["kind"] == "solve":
        wl.syst.graph_capture = True
    if case["kind"] == "adjoint":
        for _ in range(20):
            if wl.syst.do_newton(1e-10, lu_mode=state["lu"])[0]:
                break
        state["expr"] = "integ(dn(%s))" % wl.unknowns[0][0]
    return state


def _run_solve(state):
    wl = state["wl"]
    # from the initial guess, with nothing kept from an earlier solve
    wl.restore()
    wl.syst.cache_tangents(False)
    wl.syst.cache_tangents(True)
    wl.syst.reset_pivot_order()
    for _ in range(20):
        done, err = wl.syst.do_newton(1e-10, lu_mode=state["lu"])
        if done:
            return wl.download()
    raise RuntimeError("no convergence: |F| = %g" % err)


def _run_step(state):
    wl = state["wl"]
    wl.restore()
    wl.syst.reset_pivot_order()
    done, err = wl.syst.do_newton(1e-10, lu_mode=state["lu"])
    return [err, wl.download()]


def _run_adjoint(state):
    syst = state["wl"].syst
    scale = -1.0 / (2.0 * math.pi)
    q, g = syst.integral_gradient(state["expr"], "inf")
    dqdp, lam = syst.adjoint(scale * g, "pi", reuse_factors=True)
    return [scale * q, g, dqdp, lam]


# --------------------------------------------------------------- dense LU --
def _lu_data(case, seed):
    """A regular matrix whose rows span six decades, as a spectral Jacobian's
    (second derivatives beside boundary rows), and a right-hand side."""
    n = case["n"]
    dev = "cuda:0" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device=dev).manual_seed(seed)
    a = torch.randn((n, n), generator=g, device=dev, dtype=torch.float64) / math.sqrt(n)
    a.diagonal().add_(torch.where(torch.rand(n, generator=g, device=dev) < 0.5, -2.0, 2.0).double())
    a *= 10.0 ** (6.0 * torch.rand((n, 1), generator=g, device=dev, dtype=torch.float64) - 3.0)
    b = a @ torch.randn(n, generator=g, device=dev, dtype=torch.float64)
    return a, b


def _prepare_lu(case, seed):
    from kadath_frontera_gb300.kadath import DenseLU
    a, b = _lu_data(case, seed)
    lu = DenseLU()
    return {"kind": "lu", "n": case["n"], "a": a.t().contiguous(), "b": b, "x": torch.empty_like(b), "lu": lu,
            "stream": torch.cuda.ExternalStream(lu.ctx.stream_ptr)}


def _run_lu(state):
    from kadath_frontera_gb300.kadath import KD_LU_TF32_IR
    n = state["n"]
    with torch.cuda.stream(state["stream"]):
        state["x"].copy_(state["b"])
    # column-major: the transposed copy's rows are the matrix's columns
    state["lu"].factor(state["a"].data_ptr(), n, n, KD_LU_TF32_IR)
    state["lu"].solve(state["x"].data_ptr())
    return state["x"]


# ------------------------------------------------------------------- all ---
def prepare(case, seed):
    kind = case["kind"]
    if kind == "transform":
        return _prepare_transform(case, seed)
    if kind == "points":
        return _prepare_points(case, seed)
    if kind == "lu":
        return _prepare_lu(case, seed)
    return _prepare_system(case, seed)


def run(state):
    kind = state["kind"]
    if kind == "transform":
        state["ctx"].check(state["call"](state["ctx"].h, state["n"], state["descs"]))
        return state["outs"]
    if kind == "points":
        from kadath_frontera_gb300 import kadath
        if state["host"]:
            return kadath.val_points(state["fields"], state["xyz"])
        out = state["out"]
        kadath.val_points_device(state["fields"], state["xyz"].data_ptr(), out.data_ptr(), out.shape[1])
        return out
    if kind == "residual":
        return state["wl"].syst.sec_member()
    return {"solve": _run_solve, "step": _run_step, "adjoint": _run_adjoint, "lu": _run_lu}[kind](state)


def exact(case, seed):
    if case["kind"] == "transform":
        forward = case["dir"] == "coef"
        return [c if forward else v for c, v in _transform_data(case, seed)]
    if case["kind"] == "points":
        return _exact_points(case, seed)
    if case["kind"] == "lu":
        a, b = _lu_data(case, seed)
        return torch.linalg.solve(a, b)
    # no closed form for a system's residual, iterates and gradients
    return None


def work(case):
    kind = case["kind"]
    if kind == "lu":
        n = case["n"]
        return {"bytes": 8.0 * n * n + 16.0 * n, "flops": 2.0 * n ** 3 / 3.0}
    nr, nt, np_ = case["nr"], case["nt"], case["np"]
    vals, cofs = nr * nt * np_, nr * nt * (np_ + 2)
    # one separable transform: a small product along phi, theta and r
    one = 2.0 * nr * nt * np_ * (np_ + 2) + 2.0 * cofs * (nt + nr)
    if kind == "transform":
        n = case["domains"] * case["batch"]
        return {"bytes": 8.0 * n * (vals + cofs), "flops": n * one}
    if kind == "points":
        # coefficients of the series that do not vanish: np of np + 2 in phi
        n, f = case["points"], case["fields"]
        return {"bytes": n * (24.0 + 8.0 * f) + 8.0 * f * cofs * (len(STAR_BOUNDS) + 1), "flops": 2.0 * n * f * vals}
    doms = {"toy": 3, "star": 6, "star_vector": 6, "star_large": 12}[case["system"]]
    unknowns = 1 if case["system"] == "toy" else 5
    fields = doms * unknowns
    # each equation needs its unknowns' coefficients, three second
    # derivatives and the way back to values or coefficients
    residual = {"bytes": 8.0 * fields * (vals + cofs), "flops": 6.0 * one * fields}
    if kind == "residual":
        return residual
    n = 0.87 * fields * vals  # the coefficients that regularity leaves free
    lu = 2.0 * n ** 3 / 3.0
    if kind == "step":
        return {"bytes": 16.0 * n * n, "flops": lu + residual["flops"] * (1 + vals)}
    if kind == "solve":
        return {"bytes": 48.0 * n * n, "flops": 3.0 * lu + residual["flops"] * (4 + 3 * vals)}
    # adjoint: the Jacobian written and read, the triangles read
    return {"bytes": 20.0 * n * n, "flops": 8.0 * n * n + residual["flops"] * (1 + vals)}
