"""The work whose speed this repository is measured by: calls a coupled-cluster program makes.

Each case goes through a public entry point of scess_gb300 (Context / State methods) on host
arrays in the reference's layout, as a user's program calls it.  Integrals come from seeded
density-fitting factors whose scale keeps the CCSD iteration convergent (convergent_sigma), and
fixed amplitudes are first-order doubles with small singles, so that every path meets values of
the sizes it meets in a real solve.  exact() restates each path in torch float64, on the GPU where
there is one.

Kinds (a case is a kind, its sizes and its precision):
  solve        SolveRCCSD_DIIS: the whole drop-in call, from the eri or from DF factors
  iterate      n iterations on a resident state from given amplitudes, amplitudes read back
  step         one iteration and (T) on a resident state: the step bench.py times
  triples      RCCSD_TriplesCorrection: the whole drop-in call, from the eri or from DF factors
  vjp          gradient of the residual in t1, t2 and the DF factors
  triples_vjp  gradient of E_(T) in t1, t2 and the DF factors
  transform    AO -> MO transform of the two-electron integrals
"""
import math

import numpy as np
import torch

import scess_gb300 as scess
from scess_gb300.cc import default_context
from scess_gb300.synthetic import convergent_sigma


def listed():
    return [
        # H2O/cc-pVDZ's size: the smallest drop-in solve users and the tests run (latency, launches)
        {"name": "solve_fp64_o5_v19", "kind": "solve", "o": 5, "v": 19, "precision": "fp64", "df": False},
        # a ten-electron-pair molecule solved from DF factors in the fast mode
        {"name": "solve_mixed_df_o10_v90", "kind": "solve", "o": 10, "v": 90, "precision": "mixed", "df": True},
        # three iterations (DIIS turns on at the third) of the default precision at the adjoint workload's size
        {"name": "iterate_fp64_o10_v90", "kind": "iterate", "o": 10, "v": 90, "precision": "fp64", "n": 3},
        # the same at the largest size whose FP64 iterations still take about a second
        {"name": "iterate_fp64_o16_v140", "kind": "iterate", "o": 16, "v": 140, "precision": "fp64", "n": 3},
        # the headline step: one mixed iteration and (T) at o=20 v=180
        {"name": "step_mixed_o20_v180", "kind": "step", "o": 20, "v": 180, "precision": "mixed"},
        # (T) of the smallest molecule, whole call
        {"name": "triples_fp64_o5_v19", "kind": "triples", "o": 5, "v": 19, "precision": "fp64", "df": False},
        # (T) in the default precision at an ordinary size
        {"name": "triples_fp64_df_o10_v90", "kind": "triples", "o": 10, "v": 90, "precision": "fp64", "df": True},
        # (T) in the fast mode with odd orbital counts (no multiple of any tile)
        {"name": "triples_mixed_df_o13_v117", "kind": "triples", "o": 13, "v": 117, "precision": "mixed", "df": True},
        # gradients: the residual's and E_(T)'s, with respect to amplitudes and DF factors
        {"name": "vjp_fp64_o8_v47", "kind": "vjp", "o": 8, "v": 47, "precision": "fp64"},
        {"name": "triples_vjp_fp64_o6_v31", "kind": "triples_vjp", "o": 6, "v": 31, "precision": "fp64"},
        # integral transforms: default precision with ragged sizes, fast mode with fewer MOs than AOs
        {"name": "transform_fp64_n73", "kind": "transform", "nao": 73, "nmo": 73, "precision": "fp64"},
        {"name": "transform_mixed_n112_m96", "kind": "transform", "nao": 112, "nmo": 96, "precision": "mixed"},
    ]


# (o, v) ranges of each kind's drawn cases; the upper ends are at or below the listed sizes
_RANGE = {"solve": ((3, 10), (12, 90)), "iterate": ((4, 16), (18, 140)), "step": ((8, 20), (60, 180)),
          "triples": ((4, 13), (15, 96)), "vjp": ((4, 10), (18, 56)), "triples_vjp": ((3, 7), (12, 34))}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "iterate", "step", "triples", "triples", "vjp", "triples_vjp", "transform"])
    precision = "mixed" if kind == "step" else rng.choice(["fp64", "fp64", "mixed"])
    if kind == "transform":
        nao = _log_int(rng, 24, 112 if precision == "mixed" else 80)
        return {"kind": kind, "nao": nao, "nmo": max(16, nao - rng.randrange(0, nao // 6 + 1)), "precision": precision}
    (o0, o1), (v0, v1) = _RANGE[kind]
    case = {"kind": kind, "o": _log_int(rng, o0, o1), "v": _log_int(rng, v0, v1), "precision": precision}
    if kind in ("solve", "triples"):
        case["df"] = case["v"] > 40 or rng.random() < 0.5
    if kind == "solve" and precision == "fp64":
        case["v"] = min(case["v"], 64)
    if kind == "triples" and precision == "fp64":
        case["o"] = min(case["o"], 10)
    if kind == "iterate":
        case["n"] = rng.choice([1, 2, 3])
    return case


# ---------------------------------------------------------------------------------------------
# inputs

_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _gen(seed):
    return torch.Generator(device=_DEV).manual_seed(int(seed))


def _host(x):
    """A tensor indexed [p, q, ...] as a NumPy array with the same indices in column-major memory."""
    return x.permute(*reversed(range(x.ndim))).contiguous().cpu().numpy().T


def _inputs(case, seed):
    """(eps, B[Q,p,q], t1[i,a], t2[i,j,a,b]) as torch float64 tensors."""
    o, v = case["o"], case["v"]
    n, naux = o + v, 3 * (o + v)
    g = _gen(seed)
    rand = lambda *s: torch.rand(*s, generator=g, device=_DEV, dtype=torch.float64)  # noqa: E731
    normal = lambda *s: torch.randn(*s, generator=g, device=_DEV, dtype=torch.float64)  # noqa: E731
    eps = torch.cat([torch.sort(-1.5 + 1.2 * rand(o)).values, torch.sort(0.2 + 2.8 * rand(v)).values])
    x = normal(naux, n, n) * convergent_sigma(o, v)
    B = torch.triu(x) + torch.triu(x, 1).transpose(1, 2)
    d1 = eps[:o, None] - eps[None, o:]
    t1 = 0.003 * normal(o, v) / d1
    d2 = d1[:, None, :, None] + d1[None, :, None, :]
    Bov = B[:, :o, o:]
    t2 = torch.einsum("Qia,Qjb->ijab", Bov, Bov) / d2
    return eps, B, t1, t2


def _eri(B):
    return torch.einsum("Qpr,Qqs->pqrs", B, B)


def _transform_inputs(case, seed):
    """AO integrals with their 8-fold symmetry and decaying blocks, and orthonormal coefficients."""
    n, m = case["nao"], case["nmo"]
    g = _gen(seed)
    x = torch.randn(n, n, n, generator=g, device=_DEV, dtype=torch.float64)
    at = torch.arange(n, device=_DEV, dtype=torch.float64)
    x = (x + x.transpose(1, 2)) * torch.exp(-8.0 * (at[:, None] - at[None, :]).abs() / n)
    tei = torch.einsum("Qpq,Qrs->pqrs", x, x) / n
    C = torch.linalg.qr(torch.randn(n, n, generator=g, device=_DEV, dtype=torch.float64))[0][:, :m]
    return tei, C


def _cotangents(case, seed):
    o, v = case["o"], case["v"]
    g = _gen(seed + 104729)
    g1 = torch.randn(o, v, generator=g, device=_DEV, dtype=torch.float64)
    g2 = torch.randn(o, o, v, v, generator=g, device=_DEV, dtype=torch.float64)
    return g1, 0.5 * (g2 + g2.permute(1, 0, 3, 2))


def prepare(case, seed):
    kind = case["kind"]
    ctx = default_context()
    s = {"case": case, "ctx": ctx, "kind": kind, "precision": case["precision"]}
    if kind == "transform":
        tei, C = _transform_inputs(case, seed)
        s.update(tei=_host(tei), C=_host(C))
        return s
    eps, B, t1, t2 = _inputs(case, seed)
    s.update(eps=_host(eps), o=case["o"], t1=_host(t1), t2=_host(t2))
    if kind == "solve" or kind == "triples":
        s["ints"] = {"B": _host(B)} if case["df"] else {"eri": _host(_eri(B))}
    elif kind == "iterate" or kind == "step":
        # the program's resident state: integrals and DIIS subspace stay on the GPU
        s["state"] = ctx.state(eps=s["eps"], nocc=s["o"], B=_host(B), precision=s["precision"])
    else:
        s["B"] = _host(B)
        if kind == "vjp":
            s["g1"], s["g2"] = (_host(x) for x in _cotangents(case, seed))
    return s


def run(s):
    kind, ctx, p = s["kind"], s["ctx"], s["precision"]
    if kind == "solve":
        w = ctx.solve(eps=s["eps"], nocc=s["o"], precision=p, **s["ints"])
        return {"E": w.E_CCSD, "t1": w.t1, "t2": w.t2}
    if kind == "iterate":
        st = s["state"]
        st.set_amplitudes(s["t1"], s["t2"])
        st.iterate(s["case"]["n"])
        t1, t2 = st.amplitudes()
        return {"t1": t1, "t2": t2}
    if kind == "step":
        st = s["state"]
        st.set_amplitudes(s["t1"], s["t2"])
        st.iterate(1)
        et, _ = st.triples(p)
        t1, t2 = st.amplitudes()
        return {"E_T": et, "t1": t1, "t2": t2}
    if kind == "triples":
        return {"E_T": ctx.triples(eps=s["eps"], nocc=s["o"], t1=s["t1"], t2=s["t2"], precision=p, **s["ints"])}
    if kind == "vjp":
        g1, g2, gB = ctx.residual_vjp(None, s["o"], s["t1"], s["t2"], s["g1"], s["g2"], precision=p, B=s["B"],
                                      want_integrals=True)
        return {"g_t1": g1, "g_t2": g2, "g_B": gB}
    if kind == "triples_vjp":
        et, g1, g2, gB = ctx.triples_vjp(eps=s["eps"], nocc=s["o"], t1=s["t1"], t2=s["t2"], B=s["B"],
                                         want_integrals=True, precision=p)
        return {"E_T": et, "g_t1": g1, "g_t2": g2, "g_B": gB}
    return {"eri": ctx.transform_tei(s["tei"], s["C"], chem_to_phys=True, precision=p)}


# ---------------------------------------------------------------------------------------------
# the work no implementation can do without


def _flops_iteration(o, v):
    return (2.0 * o**2 * v**4 + 4.0 * o * v**4 + 16.0 * o**3 * v**3 + 16.0 * o**2 * v**3 + 4.0 * o * v**3
            + 24.0 * o**3 * v**2 + 4.0 * o**4 * v**2 + 4.0 * o**4 * v)


def _flops_triples(o, v):
    return v * (v + 1) * (v + 2) / 6.0 * 12.0 * o**3 * (v + o)


def work(case):
    kind = case["kind"]
    if kind == "transform":
        n, m = case["nao"], case["nmo"]
        flops = 2.0 * (n**4 * m + n**3 * m**2 + n**2 * m**3 + n * m**4)
        return {"bytes": 8.0 * (n**4 + n * m + m**4), "flops": flops}
    o, v = case["o"], case["v"]
    n = o + v
    amp = 8.0 * (o * v + o * o * v * v)
    ints = 8.0 * (3 * n**3 if case.get("df", True) else n**4)
    # the integral blocks one iteration reads
    blocks = 8.0 * (v**4 + o * v**3 + 3 * o**2 * v**2 + o**3 * v + o**4)
    it, tr = _flops_iteration(o, v), _flops_triples(o, v)
    # integrals from B: (vv|vv), (ov|vv), the (oo|vv)-sized ones, (oo|ov)
    form = 6.0 * n * (v**4 + o * v**3 + 3 * o**2 * v**2 + o**3 * v) if case.get("df", True) else 0.0
    form_t = 6.0 * n * (o * v**3 + o**2 * v**2 + o**3 * v) if case.get("df", True) else 0.0
    if kind == "solve":
        steps = 12  # iterations to convergence, about
        return {"bytes": ints + amp + steps * blocks, "flops": form + steps * it}
    if kind == "iterate":
        return {"bytes": 2 * amp + case["n"] * blocks, "flops": case["n"] * it}
    if kind == "step":
        return {"bytes": 2 * amp + blocks, "flops": it + tr + form_t}
    if kind == "triples":
        return {"bytes": ints + amp, "flops": form_t + tr}
    if kind == "vjp":
        return {"bytes": 2 * ints + 3 * amp, "flops": 3 * (it + form)}
    return {"bytes": 2 * ints + 2 * amp, "flops": 3 * (tr + form_t)}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits, in plain torch


def _blocks(B, o):
    e = torch.einsum
    oo, ov, vv = B[:, :o, :o], B[:, :o, o:], B[:, o:, o:]
    return {"ovov": e("Qkc,Qld->kcld", ov, ov), "oovv": e("Qki,Qac->kiac", oo, vv),
            "ovvo": e("Qkc,Qai->kcai", ov, B[:, o:, :o]),
            "ovvv": e("Qkd,Qac->kdac", ov, vv), "ovoo": e("Qlc,Qki->lcki", ov, oo), "oooo": e("Qki,Qlj->klij", oo, oo),
            "vvvv": e("Qac,Qbd->abcd", vv, vv)}


def _residual(b, t1, t2, literal=True):
    """The closed-shell CCSD residual numerators (spin-adapted, canonical orbitals).  The dressing of
    the particle ladder by t1 is two terms, or (not literal) one of them and its transpose: equal for
    t2(ijab) = t2(jiba), with gradients that differ by a transposition."""
    e = torch.einsum
    ovov, oovv, ovvo, ovvv, ovoo = b["ovov"], b["oovv"], b["ovvo"], b["ovvv"], b["ovoo"]
    both = lambda x: x + x.permute(1, 0, 3, 2)  # noqa: E731
    tau = t2 + e("ia,jb->ijab", t1, t1)
    L = 2 * ovov - ovov.permute(0, 3, 2, 1)
    Foo, Fvv, Fov = e("kcld,ilcd->ki", L, tau), -e("kcld,klad->ac", L, tau), e("kcld,ld->kc", L, t1)
    Lo = 2 * ovoo - ovoo.permute(2, 1, 0, 3)
    Lv = 2 * ovvv - ovvv.permute(0, 3, 2, 1)
    r1 = e("ac,ic->ia", Fvv, t1) - e("ki,ka->ia", Foo, t1) + e("kc,kica->ia", Fov, 2 * t2 - t2.transpose(0, 1))
    r1 = r1 + e("ki,ka->ia", e("kc,ic->ki", Fov, t1), t1)
    r1 = r1 + 2 * e("kcai,kc->ia", ovvo, t1) - e("kiac,kc->ia", oovv, t1)
    r1 = r1 + e("kdac,ikcd->ia", Lv, tau) - e("lcki,klac->ia", Lo, tau)
    X = e("iacb,jc->ijab", ovvv, t1) - e("kibj,ka->ijab", e("kibc,jc->kibj", oovv, t1), t1)
    X = X - e("akij,kb->ijab", e("kcai,jc->akij", ovvo, t1) + ovoo.permute(1, 3, 0, 2), t1)
    Loo, Lvv = Foo + e("lcki,lc->ki", Lo, t1), Fvv + e("kdac,kd->ac", Lv, t1)
    Woooo = b["oooo"] + e("lcki,jc->klij", ovoo, t1) + e("kclj,ic->klij", ovoo, t1) + e("kcld,ijcd->klij", ovov, tau)
    Wvoov = ovvo.permute(2, 0, 3, 1) + e("kcad,id->akic", ovvv, t1) - e("kcli,la->akic", ovoo, t1)
    Wvoov = Wvoov - 0.5 * e("ldkc,ilda->akic", ovov, t2) - 0.5 * e("lckd,ilad->akic", ovov, t2) + e("ldkc,ilad->akic", ovov, t2)
    Wvoov = Wvoov - e("lkci,la->akic", e("ldkc,id->lkci", ovov, t1), t1)
    Wvovo = oovv.permute(2, 0, 3, 1) + e("kdac,id->akci", ovvv, t1) - e("lcki,la->akci", ovoo, t1)
    Wvovo = Wvovo - 0.5 * e("lckd,ilda->akci", ovov, t2) - e("lcki,la->akci", e("lckd,id->lcki", ovov, t1), t1)
    r2 = ovov.permute(0, 2, 1, 3) + e("klij,klab->ijab", Woooo, tau) + e("abcd,ijcd->ijab", b["vvvv"], tau)
    dressed = e("ka,kbij->ijab", t1, e("kcbd,ijcd->kbij", ovvv, tau))
    if literal:
        r2 = r2 - dressed - e("kb,kaij->ijab", t1, e("kdac,ijcd->kaij", ovvv, tau))
    else:
        X = X - dressed
    X = X + e("ac,ijcb->ijab", Lvv, t2) - e("ki,kjab->ijab", Loo, t2)
    X = X + 2 * e("akic,kjcb->ijab", Wvoov, t2) - e("akci,kjcb->ijab", Wvovo, t2)
    X = X - e("akic,kjbc->ijab", Wvoov, t2) - e("bkci,kjac->ijab", Wvovo, t2)
    return r1, r2 + both(X)


def _energy(b, t1, t2):
    g = b["ovov"].permute(0, 2, 1, 3)
    return float(((2 * g - g.transpose(2, 3)) * (t2 + torch.einsum("ia,jb->ijab", t1, t1))).sum())


def _denominators(eps, o):
    d1 = eps[:o, None] - eps[None, o:]
    return d1, d1[:, None, :, None] + d1[None, :, None, :]


def _iterate(b, eps, o, t1, t2, n, until=None):
    """n Jacobi iterations with DIIS (8 vectors, from the third); or until (dE, rms) are met."""
    d1, d2 = _denominators(eps, o)
    amps, errs, last = [], [], math.inf
    for it in range(n):
        r1, r2 = _residual(b, t1, t2)
        n1, n2 = r1 / d1, r2 / d2
        amp = torch.cat([n1.reshape(-1), n2.reshape(-1)])
        err = amp - torch.cat([t1.reshape(-1), t2.reshape(-1)])
        amps, errs = (amps + [amp])[-8:], (errs + [err])[-8:]
        if it >= 2:
            k = len(errs)
            G = torch.tensor([[float(x @ y) for y in errs] for x in errs], dtype=torch.float64)
            M = -torch.ones(k + 1, k + 1, dtype=torch.float64)
            M[:k, :k], M[k, k] = G / G.abs().max(), 0.0
            c = torch.linalg.solve(M, torch.tensor([0.0] * k + [-1.0], dtype=torch.float64))[:k]
            amp = sum(float(ci) * a for ci, a in zip(c, amps))
        t1, t2 = amp[: t1.numel()].view_as(t1), amp[t1.numel():].view_as(t2)
        if until is not None:
            E = _energy(b, t1, t2)
            if abs(E - last) < until[0] and float(err.norm()) / math.sqrt(err.numel()) < until[1]:
                break
            last = E
    return t1, t2


def _triples(B, eps, o, t1, t2):
    """E_(T) from W and V over all a >= b >= c, one leading virtual a at a time."""
    e = torch.einsum
    v = eps.numel() - o
    ov, oo, vv = B[:, :o, o:], B[:, :o, :o], B[:, o:, o:]
    ovvv, ovoo, ovov = e("Qia,Qbf->iabf", ov, vv), e("Qia,Qmj->iamj", ov, oo), e("Qia,Qjb->iajb", ov, ov)
    ev, eo = eps[o:], eps[:o]
    e3 = eo[:, None, None] + eo[None, :, None] + eo[None, None, :]
    total = 0.0
    for a in range(v):
        m = a + 1  # b, c <= a

        # w^{xyz}_{ijk} = sum_f (ix|yf) t2(k,j,z,f) - sum_m (ix|mj) t2(m,k,y,z), symmetrised over the
        # six simultaneous permutations of (ia), (jb), (kc); W[b, c, i, j, k]
        W = e("iyf,kjzf->yzijk", ovvv[:, a, :m, :], t2[:, :, :m, :]) - e("imj,mkyz->yzijk", ovoo[:, a], t2[:, :, :m, :m])
        W = W + e("izf,jkyf->yzijk", ovvv[:, a, :m, :], t2[:, :, :m, :]) - e("imk,mjzy->yzijk", ovoo[:, a], t2[:, :, :m, :m])
        W = W + e("jyf,kizf->yzijk", ovvv[:, :m, a, :], t2[:, :, :m, :]) - e("jymi,mkz->yzijk", ovoo[:, :m], t2[:, :, a, :m])
        W = W + e("jyzf,ikf->yzijk", ovvv[:, :m, :m, :], t2[:, :, a, :]) - e("jymk,miz->yzijk", ovoo[:, :m], t2[:, :, :m, a])
        W = W + e("kzf,jiyf->yzijk", ovvv[:, :m, a, :], t2[:, :, :m, :]) - e("kzmi,mjy->yzijk", ovoo[:, :m], t2[:, :, a, :m])
        W = W + e("kzyf,ijf->yzijk", ovvv[:, :m, :m, :], t2[:, :, a, :]) - e("kzmj,miy->yzijk", ovoo[:, :m], t2[:, :, :m, a])
        V = e("i,jykz->yzijk", t1[:, a], ovov[:, :m, :, :m]) + e("jy,ikz->yzijk", t1[:, :m], ovov[:, a, :, :m])
        V = V + e("kz,ijy->yzijk", t1[:, :m], ovov[:, a, :, :m])
        Y = W + V
        r3 = 4 * Y + Y.permute(0, 1, 4, 2, 3) + Y.permute(0, 1, 3, 4, 2)
        r3 = r3 - 2 * (Y.permute(0, 1, 4, 3, 2) + Y.permute(0, 1, 2, 4, 3) + Y.permute(0, 1, 3, 2, 4))
        d = e3[None, None] - (ev[a] + ev[:m, None] + ev[None, :m])[:, :, None, None, None]
        per = (W * r3 / d).sum(dim=(2, 3, 4))
        w = torch.ones(m, m, device=B.device, dtype=torch.float64)
        idx = torch.arange(m, device=B.device)
        w = torch.where(idx[None, :] > idx[:, None], torch.zeros_like(w), w)  # c <= b
        same = (idx[:, None] == a).to(torch.int64) + (idx[None, :] == idx[:, None]).to(torch.int64)
        w = torch.where(same == 2, w / 6, torch.where(same == 1, w / 2, w))
        total = total + 2 * (w * per).sum()
    return total


def exact(case, seed):
    kind = case["kind"]
    if kind == "transform":
        x, C = _transform_inputs(case, seed)
        for _ in range(4):  # each index in turn
            x = torch.tensordot(x, C, dims=([0], [0]))
        return {"eri": x.permute(0, 2, 1, 3)}
    o, v = case["o"], case["v"]
    eps, B, t1, t2 = _inputs(case, seed)
    if kind == "solve":
        _, d2 = _denominators(eps, o)
        b = _blocks(B, o)
        g = b["ovov"].permute(0, 2, 1, 3) / d2
        t1, t2 = _iterate(b, eps, o, torch.zeros_like(t1), g, 60, until=(1e-10, 1e-8))
        return {"E": _energy(b, t1, t2), "t1": t1, "t2": t2}
    if kind == "iterate":
        t1, t2 = _iterate(_blocks(B, o), eps, o, t1, t2, case["n"])
        return {"t1": t1, "t2": t2}
    if kind == "step":
        t1, t2 = _iterate(_blocks(B, o), eps, o, t1, t2, 1)
        et = float(_triples(B, eps, o, t1, t2)) if _flops_triples(o, v) < 1e12 else None
        return {"E_T": et, "t1": t1, "t2": t2}
    if kind == "triples":
        return {"E_T": float(_triples(B, eps, o, t1, t2))}
    for x in (t1, t2, B):
        x.requires_grad_(True)
    if kind == "vjp":
        g1, g2 = _cotangents(case, seed)
        r1, r2 = _residual(_blocks(B, o), t1, t2, literal=case["precision"] == "fp64")
        gt1, gt2, gB = torch.autograd.grad((g1 * r1).sum() + (g2 * r2).sum(), (t1, t2, B))
        return {"g_t1": gt1, "g_t2": gt2, "g_B": gB}
    et = _triples(B, eps, o, t1, t2)
    gt1, gt2, gB = torch.autograd.grad(et, (t1, t2, B))
    return {"E_T": float(et), "g_t1": gt1, "g_t2": gt2, "g_B": gB}
