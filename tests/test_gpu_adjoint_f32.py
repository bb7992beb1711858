"""The reverse sweep on fp32 fields against a restatement of it in FP64 whose every stored field is rounded to f32,
run on the states that the steps went through.

Both form a value in FP64 from the same f32 fields and round it once, so they differ where the order of an FP64
sum turns a rounding: one value by 2^-24 of itself.  Bar: dE/dK within 1e-7 of its largest value (a rounding turned
in the largest term), which a field stored one operation too early or too late, or a wrong neighbour, does not meet."""
import math

import numpy as np
import pytest

import nm_adjoint as adj
import oracle as orc

pytestmark = pytest.mark.gpu


def R(x):
    return np.asarray(x).astype(np.float32).astype(np.float64)


def color(mu, muf, h2, c, par):
    out = mu.copy()
    s = sum(adj._nb(mu, d) for d in adj._SH)
    on = par == c
    adj._in(muf)[on] = R(adj._in(muf)[on] + h2 / 6.0 * adj._in(mu)[on])
    adj._in(out)[on] = 0.0
    adj._in(out)[~on] = R(adj._in(mu)[~on] + s[~on] / 6.0)
    return out, muf


def vcycle(mu, S, h, levels, pre, post, sweeps):
    h2, par = h * h, adj._colors(S)
    if levels == 1:  # in FP64 from first to last
        _, muf = adj.adj_vcycle(mu, S, h, 1, pre, post, sweeps)
        return mu, R(muf)
    muf = np.zeros_like(mu)
    for _ in range(post):
        for c in (1, 0):
            mu, muf = color(mu, muf, h2, c, par)
    SC = (S - 1) // 2 + 1
    _, mufc = vcycle(R(8.0 * adj._full_weighting(mu, SC)), SC, 2 * h, levels - 1, pre, post, sweeps)
    mur = R(adj._trilinear(mufc, S) / 8.0)
    muf = R(muf + mur)
    mu = mu.copy()
    adj._in(mu)[...] = R(adj._in(mu) + (sum(adj._nb(mur, d) for d in adj._SH) - 6.0 * adj._in(mur)) / h2)
    for _ in range(pre):
        for c in (1, 0):
            mu, muf = color(mu, muf, h2, c, par)
    return mu, muf


def update(u, K, P, L, half_dv, dt):
    """The f32 update, operation by operation."""
    f = np.float32
    u, K, P = f(u), f(K), f(P)
    c, lc = adj._in(u), adj._in(L)
    s = None
    for d in adj._SH:
        x = np.where(adj._nb(L, d) == lc, adj._nb(u, d), c)
        s = x if s is None else s + x
    lap = s - f(6) * c
    out = np.zeros_like(u)
    adj._in(out)[...] = (c + f(half_dv) * lap) + (f(dt) * (adj._in(K) - f(2) * adj._in(P))) * c
    return out.astype(np.float64)


# Both row alignments (S = 1 and 3 mod 4), V-cycles closer and further apart than the steps whose sums run
# together, sweeps other than one a side, and tails of two, three and four levels (16-8, 16-8-4, 16-8-4-2).
@pytest.mark.parametrize("NN,opts,steps", [(16, {}, 9), (22, {}, 9), (18, dict(poisson_interval=7), 15), (20, dict(mg_pre=2), 6),
                                           (32, {}, 9), (48, {}, 6), (32, dict(mg_levels=4), 6), (32, dict(mg_levels=5), 6),
                                           (24, dict(mg_levels=4), 6)])
def test_reverse_sweep_of_f32_fields(NN, opts, steps):
    from realmolecule_b200 import Context
    h = 7.2 / NN
    N2, d = NN / 2, 1.4 / 2 / h
    rows = [{"i": N2 - d, "j": N2, "k": N2 + 0.2, "Z": 0.0, "Z_nuc": 1.0},
            {"i": N2 + d, "j": N2 + 0.3, "k": N2, "Z": 0.0, "Z_nuc": 1.0},
            {"i": N2 - d + 0.05, "j": N2, "k": N2, "Z": 1.0, "Z_nuc": 0.0},
            {"i": N2 + d - 0.05, "j": N2, "k": N2, "Z": 1.0, "Z_nuc": 0.0}]
    kw = dict(label_until=1, norm_interval=1, poisson_interval=4)
    kw.update(opts)
    ctx = Context(NN, NN * h, rows, flavor="new", precision="mixed", **kw)
    ctx.initialize()
    S, shp, n = NN + 1, (NN + 1,) * 3, len(rows)
    levels = ctx.info().mg_levels
    pre, post = kw.get("mg_pre", 1), kw.get("mg_post", 1)
    K = ctx.download_K().reshape(shp)
    K64 = orc.NewMethodDriver(NN, NN * h, rows).K.reshape(shp)
    Z = np.array([r["Z"] for r in rows])
    half_dv, dt, h3 = 0.1, 0.2 * h * h, h ** 3
    get = lambda: {k: v.reshape(shp) for k, v in ctx.download(psi=True, P=True).items()}
    ctx.set_adjoint_window(steps)
    recs, st = [], get()
    L = st["label"]
    for s in range(1, steps + 1):
        ctx.step(1)
        new = get()
        psi = st["psi"].astype(np.float64)
        raw = update(psi, K, new["P"], L, half_dv, dt)
        N = np.bincount(L.ravel(), weights=(raw ** 2).ravel() * h3, minlength=n)
        c = np.where((Z > 0) & (N > 0), np.sqrt(Z / np.where(N > 0, N, 1.0)), 1.0)
        assert np.abs(R(c[L] * raw) - new["psi"]).max() <= 2.0 ** -23 * np.abs(new["psi"]).max()  # the step restated
        recs.append({"psi": psi, "P": new["P"].astype(np.float64), "vc": s % kw["poisson_interval"] == 0, "c": c})
        st = new
    _, g = ctx.adjoint(forces=False, potential=True)
    ctx.close()

    psi, P = st["psi"].astype(np.float64), st["P"].astype(np.float64)
    u, pc = adj._in(psi), adj._in(P)
    AP = (6.0 * pc - sum(adj._nb(P, d) for d in adj._SH)) / (h * h)
    lab = adj._in(L).ravel()
    per = lambda x: np.bincount(lab, weights=np.ravel(x), minlength=n)
    # the readout's sums: every same-label edge once (edges to a face point of the domain included)
    T = np.zeros(n)
    for a in range(3):
        lo, hi = np.take(L, range(S - 1), a), np.take(L, range(1, S), a)
        e = np.where(lo == hi, np.diff(psi, axis=a) ** 2, 0.0)
        sl = tuple(slice(1, -1) if b != a else slice(None) for b in range(3))
        T += np.bincount(lo[sl].ravel(), weights=0.5 * h * e[sl].ravel(), minlength=n)
    N, VK, Pr = per(u * u * h3), per(-adj._in(K64) * u * u * h3), per(pc * u * u * h3)
    w = np.where((Z > 0) & (N > 0), Z / np.where(N > 0, N, 1.0), 1.0)
    qn = np.where(N > 0, (T + VK + 2.0 * Pr) / np.where(N > 0, N, 1.0), 0.0)
    wl, ql = w[adj._in(L)], qn[adj._in(L)]
    lam, muP, gK = np.zeros(shp), np.zeros(shp), np.zeros(shp)
    adj._in(lam)[...] = R(wl * (-h * adj._same_label_lap(psi, L) + 2.0 * h3 * u * (2.0 * pc - adj._in(K64) - ql)))
    adj._in(muP)[...] = R(2.0 * wl * h3 * u * u - h3 / math.pi * AP)
    adj._in(gK)[...] = -wl * h3 * u * u
    K = K.astype(np.float64)
    for r in range(steps - 1, -1, -1):
        rec = recs[r]
        lam = R(adj._adj_norm(recs[r + 1]["psi"] if r + 1 < steps else psi, lam, rec["c"], L, Z, h3))
        lt, pp = adj._in(lam), adj._in(rec["psi"])
        out = np.zeros(shp)
        adj._in(out)[...] = R(lt + half_dv * adj._same_label_lap(lam, L) + dt * (adj._in(K) - 2.0 * adj._in(rec["P"])) * lt)
        adj._in(gK)[...] += dt * pp * lt
        adj._in(muP)[...] = R(adj._in(muP) - 2.0 * dt * pp * lt)
        lam = out
        if rec["vc"]:
            muP, muf = vcycle(muP, S, h, levels, pre, post, 16)
            adj._in(lam)[...] = R(adj._in(lam) + 4.0 * math.pi * pp * adj._in(muf))
    assert np.abs(g - gK.ravel()).max() <= 1e-7 * np.abs(gK).max()
