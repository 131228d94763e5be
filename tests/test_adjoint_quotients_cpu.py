"""The reverse-mode operators of the 2-D adjoint (tenjin_gb300/csrc/tj_adjoint_local.h)
against the same derivatives written out in Python floats with one division per
quotient, on seeded states: the same bits. The limiter's branch and its extrapolation
likewise, over zeros, subnormal and huge numbers, infinities and NaN. A quotient formed as a product with a
reciprocal rounds twice, so an operator that does so is further from the exact
derivative than this and differs here. No tolerance: both sides are IEEE binary64
in one order of operations (compiled without contraction)."""
import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "tenjin_gb300", "csrc")
MM = 4
D = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("tja") / "libtja.so")
    subprocess.run(["g++", "-O1", "-std=c++14", "-ffp-contract=off", "-shared", "-fPIC", "-I" + CSRC,
                    os.path.join(HERE, "adjoint_local_harness.cpp"), "-o", out], check=True)
    L = ctypes.CDLL(out)
    d, i = ctypes.c_double, ctypes.c_int
    L.h_thinc.argtypes = [D, i, d, d, d, D]
    L.h_thinc_rev.argtypes = [D, i, d, d, d, d, d, D]
    L.h_muscl.argtypes = [d, d, d, D]
    L.h_muscl_rev.argtypes = [d, d, d, d, d, D]
    return L


def p(a):
    return a.ctypes.data_as(D)


def _eos(M):
    e = np.zeros(3 * MM)
    e[:M] = [3.4, 0.4, 1.1, 2.0][:M]
    e[MM:MM + M] = [-4.4 * 6e8, 0.0, -1.4e7, 0.0][:M]
    e[2 * MM:2 * MM + M] = [1.2e5, 3e4, 0.0, 5e4][:M]
    return e


def _prim(M, rng):
    x = np.zeros(2 * MM + 3)
    a = rng.uniform(0.2, 0.8, M)
    x[:M] = a / a.sum()
    x[MM:MM + M] = [1000.0, 1.2, 800.0, 50.0][:M] * rng.uniform(0.8, 1.2, M)
    x[2 * MM:2 * MM + 2] = rng.uniform(-60, 60, 2)
    x[2 * MM + 2] = rng.uniform(1e5, 3e8)
    return x


def _adjoint(n, M, blocks, rng):
    v = rng.standard_normal(n)
    for b in range(blocks):
        v[b * MM + M:(b + 1) * MM] = 0.0
    return v


def _face_state_rev(M, e, x, l):
    G, pr, er = e[:MM], e[MM:2 * MM], e[2 * MM:]
    a, rk, u, pp = x[:MM], x[MM:2 * MM], x[2 * MM:2 * MM + 2], x[2 * MM + 2]
    ar, rho = [0.0] * M, 0.0
    for m in range(M):
        ar[m] = a[m] * rk[m]
        rho += ar[m]
    invG = A = xit = 0.0
    xi, c2, v = [0.0] * M, [0.0] * M, [0.0] * M
    for m in range(M):
        invG += a[m] / G[m]
        xi[m] = 1.0 / G[m]
        c2[m] = pp * (G[m] + 1.0) / rk[m] - pr[m] / rk[m]
        v[m] = xi[m] * c2[m] * ar[m] / rho
        A += v[m] if 0.0 < v[m] else 0.0
        xit += xi[m] * a[m]
    c = math.sqrt((1e-6 if A <= 0.0 else A) / xit)
    la, lar, lrk = list(l[:M]), list(l[MM:MM + M]), [0.0] * M
    lrho, lru, lu, lE, lp, lc = l[2 * MM], l[2 * MM + 1:2 * MM + 3], list(l[2 * MM + 3:2 * MM + 5]), *l[2 * MM + 5:2 * MM + 8]
    gG, gp, ge = [0.0] * M, [0.0] * M, [0.0] * M
    lA = 0.0 if A <= 0.0 else lc / (2.0 * c * xit)
    lxit = -lc * c / (2.0 * xit)
    for m in range(M):
        lxi = lxit * a[m]
        la[m] += lxit * xi[m]
        if 0.0 < v[m]:
            lc2 = lA * xi[m] * ar[m] / rho
            lar[m] += lA * xi[m] * c2[m] / rho
            lrho += -lA * v[m] / rho
            lxi += lA * c2[m] * ar[m] / rho
            lp += lc2 * (G[m] + 1.0) / rk[m]
            lrk[m] += -lc2 * c2[m] / rk[m]
            gG[m] += lc2 * pp / rk[m]
            gp[m] += -lc2 / rk[m]
        gG[m] += -lxi * xi[m] * xi[m]
    lp += lE * invG
    for m in range(M):
        la[m] += lE * (pp - pr[m]) / G[m]
        gG[m] += -lE * (pp - pr[m]) * a[m] / (G[m] * G[m])
        gp[m] += -lE * a[m] / G[m]
        ge[m] += lE * ar[m]
        lar[m] += lE * er[m]
    for r in range(2):
        lrho += lE * 0.5 * u[r] * u[r] + lru[r] * u[r]
        lu[r] += lE * rho * u[r] + lru[r] * rho
    for m in range(M):
        lar[m] += lrho
        la[m] += lar[m] * rk[m]
        lrk[m] += lar[m] * a[m]
    return la, lrk, lu, lp, gG, gp, ge


@pytest.mark.parametrize("M", [1, 2, 4])
def test_face_state_rev(lib, M):
    rng = np.random.default_rng(40 + M)
    e = _eos(M)
    for _ in range(50):
        x, l = _prim(M, rng), _adjoint(2 * MM + 8, M, 2, rng)
        lx, g = np.zeros(2 * MM + 3), np.zeros(3 * MM)
        lib.h_face_state_rev(M, p(e), p(x), 0, p(l), p(lx), p(g))
        la, lrk, lu, lp, gG, gp, ge = _face_state_rev(M, e.tolist(), x.tolist(), l.tolist())
        assert lx[:M].tolist() == la and lx[MM:MM + M].tolist() == lrk
        assert lx[2 * MM:].tolist() == lu + [lp]
        assert g[:M].tolist() == gG and g[MM:MM + M].tolist() == gp and g[2 * MM:2 * MM + M].tolist() == ge


def _hllc_rev(M, L, R, d, lF):
    """L, R, and the adjoints returned: dicts of a[M], ar[M], rho, ru[2], u[2], E, p, c."""
    uL, uR = L["u"][d], R["u"][d]
    x1, x2 = abs(uL) + L["c"], abs(uR) + R["c"]
    SR = x2 if x1 < x2 else x1
    SL = -SR
    Num = R["p"] - L["p"] + L["ru"][d] * (SL - uL) - R["ru"][d] * (SR - uR)
    Den = L["rho"] * (SL - uL) - R["rho"] * (SR - uR)
    Ss = Num / Den
    side = 0 if SL >= 0.0 or Ss >= 0.0 else 1
    hllc = not (SL >= 0.0) if side == 0 else SR >= 0.0
    zero = lambda: dict(a=[0.0] * M, ar=[0.0] * M, rho=0.0, ru=[0.0, 0.0], u=[0.0, 0.0], E=0.0, p=0.0, c=0.0)
    lL, lR = zero(), zero()
    K, lK = (R, lR) if side else (L, lL)
    SK, uK = (SR if side else SL), K["u"][d]
    guard = Ss - uK == 0.0 and Ss != 0.0
    mult = 1.0 if guard else (SK - uK) / (SK - Ss)
    ars, rs = [0.0] * M, 0.0
    for m in range(M):
        ars[m] = mult * K["ar"][m]
        rs += ars[m]
    rus = [0.0, 0.0]
    rus[d] = mult * K["rho"] * Ss
    rus[1 - d] = mult * K["ru"][1 - d]
    vsd = rus[d] / rs
    D1, D2 = Ss - uK, K["rho"] * Ss + K["p"] / (SK - uK)
    W = K["E"] + D1 * D2
    Es = mult * W
    w = SK if hllc else 0.0
    lSs, lSK, luK, lmult, lvsd = lF["Ss"], 0.0, 0.0, 0.0, 0.0
    lars, lrus = [0.0] * M, [0.0, 0.0]
    for m in range(M):
        lK["a"][m] += lF["Fa"][m] * vsd
        lvsd += lF["Fa"][m] * K["a"][m]
    for m in range(M):
        lK["ar"][m] += lF["Far"][m] * (uK - w)
        luK += lF["Far"][m] * K["ar"][m]
        lars[m] = lF["Far"][m] * w
        if hllc:
            lSK += lF["Far"][m] * (ars[m] - K["ar"][m])
    for r in range(2):
        lK["ru"][r] += lF["Fru"][r] * (uK - w)
        luK += lF["Fru"][r] * K["ru"][r]
        if r == d:
            lK["p"] += lF["Fru"][r]
        lrus[r] = lF["Fru"][r] * w
        if hllc:
            lSK += lF["Fru"][r] * (rus[r] - K["ru"][r])
    lK["E"] += lF["FE"] * (uK - w)
    lK["p"] += lF["FE"] * uK
    luK += lF["FE"] * (K["E"] + K["p"])
    lEs = lF["FE"] * w
    if hllc:
        lSK += lF["FE"] * (Es - K["E"])
    lrus[d] += lvsd / rs
    lrs = -lvsd * vsd / rs
    for m in range(M):
        lars[m] += lrs
    for m in range(M):
        lmult += lars[m] * K["ar"][m]
        lK["ar"][m] += lars[m] * mult
    lmult += lrus[d] * K["rho"] * Ss
    lK["rho"] += lrus[d] * mult * Ss
    lSs += lrus[d] * mult * K["rho"]
    lmult += lrus[1 - d] * K["ru"][1 - d]
    lK["ru"][1 - d] += lrus[1 - d] * mult
    lmult += lEs * W
    lW = lEs * mult
    lK["E"] += lW
    lD1, lD2 = lW * D2, lW * D1
    lSs += lD1
    luK -= lD1
    lK["rho"] += lD2 * Ss
    lSs += lD2 * K["rho"]
    lK["p"] += lD2 / (SK - uK)
    lSK += -lD2 * K["p"] / ((SK - uK) * (SK - uK))
    luK += lD2 * K["p"] / ((SK - uK) * (SK - uK))
    if not guard:
        den = SK - Ss
        lSK += lmult * (uK - Ss) / (den * den)
        luK += -lmult / den
        lSs += lmult * mult / den
    lSL, lSR = (0.0, lSK) if side else (lSK, 0.0)
    lK["u"][d] += luK
    lNum, lDen = lSs / Den, -lSs * Ss / Den
    lR["p"] += lNum
    lL["p"] -= lNum
    lL["ru"][d] += lNum * (SL - uL)
    lSL += lNum * L["ru"][d]
    lL["u"][d] -= lNum * L["ru"][d]
    lR["ru"][d] -= lNum * (SR - uR)
    lSR -= lNum * R["ru"][d]
    lR["u"][d] += lNum * R["ru"][d]
    lL["rho"] += lDen * (SL - uL)
    lSL += lDen * L["rho"]
    lL["u"][d] -= lDen * L["rho"]
    lR["rho"] -= lDen * (SR - uR)
    lSR -= lDen * R["rho"]
    lR["u"][d] += lDen * R["rho"]
    lSR -= lSL
    if x1 < x2:
        lR["u"][d] += lSR * ((uR > 0.0) - (uR < 0.0))
        lR["c"] += lSR
    else:
        lL["u"][d] += lSR * ((uL > 0.0) - (uL < 0.0))
        lL["c"] += lSR
    return side, lL, lR


def _fs(M, z):
    z = z.tolist()
    return dict(a=z[:M], ar=z[MM:MM + M], rho=z[2 * MM], ru=z[2 * MM + 1:2 * MM + 3], u=z[2 * MM + 3:2 * MM + 5],
                E=z[2 * MM + 5], p=z[2 * MM + 6], c=z[2 * MM + 7])


@pytest.mark.parametrize("M", [1, 2, 4])
@pytest.mark.parametrize("d", [0, 1])
def test_hllc_rev(lib, M, d):
    rng = np.random.default_rng(60 + 10 * M + d)
    e, sides = _eos(M), set()
    for _ in range(50):
        S = []
        for _ in range(2):
            o = np.zeros(2 * MM + 8)
            lib.h_face_state(M, p(e), p(_prim(M, rng)), 0, p(o))
            S.append(o)
        lf = _adjoint(2 * MM + 4, M, 2, rng)
        lL, lR = np.zeros(2 * MM + 8), np.zeros(2 * MM + 8)
        lib.h_hllc_rev(M, p(S[0]), p(S[1]), d, p(lf), p(lL), p(lR))
        f = lf.tolist()
        side, wL, wR = _hllc_rev(M, _fs(M, S[0]), _fs(M, S[1]), d,
                                 dict(Fa=f[:M], Far=f[MM:MM + M], Fru=f[2 * MM:2 * MM + 2], FE=f[2 * MM + 2], Ss=f[2 * MM + 3]))
        sides.add(side)
        assert _fs(M, lL) == wL and _fs(M, lR) == wR
    assert sides == {0, 1}


@pytest.mark.parametrize("M", [1, 2, 4])
def test_c2p_rev(lib, M):
    rng = np.random.default_rng(80 + M)
    e = _eos(M)
    G, pr, er = (e[k * MM:(k + 1) * MM].tolist() for k in range(3))
    for _ in range(50):
        carried = np.zeros(3 * MM + 7)
        lib.h_p2c(M, p(e), p(_prim(M, rng)), p(carried))
        c = np.concatenate([carried[:2 * MM], carried[3 * MM + 1:3 * MM + 3], carried[3 * MM + 5:3 * MM + 6]])
        l = _adjoint(3 * MM + 7, M, 3, rng)
        mu, g = np.zeros(2 * MM + 3), np.zeros(3 * MM)
        lib.h_c2p_rev(M, p(e), p(c), p(l), p(mu), p(g))
        a, ar, ru, E = c[:M].tolist(), c[MM:MM + M].tolist(), c[2 * MM:2 * MM + 2].tolist(), float(c[2 * MM + 2])
        la, lar, lrk, rest = l[:M].tolist(), l[MM:MM + M].tolist(), l[2 * MM:2 * MM + M].tolist(), l[3 * MM:].tolist()
        lrho, lru, lu, lE, lp = rest[0], rest[1:3], rest[3:5], rest[5], rest[6]
        rho, rk, u, ke = 0.0, [ar[m] / a[m] for m in range(M)], [0.0, 0.0], 0.0
        for m in range(M):
            rho += ar[m]
        for r in range(2):
            u[r] = ru[r] / rho
            ke += 0.5 * rho * u[r] * u[r]
        invG = ent = pnt = 0.0
        for m in range(M):
            invG += a[m] / G[m]
            ent += er[m] * ar[m]
            pnt += pr[m] * a[m] / G[m]
        pp = (E - ke - ent + pnt) / invG
        lN, lD = lp / invG, -lp * pp / invG
        wa, war = [0.0] * M, [0.0] * M
        for m in range(M):
            wa[m] = la[m] - lrk[m] * rk[m] / a[m] + lN * pr[m] / G[m] + lD / G[m]
            war[m] = lar[m] + lrk[m] / a[m] - lN * er[m]
        wru = [0.0, 0.0]
        for r in range(2):
            t = lu[r] - lN * rho * u[r]
            lrho += -lN * 0.5 * u[r] * u[r]
            wru[r] = lru[r] + t / rho
            lrho += -t * u[r] / rho
        assert mu[:M].tolist() == wa and mu[MM:MM + M].tolist() == [war[m] + lrho for m in range(M)]
        assert mu[2 * MM:].tolist() == wru + [lE + lN]
        assert g[:M].tolist() == [0.0 - (lN * pr[m] + lD) * a[m] / (G[m] * G[m]) for m in range(M)]
        assert g[MM:MM + M].tolist() == [lN * a[m] / G[m] for m in range(M)]


def _thinc_rev(s, d, beta0, dx, dy, lL, lR):
    eps = 1e-20
    aL, aR, a0 = (s[0][1], s[2][1], s[1][1]) if d == 0 else (s[1][0], s[1][2], s[1][1])
    mn = aR if aR < aL else aL
    mx = (aR if aL < aR else aL) - mn
    theta = float((0.0 < aR - aL) - (aR - aL < 0.0))
    C = (a0 - mn + eps) / (mx + eps)
    nx = -1.0 / (8.0 * dx) * (s[2][2] + 2.0 * s[2][1] + s[2][0] - s[0][2] - 2.0 * s[0][1] - s[0][0])
    ny = -1.0 / (8.0 * dy) * (s[2][2] + 2.0 * s[1][2] + s[0][2] - s[0][0] - 2.0 * s[1][0] - s[2][0])
    norm = math.sqrt(nx * nx + ny * ny)
    nd = nx if d == 0 else ny
    beta = abs(nd / norm) * beta0 + 0.01
    ch, th = math.cosh(beta), math.tanh(beta)
    B = math.exp(theta * beta * ((2.0 * C) - 1.0))
    A = ((B / ch) - 1.0) / th
    q = 1.0 + A * th
    T = (th + A) / q
    lmn = lL + lR
    lmx = lL * 0.5 * (1.0 + theta * A) + lR * 0.5 * (1.0 + theta * T)
    lA = lL * (mx / 2.0) * theta
    lT = lR * (mx / 2.0) * theta
    lt = lT * (1.0 - A * A) / (q * q)
    lA += lT * (1.0 - th * th) / (q * q)
    lB = lA / (ch * th)
    lch = -lA * B / (ch * ch * th)
    lt += -lA * A / th
    lbeta = lB * B * theta * (2.0 * C - 1.0)
    lC = lB * B * theta * beta * 2.0
    lbeta += lch * th * ch
    lbeta += lt * (1.0 - th * th)
    lnvc = lbeta * beta0
    la0 = lC / (mx + eps)
    lmn -= lC / (mx + eps)
    lmx -= lC * C / (mx + eps)
    lmn -= lmx
    ls = [[0.0] * 3 for _ in range(3)]
    laL, laR = (lmx, lmn) if aR < aL else (lmn, lmx)
    for (i, j), v in ((((0, 1), laL), ((2, 1), laR)) if d == 0 else (((1, 0), laL), ((1, 2), laR))):
        ls[i][j] += v
    ls[1][1] += la0
    sg = float((nd > 0.0) - (nd < 0.0))
    n3 = norm * norm * norm
    lnx = lnvc * sg * ((1.0 if d == 0 else 0.0) / norm - nd * nx / n3)
    lny = lnvc * sg * ((1.0 if d == 1 else 0.0) / norm - nd * ny / n3)
    cx, cy = -1.0 / (8.0 * dx) * lnx, -1.0 / (8.0 * dy) * lny
    for i, j, v in ((2, 2, cx + cy), (2, 1, 2.0 * cx), (2, 0, cx - cy), (0, 2, -cx + cy), (0, 1, -2.0 * cx),
                    (0, 0, -cx - cy), (1, 2, 2.0 * cy), (1, 0, -2.0 * cy)):
        ls[i][j] += v
    return [v for row in ls for v in row]


@pytest.mark.parametrize("d", [0, 1])
def test_thinc_candidate_rev(lib, d):
    rng = np.random.default_rng(90 + d)
    done = 0
    while done < 50:
        ang, off = rng.uniform(0, 2 * np.pi), rng.uniform(-0.6, 0.6)
        ii, jj = np.meshgrid([-1, 0, 1], [-1, 0, 1], indexing="ij")
        s = 0.5 * (1 + np.tanh(1.3 * (np.cos(ang) * ii + np.sin(ang) * jj - off)))
        s = np.ascontiguousarray(1e-6 + (1 - 2e-6) * s)
        if not lib.h_thinc(p(s), d, 1.6, 1.0 / 512, 1.0 / 300, p(np.zeros(2))):
            continue
        lL, lR = rng.standard_normal(2)
        ls = np.zeros(9)
        lib.h_thinc_rev(p(s), d, 1.6, 1.0 / 512, 1.0 / 300, lL, lR, p(ls))
        assert ls.tolist() == _thinc_rev(s.tolist(), d, 1.6, 1.0 / 512, 1.0 / 300, float(lL), float(lR))
        done += 1


def _muscl_branch(um, u0, up):
    with np.errstate(all="ignore"):
        um, u0, up, two = np.float64(um), np.float64(u0), np.float64(up), np.float64(2.0)
        r = (u0 - um) / (up - u0)
        if np.isinf(r) or np.isnan(r):
            r = np.float64(0.0)
        if r <= 0.0:
            return 0
        return 1 if two * r / (1.0 + r) < two / (1.0 + r) else 2


def _limiter_inputs():
    v = [0.0, -0.0, 1.0, -1.0, 1.0 + 2.0 ** -52, 1.0 - 2.0 ** -50, 2.0, 1.0 / 3.0, 5e-324, -5e-324, 1e-320,
         2.2250738585072014e-308, 1e-200, 1e200, 1e300, -1e300, 1.7976931348623157e308, -1.7976931348623157e308, math.inf, -math.inf, math.nan]
    rng = np.random.default_rng(5)
    cases = [(a, b, c) for a in v for b in v for c in v]
    cases += [tuple(x) for x in rng.standard_normal((4000, 3)) * 10.0 ** rng.integers(-323, 300, (4000, 1))]
    cases += [(1.0 - k * 2.0 ** -53, 1.0, 1.0 + j * 2.0 ** -52) for k in range(9) for j in range(9)]
    return cases


def _same(a, b):
    return (np.isnan(a) and np.isnan(b)) or np.float64(a).tobytes() == np.float64(b).tobytes()


def test_muscl_extrapolation(lib):
    """The limited extrapolation in the reference's order (hllc.cpp:527-568): two quotients, the
    smaller one, and each factor of one half as a product of its own."""
    f = np.float64
    out = np.zeros(2)
    for um, u0, up in _limiter_inputs():
        lib.h_muscl(um, u0, up, p(out))
        with np.errstate(all="ignore"):
            a, b, c = f(um), f(u0), f(up)
            r = (b - a) / (c - b)
            phi = f(0.0)
            if not (np.isinf(r) or np.isnan(r) or r <= 0.0):
                x, y = f(2.0) / (f(1.0) + r), f(2.0) * r / (f(1.0) + r)
                phi = y if y < x else x
            g = phi * f(0.5) * (c - a)
            want = b - f(0.5) * g, b + f(0.5) * g
        assert _same(out[0], want[0]) and _same(out[1], want[1]), (um, u0, up)


def test_muscl_branch(lib):
    """The active piece of the limiter (hllc.cpp:527-568): the reverse of L = R = u0 (0), of the
    slope u0 - um (1) and of up - u0 (2), told apart by the adjoint of um and up."""
    out = np.zeros(3)
    for um, u0, up in _limiter_inputs():
        lib.h_muscl_rev(um, u0, up, 0.0, 2.0, p(out))
        got = 1 if out[0] != 0.0 else 2 if out[2] != 0.0 else 0
        assert got == _muscl_branch(um, u0, up), (um, u0, up)
