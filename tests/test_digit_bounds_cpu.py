"""Soundness of the digit pass's certified bounds (ct_digits.cuh) on the CPU, operation by operation in numpy:
the kernel value of kernel_mid2 within kKvErr (plus the term for the rounding of the scaled coordinates) of an
extended-precision evaluation, and the dot of the kept digit products within e0 + e1 (|v_q| + |v_c|) of the
exact dot.  A candidate is discarded on these bounds alone.

An FMA is taken as the exact FP64 product plus one FP64 addition, rounded to FP32; rsqrt.approx at both ends of
2^-22 around the root.  The tolerances are the constants of the kernel.
"""
import numpy as np
import pytest

F4 = np.float32
KKV_ERR = 4e-10


def fma(a, b, c):
    a, b, c = (np.asarray(x, np.float64) for x in (a, b, c))
    return (a * b + c).astype(F4)


def add(a, b):
    return (np.asarray(a, F4) + np.asarray(b, F4)).astype(F4)


def mul(a, b):
    return (np.asarray(a, F4) * np.asarray(b, F4)).astype(F4)


def two_sum(a, b):
    s = add(a, b)
    z = add(s, -a)
    return s, add(add(a, -add(s, -z)), add(b, -z))


def split(x):
    h = F4(x)
    return h, F4(np.float64(x) - np.float64(h))


def scaled(x, il):
    """df_mulf of the double-float scale and an f32 coordinate."""
    p = mul(il[0], x)
    e = fma(il[1], x, fma(il[0], x, -p))
    s = add(p, e)
    return s, add(e, -add(s, -p))


def kernel_mid(xq, xc, il, kt, end):
    S = np.zeros(len(xq), F4)
    C = S.copy()
    for a in range(xq.shape[1]):
        qh, ql = scaled(xq[:, a], il[a])
        ch, cl = scaled(xc[:, a], il[a])
        s0, e = two_sum(ch, -qh)
        l0 = add(e, add(cl, -ql))
        s = add(s0, l0)
        l = add(l0, -add(s, -s0))
        p = mul(s, s)
        pe = fma(add(s, s), l, fma(s, s, -p))
        S, se = two_sum(S, p)
        C = add(add(C, pe), se)
    if kt == 1:
        S = np.maximum(S, F4(1e-30))
        r = (1.0 / np.sqrt(S.astype(np.float64)) * (1 + end * 2.0 ** -22)).astype(F4)
        h = mul(S, r)
        C = mul(add(fma(-h, h, S), C), mul(r, F4(0.5)))
        S = h
    C = np.where(S > F4(86), F4(0), C)
    S = np.minimum(S, F4(86))
    kL1 = F4(2839.0 / 65536.0)
    kL2 = F4(np.log(2.0) / 16 - 2839.0 / 65536.0)
    n = add(fma(S, F4(-23.083120654223414), F4(12582912.0)), F4(-12582912.0))
    r0 = fma(n, -kL1, -S)
    rl = fma(n, -kL2, -C)
    rs = add(r0, rl)
    er = add(rl, -add(rs, -r0))
    w = fma(rs, F4(1 / 120), F4(1 / 24))
    w = fma(rs, w, F4(1 / 6))
    w = fma(rs, w, F4(0.5))
    pl = fma(mul(rs, rs), w, er)
    T = np.exp2(np.arange(16) / 16.0)
    ni = n.astype(np.int64)
    th = T.astype(F4)[ni & 15]
    tl = (T - T.astype(F4).astype(np.float64)).astype(F4)[ni & 15]
    f = np.exp2((ni >> 4).astype(np.float64)).astype(F4)
    p = mul(th, rs)
    pe = fma(th, rs, -p)
    s = add(th, p)
    e = add(p, add(th, -s))
    lo = add(fma(tl, rs, tl), fma(th, pl, add(e, pe)))
    if kt == 0:
        return mul(s, f), mul(lo, f)
    k3h = F4(1 / 3)
    k3l = F4(1 / 3 - np.float64(k3h))
    q = mul(S, S)
    qe = fma(add(S, S), C, fma(S, S, -q))
    u = mul(q, k3h)
    ue = fma(qe, k3h, fma(q, k3l, fma(q, k3h, -u)))
    s1, e1 = two_sum(np.ones_like(S), S)
    s2, e2 = two_sum(s1, u)
    pol = add(add(e1, e2), add(C, ue))
    k = mul(s2, s)
    ke = fma(pol, s, fma(s2, lo, fma(s2, s, -k)))
    return mul(k, f), mul(ke, f)


@pytest.mark.parametrize("kt", [0, 1])
@pytest.mark.parametrize("d", [1, 3, 8])
@pytest.mark.parametrize("scale", [1e-3, 0.03, 0.3, 1.0, 3.0, 10.0, 1000.0])
def test_kernel_value_within_its_bound(kt, d, scale):
    rng = np.random.default_rng(int(1000 * scale) + 10 * d + kt)
    n = 20000
    xq = (rng.standard_normal((n, d)) * scale).astype(F4)
    xc = (rng.standard_normal((n, d)) * scale).astype(F4)
    if scale >= 10:  # far points have kernel values of 0: near ones at large coordinates
        xc = (xq + rng.standard_normal((n, d)) * rng.choice([1e-3, 0.1, 1.0, 3.0], (n, 1))).astype(F4)
    xc[:10] = xq[:10]
    ls = rng.uniform(0.5, 2.0, d)
    il64 = 1.0 / ls
    x = (xq.astype(np.longdouble) - xc.astype(np.longdouble)) * il64.astype(np.longdouble)
    d2 = (x * x).sum(axis=1)
    if kt == 0:
        ref = np.exp(-d2 / 2)
        il = [split(v * np.sqrt(0.5)) for v in il64]
    else:
        a = np.sqrt(5 * d2)
        ref = (1 + a + a * a / 3) * np.exp(-a)
        il = [split(v * np.sqrt(5.0)) for v in il64]
    xmax = np.abs(xq * il64).max(axis=1) + np.abs(xc * il64).max()
    for end in (-1, 1):
        kh, kl = kernel_mid(xq, xc, il, kt, end)
        err = np.abs(kh.astype(np.longdouble) + kl.astype(np.longdouble) - ref)
        assert np.all(err <= KKV_ERR + 1e-13 * d * xmax), float(err.max())


def digits(v, e):
    x = v.astype(np.float64) * 2.0 ** (6 - e)
    out = []
    for _ in range(5):
        a = np.rint(x)
        assert np.abs(a).max() <= 64
        out.append(a)
        x = (x - a) * 128.0
    return out


@pytest.mark.parametrize("m", [32, 256, 800])
@pytest.mark.parametrize("kind", ["normal", "spikes", "wide", "tiny"])
def test_digit_dot_within_its_bound(m, kind):
    rng = np.random.default_rng(m)
    n = 120
    v = rng.standard_normal((n, m)) / np.sqrt(m)
    if kind == "spikes":
        v *= rng.random((n, m)) < 0.03
        v[:, 0] = rng.choice([-0.99999, 0.99999], n)
    elif kind == "wide":
        v *= 10.0 ** rng.uniform(-8, 3, (n, 1))
    elif kind == "tiny":
        v *= 1e-17
    v = v.astype(F4)
    norm = np.sqrt((v.astype(np.float64) ** 2).sum(axis=1))
    _, e = np.frexp(F4(norm.max() * (1 + 1e-6)) * F4(0.9924))
    e = max(int(e), -50)
    sc = 2.0 ** e
    dg = digits(v, e)
    e0 = 4.7 * m * 2.0 ** -42 * sc * sc + 1e-12 * sc * sc
    e1 = 1.02 * 2.0 ** -35 * sc * np.sqrt(m)
    o = []
    for s in range(6):
        acc = np.zeros((n, n))
        for i in range(5):
            if 0 <= s - i < 5:
                acc += dg[i] @ dg[s - i].T
        assert np.abs(acc).max() < 2 ** 24  # exact in FP32
        o.append(-(acc * 2.0 ** (-12 - 7 * s) * sc * sc).astype(F4))
    b1, a1 = two_sum(o[0], o[1])
    dh, a2 = two_sum(b1, o[2])
    dl = add(add(a1, a2), add(o[3], add(o[4], o[5])))
    exact = np.zeros((n, n), np.longdouble)
    for c in range(m):  # products of two FP32 values are exact
        exact += np.outer(v[:, c].astype(np.longdouble), v[:, c].astype(np.longdouble))
    err = np.abs(dh.astype(np.longdouble) + dl.astype(np.longdouble) + exact)
    assert np.all(err <= e0 + e1 * (norm[:, None] + norm[None, :])), float(err.max())
