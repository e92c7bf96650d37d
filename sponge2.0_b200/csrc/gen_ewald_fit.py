"""Generates ewald_fit.h: rational approximations of the two smooth Ewald
kernels the pair kernel evaluates in FP32.

With z = beta*r and w = z^2 the real-space Coulomb force and energy are

    F_c / (q_i q_j) = r^-3 [erfc(z) + 2z/sqrt(pi) e^-z^2] = r^-3 - beta^3 K(w)
    E_c / (q_i q_j) = erfc(z)/r                          = r^-1 - beta   M(w)

    K(w) = [erf(z) - 2z/sqrt(pi) e^-z^2] / z^3     (entire, even in z)
    M(w) = erf(z) / z                               (entire, even in z)

Both are fitted on w in [0, W_MAX] as P(x)/Q(x), x = w/W_MAX: degrees (5,5),
in double: for the scalar kernels by iteratively reweighted linear least
squares on the relative error (Loeb's method); for the packed cluster-pair
kernel by the same linearisation with Lawson's weights, which drive the
largest absolute error down (minimax: 7e-9 for K, 1e-9 for M, below what FP32
resolves), scaled to monic denominators.  Degrees (4,5) would save the packed
kernel an instruction, but their 6e-8 is one-sided over whole ranges of r and
moved the forces' error against 64 bits from 8e-7 to 1.0e-6 relative RMS.
W_MAX = 12.25 covers beta*rc <= 3.5, i.e. a direct-space
tolerance down to ~1e-7 at rc = 10.  Run from this directory:
``python gen_ewald_fit.py > ewald_fit.h``.
"""
import numpy as np
from scipy.special import erf

W_MAX = 12.25
DEG = 5


def K(w):
    z = np.sqrt(w)
    out = np.empty_like(w)
    small = z < 1e-3
    zz = z[~small]
    out[~small] = (erf(zz) - 2 * zz / np.sqrt(np.pi) * np.exp(-zz * zz)) / zz ** 3
    ws = w[small]
    out[small] = 2 / np.sqrt(np.pi) * (2 / 3 - 2 * ws / 5 + ws * ws / 7 - ws ** 3 / 27)
    return out


def M(w):
    z = np.sqrt(w)
    out = np.empty_like(w)
    small = z < 1e-4
    out[~small] = erf(z[~small]) / z[~small]
    out[small] = 2 / np.sqrt(np.pi) * (1 - w[small] / 3)
    return out


def ratfit(f, m=DEG, n=DEG, iters=40):
    w = np.linspace(0, W_MAX, 12001)
    y = f(w)
    x = w / W_MAX
    wq = np.ones_like(x)
    for _ in range(iters):
        A = np.hstack([np.vander(x, m + 1, increasing=True),
                       -(y[:, None]) * np.vander(x, n + 1, increasing=True)[:, 1:]])
        scale = (wq * np.abs(y))[:, None]
        sol, *_ = np.linalg.lstsq(A / scale, y / scale[:, 0], rcond=None)
        p = sol[:m + 1]
        q = np.concatenate([[1.0], sol[m + 1:]])
        wq = np.abs(np.polyval(q[::-1], x))
    xf = x.astype(np.float32)
    pf = p.astype(np.float32)
    qf = q.astype(np.float32)
    P = np.full_like(xf, pf[-1])
    for k in pf[-2::-1]:
        P = P * xf + k
    Q = np.full_like(xf, qf[-1])
    for k in qf[-2::-1]:
        Q = Q * xf + k
    err = np.abs((P / Q).astype(np.float64) - y).max()
    return pf, qf, err


def horner32(c, x):
    """Horner's rule with fused multiply-adds in FP32."""
    r = np.full_like(x, np.float32(c[-1]))
    for k in c[-2::-1]:
        r = (r.astype(np.float64) * x.astype(np.float64) + np.float64(np.float32(k))).astype(np.float32)
    return r


def minimax(f, m, n, iters=60):
    w = W_MAX * (1 - np.cos(np.linspace(0, np.pi, 6001))) / 2
    y = f(w)
    x = w / W_MAX
    lawson, wq = np.ones_like(x), np.ones_like(x)
    best = (np.inf, None, None)
    for it in range(iters):
        A = np.hstack([np.vander(x, m + 1, increasing=True),
                       -(y[:, None]) * np.vander(x, n + 1, increasing=True)[:, 1:]])
        scale = lawson / np.abs(wq)
        sol, *_ = np.linalg.lstsq(A * scale[:, None], y * scale, rcond=None)
        p, q = sol[:m + 1], np.concatenate([[1.0], sol[m + 1:]])
        wq = np.polyval(q[::-1], x)
        err = np.abs(np.polyval(p[::-1], x) / wq - y)
        if err.max() < best[0]:
            best = (err.max(), p, q)
        if it > 8:
            lawson = lawson * (err / err.max() + 1e-3) ** 0.5
            lawson /= lawson.max()
    _, p, q = best
    # the packed kernel's denominators are monic: their first step is an
    # addition with one constant operand
    p, q = p / q[-1], q / q[-1]
    w = np.linspace(0, W_MAX, 200001)
    xf = (w / W_MAX).astype(np.float32)
    r = (horner32(p, xf) * (np.float32(1) / horner32(q, xf))).astype(np.float64)
    return p, q, np.abs(r - f(w)).max()


def main():
    kp, kq, kerr = ratfit(K)
    mp, mq, merr = ratfit(M)
    kp2, kq2, kerr2 = minimax(K, DEG, DEG)
    mp2, mq2, merr2 = minimax(M, DEG, DEG)
    fmt = lambda a: ", ".join(f"{float(v):.9e}f" for v in a)
    print("// Generated by gen_ewald_fit.py -- do not edit.")
    print(f"// K(w) max abs error {kerr:.2e} (K(0)=0.752), M(w) max abs error {merr:.2e} (M(0)=1.128),")
    print(f"// FP32 Horner evaluation on w in [0, {W_MAX}]; the packed kernel's minimax fits")
    print(f"// K {kerr2:.2e}, M {merr2:.2e}.")
    print("#pragma once")
    print(f"#define SPGNB_EWALD_W_MAX {W_MAX}f")
    print(f"#define SPGNB_EWALD_INV_W_MAX {1.0 / W_MAX:.9e}f")
    print(f"static __constant__ float kEwaldKP[{DEG + 1}] = {{{fmt(kp)}}};")
    print(f"static __constant__ float kEwaldKQ[{DEG + 1}] = {{{fmt(kq)}}};")
    print(f"static __constant__ float kEwaldMP[{DEG + 1}] = {{{fmt(mp)}}};")
    print(f"static __constant__ float kEwaldMQ[{DEG + 1}] = {{{fmt(mq)}}};")
    # the same coefficients as (c, c) pairs: operands of packed FP32x2 arithmetic
    fmt2 = lambda a: ", ".join(f"{{{float(v):.9e}f, {float(v):.9e}f}}" for v in a)
    for name, a in (("KP", kp2), ("KQ", kq2), ("MP", mp2), ("MQ", mq2)):
        print(f"static __constant__ float2 kEwald{name}2[{len(a)}] = {{{fmt2(a)}}};")
        print(f"static const double kEwald{name}Host[{len(a)}] = {{{', '.join(repr(float(v)) for v in a)}}};")


if __name__ == "__main__":
    main()
