"""The fused float-float sums of the FP32D patch (Dot2, cell_offsets in
rbc3d_gb300/csrc/selfff.cu), restated in exact rational arithmetic rounded to
float32 where the kernel rounds: the theta part of two columns (four terms
each), then the phi part of a point from them.  In a fused step t = RN(s + w v)
from a sum s kept at off/2 .. 3 off/2 with |w v| <= off/2, the difference s - t
must be exact, so that RN(w v + (s - t)) is what t lost, to one rounding."""
import math
from fractions import Fraction

import numpy as np
import pytest


def rn(v):
    """Fraction -> the nearest float32 (ties to even), as a Fraction; normal range."""
    if v == 0:
        return Fraction(0)
    e = math.frexp(float(abs(v)))[1]
    for k in (e - 1, e, e + 1):  # 2^(k-1) <= |v| < 2^k
        if Fraction(2) ** (k - 1) <= abs(v) < Fraction(2) ** k:
            e = k
    unit = Fraction(2) ** (e - 24)
    return round(v / unit) * unit


def split(v):
    h = Fraction(float(np.float32(v)))
    return h, Fraction(float(np.float32(v - float(h))))


class Dot2:
    def __init__(self, off):
        self.off, self.s, self.c = off, off, Fraction(0)

    def add(self, w, v, fast):
        (wh, wl), (vh, vl) = w, v
        if fast:
            assert self.off / 2 <= self.s <= 3 * self.off / 2 and abs(wh * vh) <= self.off / 2
            t = rn(self.s + wh * vh)
            assert rn(self.s - t) == self.s - t  # exact
            lost = rn(wh * vh + (self.s - t))
            assert self.off / 2 <= t <= 3 * self.off / 2
        else:  # product and TwoSum
            p = rn(wh * vh)
            e = rn(wh * vh - p)
            t = rn(self.s + p)
            bb = rn(t - self.s)
            lost = rn(rn(rn(self.s - rn(t - bb)) + rn(p - bb)) + e)
        self.s = t
        self.c = rn(self.c + wh * vl)
        self.c = rn(self.c + wl * vh)
        self.c = rn(self.c + lost)

    def drop(self):
        assert rn(self.s - self.off) == self.s - self.off  # exact
        self.s -= self.off


def dot(off, deriv, value, full):
    """deriv, value: (weight, operand) pairs; full: every term from the offset"""
    d = Dot2(off)
    for w, v in deriv:
        d.add(w, v, True)
    if not full:
        d.drop()
    for w, v in value:
        d.add(w, v, full)
    if full:
        d.drop()
    return d.s, d.c


def offset(b):
    return Fraction(2) ** math.frexp(2 * 1.01 * b)[1]


def weights(s, h):
    return [1 - s * s * (3 - 2 * s), s * s * (3 - 2 * s), h * s * (1 + s * (-2 + s)), h * s * s * (-1 + s)]


@pytest.mark.parametrize("full", [False, True])
def test_theta_and_phi_parts(full):
    """full: densities and normals; else positions, whose offset covers the
    derivative terms only and whose value terms are added by TwoSum."""
    rng = np.random.default_rng(7 + full)
    hx = hy = 2 * math.pi / 50
    worst = 0.0
    for trial in range(200):
        scale = 10.0 ** rng.uniform(-3, 1)
        v = np.zeros((2, 2, 4))  # row, column, slot u u_th u_ph u_thph
        v[..., 0] = scale * rng.uniform(-1.5, 1.5, (2, 2))
        v[..., 1:] = scale * rng.uniform(-15, 15, (2, 2, 3))
        if trial % 4 == 0:  # near-cancelling interpolant
            v[..., 0] -= v[..., 0].mean()
        u, ut, up, utp = np.abs(v).max(axis=(0, 1)) * (1 + rng.uniform(0, 3))  # the cell's bounds
        D, U = up + hx / 4 * utp, u + hx / 4 * ut
        ou, od = offset(U if full else hx / 4 * ut), offset(D)
        op = offset(U + hy / 4 * D if full else hy / 4 * D)
        x, y = weights(rng.uniform(), hx), weights(rng.uniform(), hy)
        xs, ys = [split(w) for w in x], [split(w) for w in y]
        Us, Ds = [], []
        for j in range(2):
            n = [[split(v[i, j, k]) for k in range(4)] for i in range(2)]
            Us.append(dot(ou, [(xs[2], n[0][1]), (xs[3], n[1][1])], [(xs[0], n[0][0]), (xs[1], n[1][0])], full))
            Ds.append(dot(od, [(xs[2], n[0][3]), (xs[3], n[1][3])], [(xs[0], n[0][2]), (xs[1], n[1][2])], True))
        s, c = dot(op, [(ys[2], Ds[0]), (ys[3], Ds[1])], [(ys[0], Us[0]), (ys[1], Us[1])], full)
        w = np.array([[[x[i] * y[j], x[2 + i] * y[j], x[i] * y[2 + j], x[2 + i] * y[2 + j]] for j in range(2)]
                      for i in range(2)])
        ref = float(U + hy / 4 * D) if full else np.abs(w * v).sum()
        worst = max(worst, abs(float(s + c) - float(np.sum(w * v))) / ref)
    # the sums' lost parts, up to 2^-24 of the offset, are summed in float32:
    # 2^-48 of up to 4 bounds a term, 12 terms a value, 2e-13; the positions'
    # offsets are not small against their sum of |w v| where the bounds are four
    # times the stencil's, and stay within the figure of test_ff_arith
    assert worst < (1e-12 if full else 5e-12), worst
