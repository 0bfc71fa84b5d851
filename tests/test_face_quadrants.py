"""Index arithmetic of face_kernel (ard_face.cuh), mirrored on the CPU.

The mirror restates the kernel's shared-memory regions (sized as face_smem
sizes them, poisoned with NaN), its staging, the two half-size products per
quadrant and its output indices, for whole, one-output and split jobs, both
directions, aligned and unaligned extents and row pitches.  It asserts that
every access stays inside its region, that no poisoned value is used, that
every output is written once, and that the result is the full 2D transform
(products with the dense C / Ci matrices) to FP64 rounding.
"""
import itertools

import numpy as np
import pytest

half = lambda n: (n + 1) >> 1
half4 = lambda n: (half(n) + 3) & ~3


def pitch(n):
    n4 = half4(n)
    return n4 + (0 if n4 & 7 else 4)


def basis(n, ci):
    k, j = np.arange(n)[:, None], np.arange(n)[None, :]
    c = 2.0 * np.cos(np.pi * (((2 * j + 1) * k) % (4 * n)) / (2.0 * n))
    if ci:
        c[0] *= 0.5
    return c


def tables(n, ci):
    """Hr[p][m][j], Hf[p][j][m], rows of pitch half4, zero padded (flat)."""
    b, h, h4 = basis(n, ci), half(n), half4(n)
    hr, hf = np.zeros((2, h, h4)), np.zeros((2, h, h4))
    for p, m, j in itertools.product(range(2), range(h), range(h)):
        if 2 * m + p < n:
            hr[p, m, j] = hf[p, j, m] = b[2 * m + p, j]
    return hr.ravel(), hf.ravel()


class Region:
    """A shared-memory region: bounds-checked, NaN until written."""

    def __init__(self, n):
        self.v = np.full(n, np.nan)

    def get(self, i):
        assert 0 <= i < len(self.v), (i, len(self.v))
        x = self.v[i]
        assert not np.isnan(x), "read of an unwritten element"
        return x

    def put(self, i, x):
        assert 0 <= i < len(self.v), (i, len(self.v))
        self.v[i] = x

    def row(self, i, n):
        assert 0 <= i and i + n <= len(self.v), (i, n, len(self.v))
        r = self.v[i:i + n]
        assert not np.isnan(r).any(), "read of an unwritten element"
        return r


def shape(J, h, inv):
    no, o0 = (2 if J["which"] == 0 else 1), (1 if J["which"] == 2 else 0)
    npu, pu0, c0, nc = 2, 0, J["u0"] >> 1, (J["ub"] + 1) >> 1
    if J["split"] and not inv:
        npu, pu0 = 1, h
    elif J["split"]:
        first = (((nc + 1) >> 1) + 3) & ~3
        if h:
            c0, nc = c0 + first, max(0, nc - first)
        else:
            nc = min(nc, first)
    return no, o0, npu, pu0, c0, nc


def run_job(J, h, inv, X, tabA, tabB, out, count):
    V, U, ld = J["V"], J["U"], J["ld"]
    no, o0, npu, pu0, c0, nc = shape(J, h, inv)
    if nc <= 0:
        return
    hv, hu, hv4, hu4, fp, ap = half(V), half(U), half4(V), half4(U), pitch(U), pitch(V)
    nq = (nc + 3) >> 2
    ncp, units = 4 * nq, no * 2 * npu
    F = Region(max(units * hv * fp, units * hv * ncp if inv else 0))
    A, B, Tm = Region(2 * hv * ap), Region(npu * hu4 * ncp), Region(units * hv4 * ncp)
    for row, q in itertools.product(range(2 * hv), range(hv4 >> 2)):
        for e in range(4):
            A.put(row * ap + 4 * q + e, tabA[row * hv4 + 4 * q + e])
    for p, j, c in itertools.product(range(npu), range(hu4), range(nq)):
        ok = j < hu and c0 + 4 * c < hu4
        for e in range(4):
            B.put((p * hu4 + j) * ncp + 4 * c + e, tabB[((pu0 + p) * hu + j) * hu4 + c0 + 4 * c + e] if ok else 0.0)
    for u in range(units):
        for i in range((hv4 - hv) * ncp):
            Tm.put((u * hv4 + hv) * ncp + i, 0.0)

    def x(layer, r, u):
        assert 0 <= r < V and 0 <= u < U
        return X[layer][r * ld + u]

    if not inv:
        for r, q in itertools.product(range(hv), range(hu4 >> 2)):
            r2 = V - 1 - r
            for e in range(4):
                j = 4 * q + e
                for o in range(o0, o0 + no):
                    sg = -1.0 if o else 1.0
                    get = lambda rr, u: (x(0, rr, u) + sg * x(1, rr, u)) if j < hu else 0.0
                    e0, e1 = [], []
                    for rr in (r, r2):
                        a, b = get(rr, j), get(rr, U - 1 - j)
                        mid = 2 * j + 1 == U
                        e0.append(a if mid else a + b)
                        e1.append(0.0 if mid else a - b)
                    for p in range(pu0, pu0 + npu):
                        a, b = (e1 if p else e0)
                        base = ((o - o0) * 2 * npu + p - pu0) * hv * fp + r * fp + j
                        F.put(base, a if r == r2 else a + b)
                        F.put(base + npu * hv * fp, 0.0 if r == r2 else a - b)
    else:
        for kv, q in itertools.product(range(2 * hv), range(hu4 >> 1)):
            for o in range(o0, o0 + no):
                sg = -1.0 if o else 1.0
                w = [(x(0, kv, 4 * q + e) + sg * x(1, kv, 4 * q + e)) if kv < V and 4 * q + e < U else 0.0
                     for e in range(4)]
                base = (((o - o0) * 2 + (kv & 1)) * 2) * hv * fp + (kv >> 1) * fp + 2 * q
                F.put(base, w[0])
                F.put(base + 1, w[2])
                F.put(base + hv * fp, w[1])
                F.put(base + hv * fp + 1, w[3])

    def product(K, lp, L, l_of, R, r_of, put):
        for u in range(units):
            for r, ct in itertools.product(range(hv), range(nq)):
                l = L.row(l_of(u) + r * lp, K)
                acc = np.zeros(4)
                for k in range(K):
                    acc += l[k] * R.row(r_of(u) + k * ncp + 4 * ct, 4)
                put(u, r, 4 * ct, acc)

    def to_t(u, r, c, v):
        for e in range(4):
            Tm.put((u * hv4 + r) * ncp + c + e, v[e])

    product(hu4, fp, F, lambda u: u * hv * fp, B, lambda u: (u % npu) * hu4 * ncp, to_t)
    a_of, t_of = (lambda u: (u // npu % 2) * hv * ap), (lambda u: u * hv4 * ncp)

    def store(o, r, u, v):
        assert 0 <= r < V and 0 <= u < U
        out[o][r, u] = v
        count[o][r, u] += 1

    if not inv:
        def to_out(u, r, c, v):
            pu, pv, o = pu0 + u % npu, u // npu % 2, o0 + u // (2 * npu)
            kv, ku = 2 * r + pv, 2 * (c0 + c) + pu
            if kv >= V:
                return
            for e in range(4):
                if c + e < nc and ku + 2 * e < U:
                    store(o, kv, ku + 2 * e, v[e])
        product(hv4, ap, A, a_of, Tm, t_of, to_out)
    else:
        O = Region(len(F.v))   # the result quadrants take the layers' place

        def to_o(u, r, c, v):
            for e in range(4):
                O.put((u * hv + r) * ncp + c + e, v[e])
        product(hv4, ap, A, a_of, Tm, t_of, to_o)
        for o, r, c in itertools.product(range(no), range(hv), range(ncp)):
            u = c0 + c
            u2, r2 = U - 1 - u, V - 1 - r
            if c >= nc or u >= hu:
                continue
            ee, eo, oe, oo = (O.get((o * 4 * hv + r) * ncp + c + k * hv * ncp) for k in range(4))
            store(o0 + o, r, u, ee + oe + eo + oo)
            if u2 != u:
                store(o0 + o, r, u2, ee + oe - eo - oo)
            if r2 != r:
                store(o0 + o, r2, u, ee - oe + eo - oo)
                if u2 != u:
                    store(o0 + o, r2, u2, ee - oe - eo + oo)


@pytest.mark.parametrize("V,U,ld", [(6, 6, 6), (7, 9, 9), (12, 33, 36), (13, 34, 36), (8, 40, 40), (9, 65, 68)])
@pytest.mark.parametrize("inv", [False, True])
@pytest.mark.parametrize("form", ["whole", "outputs", "split"])
def test_quadrants_are_the_full_transform(V, U, ld, inv, form):
    rng = np.random.default_rng(V * 100 + U)
    X = [np.full(V * ld, np.nan) for _ in range(2)]
    D = [rng.standard_normal((V, U)) for _ in range(2)]
    for k in range(2):
        X[k].reshape(V, ld)[:, :U] = D[k]
    for ci in (False, True):
        hrV, hfV = tables(V, ci)
        hrU, hfU = tables(U, ci)
        tabA, tabB = (hfV, hrU) if inv else (hrV, hfU)
        out = [np.full((V, U), np.nan) for _ in range(2)]
        count = [np.zeros((V, U), int) for _ in range(2)]
        for u0 in range(0, U, 32):
            for which in ((0,) if form == "whole" else (1, 2)):
                J = dict(V=V, U=U, ld=ld, u0=u0, ub=min(32, U - u0), which=which, split=1 if form == "split" else 0)
                for h in ((0, 1) if form == "split" else (0,)):
                    run_job(J, h, inv, X, tabA, tabB, out, count)
        bV, bU = basis(V, ci), basis(U, ci)
        for o in range(2):
            W = D[0] - D[1] if o else D[0] + D[1]
            want = bV.T @ W @ bU if inv else bV @ W @ bU.T
            assert (count[o] == 1).all()
            assert np.abs(out[o] - want).max() < 1e-11 * np.abs(want).max()
