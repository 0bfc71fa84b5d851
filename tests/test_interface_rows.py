"""Addresses of the interface kernels (side_row, ard_kernels.cuh), mirrored on
the CPU, against the general rule of which shell layer owns a cell (X layers own
what they touch, then Y layers, then Z layers: shell_index).

For every interface axis, both sides, extents from the smallest partition up and
every face cell, the base plus its layer and row steps is the offset of the
owner's element, over items as the layout cuts them: rows on an air side's Y
shell alone, any number of other rows together."""
import itertools

import pytest


def face_layer(c, n):
    return c if c < 3 else (c - (n - 6) if c >= n - 3 else -1)


class Air:
    def __init__(self, w, h, d):
        self.w, self.h, self.d, self.wp = w, h, d, (w + 3) // 4 * 4
        self.fx = 1000
        self.fy = self.fx + 6 * d * h
        self.fz = self.fy + 6 * d * self.wp

    def shell_index(self, x, y, z):
        l = face_layer(x, self.w)
        if l >= 0:
            return self.fx + (l * self.d + z) * self.h + y
        l = face_layer(y, self.h)
        if l >= 0:
            return self.fy + (l * self.d + z) * self.wp + x
        l = face_layer(z, self.d)
        return self.fz + (l * self.h + y) * self.wp + x if l >= 0 else -1


def side_row(S, axis, lo, u, v):
    """(f, fk, fv) of an air side, as the kernel forms them."""
    ext = (S.w, S.h, S.d)[axis]
    c0, l0 = (ext - 3, 3) if lo else (0, 0)
    if axis == 0:
        return S.fx + (l0 * S.d + v) * S.h + u, S.d * S.h, S.h
    l = face_layer(u, S.w)
    if l >= 0:
        if axis == 1:
            return S.fx + (l * S.d + v) * S.h + c0, 1, S.h
        return S.fx + (l * S.d + c0) * S.h + v, S.h, 1
    if axis == 1:
        return S.fy + (l0 * S.d + v) * S.wp + u, S.d * S.wp, S.wp
    l = face_layer(v, S.h)
    if l >= 0:
        return S.fy + (l * S.d + c0) * S.wp + u, S.wp, 0
    return S.fz + (l0 * S.h + v) * S.wp + u, S.h * S.wp, S.wp


@pytest.mark.parametrize("extent", [(6, 6, 6), (7, 9, 6), (13, 8, 11), (12, 6, 17)])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("lo", [False, True])
@pytest.mark.parametrize("n", [1, 2, 4])
def test_rows_reach_the_owning_layer(extent, axis, lo, n):
    S = Air(*extent)
    ext = extent[axis]
    nu, nv = ((S.h, S.d), (S.w, S.d), (S.w, S.h))[axis]
    alone = lambda v: axis == 2 and face_layer(v, S.h) >= 0
    v, seen = 0, 0
    while v < nv:
        k = 1
        while not alone(v) and k < n and v + k < nv and not alone(v + k):
            k += 1
        for u, r, m in itertools.product(range(nu), range(k), range(3)):
            f, fk, fv = side_row(S, axis, lo, u, v)
            c = ext - 3 + m if lo else m
            x, y, z = ((c, u, v + r), (u, c, v + r), (u, v + r, c))[axis]
            assert f + m * fk + r * fv == S.shell_index(x, y, z)
            seen += 1
        v += k
    assert seen == nu * nv * 3
