"""Coarse-graining by tiles of points (k_cg_gather): grids whose last tiles are
not full, and contacts across a periodic boundary (a list of their own).

A grid evaluated in two parts along one dimension must give the whole grid's
points: the tiles, chunks and blocks fall differently, the sums are the same
ones in another order (1e-10 of each field's largest value, the tolerance of
the coarse-graining tests). Volume fraction and density are also summed here
directly over the particles.
"""
import math

import numpy as np
import pytest

import cases
from mercurydpm_fork_b200 import _abi

pytestmark = pytest.mark.gpu
WIDTH = 1e-3


def _close(a, b):
    scale = np.abs(b).max(axis=0)
    assert np.all(np.abs(a - b).max(axis=0) <= 1e-10 * scale + 1e-300)


@pytest.mark.parametrize("coord,n,cut", [("XZ", (4, 1, 5), 2), ("XZ", (7, 1, 9), 3), ("XZ", (13, 1, 2), 6),
                                         ("XYZ", (5, 4, 3), 2), ("XYZ", (4, 3, 7), 2)])
def test_parts_of_a_grid_give_the_grid(gpu, coord, n, cut):
    sc = cases.small_chute()  # periodic in x and y
    e = sc.engine()
    e.step(20)
    st, c = e.download(), e.contacts()
    assert c["periodic"].sum() > 10
    code = _abi.DEM_CG_XZ if coord == "XZ" else _abi.DEM_CG_XYZ
    lo = np.array([0.0, 0.0, float(sc.instance.domain_min[2])])
    hi = np.array([sc.instance.periodic_max[0], sc.instance.periodic_max[1], float(st["position"][:, 2].max()) + 1e-3])
    whole = e.cg(code, n, lo, hi, WIDTH).reshape(n + (-1,))
    for axis in (0, 2):
        k = min(cut, n[axis] - 1)
        if k < 2 or n[axis] - k < 2:  # a single point has no range test
            continue
        at = lo[axis] + (hi[axis] - lo[axis]) / n[axis] * k
        for first, last in ((0, k), (k, n[axis])):
            m, a, b = list(n), lo.copy(), hi.copy()
            m[axis] = last - first
            a[axis], b[axis] = (lo[axis], at) if first == 0 else (at, hi[axis])
            part = e.cg(code, m, a, b, WIDTH).reshape(tuple(m) + (-1,))
            want = np.take(whole, range(first, last), axis=axis)
            _close(part.reshape(-1, part.shape[-1]), want.reshape(-1, part.shape[-1]))
    # volume fraction and density by direct sums
    e.close()
    move = sc.inv_mass > 0
    x, r, mass = st["position"][move], sc.radius[move], 1.0 / sc.inv_mass[move]
    dims = [0, 2] if coord == "XZ" else [0, 1, 2]
    pts = np.stack(np.meshgrid(*[lo[k] + (np.arange(n[k]) + 0.5) * (hi[k] - lo[k]) / n[k] for k in range(3)], indexing="ij"),
                   -1).reshape(-1, 3)
    one, ratio = 1.0 / (math.sqrt(2 * math.pi) * WIDTH), 3.0
    if coord == "XZ":
        pre = one ** 2 / (1 - math.exp(-0.5 * ratio ** 2)) / (hi[1] - lo[1])
    else:
        pre = one ** 3 / (math.erf(ratio / math.sqrt(2)) - math.sqrt(2 / math.pi) * ratio * math.exp(-0.5 * ratio ** 2))
    d2 = ((pts[:, None, dims] - x[None, :, dims]) ** 2).sum(2)
    phi = np.where(d2 > (ratio * WIDTH) ** 2, 0.0, pre * np.exp(-d2 / (2 * WIDTH ** 2)))
    _close(whole.reshape(len(pts), -1)[:, :2], phi @ np.stack([4 / 3 * math.pi * r ** 3, mass], 1))
