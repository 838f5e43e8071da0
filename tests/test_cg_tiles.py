"""Coarse-graining by tiles of points (k_cg_gather): grids whose last tiles are
not full, and contacts across a periodic boundary (a list of their own).

A grid evaluated in two parts along one dimension must give the whole grid's
points: the tiles, chunks and blocks fall differently, the sums are the same
ones in another order (1e-10 of each field's largest value, the tolerance of
the coarse-graining tests). Volume fraction and density are also summed here
directly over the particles.

Grids of some hundred tiles and more, which no block splits, are compared point
by point with coarser grids whose points are among theirs, and one whose fields
take more workspace than a handle keeps is evaluated as well.
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


@pytest.mark.parametrize("coord,n,k", [("XZ", (60, 1, 90), 3), ("XZ", (61, 1, 83), 1), ("XYZ", (18, 18, 21), 3),
                                       ("XYZ", (33, 9, 27), 3)])
def test_grids_of_unsplit_tiles_hold_the_points_of_split_ones(gpu, coord, n, k):
    """A block takes a whole tile where there are more than four tiles an SM. The
    points of a grid k times coarser in every direction (k odd) are every k-th
    of it, from (k - 1) / 2; for k = 1 its first rows are a grid of their own."""
    sc = cases.small_chute()
    e = sc.engine()
    e.step(20)
    top = float(e.download()["position"][:, 2].max()) + 1e-3
    lo = np.array([0.0, 0.0, float(sc.instance.domain_min[2])])
    hi = np.array([sc.instance.periodic_max[0], sc.instance.periodic_max[1], top])
    code = _abi.DEM_CG_XZ if coord == "XZ" else _abi.DEM_CG_XYZ
    tile = (2, 1, 4) if coord == "XZ" else (2, 2, 2)
    assert np.prod([-(-a // t) for a, t in zip(n, tile)]) > 4 * 148
    whole = e.cg(code, n, lo, hi, WIDTH).reshape(n + (-1,))
    np.testing.assert_array_equal(whole.reshape(-1, whole.shape[-1]), e.cg(code, n, lo, hi, WIDTH))
    if k > 1:
        m = tuple(-(-a // k) if a > 1 else 1 for a in n)
        assert all(a % k == 0 for a in n if a > 1)
        part = e.cg(code, m, lo, hi, WIDTH).reshape(m + (-1,))
        want = whole[tuple(slice((k - 1) // 2, None, k) if a > 1 else slice(None) for a in n)]
    else:
        m, b = (5,) + n[1:], hi.copy()
        b[0] = lo[0] + (hi[0] - lo[0]) / n[0] * 5
        part, want = e.cg(code, m, lo, b, WIDTH).reshape(m + (-1,)), whole[:5]
    e.close()
    assert np.abs(part[..., 11]).max() > 0
    _close(part.reshape(-1, part.shape[-1]), want.reshape(-1, want.shape[-1]))


def test_fields_larger_than_the_kept_workspace(gpu):
    """2.5 million points are 577 MB of fields: workspace taken for the call."""
    sc = cases.compressed_box(n=60)
    e = sc.engine()
    e.step(5)
    lo, hi = (0.0, 0.0, 0.0), (0.01, 0.01, 0.04)
    n = (117, 117, 183)
    before = e.memory()["device_bytes"]
    fine = e.cg(_abi.DEM_CG_XYZ, n, lo, hi, WIDTH).reshape(n + (-1,))
    assert fine.nbytes > 512 << 20 and e.memory()["device_bytes"] == before
    m = tuple(a // 3 for a in n)
    _close(e.cg(_abi.DEM_CG_XYZ, m, lo, hi, WIDTH), fine[1::3, 1::3, 1::3].reshape(-1, fine.shape[-1]))
    assert e.memory()["device_bytes"] > before  # the smaller grid's is kept
    assert e.reduce()["n_contacts"] > 50
    e.close()
