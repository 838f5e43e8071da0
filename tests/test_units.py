"""The force evaluation's unit list (k_units): one thread per pair or wall
candidate, chunks of whole warps per block, contacts compacted per block.

Sizes where a chunk, a warp or a block is not full, from a lone pair to
several blocks, against the oracle: contact pairs exact, per-contact forces
bit-exact at the initial evaluation, and the first steps (in which springs of
the initial evaluation may be kept without a contact) within the parity
tests' tolerances. A list of one wall candidate and no pair, and none at all,
run too; a run is bit-identical under every chunk size.
"""
import numpy as np
import pytest

import cases
import harness as H
from mercurydpm_fork_b200 import scenarios

pytestmark = pytest.mark.gpu


def _box(n, spacing=0.995):
    nx = max(1, round(n ** (1 / 3)))
    nz = -(-n // (nx * nx))
    edge = lambda k: k * spacing * (1 + 1e-9)
    return scenarios.settling_box(n=n, seed=n, box=(edge(nx), edge(nx), edge(nz)), spacing=spacing, jitter=0.004, vstd=0.05)


@pytest.mark.parametrize("n", [1, 2, 3, 11, 12, 43, 130, 1000, 2777])
def test_sizes_around_warps_and_chunks(gpu, n):
    sc = _box(n)
    g, o = H.run_gpu(sc, 0), H.run_oracle(sc, 0)
    assert H.pair_set(g["contacts"]) == H.pair_set(o["contacts"]) and len(o["contacts"]["id_p"]) > 0
    np.testing.assert_array_equal(g["contacts"]["force"], o["contacts"]["force"])
    np.testing.assert_array_equal(g["contacts"]["springs"], o["contacts"]["springs"])
    for steps in (1, 2, 20):
        g, o = H.run_gpu(sc, steps), H.run_oracle(sc, steps)
        assert H.pair_set(g["contacts"]) == H.pair_set(o["contacts"])
        assert H.rel_err(g["position"], o["position"], 1e-3) < 1e-13
        for k in ("velocity", "force", "torque"):
            assert H.rel_err(g[k], o[k]) < 1e-9, k
        assert H.rel_err(g["contacts"]["springs"], o["contacts"]["springs"]) < 1e-9


def test_no_unit_at_all(gpu):
    sc = scenarios.settling_box(n=8, seed=1, box=(20, 20, 40), spacing=4.0)
    g, o = H.run_gpu(sc, 5), H.run_oracle(sc, 5)
    assert len(g["contacts"]["id_p"]) == 0
    np.testing.assert_array_equal(g["position"], o["position"])


@pytest.mark.parametrize("case", ["small_chute", "small_drum", "triangle_mesh"])
def test_chunk_size_changes_nothing(gpu, case):
    sc = getattr(cases, case)()
    runs = []
    for block in (64, 128, 256):
        e = sc.engine()
        e.set_tuning(detect_block=block, contacts_blocks_per_sm=3 if block == 256 else 5, sum_block=128)
        e.step(30)
        runs.append(dict(e.download(), springs=e.contacts()["springs"]))
        e.close()
    for other in runs[1:]:
        for k in ("position", "velocity", "angular_velocity", "springs"):
            np.testing.assert_array_equal(other[k], runs[0][k], err_msg=k)


@pytest.mark.parametrize("share", [0.024, 0.2])
def test_wall_that_translates_into_the_bed(gpu, share):
    """A lid that starts out of reach of every sphere's list and comes down by
    `share` of the skin a step: its list holds for the steps it is made for."""
    sc = scenarios.settling_box(n=216, seed=3, box=(6 * 0.999, 6 * 0.999, 6 * 0.999), spacing=0.999 * (1 - 1e-9),
                                jitter=0.0, vstd=0.0)
    r = float(sc.radius[0])
    skin, gap = 0.4 * r, 0.7 * r
    lid = sc.walls[5]
    lid.position[2] += gap
    lid.velocity[2] = -share * skin / sc.time_step
    steps = int(1.1 * gap / (share * skin))
    g, o = H.run_gpu(sc, steps), H.run_oracle(sc, steps)
    assert ((o["contacts"]["is_wall"] == 1) & (o["contacts"]["id_i"] == 5)).sum() > 0
    assert H.pair_set(g["contacts"]) == H.pair_set(o["contacts"])
    assert H.rel_err(g["position"], o["position"], 1e-3) < 1e-13
    for k in ("velocity", "force"):
        assert H.rel_err(g[k], o[k]) < 1e-9, k


@pytest.mark.parametrize("l_d,skin", [(50.0, 0.05), (50.0, 0.0501), (31.0, 0.05)])
def test_lists_are_symmetric_at_the_edge_of_the_reach(gpu, l_d, skin):
    """Spheres 1.05 diameters apart with a skin of 0.05: thousands of pairs lie
    within the FP32 test's margin of the reach, some of them with a cell boundary
    in between. A list that one partner alone holds is an error of the run."""
    n = 50_000 if l_d > 40 else 20_000
    sc = scenarios.triangle_floor(n=n, seed=1, drop_d=0.02, v0=0.5, l_d=l_d)
    e = sc.engine(skin=skin * 1e-3)
    e.step(150)
    x, rebuilds = e.download()["position"], e.stats()["rebuilds"]
    e.close()
    assert rebuilds >= 3
    e = sc.engine()
    e.step(150)
    assert H.rel_err(x, e.download()["position"], 1e-3) < 1e-13
    e.close()
