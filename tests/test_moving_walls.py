"""Moving walls that reach spheres at rest long after the last list rebuild,
against the CPU oracle.

A rebuild files a moving wall with the spheres it can reach in a number of time
steps (256 in systems of this size, more for a slow wall) and the lists are made
anew after as many. A bed of spheres that do not touch, without gravity, gives no
other reason to rebuild: a wall hangs 0.7 radii above it (the skin is 0.4) and
falls, or turns about a position 6 diameters beside it (off its own axis), or
both, so that its first contact comes soon after the first rebuild, just before
those steps are over, or after a rebuild made because of them. Positions agree to 1e-13 of a diameter, velocities, forces and springs to
1e-9 relative, as in the parity tests over short horizons.
"""
import dataclasses

import numpy as np
import pytest

import harness as H
from mercurydpm_fork_b200 import scenarios
from mercurydpm_fork_b200.engine import axisymmetric_wall, infinite_wall, intersection_wall

pytestmark = pytest.mark.gpu

D = 1e-3
R = 0.5 * D
GAP = 0.7 * R


def _bed():
    """6 x 6 x 6 spheres 1.3 diameters apart about the origin, at rest."""
    sc = scenarios.settling_box(n=216, seed=1, box=(6 * 1.3, 6 * 1.3, 6 * 1.3), spacing=1.3 * (1 - 1e-9), jitter=0.0, vstd=0.0)
    sc.position -= 0.5 * (sc.position.min(0) + sc.position.max(0))
    sc.instance = dataclasses.replace(sc.instance, gravity=(0, 0, 0), domain_min=(-6 * D,) * 3, domain_max=(6 * D,) * 3)
    return sc


def _wall(kind, motion, steps_to_reach, dt, top):
    z = top + GAP
    pivot = (-6 * D, 0, z)
    s = GAP / steps_to_reach / dt  # speed of approach at the bed's far end
    reach = 6 * D + 2.5 * 1.3 * D
    v = (0, 0, -s if motion == "falls" else (-0.5 * s if motion == "both" else 0))
    om = (0, (s if motion == "turns" else 0.5 * s) / reach, 0) if motion != "falls" else (0, 0, 0)
    kw = dict(velocity=v, angular_velocity=om)
    if kind == "plane":
        return infinite_wall((0, 0, 1), pivot, **kw)
    if kind == "disk":  # a flat cylinder about the z axis through the pivot
        return axisymmetric_wall((0, 0, 1), [((-1, 0, 0), (20 * D, 0, 0)), ((0, 0, 1), (0, 0, 0)), ((0, 0, -1), (0, 0, 4 * D))],
                                 position=pivot, **kw)
    faces = [((0, 0, 1), (0, 0, 0)), ((0, 0, -1), (0, 0, 4 * D)), ((1, 0, 0), (-D, 0, 0)), ((-1, 0, 0), (20 * D, 0, 0))]
    return intersection_wall(faces, position=pivot, **kw)


def _compare(g, o, key):
    assert H.pair_set(g["contacts"]) == H.pair_set(o["contacts"]), key
    assert H.rel_err(g["position"], o["position"], D) < 1e-13, key
    for k in ("velocity", "force"):
        assert H.rel_err(g[k], o[k]) < 1e-9, (k, key)
    assert H.rel_err(g["contacts"]["springs"], o["contacts"]["springs"]) < 1e-9, key


def _scenario(kind, motion, steps_to_reach):
    sc = _bed()
    sc.walls = [_wall(kind, motion, steps_to_reach, sc.time_step, float(sc.position[:, 2].max()) + R)]
    return sc


@pytest.mark.parametrize("steps_to_reach", [13.4, 118, 248, 400])
@pytest.mark.parametrize("motion", ["falls", "turns", "both"])
@pytest.mark.parametrize("kind", ["plane", "disk", "block"])
def test_wall_that_arrives_between_rebuilds(gpu, kind, motion, steps_to_reach):
    sc = _scenario(kind, motion, steps_to_reach)
    seen = 0
    for steps in (int(1.02 * steps_to_reach), int(1.06 * steps_to_reach), int(1.12 * steps_to_reach)):
        g, o = H.run_gpu(sc, steps), H.run_oracle(sc, steps)
        _compare(g, o, steps)
        seen += int((o["contacts"]["is_wall"] == 1).sum())
    assert seen >= 6


def test_calls_of_a_few_steps(gpu):
    """The age of the lists counts steps, whatever the calls they come in."""
    sc = _scenario("block", "turns", 258)
    e = sc.engine()
    rebuilds = 0
    for _ in range(67):
        e.step(4)
        rebuilds += e.stats()["rebuilds"]
    g = dict(e.download(), force=e.forces()[0], contacts=H.sort_contacts(e.contacts()))
    e.close()
    o = H.run_oracle(sc, 268)
    assert (o["contacts"]["is_wall"] == 1).sum() >= 3 and rebuilds >= 2
    _compare(g, o, "calls")


@pytest.mark.parametrize("motion", ["falls", "turns"])
def test_periodic_box(gpu, motion):
    """The bed drifts over the seams of its periodic box while the wall comes."""
    sc = _scenario("plane", motion, 125)
    half = 3 * 1.3 * D
    sc.instance = dataclasses.replace(sc.instance, periodic_mask=0b011, periodic_min=(-half, -half, 0),
                                      periodic_max=(half, half, 0))
    sc.position[:, 0] += 0.6 * D
    sc.position[:, 1] += 0.55 * D
    sc.velocity[:] = (0.125, 0.25, 0.0)
    seen = 0
    for steps in (115, 128, 145):
        g, o = H.run_gpu(sc, steps), H.run_oracle(sc, steps)
        _compare(g, o, steps)
        seen += int((o["contacts"]["is_wall"] == 1).sum())
    assert seen >= 6


def test_batch_of_moving_and_standing_walls(gpu):
    members = [_scenario("block", "turns", 118), _scenario("disk", "falls", 14), _scenario("plane", "both", 60), _bed()]
    members[3].walls = []
    b = scenarios.batch(members)
    for steps in (16, 66, 126):
        e = b.engine()
        e.step(steps)
        pos, f, c = e.download()["position"], e.forces()[0], e.contacts()
        e.close()
        for k, m in enumerate(members):
            o = H.run_oracle(m, steps)
            sl = b.member_slice(k)
            assert H.rel_err(pos[sl], o["position"], D) < 1e-13, (steps, k)
            assert H.rel_err(f[sl], o["force"]) < 1e-9, (steps, k)
            here = (c["id_p"] >= sl.start) & (c["id_p"] < sl.stop)
            assert here.sum() == len(o["contacts"]["id_p"]), (steps, k)
