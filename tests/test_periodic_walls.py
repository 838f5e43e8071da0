"""Walls and triangle meshes in periodic boxes: spheres that a drift carries
across a seam between two list rebuilds meet what stands on the far side.

The list rebuild files the walls near a particle, and walls do not repeat with
the period, so those near the particle's image count as well. Spheres start a
few hundredths of a diameter before both seams and cross them at 1 m/s (0.002
diameters a step) well before their first rebuild (half the skin, 50 steps). The
CPU oracle has no triangle walls: a flat mesh of one group without friction
acts as an infinite wall, and a mesh in relief is compared with the engine's
own run at a skin so small that every few steps rebuild.
"""
import dataclasses

import numpy as np
import pytest

import cases
import harness as H
from mercurydpm_fork_b200 import scenarios
from mercurydpm_fork_b200.engine import axisymmetric_wall, infinite_wall, intersection_wall

pytestmark = pytest.mark.gpu

D = 1e-3
L = 10 * D
STEP = 0.002 * D  # lateral travel of a time step (1 m/s x 2 us)


def _sliding_floor(sign, amplitude_d, mu):
    """9 x 9 spheres pressed on the mesh by a strong gravity, the outer rows
    0.03 and 0.05 diameters before the seams they move towards."""
    sc = scenarios.triangle_floor(n=81, l_d=10.0, amplitude_d=amplitude_d, vstd=0.0, drop_d=0.0)
    g = 2000.0
    sc.instance = dataclasses.replace(sc.instance, gravity=(0, 0, -g))
    sc.species = [scenarios.linear_sliding_species(1e-4, 0.8, 1.0 / sc.inv_mass[0], mu)]
    edge = sc.position.max(0) if sign > 0 else sc.position.min(0)
    seam = L if sign > 0 else 0.0
    sc.position[:, 0] += seam - sign * 0.03 * D - edge[0]
    sc.position[:, 1] += seam - sign * 0.05 * D - edge[1]
    # on the mesh, a little deeper than at rest, so that the first step lifts them
    reach = sc.radius[0] - 1.2 * g / (sc.inv_mass[0] * sc.species[0].stiffness)
    corners = [[np.array(w.faces[k][:3]) for k in range(3)] for w in sc.walls]
    lo, hi = np.zeros(sc.n), np.full(sc.n, 2 * D)
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        x = np.column_stack([sc.position[:, :2], mid])
        free = np.min([cases.point_triangle_distance(x, *t) for t in corners], axis=0) > reach
        lo, hi = np.where(free, lo, mid), np.where(free, mid, hi)
    sc.position[:, 2] = hi
    sc.velocity[:, 0], sc.velocity[:, 1], sc.velocity[:, 2] = sign * 1.0, sign * 0.8, 0.0
    return sc


def _per_particle(c, n, key):
    out = np.zeros((n,) + c[key].shape[1:])
    np.add.at(out, c["id_p"], c[key])
    return out


@pytest.mark.parametrize("sign", [1, -1])
def test_flat_mesh_across_the_seams_is_an_infinite_wall(gpu, sign):
    sc = _sliding_floor(sign, 0.0, 0.0)
    flat = dataclasses.replace(sc, walls=[infinite_wall((0, 0, -1), (0, 0, 0))])
    for steps in (0, 10, 17, 20, 35, 70, 110):
        g, o = H.run_gpu(sc, steps), H.run_oracle(flat, steps)
        assert (o["contacts"]["is_wall"] == 1).all() and len(o["contacts"]["id_p"]) == sc.n
        # one triangle each, whichever it is
        assert sorted(g["contacts"]["id_p"].tolist()) == sorted(o["contacts"]["id_p"].tolist()), steps
        # 110 steps of rounding on coordinates of 10 diameters: 1.2e-13 of a diameter
        assert H.rel_err(g["position"], o["position"], D) < 1e-12, steps
        assert H.rel_err(g["force"], o["force"]) < 1e-9, steps
        f = [_per_particle(x["contacts"], sc.n, "force") for x in (g, o)]
        assert H.rel_err(f[0], f[1]) < 1e-9, steps
        if steps in (20, 35):
            assert g["stats"]["rebuilds"] == 1, "the crossing is meant to fall between two rebuilds"
            wrapped = np.abs(g["position"][:, :2] - sc.position[:, :2]).max(1) > 0.5 * L
            assert wrapped.sum() >= 9


@pytest.mark.parametrize("sign", [1, -1])
def test_mesh_in_relief_across_the_seams_at_any_rebuild_interval(gpu, sign):
    """Grouped triangles with friction: contacts, springs and forces of a run
    whose crossings fall between rebuilds are those of one that rebuilds every
    few steps."""
    sc = _sliding_floor(sign, 0.3, 0.5)
    for steps in (17, 20, 45, 110):
        g, r = H.run_gpu(sc, steps), H.run_gpu(sc, steps, skin=6.5 * STEP)
        assert r["stats"]["rebuilds"] > 2 * g["stats"]["rebuilds"]
        assert H.pair_set(g["contacts"]) == H.pair_set(r["contacts"]), steps
        for k in ("position", "velocity", "force", "torque"):
            np.testing.assert_array_equal(g[k], r[k], err_msg=f"{k} at {steps}")
        for k in ("overlap", "springs"):
            np.testing.assert_array_equal(g["contacts"][k], r["contacts"][k], err_msg=f"{k} at {steps}")


def _wall(kind, slow):
    near = 0.47 * D  # its side: 0.03 diameters into a sphere at the lower seam
    v = (-0.5, 0, 0) if slow else (0, 0, 0)
    if kind == "block":
        return intersection_wall([((1, 0, 0), (near, 0, 0)), ((-1, 0, 0), (4 * D, 0, 0)), ((0, 0, -1), (0, 0, 0))],
                                 velocity=v)
    if kind == "disk":
        return axisymmetric_wall((0, 0, 1), [((-1, 0, 0), (2 * D, 0, 0)), ((0, 0, -1), (0, 0, 0))],
                                 position=(near + 2 * D, L / 2, 0), velocity=v)
    return infinite_wall((-1, 0, -0.02), (-0.47 * D, 0, 0), velocity=v)  # leans over the lower seam


@pytest.mark.parametrize("slow", [False, True])
@pytest.mark.parametrize("kind", ["block", "disk", "plane"])
def test_finite_walls_across_a_seam(gpu, kind, slow):
    """A standing or slowly translating wall behind the lower x seam, spheres
    coming over the upper one at several heights: its faces and edges."""
    sc = scenarios.triangle_floor(n=27, l_d=10.0, amplitude_d=0.0, vstd=0.0)
    sc.walls = [_wall(kind, slow)]
    j = np.arange(27)
    sc.position[:, 0] = L - (0.03 + 0.001 * (j % 9)) * D
    sc.position[:, 1] = (0.6 + 1.09 * (j % 9)) * D
    sc.position[:, 2] = (-2.2 + 0.07 * (j % 9) + 1.2 * (j // 9)) * D
    sc.velocity[:] = (1.0, 0.1, 0.05)
    sc.instance = dataclasses.replace(sc.instance, gravity=(0, 0, 0), domain_min=(0, 0, -4 * D), domain_max=(L, L, 4 * D))
    seen = 0
    for steps in (0, 14, 17, 20, 30, 45, 80):
        g, o = H.run_gpu(sc, steps), H.run_oracle(sc, steps)
        assert H.pair_set(g["contacts"]) == H.pair_set(o["contacts"]), steps
        assert H.rel_err(g["position"], o["position"], D) < 1e-12, steps
        assert H.rel_err(g["force"], o["force"]) < 1e-9, steps
        assert H.rel_err(g["contacts"]["springs"], o["contacts"]["springs"]) < 1e-9, steps
        if steps in (20, 30):
            assert g["stats"]["rebuilds"] == 1
        seen += int((o["contacts"]["is_wall"] == 1).sum())
    assert seen > 5
