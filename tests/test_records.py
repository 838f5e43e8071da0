"""Contact downloads ordered on the device (dem_records.cuh): particle pairs
before wall contacts, each by (id of P, id of I or the caller's wall index),
signed ids included; the geometry in the same order; forces in the caller's
order. Against the oracle's contacts of the same particles under plain ids."""
import dataclasses

import numpy as np
import pytest

import cases
import harness as H
from test_units import _box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, -400, -(1 << 31), (1 << 31) - 1000])
@pytest.mark.parametrize("touches_walls", [False, True])
def test_order_of_contacts_with_any_ids(gpu, offset, touches_walls):
    sc = _box(1000) if touches_walls else cases.compressed_box()
    ids = (np.arange(sc.n) + offset).astype(np.int32)
    o = H.run_oracle(sc, 0)
    e = dataclasses.replace(sc, ids=ids).engine()
    e.step(0)
    c, geo, (f, t) = e.contacts(), e.contact_geometry(), e.forces()
    short = dict(n=e.counts())
    e.close()
    key = np.lexsort((c["id_i"], c["id_p"], c["is_wall"]))
    np.testing.assert_array_equal(key, np.arange(len(key)))
    pairs = c["is_wall"] == 0
    assert pairs.sum() > 1000 and ((~pairs).sum() > 10) == touches_walls
    assert short["n"]["contacts"] == pairs.sum() and short["n"]["wall_contacts"] == (~pairs).sum()
    oc = H.sort_contacts(o["contacts"])
    np.testing.assert_array_equal(c["id_p"], oc["id_p"] + offset)
    np.testing.assert_array_equal(np.where(pairs, c["id_i"] - offset, c["id_i"]), oc["id_i"])
    np.testing.assert_array_equal(c["force"], oc["force"])
    np.testing.assert_array_equal(c["springs"], oc["springs"])
    assert H.rel_err(f, o["force"]) < 1e-14 and H.rel_err(t, o["torque"]) < 1e-14
    # the geometry's rows belong to the contacts' rows: the normal part of the force
    along = np.einsum("ij,ij->i", c["force"] - geo["tangential_force"], geo["normal"])
    np.testing.assert_allclose(along[:, None] * geo["normal"], c["force"] - geo["tangential_force"],
                               atol=1e-12 * np.abs(c["force"]).max())


def test_downloads_on_a_full_device(gpu):
    """Where no workspace is to be had, contacts, geometry and counts are the same
    (sorted on the host), calls that need one say so, and the handle works on."""
    from mercurydpm_fork_b200 import _abi
    from mercurydpm_fork_b200.engine import DemError, lib
    sc = _box(1000)
    e = sc.engine()
    e.step(5)
    box = (0, 0, 0), (0.01, 0.01, 0.01)
    want = e.contacts(), e.contact_geometry(), e.counts(), e.reduce(), e.cg(_abi.DEM_CG_O, (1, 1, 1), *box, 1e-3)
    assert lib().dem_selftest_workspace_limit(e._h, 0) == 0
    got = e.contacts(), e.contact_geometry(), e.counts()
    for a, b in zip(got[:2], want[:2]):
        assert a.keys() == b.keys()
        for k in a:
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    assert got[2] == want[2]
    for call in (e.reduce, lambda: e.cg(_abi.DEM_CG_O, (1, 1, 1), *box, 1e-3)):
        with pytest.raises(DemError) as err:
            call()
        assert err.value.code == _abi.DEM_ERR_CUDA
    e.step(5)
    after = e.contacts()
    assert lib().dem_selftest_workspace_limit(e._h, (1 << 64) - 1) == 0
    for k, v in e.contacts().items():
        np.testing.assert_array_equal(after[k], v, err_msg=k)
    assert e.reduce()["n_contacts"] == (after["is_wall"] == 0).sum()
    e.close()


def test_kept_workspace_is_reported_and_given_back(gpu):
    """The workspace of a simulation counts in memory() and goes with its arrays."""
    big, small = _box(2777), _box(130)
    small = dataclasses.replace(small, instance=big.instance, walls=big.walls)  # the same domain: the same cells
    sizes = lambda sc: (sc.position, sc.velocity, sc.radius, sc.inv_mass, sc.inv_inertia, sc.species_index, sc.ids)
    fresh = small.engine()
    e = big.engine()
    held = e.memory()["device_bytes"]
    e.step(0)
    e.contacts()
    assert e.memory()["device_bytes"] > held
    e.upload(*sizes(small))
    assert e.memory()["device_bytes"] == fresh.memory()["device_bytes"]
    e.step(3)
    fresh.step(3)
    np.testing.assert_array_equal(e.download()["position"], fresh.download()["position"])
    e.close()
    fresh.close()
