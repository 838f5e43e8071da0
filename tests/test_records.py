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
