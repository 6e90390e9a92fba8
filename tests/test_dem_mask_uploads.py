"""When a Dirichlet mask goes to a context: at once, and again whenever its array can have changed.
The context is a stand-in that keeps what it is given."""
import copy
import ctypes
import pickle

import numpy as np
import pytest

from topomax_gb300 import dem
from topomax_gb300.designs import ElasticityParameters, Side

MESH = dem.Mesh(5, 3, 2.0, 1.0)
SIZE = 2 * 6 * 4


class _Context:
    def __init__(self):
        self.ptr, self.mask_version, self.mask_uploads, self.lib = None, None, 0, self

    def check(self, rc):
        assert rc == 0

    def topo_dem_set_mask(self, _, address):
        self.held = np.ctypeslib.as_array(ctypes.cast(address, ctypes.POINTER(ctypes.c_float)), (SIZE,)).copy()
        return 0

    def uses(self, enf):
        enf._install(self)
        return np.array_equal(self.held, enf._mask.ravel()[:SIZE])


def _enforcer(device, side=Side.LEFT):
    return dem.ElasticityEnforcer(ElasticityParameters(
        fixed_sides=[side], body_force=None, tractions=None, filter_radius=0.05, young_modulus=1.0,
        poisson_ratio=0.3), MESH, device=device)


def test_a_private_mask_is_uploaded_once():
    c, a, b = _Context(), _enforcer("meta"), _enforcer("meta", Side.TOP)
    for k, enf in enumerate((a, a, b, b, a)):
        assert c.uses(enf) and c.mask_uploads == (1, 1, 2, 2, 3)[k]


def test_mask_host_can_be_replaced():
    c, enf = _Context(), _enforcer("meta")
    assert c.uses(enf)
    new = np.linspace(0.0, 1.0, SIZE, dtype=np.float32).reshape(-1, 2)
    enf.mask_host = new
    assert c.uses(enf) and np.array_equal(c.held, new.ravel())
    new[3] = 7.0  # the array stays its owner's
    assert c.uses(enf) and c.held[6] == 7.0
    enf.mask_host = new.astype(np.float64).T[::-1].T
    assert c.uses(enf) and np.array_equal(c.held, new[:, ::-1].ravel())
    with pytest.raises(ValueError):
        enf.mask_host = new[:-1]


def test_writes_through_a_cpu_tensor_take_effect():
    c, enf = _Context(), _enforcer("cpu")
    for v in (0.25, 0.5):
        assert c.uses(enf)
        enf.zero_enforcer[1, 0] = v
    assert c.uses(enf) and c.held[2] == 0.5


def test_shallow_copies_share_the_array_and_its_state():
    c, enf = _Context(), _enforcer("meta")
    twin = copy.copy(enf)
    assert c.uses(twin) and c.uses(enf) and c.mask_uploads == 1
    enf.mask_host[0] = 3.0
    assert c.uses(twin) and c.held[0] == 3.0


@pytest.mark.parametrize("duplicate", [copy.deepcopy, lambda e: pickle.loads(pickle.dumps(e))])
def test_separate_copies_have_masks_of_their_own(duplicate):
    c, enf = _Context(), _enforcer("meta")
    assert c.uses(enf)
    enf._dem = None
    other = duplicate(enf)
    other.mask_host[0] = 3.0
    assert c.uses(other) and c.held[0] == 3.0 and c.uses(enf) and c.held[0] != 3.0
    third = duplicate(enf)
    third._mask = third._mask + 1.0  # contents that differ under a number of their own
    assert c.uses(third)
