"""The C record of a tube (Tube.to_c) takes and refuses the values that
assignment to the fields of a kaos_tube_c does."""
import ctypes as C

import numpy as np
import pytest

from kaos_b200 import grids
from kaos_b200.model_input import KaosTube


def _tube():
    return grids.config_small(n_particles=200)[2]


@pytest.mark.parametrize("name,value", [("pG", None), ("sumdsICR", "x"), ("nq", 6.0),
                                        ("capacity", 10.5)])
def test_record_refuses(name, value):
    t = _tube()
    setattr(t, name, value)
    with pytest.raises((TypeError, ValueError)):
        t.to_c()


@pytest.mark.parametrize("value", [np.float32(2.5), 2, np.float64(2.5), "2.5", True])
def test_record_takes(value):
    t = _tube()
    t.pG = t.ms = value
    t.nq = np.int64(t.nq)
    c = t.to_c()
    assert c.pG == float(value) and c.ms == float(value) and c.nq == t.nq
    assert C.sizeof(c) == C.sizeof(KaosTube)
