"""Sizes and values at which the kernels' special paths can go wrong, against the oracle.

EXACT float must equal the oracle bit for bit: divisors of every kind (a power of two,
one whose reciprocal formula fails its check) at amplitudes down to subnormals.
"""
import numpy as np
import pytest

from rockseis_b200 import abi
from rockseis_b200.rockseis import ModellingAcoustic2D, ModellingElastic2D
from tests.cases import Case2D

pytestmark = pytest.mark.gpu


def traces(c):
    cls = ModellingAcoustic2D if c.physics == abi.ACOUSTIC2D else ModellingElastic2D
    mod = cls(c.model, c.src, c.order, 1)
    (mod.setRecP if c.rec.field == abi.PRESSURE else mod.setRecVx)(c.rec)
    assert mod.run() == 1
    return c.rec.data


@pytest.mark.parametrize("dx,amp", [(10.0, 1.0), (8.0, 1.0), (16.0, 1e-30), (9.00014782, 1.0), (9.00014782, 1e-32),
                                    (7.3, 1e-34), (12.5, 1e-38)])
@pytest.mark.parametrize("physics", [abi.ACOUSTIC2D, abi.ELASTIC2D])
def test_exact_division(require_gpu, physics, dx, amp):
    # 9.00014782 fails the check of the two-operation quotient and takes the double one throughout
    c = Case2D(physics, nx=57, nz=49, nt=180, dx=dx, scoord=(30.3 * dx, 2.7 * dx))
    c.src.data *= np.float32(amp)
    want = c.oracle_traces()
    assert np.abs(want).max() > 0
    assert np.array_equal(traces(c), want)
