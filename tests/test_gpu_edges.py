"""Sizes and values at which the kernels' special paths can go wrong, against the oracle.

EXACT float must equal the oracle bit for bit: divisors of every kind (a power of two,
one whose reciprocal formula fails its check) at amplitudes down to subnormals, C-PML
strips and array ends off every vector and tile boundary, more sources and receivers than
threads.
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
                                    (12.5, 1e-34)])
@pytest.mark.parametrize("physics", [abi.ACOUSTIC2D, abi.ELASTIC2D])
def test_exact_division(require_gpu, physics, dx, amp):
    # 9.00014782 fails the check of the two-operation quotient and takes the double one throughout
    c = Case2D(physics, nx=57, nz=49, nt=180, dx=dx, scoord=(30.3 * dx, 2.7 * dx))
    c.src.data *= np.float32(amp)
    want = c.oracle_traces()
    assert np.abs(want).max() > 0
    assert np.array_equal(traces(c), want)


@pytest.mark.parametrize("physics", [abi.ACOUSTIC2D, abi.ELASTIC2D])
@pytest.mark.parametrize("nx,nz,lpml,order,fs", [(15, 16, 1, 8, 0), (38, 17, 3, 8, 1), (31, 33, 5, 5, 0), (64, 16, 13, 8, 1),
                                                 (7, 40, 30, 8, 0), (121, 9, 20, 2, 0)])
def test_strips_and_edges_bitwise(require_gpu, physics, nx, nz, lpml, order, fs):
    # strips that start and end off the vectors' boundaries, and tiles that hold both of an axis' ends
    c = Case2D(physics, nx=nx, nz=nz, lpml=lpml, order=order, fs=fs, nt=90, scoord=(10.0 * nx / 2 + 3.3, 23.7),
               rfield=abi.VX if physics == abi.ELASTIC2D else abi.PRESSURE)
    assert np.array_equal(traces(c), c.oracle_traces())


def test_more_points_than_threads(require_gpu):
    # 1200 receivers, and 90 sources of which thirds share a cell (their contributions add in trace order)
    sc = np.array([(100.0 + 7.3 * (k // 3), 31.7) for k in range(90)])
    c = Case2D(abi.ACOUSTIC2D, nx=121, nz=41, nt=70, scoord=sc, nrec=1200, rdx=0.97)
    c.src.data *= np.linspace(0.5, 1.5, len(sc), dtype=np.float32)[:, None]
    assert np.array_equal(traces(c), c.oracle_traces())
