"""Sizes and values at which the kernels' special paths can go wrong, against the oracle.

EXACT float must equal the oracle bit for bit: divisors of every kind (a power of two,
one whose reciprocal formula fails its check) at amplitudes down to subnormals, C-PML
strips and array ends off every vector and tile boundary, more sources and receivers than
threads, z-chunks of every remainder.  FAST must lie within float rounding of the oracle at
the same sizes, and no tile or z-chunk may change a bit of it.  The elastic 3D float
kernels, which the oracle does not cover, are held to the FP64 propagator's other kernels.
"""
import numpy as np
import pytest

from rockseis_b200 import abi, synth
from rockseis_b200.rockseis import Data3D, ModelElastic3D, ModellingAcoustic2D, ModellingElastic2D, Plan
from tests.cases import Case2D, rel_l2
from tests.test_gpu_modelling_3d import Case3D

pytestmark = pytest.mark.gpu


# FAST against the oracle: float sums in another order and with fused multiply-adds, some 30
# roundings of 2^-24 a step and point that add up like a random walk over at most 90 steps of
# amplitudes of the traces' own size: sqrt(30 * 90) * 6e-8 = 3e-6 (measured: 1e-7 to 3.4e-7)
FAST_TOL = 3e-6


def traces(c, tile=-1, precision=None):
    cls = ModellingAcoustic2D if c.physics == abi.ACOUSTIC2D else ModellingElastic2D
    mod = cls(c.model, c.src, c.order, 1, precision)
    mod.tile = tile
    c.rec.data[:] = 0
    (mod.setRecP if c.rec.field == abi.PRESSURE else mod.setRecVx)(c.rec)
    assert mod.run() == 1
    return c.rec.data.copy()


@pytest.mark.parametrize("dx,amp", [(10.0, 1.0), (8.0, 1.0), (16.0, 1e-30), (9.00014782, 1.0), (9.00014782, 1e-32),
                                    (7.3, 1e-34), (12.5, 1e-34), (12.5, 1e-38)])
@pytest.mark.parametrize("physics", [abi.ACOUSTIC2D, abi.ELASTIC2D])
def test_exact_division(require_gpu, physics, dx, amp):
    # 9.00014782 fails the check of the two-operation quotient and takes the double one throughout;
    # at 1e-38 every elastic velocity is below the smallest subnormal; 7.3 needs the shorter time step
    c = Case2D(physics, nx=57, nz=49, nt=180, dx=dx, dt=1e-3 if dx >= 8 else 8e-4, scoord=(30.3 * dx, 2.7 * dx))
    c.src.data *= np.float32(amp)
    want = c.oracle_traces()
    assert np.abs(want).max() > 0 or (physics == abi.ELASTIC2D and amp == 1e-38)
    assert np.array_equal(traces(c), want)


# padded grids of more than twice the order: on smaller ones the oracle, like the reference, reads
# outside its arrays
SIZES_2D = [(9, 11, 1, 4, 0), (15, 16, 1, 8, 0), (38, 17, 3, 8, 1), (31, 33, 5, 5, 0), (64, 16, 13, 8, 1), (7, 40, 30, 8, 0),
            (121, 9, 20, 2, 0)]


def strips_case(physics, nx, nz, lpml, order, fs):
    return Case2D(physics, nx=nx, nz=nz, lpml=lpml, order=order, fs=fs, nt=90, scoord=(10.0 * nx / 2 + 3.3, 23.7),
                  rfield=abi.VX if physics == abi.ELASTIC2D else abi.PRESSURE)


@pytest.mark.parametrize("tile", [9, 10])   # the two float defaults: two rows a thread, one row
@pytest.mark.parametrize("physics", [abi.ACOUSTIC2D, abi.ELASTIC2D])
@pytest.mark.parametrize("nx,nz,lpml,order,fs", SIZES_2D)
def test_strips_and_edges_bitwise(require_gpu, physics, nx, nz, lpml, order, fs, tile):
    # strips that start and end off the vectors' boundaries, and tiles that hold both of an axis' ends
    c = strips_case(physics, nx, nz, lpml, order, fs)
    assert np.array_equal(traces(c, tile), c.oracle_traces())


@pytest.mark.parametrize("physics", [abi.ACOUSTIC2D, abi.ELASTIC2D])
@pytest.mark.parametrize("nx,nz,lpml,order,fs", SIZES_2D)
def test_strips_and_edges_fast(require_gpu, physics, nx, nz, lpml, order, fs):
    # streamed z sums and reduced-order rows in place of the exact mode's pairs
    c = strips_case(physics, nx, nz, lpml, order, fs)
    two, one = traces(c, 9, abi.F32_FAST), traces(c, 10, abi.F32_FAST)
    assert np.array_equal(two, one)
    assert rel_l2(two, c.oracle_traces()) <= FAST_TOL


def test_more_points_than_threads(require_gpu):
    # 1200 receivers, and 90 sources of which thirds share a cell (their contributions add in trace order)
    sc = np.array([(100.0 + 7.3 * (k // 3), 31.7) for k in range(90)])
    c = Case2D(abi.ACOUSTIC2D, nx=121, nz=41, nt=70, scoord=sc, nrec=1200, rdx=0.97)
    c.src.data *= np.linspace(0.5, 1.5, len(sc), dtype=np.float32)[:, None]
    assert np.array_equal(traces(c), c.oracle_traces())


SIZES_3D = [(33, 9, 8, 5, 8), (20, 26, 21, 3, 6), (24, 20, 34, 7, 8)]


@pytest.mark.parametrize("zchunk", [0, 1, 2, 3, 16])
@pytest.mark.parametrize("nx,ny,nz,lpml,order", SIZES_3D)
def test_acoustic3d_chunks_and_strips_bitwise(require_gpu, nx, ny, nz, lpml, order, zchunk):
    c = Case3D(nx=nx, ny=ny, nz=nz, lpml=lpml, order=order, nt=60, fs=nz % 2, scoord=(103.3, 41.9, 32.2))
    assert np.array_equal(c.gpu(zchunk=zchunk), c.oracle())


@pytest.mark.parametrize("nx,ny,nz,lpml,order", SIZES_3D)
def test_acoustic3d_chunks_and_strips_fast(require_gpu, nx, ny, nz, lpml, order):
    c = Case3D(nx=nx, ny=ny, nz=nz, lpml=lpml, order=order, nt=60, fs=nz % 2, scoord=(103.3, 41.9, 32.2))
    want = c.gpu(precision=abi.F32_FAST)
    assert rel_l2(want, c.oracle()) <= FAST_TOL
    for zchunk in (1, 2, 3, 16):
        assert np.array_equal(c.gpu(precision=abi.F32_FAST, zchunk=zchunk), want)


def elastic3d(prec, nx, ny, nz, lpml, fs, zchunk=0, order=8, nt=60):
    rng = np.random.default_rng(3)
    m = ModelElastic3D(nx, ny, nz, lpml, 10.0, 10.0, 10.0, 0.0, 0.0, 0.0, fs, prec)
    m.createModel()
    vp = (1800 + 1200 * np.linspace(0, 1, nz)[:, None, None] * rng.uniform(0.9, 1.1, (nz, ny, nx))).astype(np.float32)
    m.Vp[:], m.Vs[:], m.R[:] = vp, vp / np.float32(1.8), 310 * vp.astype(np.float64) ** 0.25
    src = Data3D(1, nt, 1e-3, 0.0, prec)
    src.scoords[:] = [[5.3 * nx, 4.9 * ny, 32.2]]
    src.data[:] = 1e9 * synth.ricker(nt, 1e-3, 25.0)[None, :]
    src.makeMap(m, 0)
    rec = Data3D(12, nt, 1e-3, 0.0, prec)
    rec.gcoords[:] = np.stack([np.linspace(25.0, 10.0 * (nx - 3), 12), np.linspace(15.5, 10.0 * (ny - 3), 12), np.full(12, 14.2)], 1)
    rec.setField(abi.VZ)
    rec.makeMap(m, 1)
    p = Plan([m], [src], [rec], order, prec, zchunk=zchunk)
    p.run()
    return p.read_traces(0).astype(np.float64)


@pytest.mark.parametrize("nx,ny,nz,lpml,fs,order", [(34, 21, 23, 7, 0, 8), (25, 33, 16, 10, 1, 8), (40, 18, 19, 5, 0, 5)])
def test_elastic3d_float_against_fp64(require_gpu, nx, ny, nz, lpml, fs, order):
    # float propagation over 60 steps of 18 derivatives; both float arithmetics were 2e-7 to 2e-6
    # off the FP64 propagator (whose kernels are other ones) at these sizes
    want = elastic3d(abi.F64, nx, ny, nz, lpml, fs, order=order)
    exact = elastic3d(abi.F32_EXACT, nx, ny, nz, lpml, fs, order=order)
    assert rel_l2(exact, want) < 1e-5
    assert rel_l2(elastic3d(abi.F32_FAST, nx, ny, nz, lpml, fs, order=order), want) < 1e-5
    for zchunk in (1, 3, 16):
        assert np.array_equal(elastic3d(abi.F32_EXACT, nx, ny, nz, lpml, fs, zchunk, order), exact)
