"""Focal-series gradients at the checkpoint strides where the segments differ:
a last segment of one slice, of all but one, equal segments and one segment.
Each against the FP64 oracle (the tolerance of test_gpu_adjoint.py) and, as
every stride recomputes the same waves, against the single segment."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu
GRAD_TOL = 1e-4


def rel_l2(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


@pytest.fixture(scope="module")
def case(oracle_mod):
    from cudamultislice_b200 import ManagedMultisliceSimulation, build, structures

    build.build(verbose=False)
    Z, x, y, z = structures.srtio3(2, 2, 3)
    rng = np.random.default_rng(8)
    x, y = ((a + rng.normal(0, 0.05, a.size)).astype(np.float32) for a in (x, y))
    eng, orc = ManagedMultisliceSimulation(), oracle_mod.OracleSimulation()
    for s in (eng, orc):
        s.SetAtoms(Z, x, y, z)
        s.UploadBinnedAtoms()
        s.GetParameterisation(FPARAMS)
        s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
        s.SetCalculationVariables(0.1, -500.0, 64, 64, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 2.0, 2.0)
        s.PreCalculateFrequencies()
        s.InitialiseWavefunctions(1.9525)
    assert eng.GetSlices(True) >= 7
    defoci = np.array([-400.0, 300.0], np.float32)
    T = (np.random.default_rng(1).random((2, 64, 64)) * 0.5 + 0.75).astype(np.float32)
    ref = orc.FocalGrad(defoci, T.astype(np.float64), 7)
    orc.close()
    eng.SetCheckpoint(7)
    yield eng, defoci, T, ref, eng.FocalSeriesGrad(defoci, T, 7)
    eng.close()


@pytest.mark.parametrize("stride", [1, 2, 3, 4, 6, 7])
def test_strides_against_the_oracle(case, stride):
    eng, defoci, T, ref, single = case
    eng.SetCheckpoint(stride)
    L, gV, gxy = eng.FocalSeriesGrad(defoci, T, 7)
    assert abs(L - ref[0]) / ref[0] < 1e-5
    assert rel_l2(gV, ref[1]) < GRAD_TOL and rel_l2(gxy, ref[2]) < GRAD_TOL
    assert rel_l2(gV, single[1]) < 1e-6 and rel_l2(gxy, single[2]) < 1e-6
