"""Position adjoint of slices at and beyond the box's lower end.

The last conventional slice can begin up to one slice thickness above the
bottom of the box and its sub-planes then lie below it: with thick slices its
z-bin window holds no bin at all.  Such a slice adds nothing to dL/dxy; the
others are the oracle's, to the gradient tolerance of test_gpu_adjoint.py."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu
GRAD_TOL = 1e-4


def rel_l2(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


# windows past the bins by three, by one, exactly at their end, and not empty
@pytest.mark.parametrize("depth,dz", [(2.0, 5.0), (1.0, 4.9), (0.2, 4.1), (5.0, 4.9)])
@pytest.mark.parametrize("potential_sum", [1, 2])
def test_gradient_with_empty_last_window(oracle_mod, depth, dz, potential_sum):
    from cudamultislice_b200 import ManagedMultisliceSimulation, build

    build.build(verbose=False)
    rng = np.random.default_rng(23)
    m = 24
    Z = rng.choice([8, 22, 38], m).astype(np.int32)
    x, y, z = ((rng.random(m) * s).astype(np.float32) for s in (6.0, 6.0, depth))
    z[:2] = 0.0, depth
    eng, orc = ManagedMultisliceSimulation(), oracle_mod.OracleSimulation()
    for s in (eng, orc):
        s.SetAtoms(Z, x, y, z)
        s.UploadBinnedAtoms()
        s.GetParameterisation(FPARAMS)
        s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
        s.SetCalculationVariables(0.1, -500.0, 64, 64, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 2.0, 2.0)
        s.PreCalculateFrequencies()
        s.InitialiseWavefunctions(dz)
    S = orc.GetSlices(True)
    assert eng.GetSlices(True) == S == 2
    defoci = np.array([-400.0, 300.0], np.float32)
    T = (np.random.default_rng(1).random((2, 64, 64)) * 0.5 + 0.75).astype(np.float32)
    L0, gV0, gxy0 = orc.FocalGrad(defoci, T.astype(np.float64), S)
    eng.SetPotentialSum(potential_sum)
    for want_v in (True, False):
        L, gV, gxy = eng.FocalSeriesGrad(defoci, T, S, want_v=want_v)
        assert abs(L - L0) / L0 < 1e-5
        assert rel_l2(gxy, gxy0) < GRAD_TOL
    eng.close()
    orc.close()
