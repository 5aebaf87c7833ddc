"""After a call that the device has no memory for, the handle goes on: the
failure is that call's own status and not the next one's."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu


def test_calls_after_a_stack_that_does_not_fit():
    from cudamultislice_b200 import ManagedMultisliceSimulation, MultisliceError, build

    build.build(verbose=False)
    n = 2048
    s = ManagedMultisliceSimulation()
    s.SetAtoms(np.full(2, 6, np.int32), np.float32([20, 30]), np.float32([20, 30]), np.float32([0, 40]))
    s.UploadBinnedAtoms()
    s.GetParameterisation(FPARAMS)
    s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
    s.SetCalculationVariables(0.03, -500.0, n, n, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 2.0, 2.0)
    s.PreCalculateFrequencies()
    s.InitialiseWavefunctions(2.0)
    s.RunConventional()
    wave = s.ExitWave()
    s.InitialiseWavefunctions(0.002)  # 22,000 slices of 16 MB: 370 GB
    with pytest.raises(MultisliceError) as e:
        s.BuildPotentialStack()
    assert e.value.code == 5
    s.InitialiseWavefunctions(2.0)
    s.RunConventional()
    assert np.array_equal(s.ExitWave(), wave)
    s.close()
