"""Potentials of grids whose pixels lie so far apart that a distance squared
overflows FP32: atoms out of reach add nothing, not infinity times zero.  Every
potential sum gives the term-by-term one's values (1e-6: the sums' agreement on
the one pixel in reach)."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ps", [1e15, 1e19, 1e30, 3e37])
def test_pixels_past_the_range_of_a_square(ps):
    from cudamultislice_b200 import ManagedMultisliceSimulation, build

    build.build(verbose=False)
    V = {}
    for mode in (0, 1, 2):
        s = ManagedMultisliceSimulation()
        s.SetAtoms(np.full(30, 14, np.int32), *(np.linspace(0, 3, 30, dtype=np.float32),) * 3)
        s.UploadBinnedAtoms()
        s.GetParameterisation(FPARAMS)
        s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
        s.SetCalculationVariables(ps, -500.0, 64, 64, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 2.0, 2.0)
        s.PreCalculateFrequencies()
        s.InitialiseWavefunctions(2.0)
        s.SetPotentialSum(mode)
        S = s.BuildPotentialStack()
        V[mode] = [s.PotentialSlice(0, it) for it in range(1, S + 1)]
        s.close()
    assert max(v.max() for v in V[1]) > 100.0
    for mode in (0, 2):
        for v, ref in zip(V[mode], V[1]):
            assert np.allclose(v, ref, rtol=1e-6, atol=1e-3), mode
