"""Exit-wave error of crystals, whose slices repeat and add up rounding that is
the same in every slice, on grids of several sizes and pixel sizes.

The limit is half an FP32 ulp a slice, all of one sign: S 2^-25, 1.5e-6 for
52 slices.  Unit factors whose modulus or angle is off systematically exceed
it."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ps", [(128, 0.045), (256, 0.03), (256, 0.045)])
def test_crystal_wave_error(oracle_mod, n, ps):
    from cudamultislice_b200 import ManagedMultisliceSimulation, build, structures

    build.build(verbose=False)
    cells = max(1, round(n * ps / 3.905))
    Z, *pos = structures.srtio3(cells, cells, 25)
    rng = np.random.default_rng(2)
    pos = [(a + rng.normal(0.0, 0.08, a.size)).astype(np.float32) for a in pos]
    eng, orc = ManagedMultisliceSimulation(), oracle_mod.OracleSimulation()
    for s in (eng, orc):
        s.SetAtoms(Z, *pos)
        s.UploadBinnedAtoms()
        s.GetParameterisation(FPARAMS)
        s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1.2e7, 0.1, 30.0, 20.0)
        s.SetCalculationVariables(ps, -500.0, n, n, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 2.0, 2.0)
        s.PreCalculateFrequencies()
        s.InitialiseWavefunctions(1.9525)
    ref = orc.run_conventional()
    S = eng.GetSlices(True)
    for loop in (True, False):
        eng.SetSliceLoop(loop)
        eng.RunConventional()
        eng.RunConventional()
        e = np.linalg.norm(eng.ExitWave().astype(np.complex128) - ref) / np.linalg.norm(ref)
        print(n, ps, loop, S, f"{e:.3e}")
        assert e < S * 2.0 ** -25
    eng.close()
    orc.close()
