"""The separable potential where the cut-off is a tie: pixels at which
fl(fl(dx^2 + dy^2) + dz^2) of an atom and sub-plane is 5 or the number below it
only by the rounding of each operation.  A sum formed with one rounding less
includes or leaves out such a plane, worth its value at sqrt(5) A (at least 3e-6
of the slice's maximum here); everything else agrees with FP64 to 8e-7 of the
maximum.  About one pixel in a million ties, so many slices are compared."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,Z,n,ps,dz", [
    ("carbon", [6], 256, 0.05, 2.0), ("oxide", [8, 22, 38], 384, 0.03, 1.2), ("nitride", [7, 31], 256, 0.05, 2.0)])
def test_planes_at_the_cutoff(oracle_mod, name, Z, n, ps, dz):
    from cudamultislice_b200 import ManagedMultisliceSimulation, build

    build.build(verbose=False)
    wrong = []
    for seed in range(4):
        rng = np.random.default_rng(seed)
        m = int(0.08 * (n * ps) ** 2 * 16.0)
        species = rng.choice(Z, m).astype(np.int32)
        x, y, z = ((rng.random(m) * s).astype(np.float32) for s in (n * ps, n * ps, 16.0))
        eng, orc = ManagedMultisliceSimulation(), oracle_mod.OracleSimulation()
        for s in (eng, orc):
            s.SetAtoms(species, x, y, z)
            s.UploadBinnedAtoms()
            s.GetParameterisation(FPARAMS)
            s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
            s.SetCalculationVariables(ps, -500.0, n, n, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 2.0, 2.0)
            s.PreCalculateFrequencies()
            s.InitialiseWavefunctions(dz)
        eng.SetPotentialSum(2)
        for it in range(1, eng.GetSlices(True) + 1):
            ref = orc.PotentialConventional(it)
            off = np.abs(eng.PotentialSlice(0, it) - ref)
            wrong += [(seed, it, int(p), float(off.flat[p])) for p in np.flatnonzero(off > 1.5e-6 * ref.max())]
        eng.close()
        orc.close()
    assert not wrong, wrong
