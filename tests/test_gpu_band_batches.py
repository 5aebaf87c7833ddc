"""Batched slice passes that skip the band's zero butterflies against the plain
path: rasters (stored transmission, many instances) and one-by-one steps on the
line lengths and plans that take that form and on a neighbour that does not.

The signals are sums of |FFT psi|^2 over a detector: either path's waves are
within 1e-5 of FP64, so a signal is within 2 x 1e-5 of it and the two within
4e-5 of each other; waves within 2e-5."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,plan", [
    (64, 64, 0), (128, 256, 1), (256, 128, 2), (256, 256, 4), (512, 256, 0), (256, 512, 0), (512, 512, 0), (512, 512, 3),
    (512, 1024, 0), (1024, 64, 0), (128, 64, -1)])
def test_raster_and_steps(nx, ny, plan):
    from cudamultislice_b200 import ManagedMultisliceSimulation, build

    build.build(verbose=False)
    rng = np.random.default_rng(5)
    n, ps = 80, 0.08
    Z = rng.choice([6, 14, 38], n).astype(np.int32)
    x, y, z = ((rng.random(n) * s).astype(np.float32) for s in (nx * ps, ny * ps, 7.0))
    px = rng.integers(0, nx, 9).astype(np.int32)
    py = rng.integers(0, ny, 9).astype(np.int32)
    sig, waves = [], []
    for path in (0, 1):
        for stem in (True, False):
            s = ManagedMultisliceSimulation()
            s.SetSlicePath(path)
            s.SetFFTPlan(plan)
            s.SetAtoms(Z, x, y, z)
            s.UploadBinnedAtoms()
            s.GetParameterisation(FPARAMS)
            if stem:
                s.ApplyMicroscopeParameters(200.0, 0.0, 0.0, 0.0, 0.0, 0.1, 30.0, 25.0)
                s.STEMSetCalculationVariables(ps, 0.0, nx, ny, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ())
                s.PreCalculateFrequencies()
                s.STEMInitialiseWavefunctions(0, 0)
                sig.append(s.StemRaster(px, py, 5.0, 60.0, batch=8))
            else:
                s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
                s.SetCalculationVariables(ps, -500.0, nx, ny, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 2.0, 2.0)
                s.PreCalculateFrequencies()
                s.InitialiseWavefunctions(2.0)
                for i in range(1, s.GetSlices(True) + 1):
                    s.MultisliceStepConventional(i)
                waves.append(s.ExitWave())
            s.close()
    assert sig[0].min() > 0
    assert np.abs(sig[0] - sig[1]).max() < 4e-5 * np.abs(sig[1]).max()
    assert np.linalg.norm(waves[0] - waves[1]) < 2e-5 * np.linalg.norm(waves[1])
