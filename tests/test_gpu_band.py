"""The fused passes' band-limited states against the plain path.

Between fused passes only the propagator's band of frequency columns is stored;
the rest of the buffers keeps whatever was there.  Read-outs in the middle of a
run (image, diffraction accumulation, exit wave) and the steps that follow must
see zeros there, on the smallest grid, strips and the two-column staged pass.
Each path is within 1e-5 of FP64, so the two within 2e-5 of each other."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu
TOL = 2e-5


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("nx,ny,plan", [(64, 64, -1), (64, 128, 0), (256, 64, 5), (64, 2048, 1)])
def test_readouts_between_steps(nx, ny, plan):
    from cudamultislice_b200 import ManagedMultisliceSimulation, build

    build.build(verbose=False)
    rng = np.random.default_rng(3)
    n = 60
    Z = rng.choice([6, 14, 38], n).astype(np.int32)
    x, y, z = ((rng.random(n) * s).astype(np.float32) for s in (6.0, 6.0, 9.0))
    out = []
    for path in (0, 1):
        s = ManagedMultisliceSimulation()
        s.SetSlicePath(path)
        s.SetFFTPlan(plan)
        s.SetAtoms(Z, x, y, z)
        s.UploadBinnedAtoms()
        s.GetParameterisation(FPARAMS)
        s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
        s.SetCalculationVariables(0.1, -500.0, nx, ny, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 2.0, 2.0)
        s.PreCalculateFrequencies()
        s.InitialiseWavefunctions(2.0)
        s.AllocTDS()
        got = []
        for i in range(1, s.GetSlices(True) + 1):
            s.MultisliceStepConventional(i)
            if i == 2:  # from the row-frequency state
                s.SimulateImage()
                s.AddTDSWaves()
                got += [s.Image(), s.SimulateImageSeries([-300.0, 200.0])]
            if i == 3:  # real space, then the steps go on from it
                got.append(s.ExitWave())
                s.SimulateImage()
                s.AddTDSWaves()
                got.append(s.Image())
        got += [s.TDS(), s.ExitWave()]
        out.append(got)
        s.close()
    for a, b in zip(*out):
        assert rel(a, b) < TOL
