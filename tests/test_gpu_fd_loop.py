"""The finite-difference loop (one persistent launch for all steps) against the
per-pass form and the plain path, on every grid it is provided for: one step,
two, an odd count, and single steps and a second run that go on from the state
it leaves.  Both forms are FP32 transforms of the same recursion; the plain path
is held to 5e-5 of FP64 after 40 steps, so the three agree to 1e-4 here."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu
TOL = 1e-4


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n,steps", [(256, 1), (256, 7), (512, 2), (512, 9), (1024, 1), (1024, 5)])
def test_fd_loop(n, steps):
    from cudamultislice_b200 import ManagedMultisliceSimulation, build

    build.build(verbose=False)
    rng = np.random.default_rng(2)
    m = 60
    Z = rng.choice([6, 14, 38], m).astype(np.int32)
    x, y, z = ((rng.random(m) * s).astype(np.float32) for s in (8.0, 8.0, 8.0))
    runs = []
    for mode in ("loop", "passes", "plain"):
        s = ManagedMultisliceSimulation()
        s.SetSliceLoop(mode == "loop")
        s.SetSlicePath(1 if mode == "plain" else 0)
        s.SetAtoms(Z, x, y, z)
        s.UploadBinnedAtoms()
        s.GetParameterisation(FPARAMS)
        s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
        s.SetCalculationVariables(0.05, -500.0, n, n, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 0.0, 0.0)
        s.PreCalculateFrequencies()
        s.SetFDdz(0.5)
        s.InitialiseWavefunctions(2.0)
        l0 = s.LaunchCount()
        assert s.RunFD(steps) == steps
        waves = [s.ExitWave()]
        s.MultisliceStepFD(steps + 1)  # single steps go on from the state
        s.MultisliceStepFD(steps + 2)
        waves.append(s.ExitWave())
        s.RunFD(steps)  # and a run from there (its own planes 1..steps)
        waves.append(s.ExitWave())
        s.InitialiseWavefunctions(2.0)
        s.RunFD(steps)
        again = s.ExitWave()
        assert np.array_equal(again, waves[0]) or mode == "plain"
        runs.append(waves)
        s.close()
    for other in runs[1:]:
        for a, b in zip(runs[0], other):
            assert rel(a, b) < TOL
