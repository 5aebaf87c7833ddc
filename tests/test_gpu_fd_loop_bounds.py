"""The finite-difference loop against FP64, and its bounded waits.

Waves: 1e-5, the engine's accuracy target, after runs of one, some and many
steps on every grid the loop is provided for.  Waits: the hook that makes every
grid barrier expect one arrival too many runs the 20 ms bound out; the call
fails with a status, the handle asks for new waves, and the next run is right."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu
TOL = 1e-5


def pair(oracle_mod, n, ps=0.05):
    from cudamultislice_b200 import ManagedMultisliceSimulation, build

    build.build(verbose=False)
    rng = np.random.default_rng(2)
    m = 60
    Z = rng.choice([6, 14, 38], m).astype(np.int32)
    x, y, z = ((rng.random(m) * s).astype(np.float32) for s in (8.0, 8.0, 8.0))
    both = ManagedMultisliceSimulation(), oracle_mod.OracleSimulation()
    for s in both:
        s.SetAtoms(Z, x, y, z)
        s.UploadBinnedAtoms()
        s.GetParameterisation(FPARAMS)
        s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
        s.SetCalculationVariables(ps, -500.0, n, n, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 0.0, 0.0)
        s.PreCalculateFrequencies()
        s.SetFDdz(0.5)
        s.InitialiseWavefunctions(2.0)
    return both


def rel(a, b):
    return np.linalg.norm(a.astype(np.complex128) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n,steps", [(256, 1), (256, 24), (512, 24), (1024, 3)])
def test_fd_loop_against_the_oracle(oracle_mod, n, steps):
    eng, orc = pair(oracle_mod, n)
    eng.RunFD(1)  # (builds the planes; also from a state the loop left)
    eng.InitialiseWavefunctions(2.0)
    launches = eng.LaunchCount()
    eng.RunFD(steps)
    if steps == 1:
        assert eng.LaunchCount() - launches == 1  # the whole run is one launch
    for it in range(1, steps + 1):
        orc.MultisliceStepFD(it)
    assert rel(eng.ExitWave(), orc.Wave()) < TOL
    eng.close()
    orc.close()


@pytest.mark.parametrize("n", [256, 512, 1024])
def test_fd_loop_wait_bound_ends_the_launch_with_an_error(oracle_mod, n):
    from cudamultislice_b200 import MultisliceError

    eng, orc = pair(oracle_mod, n)
    eng.RunFD(3)
    good = eng.ExitWave()
    eng.InitialiseWavefunctions(2.0)
    eng.SetLoopWaitUs(20000)
    eng.SetLoopWaitTest(1)
    with pytest.raises(MultisliceError) as e:
        eng.RunFD(3)
    assert e.value.code == 3 and "grid-barrier wait ran out" in str(e.value)
    with pytest.raises(MultisliceError):
        eng.ExitWave()
    eng.SetLoopWaitTest(0)
    eng.InitialiseWavefunctions(2.0)
    eng.RunFD(3)
    assert np.array_equal(eng.ExitWave(), good)
    eng.close()
    orc.close()
