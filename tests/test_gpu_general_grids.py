"""Conventional slices of grids that are no power of two: the mixed-radix passes
against the plain path (cuFFT) and the FP64 oracle.

Each length exercises other radices (every radix alone and in products, one
pass and many, columns per CTA 2, 4 and 8, the largest length); a length with a
prime factor above 13 takes the plain path.  FP32 transforms of a few slices
are well within the 1e-5 parity tolerance of FP64."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu
TOL = 1e-5


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def setup(s, atoms, nx, ny, ps, dz=2.0):
    Z, x, y, z = atoms
    s.SetAtoms(Z, x, y, z)
    s.UploadBinnedAtoms()
    s.GetParameterisation(FPARAMS)
    s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
    s.SetCalculationVariables(ps, -500.0, nx, ny, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 2.0, 2.0)
    s.PreCalculateFrequencies()
    s.InitialiseWavefunctions(dz)


@pytest.fixture(scope="module")
def engine_cls():
    from cudamultislice_b200 import ManagedMultisliceSimulation, build

    build.build(verbose=False)
    return ManagedMultisliceSimulation


def random_specimen(n=80):
    rng = np.random.default_rng(11)
    return (rng.choice([6, 14, 38], n).astype(np.int32),
            *((rng.random(n) * s).astype(np.float32) for s in (7.0, 6.0, 9.0)))


@pytest.mark.parametrize("nx,ny", [
    (9, 12), (13, 11), (16, 24), (15, 14), (26, 33), (70, 45), (77, 91), (96, 100), (121, 169), (243, 210), (125, 343),
    (600, 450), (512, 513), (1023, 99), (384, 1296), (2187, 30), (36, 3072), (4095, 16), (74, 90), (64, 97)])
def test_mixed_radix_slices(engine_cls, oracle_mod, nx, ny):
    atoms, ps = random_specimen(), 0.12
    eng, orc = engine_cls(), oracle_mod.OracleSimulation()
    for s in (eng, orc):
        setup(s, atoms, nx, ny, ps)
    ref = orc.run_conventional()
    S = eng.RunConventional()  # beside the stack's build
    waves = [eng.ExitWave()]
    eng.RunConventional()  # over the resident stack
    waves.append(eng.ExitWave())
    for i in range(1, S + 1):  # step by step, with a read-out between
        eng.MultisliceStepConventional(i)
        if i == 2:
            eng.GetExitWave()
    waves.append(eng.ExitWave())
    eng.SetSlicePath(1)
    eng.RunConventional()
    plain = eng.ExitWave()
    for w in waves:
        assert rel(w, ref) < TOL and rel(w, plain) < TOL
    eng.close()
    orc.close()
