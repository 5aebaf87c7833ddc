"""Potential stacks built in groups of slices against one slice at a time.

The separable kernels take several consecutive slices (and instances) per
launch; a step loop without a resident stack builds each slice by itself.  Both
sum the same terms in the same order, so with one FFT plan the exit waves must
be bit-identical, whatever the group boundaries, tile remainders or grid."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine_cls():
    from cudamultislice_b200 import ManagedMultisliceSimulation, build

    build.build(verbose=False)
    return ManagedMultisliceSimulation


# slices: one, around six groups (1, 5, 6, 7), uneven last groups, more than
# sixteen slices a group; grids: square, strip, remainders against every tile
@pytest.mark.parametrize("depth,dz,nx,ny,tile", [
    (0.0, 5.0, 64, 64, -1), (4.0, 1.9, 64, 128, -1), (7.0, 2.0, 64, 64, 3), (9.0, 1.9, 128, 64, 1),
    (14.0, 0.9, 70, 45, -1), (14.0, 1.3, 33, 67, 0), (11.0, 0.12, 64, 64, 2), (8.0, 0.12, 45, 50, -1)])
def test_stack_groups_match_single_slices(engine_cls, depth, dz, nx, ny, tile):
    rng = np.random.default_rng(17)
    n = 150
    Z = rng.choice([6, 8, 22, 38], n).astype(np.int32)
    x, y, z = ((rng.random(n) * s).astype(np.float32) for s in (9.0, 8.0, max(depth, 1e-3)))
    waves = []
    for stack in (True, False):
        s = engine_cls()
        s.SetFFTPlan(0)
        s.SetBuildOverlap(False)
        s.SetAtoms(Z, x, y, z)
        s.UploadBinnedAtoms()
        s.GetParameterisation(FPARAMS)
        s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
        s.SetCalculationVariables(0.11, -500.0, nx, ny, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 2.0, 2.0)
        s.PreCalculateFrequencies()
        s.InitialiseWavefunctions(dz)
        s.SetPotentialTile(tile)
        if stack:
            S = s.RunConventional()
        else:
            S = s.GetSlices(True)
            for i in range(1, S + 1):
                s.MultisliceStepConventional(i)
        waves.append(s.ExitWave())
        s.close()
    assert np.abs(waves[0]).max() > 0
    assert np.array_equal(waves[0], waves[1]), S
