"""Read-backs and uploads that go through the pinned chunks, at the sizes where
the split changes: below the threshold, chunk remainders, one chunk more than
the helper threads take at once.  The copies must be exact."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,n", [(64, 64, 3), (300, 217, 9), (512, 512, 2), (512, 520, 9), (1024, 1024, 9)])
def test_image_series_and_targets(nx, ny, n):
    from cudamultislice_b200 import ManagedMultisliceSimulation, build

    build.build(verbose=False)
    rng = np.random.default_rng(5)
    Z = np.full(40, 14, np.int32)
    x, y, z = ((rng.random(40) * s).astype(np.float32) for s in (6.0, 6.0, 3.0))
    s = ManagedMultisliceSimulation()
    s.SetAtoms(Z, x, y, z)
    s.UploadBinnedAtoms()
    s.GetParameterisation(FPARAMS)
    s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
    s.SetCalculationVariables(0.05, -500.0, nx, ny, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 2.0, 2.0)
    s.PreCalculateFrequencies()
    s.InitialiseWavefunctions(2.0)
    S = s.RunConventional()
    df = np.linspace(-600.0, 500.0, n).astype(np.float32)
    together = s.SimulateImageSeries(df)
    for k in range(n):  # one image a call: small copies
        assert np.array_equal(together[k], s.SimulateImageSeries(df[k:k + 1])[0])
    if nx == ny:
        # the uploaded targets: their residual against themselves is exactly zero
        loss, images = s.FocalSeries(df, np.zeros_like(together), S, images=True)
        assert s.FocalSeries(df, images, S) == 0.0 and loss > 0
    s.close()
