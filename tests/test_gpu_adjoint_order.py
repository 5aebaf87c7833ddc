"""The position adjoint after potentials that are still queued.

A step past the resident stack builds its potential, and its atom tables, on
the handle's stream without waiting.  A gradient asked for behind a queue of
such steps, with targets in pinned memory (the upload does not wait either),
writes its own tables on another stream: it must come out as with an idle
handle.  The gradient's sums are FP64 atomics, equal to the last bits."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu


def test_gradient_behind_queued_single_slices():
    import torch

    from cudamultislice_b200 import ManagedMultisliceSimulation, build, structures

    build.build(verbose=False)
    Z, x, y, z = structures.srtio3(6, 6, 2)
    n, dz = 256, 0.5
    s = ManagedMultisliceSimulation()
    s.SetAtoms(Z, x, y, z)
    s.UploadBinnedAtoms()
    s.GetParameterisation(FPARAMS)
    s.ApplyMicroscopeParameters(200.0, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
    s.SetCalculationVariables(0.1, -500.0, n, n, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 2.0, 2.0)
    s.PreCalculateFrequencies()
    s.InitialiseWavefunctions(dz)
    S = s.RunConventional()
    defoci = np.array([-400.0, 300.0], np.float32)
    T = torch.from_numpy((np.random.default_rng(1).random((2, n, n)) * 0.5 + 0.75).astype(np.float32)).pin_memory().numpy()
    loss, _, ref = s.FocalSeriesGrad(defoci, T, S, want_v=False)
    for _ in range(400):
        s.MultisliceStepConventional(S + 1)
    again, _, gxy = s.FocalSeriesGrad(defoci, T, S, want_v=False)
    assert again == pytest.approx(loss, rel=1e-12)
    assert np.linalg.norm(gxy - ref) < 1e-9 * np.linalg.norm(ref)
    s.close()
