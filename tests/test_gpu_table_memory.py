"""Atom tables of the separable potential where they are large.

In a specimen thinner than the z-window every atom has a table row in every
slice.  A frozen-phonon batch of such specimens must not need one buffer for
all of them at once, and a handle without room for its tables takes fewer
buffers, then the per-sub-plane sum.  Smaller parts and fewer buffers are the
same kernels on the same tables (equal up to the order of the image's FP32
sums); the two sums of an atom's sub-planes agree to about 1e-7 of the
potential, far inside the 1e-5 of the waves."""
import numpy as np
import pytest

from tests.conftest import FPARAMS

pytestmark = pytest.mark.gpu


def film(n, side, seed=3):
    rng = np.random.default_rng(seed)
    Z = rng.choice([6, 16, 42], n).astype(np.int32)
    return Z, *((rng.random(n) * s).astype(np.float32) for s in (side, side, 0.5))


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


def handle(atoms, n=64, dz=2.0, kV=200.0):
    from cudamultislice_b200 import ManagedMultisliceSimulation, build

    build.build(verbose=False)
    s = ManagedMultisliceSimulation()
    s.SetAtoms(*atoms)
    s.UploadBinnedAtoms()
    s.GetParameterisation(FPARAMS)
    s.ApplyMicroscopeParameters(kV, -500.0, 0.0, 0.0, 1e7, 0.1, 30.0, 20.0)
    s.SetCalculationVariables(0.1, -500.0, n, n, s.GetSizeX(), s.GetSizeY(), s.GetSizeZ(), 2.0, 2.0)
    s.PreCalculateFrequencies()
    s.InitialiseWavefunctions(dz)
    return s


def test_phonon_batch_of_a_thin_specimen():
    s = handle(film(100_000, 180.0))
    diff, image = s.FrozenPhonon(7, 0, 128, 0.08, batch=128)
    diff8, image8 = s.FrozenPhonon(7, 0, 128, 0.08, batch=8)
    s.close()
    assert rel(diff, diff8) < 1e-5 and rel(image, image8) < 1e-5


@pytest.mark.parametrize("room,potential_sum", [(3.2e9, 2), (1.0e9, 1)])
def test_handle_without_room_for_its_tables(room, potential_sum):
    import torch

    from cudamultislice_b200 import MultisliceError

    atoms = film(400_000, 360.0)  # 2.1 GB of tables a slice, 6.3 GB in three buffers
    defoci = np.array([-300.0, 200.0], np.float32)
    T = (np.random.default_rng(1).random((2, 64, 64)) * 0.5 + 0.75).astype(np.float32)
    free = handle(atoms)
    S = free.RunConventional()
    waves = [free.ExitWave()]
    free.MultisliceStepConventional(1)
    waves.append(free.ExitWave())
    loss, _, gxy = free.FocalSeriesGrad(defoci, T, S, want_v=False)
    assert free.PotentialSum()[0] == 2
    free.close()

    s = handle(atoms)
    left, _ = torch.cuda.mem_get_info()
    block = torch.empty(int(left - room), dtype=torch.uint8, device="cuda")
    try:
        S = s.RunConventional()
        assert s.PotentialSum()[0] == potential_sum
        got = [s.ExitWave()]
        s.MultisliceStepConventional(1)
        got.append(s.ExitWave())
        loss1, _, gxy1 = s.FocalSeriesGrad(defoci, T, S, want_v=False)
        if potential_sum == 1:  # forced, the separable sum cannot run
            s.SetPotentialSum(2)
            with pytest.raises(MultisliceError):
                s.RunConventional()
    finally:
        del block
        torch.cuda.empty_cache()
    s.SetPotentialSum(0)
    s.RunConventional()  # and with the room back
    assert s.PotentialSum()[0] == 2 and np.array_equal(s.ExitWave(), waves[0])
    s.close()
    for a, b in zip(got, waves):
        assert rel(a.view(np.float32), b.view(np.float32)) < 1e-5
    assert loss1 == pytest.approx(loss, rel=1e-5) and rel(gxy1, gxy) < 1e-4
