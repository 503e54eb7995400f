"""EM window sizes at which the device estimator changes its form: samples per
thread (4, 12, 20, 28, 40), CTAs per cluster (1, 2, 4, 8) and the scratch form for
windows no cluster holds, with zero samples and near-ties among them."""
import numpy as np
import pytest

from microtomodenoise_b200 import DenoiseParameters, NoiseLevel, synth

pytestmark = pytest.mark.gpu


# sigma is held to the noise tests' 1e-6 relative of the oracle's
# FP64-accumulating restatement: the decisions are the same ones, and FP64 sums
# in another order differ by less than a float's rounding
REL_TOL = 1e-6


@pytest.mark.parametrize("n,mode,zwindow", [
    (1, "global", 100), (33, "global", 100), (2048, "global", 100), (2049, "global", 100), (4000, "global", 100),
    (14337, "global", 100), (57345, "global", 100), (114688, "global", 100), (114689, "global", 100),
    (3000, "z-adaptive", 3), (30000, "z-adaptive", 8), (120000, "z-adaptive", 9),
])
@pytest.mark.parametrize("flat", [False, True])
def test_sigma_at_every_window_form(gpu, port, n, mode, zwindow, flat):
    _check(port, (20, 40, 48), n, mode, zwindow, flat)


@pytest.mark.parametrize("n,zwindow", [(40000, 20), (40000, 140), (60000, 140), (100000, 190)])
def test_sigma_with_many_windows(gpu, port, n, zwindow):
    """Hundreds of slices: the shape with more samples per thread, from half
    full on."""
    _check(port, (600, 17, 18), n, "z-adaptive", zwindow, False)


@pytest.mark.parametrize("nz,n,zwindow", [(222, 88000, 100), (221, 88000, 100),  # CTAs: two waves or fewer
                                          (300, 84000, 100), (300, 88000, 100),  # 0.7 full or less
                                          (1000, 99000, 100)])                   # one CTA per window
def test_sigma_at_the_edges_of_many_windows(gpu, port, nz, n, zwindow):
    _check(port, (nz, 17, 18), n, "z-adaptive", zwindow, False)


@pytest.mark.parametrize("n,zwindow", [(60000, 140), (100000, 400)])
def test_more_clusters_than_the_gpu_holds(gpu, n, zwindow):
    """Hundreds of windows of two and of eight CTAs each: clusters start as others
    end, their CTAs at different times, and every run gives the same sigma."""
    vol = synth.small_case((600, 17, 18), seed=3)
    dp = DenoiseParameters(noise_mode="z-adaptive", zwindow=zwindow)
    runs = []
    nl = NoiseLevel(n, 15, vol.shape, seed=1)
    for _ in range(6):
        runs.append(nl.get_noiselevel(vol, dp))
    nl.close()
    assert all(np.array_equal(r, runs[0]) for r in runs)


def _check(port, shape, n, mode, zwindow, flat):
    vol = synth.small_case(shape, seed=n % 97)
    if flat:
        vol[:, :24] = 0.5  # patches of std 0 are excluded, whole windows may be empty
        vol[7:11] = 0.25
    nl = NoiseLevel(n, 15, vol.shape, seed=n)
    dp = DenoiseParameters(noise_mode=mode, zwindow=zwindow)
    got = nl.get_noiselevel(vol, dp)
    ps, samples = nl.patchstd(), nl.samples()
    nl.close()
    want = port.noise_from_patchstd(ps, samples, vol.shape, mode, zwindow=zwindow, f64acc=True)
    assert np.all(np.abs(got - want) <= REL_TOL * np.abs(want)), np.max(np.abs(got / np.maximum(want, 1e-30) - 1))
