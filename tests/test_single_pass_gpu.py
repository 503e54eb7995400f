"""The single-pass FP32 kernels, each by name. By default the paired form runs
where these ran, so the golden, odd-size and NaN cases reach them only here: they
stay the kernels of batches and of handles without a workspace. Every case also
states which kernel runs by default."""
import os
import sys

import numpy as np
import pytest

from microtomodenoise_b200 import DenoiseParameters, IterativeNLM_GPU, _lib, synth
from oracle.oracle import FilterParams

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
from cases import FILTER_CASES  # noqa: E402

pytestmark = pytest.mark.gpu

FAMILY = {"auto": "nlm_tile_f32_paired<", "tile": "nlm_tile_f32<", "ws": "nlm_tile_ws_f32<", "column": "nlm_column_f32<",
          "none": ("nlm_tile_f32<", "nlm_tile_ws_f32<", "nlm_column_f32<")}
# the default single-pass kernel ("none": a workspace no block fits), and each family
FORMS = ["auto", "none", "tile", "ws", "column"]


def run(raw, pr, sr, sigmas, form, nslices=11, aniso=1.0):
    g = IterativeNLM_GPU()
    g.configure_device(raw.shape, DenoiseParameters(radius_patchspace=pr, radius_searchspace=sr, nslices=nslices,
                                                    z_anisotropy=aniso))
    if form == "none":
        _lib.check(_lib.load().inlm_debug_pair_workspace(g._h, 1000), "pair_workspace")
    elif form != "auto":
        g.select_tile_form(form)
    assert g.describe().startswith(FAMILY[form]), g.describe()
    outs = []
    for it in range(sigmas.shape[0]):
        g.set_sigma(sigmas[it])
        g.Run_GaussianNoise(it + 1, raw if it == 0 else None)
        outs.append(g.get_result())
    assert g.describe().startswith(FAMILY[form]), g.describe()
    g.free_device()
    return np.stack(outs)


def has(form, pr, sr):
    """The column form is for patch radius 1; at patch radius 3 the warp-specialised
    kernel's buffers fit beside the box up to search radius 4."""
    return pr[:2] == (1, 1) if form == "column" else form != "ws" or pr[0] < 3 or max(sr) <= 4


SPECIALISED = [c for c in FILTER_CASES if "generic" not in c[0] and c[1][:2] != (1, 2)]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("case", SPECIALISED, ids=[c[0] for c in SPECIALISED])
def test_golden(gpu, golden_filter, case, form):
    name, pr, sr, nsl, an = case
    if not has(form, pr, sr):
        pytest.skip("no kernel of this form for these radii")
    got = run(golden_filter["raw"], pr, sr, golden_filter["sigmas"], form, nsl, an)
    assert np.array_equal(got, golden_filter[name])


@pytest.mark.parametrize("form", FORMS[1:])
@pytest.mark.parametrize("shape,pr,sr", [
    ((5, 7, 9), (1, 1, 1), (2, 2, 2)),
    ((9, 19, 41), (2, 2, 2), (3, 4, 2)),
    ((13, 9, 70), (2, 2, 1), (5, 5, 5)),
    ((17, 23, 37), (3, 3, 3), (3, 3, 3)),
    ((18, 30, 45), (3, 3, 3), (5, 5, 5)),
    ((14, 18, 33), (3, 3, 1), (2, 2, 2)),
    ((8, 8, 8), (3, 3, 2), (2, 2, 2)),
    ((3, 40, 40), (1, 1, 1), (4, 4, 4)),
    ((20, 12, 12), (1, 1, 3), (7, 7, 7)),
])
def test_odd_sizes(gpu, port, shape, pr, sr, form):
    if not has(form, pr, sr):
        pytest.skip("no kernel of this form for these radii")
    raw = synth.small_case(shape, seed=sum(shape))
    sig = np.stack([np.full(shape[0], 0.07, np.float32), np.linspace(0.03, 0.08, shape[0], dtype=np.float32)])
    want = port.denoise_f32(raw, FilterParams(search_radius=sr, patch_radius=pr), sig, all_iters=True)
    assert np.array_equal(run(raw, pr, sr, sig, form), want)


@pytest.mark.parametrize("form", FORMS[1:])
@pytest.mark.parametrize("pr,sr", [((1, 1, 1), (2, 2, 2)), ((2, 2, 2), (3, 3, 3))])
def test_nan_input(gpu, port, pr, sr, form):
    if not has(form, pr, sr):
        pytest.skip("no kernel of this form for these radii")
    rng = np.random.default_rng(11 + sum(pr))
    raw = rng.random((12, 21, 37), dtype=np.float32)
    raw[5, 10, 18] = np.nan
    raw[0, 0, 3] = np.nan
    sig = np.full((2, 12), 0.3, np.float32)
    got = run(raw, pr, sr, sig, form)
    want = port.denoise_f32(raw, FilterParams(search_radius=sr, patch_radius=pr), sig, all_iters=True)
    assert np.array_equal(got, want, equal_nan=True)
