"""The autotuner applies what it reports: the paired form where its passes were
the fastest, else the chosen single-pass configuration, by its own timings or by a
cache file. Each run is a process of its own, as the cache is read once."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import sys
import numpy as np
from microtomodenoise_b200 import DenoiseParameters, IterativeNLM_GPU, synth
from oracle.oracle import FilterParams, Port
shape, r = tuple(int(v) for v in sys.argv[1].split(",")), int(sys.argv[2])
raw = synth.small_case(shape, seed=3)
sig = np.full(shape[0], 0.06, np.float32)
g = IterativeNLM_GPU()
g.configure_device(shape, DenoiseParameters(radius_patchspace=(r,) * 3, radius_searchspace=(3, 3, 3), precision=sys.argv[3]))
print(g.autotune())
g.set_sigma(sig)
g.Run_GaussianNoise(1, raw)
print(g.describe())
if sys.argv[3] == "f32":
    want = Port().denoise_f32(raw, FilterParams(search_radius=(3, 3, 3), patch_radius=(r,) * 3), sig[None])
    assert np.array_equal(g.get_result(), want)
g.free_device()
"""

FILLS, SMALL = "40,72,130", "16,40,72"  # tiles of 32 x 8 x 8 against the SMs


def run(tmp_path, shape, radius, cache=None, precision="f32"):
    path = tmp_path / "cache.txt"
    if cache:
        path.write_text(cache + "\n")
    r = subprocess.run([sys.executable, "-c", PROGRAM, shape, str(radius), precision], cwd=ROOT, text=True,
                       capture_output=True, env={**os.environ, "INLM_AUTOTUNE_CACHE": str(path)})
    assert r.returncode == 0, r.stdout + r.stderr
    report, desc = r.stdout.strip().splitlines()[-2:]
    return report, desc, path.read_text() if path.exists() else ""


@pytest.mark.parametrize("radius,precision", [(1, "f32"), (2, "f32"), (1, "f32_fma"), (2, "f32_fma")])
def test_the_faster_form_runs(gpu, tmp_path, radius, precision):
    report, desc, saved = run(tmp_path, FILLS, radius, precision=precision)
    ms = {p.split(":")[0]: float(p.split(":")[1].split()[0]) for p in report.split("; ")[:-1]}
    fastest = min(ms, key=ms.get)
    chosen = report.split("; ")[-1]
    assert chosen.startswith("chosen paired" if fastest == "paired" else "chosen " + fastest), report
    if "paired" not in chosen or precision == "f32":  # (the fused form has a rule of its own for its column kernel)
        assert ("paired" in desc) == (fastest == "paired"), (report, desc)
    again, desc2, _ = run(tmp_path, FILLS, radius, precision=precision)  # from the file written above
    assert again == "cached; " + chosen and desc2 == desc, (again, saved)


@pytest.mark.parametrize("flags,shape,kernel", [
    (1 | 4 | 8, FILLS, "nlm_tile_f32<2,2,2> tz=16"),   # single-pass faster: it runs
    (1 | 2 | 4 | 8, FILLS, "nlm_tile_ws_f32<2,2,2>"),
    (1 | 4, FILLS, "nlm_tile_f32_paired<2,2,2>"),      # paired faster
    (1 | 4 | 8, SMALL, "nlm_tile_f32_paired<2,2,2>"),  # few tiles: the offsets are shared out
])
def test_a_cached_choice_is_applied(gpu, tmp_path, flags, shape, kernel):
    tz = 8 if flags & 2 else 16
    report, desc, _ = run(tmp_path, shape, 2, f"2 2 2 3 3 3 11 0 {tz} {flags}")
    assert report.startswith("cached; chosen ") and desc.startswith(kernel), (report, desc)


def test_a_line_without_the_paired_form_is_timed_anew(gpu, tmp_path):
    report, _, saved = run(tmp_path, FILLS, 2, "2 2 2 3 3 3 11 0 16 1")
    assert "paired: " in report and int(saved.split()[-1]) & 4, (report, saved)
