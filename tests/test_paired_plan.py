"""When the paired form runs: its plan for a workspace against the single-pass
kernel, by the library's rule for a B200 (no device needed)."""
import ctypes as C

import pytest

from microtomodenoise_b200 import DenoiseParameters, _lib

GB = 1 << 30


def plan(lib, shape, pr, sr, size):
    """(the form runs, plan's time over that of the whole volume in one chunk, bytes)"""
    cp = DenoiseParameters(radius_patchspace=(pr,) * 3, radius_searchspace=(sr,) * 3).to_c()
    out = (C.c_double * 8)()
    _lib.check(lib.inlm_debug_pair_plan((C.c_int * 3)(*shape[::-1]), C.byref(cp), int(size), out), "pair_plan")
    return bool(out[0]), out[1] / out[2], out[3]


# measured: paired and single-pass ms per pass with a workspace of so many GB
@pytest.mark.parametrize("shape,pr,sr,gb,paired,single", [
    ((256, 256, 256), 1, 10, 22, 92.9, 102.6), ((256, 256, 256), 1, 10, 16, 96.8, 102.6),
    ((256, 256, 256), 1, 10, 8, 113.7, 102.6), ((256, 256, 256), 1, 10, 4, 130.9, 102.6),
    ((256, 256, 256), 1, 10, 1, 295.8, 102.6), ((256, 256, 256), 1, 5, 2, 16.07, 17.09),
    ((256, 256, 256), 1, 5, 1, 20.03, 17.09), ((512, 512, 512), 1, 5, 4, 118.4, 136.2),
    ((512, 512, 512), 1, 5, 1, 159.3, 136.2), ((512, 512, 512), 2, 5, 2, 179.5, 286.5),
    ((512, 512, 512), 2, 5, 0.25, 327.5, 286.5), ((256, 256, 256), 2, 5, 1, 27.27, 36.15),
    ((256, 256, 256), 2, 5, 0.25, 42.45, 36.15), ((256, 256, 256), 2, 7, 2, 70.1, 105.3),
    ((256, 256, 256), 2, 7, 0.25, 249.7, 105.3), ((256, 256, 256), 3, 7, 2, 137.5, 261.7),
    ((256, 256, 256), 3, 7, 0.25, 395.9, 261.7), ((512, 512, 512), 3, 7, 2, 1118.8, 2073.3),
    ((256, 256, 256), 1, 13, 8, 224.4, 389.0),  # (the column form does not fit)
    ((61, 187, 203), 3, 7, 1, 23.8, 46.5), ((61, 187, 203), 3, 7, 0.25, 82.2, 46.5),
])
def test_the_faster_form_is_chosen(lib, shape, pr, sr, gb, paired, single):
    runs, ratio, size = plan(lib, shape, pr, sr, gb * GB)
    assert size <= gb * GB
    assert runs == (paired < single), ratio


@pytest.mark.parametrize("pr,sr,paired", [
    (1, (1, 1, 1), False), (1, (0, 0, 2), False), (1, (1, 1, 2), False), (1, (2, 2, 1), True), (1, (2, 2, 2), True),
    (2, (0, 0, 2), False), (2, (1, 1, 1), True), (3, (0, 0, 1), False), (3, (1, 1, 2), True),
])
def test_few_offsets_run_single_pass(lib, pr, sr, paired):
    cp = DenoiseParameters(radius_patchspace=(pr,) * 3, radius_searchspace=sr).to_c()
    out = (C.c_double * 8)()
    _lib.check(lib.inlm_debug_pair_plan((C.c_int * 3)(256, 256, 256), C.byref(cp), 64 * GB, out), "pair_plan")
    assert bool(out[0]) == paired


def test_less_workspace_is_never_planned_as_faster(lib):
    ratios = [plan(lib, (256, 256, 256), 2, 7, gb * GB)[1] for gb in (32, 16, 8, 4, 2, 1, 0.5, 0.25)]
    assert ratios == sorted(ratios) and ratios[0] >= 1


def test_no_room_for_the_smallest_block(lib):
    assert plan(lib, (256, 256, 256), 2, 7, 1000)[0] is False
