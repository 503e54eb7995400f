"""The paired-offset FP32 form: distances of half of the search offsets, each
used for both offsets of a pair. Bit-exact to the oracle at the edges of its
tiles, z chunks, blocks and row forms, and where it has no workspace."""
import ctypes as C
import threading

import numpy as np
import pytest

from microtomodenoise_b200 import Batch, DenoiseParameters, IterativeNLM_GPU, _lib, synth, trim_memory
from oracle.oracle import FilterParams

MB = 1 << 20


def _run(raw, pr, sr, sig, limit=0, nslices=11, precision="f32", form=None):
    g = IterativeNLM_GPU()
    g.configure_device(raw.shape, DenoiseParameters(radius_patchspace=pr, radius_searchspace=sr, nslices=nslices,
                                                    precision=precision))
    if form:
        g.select_tile_form(form)
    else:
        assert "paired" in g.describe(), g.describe()
        _lib.check(_lib.load().inlm_debug_pair_workspace(g._h, limit), "pair_workspace")
    outs = []
    for it in range(len(sig)):
        g.set_sigma(sig[it])
        g.Run_GaussianNoise(it + 1, raw if it == 0 else None)
        outs.append(g.get_result())
    desc = g.describe()
    g.free_device()
    return np.stack(outs), desc


def _run_forced(raw, pr, sr, sig, nslices=11):
    """The paired form where the single-pass kernels are the faster choice."""
    g = IterativeNLM_GPU()
    g.configure_device(raw.shape, DenoiseParameters(radius_patchspace=pr, radius_searchspace=sr, nslices=nslices))
    assert "paired" not in g.describe(), g.describe()
    _lib.check(_lib.load().inlm_debug_pair_workspace(g._h, 8 << 30), "pair_workspace")
    desc = g.describe()
    outs = []
    for it in range(len(sig)):
        g.set_sigma(sig[it])
        g.Run_GaussianNoise(it + 1, raw if it == 0 else None)
        outs.append(g.get_result())
    g.free_device()
    return np.stack(outs), desc


def _sigmas(nz):
    return np.stack([np.full(nz, 0.07, np.float32), np.linspace(0.03, 0.08, nz, dtype=np.float32)])


@pytest.mark.gpu
@pytest.mark.parametrize("shape,pr,sr,limit", [
    ((9, 19, 41), (2, 2, 2), (3, 4, 2), 0),           # one chunk, uneven search radii
    ((5, 7, 9), (1, 1, 1), (2, 2, 2), 0),             # smaller than a tile in every axis
    ((3, 40, 40), (1, 1, 1), (4, 4, 4), 0),           # fewer planes than the z halo
    ((61, 23, 70), (1, 1, 1), (4, 4, 4), 24 * MB),    # z chunks, ring wraps
    ((43, 40, 100), (2, 2, 2), (3, 3, 3), 4 * MB),    # blocks in x and y too
    ((34, 17, 45), (3, 3, 3), (3, 3, 3), 4 * MB),     # direct columns, z chunks
    ((13, 9, 70), (2, 2, 1), (5, 5, 5), 0),
    ((16, 24, 40), (1, 1, 2), (6, 6, 6), 0),
    ((12, 30, 33), (1, 1, 3), (3, 3, 3), 0),
    ((14, 18, 33), (3, 3, 1), (2, 2, 2), 0),
    ((11, 16, 32), (3, 3, 2), (4, 4, 4), 0),
    ((20, 40, 48), (1, 1, 1), (10, 10, 10), 0),       # the widest box pitch
    ((42, 66, 250), (1, 1, 1), (2, 2, 2), 0),         # eight rows per thread in the weight kernel
])
def test_paired_form_bit_exact(gpu, port, shape, pr, sr, limit):
    raw = synth.small_case(shape, seed=sum(shape))
    sig = _sigmas(shape[0])
    got, desc = _run(raw, pr, sr, sig, limit)
    assert "paired" in desc, desc
    want = port.denoise_f32(raw, FilterParams(search_radius=sr, patch_radius=pr), sig, all_iters=True)
    assert np.array_equal(got, want), f"{desc}: {np.count_nonzero(got != want)} voxels differ"


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(20, 24, 40), (42, 66, 250)])  # two and eight rows per thread
@pytest.mark.parametrize("pr,sr,nslices", [
    ((1, 1, 1), (1, 1, 2), 11), ((1, 1, 1), (1, 1, 5), 11), ((2, 2, 2), (1, 1, 2), 11),  # one offset in the end planes
    ((1, 1, 1), (0, 0, 1), 11), ((1, 1, 1), (0, 0, 2), 11), ((2, 2, 2), (0, 0, 3), 11),  # no offset at z = 0
    ((1, 1, 1), (1, 0, 3), 11), ((1, 1, 1), (0, 1, 2), 11), ((2, 2, 2), (0, 3, 2), 11), ((3, 3, 3), (3, 0, 2), 11),
    ((1, 1, 1), (2, 2, 8), 21),
])
def test_thin_search_shapes_bit_exact(gpu, port, shape, pr, sr, nslices):
    raw = synth.small_case(shape, seed=sum(sr))
    sig = _sigmas(shape[0])
    few = len(port.search_offsets(FilterParams(search_radius=sr, patch_radius=pr, nslices=nslices))) < (14 if pr[0] == 1 else 6)
    got, desc = (_run_forced if few else _run)(raw, pr, sr, sig, nslices=nslices)
    assert "paired" in desc, desc
    want = port.denoise_f32(raw, FilterParams(search_radius=sr, patch_radius=pr, nslices=nslices), sig, all_iters=True)
    assert np.array_equal(got, want), f"{desc}: {np.count_nonzero(got != want)} voxels differ"


@pytest.mark.gpu
def test_more_planes_than_a_grid_takes(gpu, port):
    """65535 planes are the largest grid in z; a stack of 65600 is one chunk."""
    raw = synth.small_case((65600, 5, 6), seed=4)
    sig = _sigmas(65600)
    got, desc = _run_forced(raw, (1, 1, 1), (1, 1, 1), sig)
    assert "paired" in desc, desc
    want = port.denoise_f32(raw, FilterParams(search_radius=(1, 1, 1), patch_radius=(1, 1, 1)), sig, all_iters=True)
    assert np.array_equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("pr,sr", [((1, 1, 1), (3, 3, 3)), ((2, 2, 2), (4, 4, 4)), ((3, 3, 3), (2, 2, 2))])
def test_paired_fused_form_equals_the_other_fused_kernels(gpu, pr, sr):
    raw = synth.small_case((21, 27, 50), seed=sum(pr) + sum(sr))
    sig = _sigmas(21)
    got, desc = _run(raw, pr, sr, sig, precision="f32_fma")
    assert "paired" in desc and "fused" in desc, desc
    want, _ = _run(raw, pr, sr, sig, precision="f32_fma", form="tile")
    assert np.array_equal(got, want)


@pytest.mark.gpu
def test_paired_form_without_room_for_its_workspace(gpu, port):
    """No workspace (a bound that fits no block, or a failing allocation): the
    single-pass kernel runs instead, and a later call has its workspace."""
    L = _lib.load()
    raw = synth.small_case((20, 24, 40), seed=5)
    sig = _sigmas(20)
    want = port.denoise_f32(raw, FilterParams(search_radius=(3, 3, 3), patch_radius=(2, 2, 2)), sig, all_iters=True)
    got, desc = _run(raw, (2, 2, 2), (3, 3, 3), sig, limit=1000)
    assert "paired" not in desc, desc
    assert np.array_equal(got, want)
    g = IterativeNLM_GPU()
    g.configure_device(raw.shape, DenoiseParameters(radius_patchspace=(2, 2, 2), radius_searchspace=(3, 3, 3)))
    for it in range(2):
        g.set_sigma(sig[it])
        # iteration 1: the offset table and the z table first, then the workspace
        L.inlm_debug_fail_allocation(2 if it == 0 else -1)
        g.Run_GaussianNoise(it + 1, raw if it == 0 else None)
        L.inlm_debug_fail_allocation(-1)
        assert np.array_equal(g.get_result(), want[it])
    assert "paired" in g.describe()
    g.free_device()


@pytest.mark.gpu
def test_a_plan_slower_than_the_single_pass_kernel_does_not_run(gpu, port):
    raw = synth.small_case((40, 64, 96), seed=7)
    sig = _sigmas(40)
    want = port.denoise_f32(raw, FilterParams(search_radius=(5, 5, 5), patch_radius=(1, 1, 1)), sig, all_iters=True)
    got, desc = _run(raw, (1, 1, 1), (5, 5, 5), sig, limit=-32 * MB)
    assert desc.startswith("nlm_column_f32<"), desc
    assert np.array_equal(got, want)
    got, desc = _run(raw, (1, 1, 1), (5, 5, 5), sig, limit=32 * MB)
    assert "paired" in desc, desc
    assert np.array_equal(got, want)


@pytest.mark.gpu
def test_first_pass_allocates_its_workspace_and_nothing_else(gpu, port):
    """Plan and tables are made when the handle is configured: a first pass takes
    a workspace (which may fail: the single-pass kernel runs) and a second nothing."""
    L = _lib.load()

    def live():
        n = C.c_int64(0)
        _lib.check(L.inlm_debug_live_allocations(C.byref(n)), "live allocations")
        return n.value

    raw = synth.small_case((20, 24, 40), seed=5)
    sig = _sigmas(20)
    want = port.denoise_f32(raw, FilterParams(search_radius=(3, 3, 3), patch_radius=(2, 2, 2)), sig, all_iters=True)
    g = IterativeNLM_GPU()
    g.configure_device(raw.shape, DenoiseParameters(radius_patchspace=(2, 2, 2), radius_searchspace=(3, 3, 3)))
    before = live()
    g.set_sigma(sig[0])
    L.inlm_debug_fail_allocation(0)
    g.Run_GaussianNoise(1, raw)
    L.inlm_debug_fail_allocation(-1)
    assert np.array_equal(g.get_result(), want[0]) and live() == before
    g.Run_GaussianNoise(1, raw)
    assert np.array_equal(g.get_result(), want[0]) and live() == before + 1
    trim_memory()  # gives the workspace up; the next pass takes another
    assert live() == before
    g.Run_GaussianNoise(1, raw)
    assert np.array_equal(g.get_result(), want[0]) and live() == before + 1
    g.set_sigma(sig[1])
    L.inlm_debug_fail_allocation(0)  # (nothing is allocated, so nothing fails)
    g.Run_GaussianNoise(2)
    L.inlm_debug_fail_allocation(-1)
    assert np.array_equal(g.get_result(), want[1]) and live() == before + 1
    assert "paired" in g.describe()
    g.free_device()


@pytest.mark.gpu
@pytest.mark.parametrize("pr,sr,form", [((1, 1, 1), (5, 5, 5), "column"), ((2, 2, 2), (4, 4, 4), None)])
def test_memory_gets_scarce_and_free_again(gpu, pr, sr, form):
    """Somebody else takes the memory between configuration and a pass: the passes
    are planned anew for what is left, or run single-pass where that plan would be
    slower; with the memory back, the handle's plan is whole."""
    torch = pytest.importorskip("torch")
    raw = synth.small_case((64, 128, 128), seed=8)
    sig = _sigmas(64)[1]
    g = IterativeNLM_GPU()
    g.configure_device(raw.shape, DenoiseParameters(radius_patchspace=pr, radius_searchspace=sr))
    g.set_sigma(sig)
    assert "paired" in g.describe()
    g.Run_GaussianNoise(1, raw)
    want = g.get_result()
    trim_memory()
    free = torch.cuda.mem_get_info()[0]
    hog = torch.empty(free - (600 << 20), dtype=torch.uint8, device="cuda")
    g.Run_GaussianNoise(1, raw)
    assert np.array_equal(g.get_result(), want)
    del hog
    torch.cuda.empty_cache()
    g.Run_GaussianNoise(1, raw)
    assert np.array_equal(g.get_result(), want)
    if form:
        g.select_tile_form(form)
        g.Run_GaussianNoise(1, raw)
        assert np.array_equal(g.get_result(), want)
    g.free_device()


@pytest.mark.gpu
def test_paired_handles_take_turns_on_one_workspace(gpu):
    L = _lib.load()
    live = C.c_int64(0)
    _lib.check(L.inlm_debug_live_allocations(C.byref(live)), "live allocations")
    before = live.value
    raw = synth.small_case((16, 24, 40), seed=6)
    sig = _sigmas(16)
    shapes = [((1, 1, 1), (4, 4, 4)), ((2, 2, 2), (2, 2, 2))]
    alone = [_run(raw, pr, sr, sig)[0] for pr, sr in shapes]
    hs = []
    for pr, sr in shapes:
        g = IterativeNLM_GPU()
        g.configure_device(raw.shape, DenoiseParameters(radius_patchspace=pr, radius_searchspace=sr))
        hs.append(g)
    for it in range(2):
        for g, want in zip(hs, alone):
            g.set_sigma(sig[it])
            g.Run_GaussianNoise(it + 1, raw if it == 0 else None)
            assert np.array_equal(g.get_result(), want[it])
    for g in hs:
        g.free_device()
    _lib.check(L.inlm_debug_live_allocations(C.byref(live)), "live allocations")
    assert live.value == before


@pytest.mark.gpu
@pytest.mark.parametrize("form,sr", [(None, (4, 4, 4)), ("tile", (3, 4))])
def test_threads_whose_launches_differ_in_shared_memory(gpu, form, sr):
    """Launches of one kernel from several threads, with more and with less dynamic
    shared memory: by the volume's depth (paired form) or the search radius."""
    jobs = [((8 + 16 * i, 40, 64), (sr[i % len(sr)],) * 3) for i in range(4)]
    handles, raws, got, errors = [], [], {}, []
    for i, (shape, s) in enumerate(jobs):
        g = IterativeNLM_GPU()
        g.configure_device(shape, DenoiseParameters(radius_patchspace=(2, 2, 2), radius_searchspace=s))
        if form:
            g.select_tile_form(form)
        g.set_sigma(_sigmas(shape[0])[1])
        handles.append(g)
        raws.append(synth.small_case(shape, seed=30 + i))
    assert len({g.describe().split("smem=")[1].split()[0] for g in handles}) > 1
    alone = []
    for g, raw in zip(handles, raws):
        g.Run_GaussianNoise(1, raw)
        alone.append(g.get_result())

    def work(i):
        try:
            for _ in range(60):
                handles[i].Run_GaussianNoise(1, raws[i])
            got[i] = handles[i].get_result()
        except _lib.InlmError as e:
            errors.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for g in handles:
        g.free_device()
    assert not errors, errors
    for i, want in enumerate(alone):
        assert np.array_equal(got[i], want), jobs[i]


@pytest.mark.gpu
@pytest.mark.parametrize("bound", [1, 0])
def test_threads_share_workspaces(gpu, bound):
    """Jobs of several threads at a time: with one workspace between them (they join
    the one that is out, pass after pass) and with one each; the pool keeps none
    beyond its bound, and none when the last handle is gone."""
    L = _lib.load()

    def live():
        n = C.c_int64(0)
        _lib.check(L.inlm_debug_live_allocations(C.byref(n)), "live allocations")
        return n.value

    before = live()
    cases = [((24, 40, 64), (2, 2, 2), (4, 4, 4)), ((24, 40, 64), (2, 2, 2), (4, 4, 4)),
             ((30, 33, 70), (1, 1, 1), (4, 4, 4)), ((16, 48, 48), (3, 3, 3), (3, 3, 3))]
    handles, raws, alone, got = [], [], [], {}
    for i, (shape, pr, sr) in enumerate(cases):
        g = IterativeNLM_GPU()
        g.configure_device(shape, DenoiseParameters(radius_patchspace=pr, radius_searchspace=sr, noise_mode="manual",
                                                    sigma=(0.06, 0.05), maxiterations=4))
        handles.append(g)
        raws.append(synth.small_case(shape, seed=20 + i))
        g.denoise(raws[i])  # (a handle's later jobs start from sigma[1])
        alone.append(g.denoise(raws[i])[0])
        assert "paired" in g.describe()
    held = live()

    def work(i):
        got[i] = [handles[i].denoise(raws[i])[0] for _ in range(12)]

    _lib.check(L.inlm_debug_pair_pool(bound), "pair_pool")
    try:
        ts = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert live() <= (held if bound else held + len(cases))
        for i, want in enumerate(alone):
            assert len(got[i]) == 12 and all(np.array_equal(o, want) for o in got[i]), cases[i]
    finally:
        L.inlm_debug_pair_pool(0)
    for g in handles:
        g.free_device()
    assert live() == before


@pytest.mark.gpu
def test_a_batch_beside_a_handle_leaves_the_pool_its_share(gpu):
    L = _lib.load()

    def live():
        n = C.c_int64(0)
        _lib.check(L.inlm_debug_live_allocations(C.byref(n)), "live allocations")
        return n.value

    raw = synth.small_case((20, 24, 40), seed=5)
    g = IterativeNLM_GPU()
    g.configure_device(raw.shape, DenoiseParameters(radius_patchspace=(2, 2, 2), radius_searchspace=(3, 3, 3)))
    g.set_sigma(_sigmas(20)[1])
    _lib.check(L.inlm_debug_pair_pool(32 * MB), "pair_pool")  # the handle's takes 11, the batch's more than 32
    try:
        b = Batch([(32, 64, 160)], [DenoiseParameters(radius_patchspace=(1, 1, 1), radius_searchspace=(4, 4, 4),
                                                      noise_mode="manual", sigma=(0.06, 0.05))])
        assert "own launch paired" in b.describe(), b.describe()
        before = live()
        for _ in range(2):
            g.Run_GaussianNoise(1, raw)
            assert live() == before + 1  # kept for the next call
        b.close()
    finally:
        L.inlm_debug_pair_pool(0)
    g.free_device()


@pytest.mark.gpu
def test_weight_step_equals_the_other_kernels_for_every_argument(gpu):
    n = C.c_int64(-1)
    _lib.check(_lib.load().inlm_debug_weight_mismatches(C.byref(n)), "weight_mismatches")
    assert n.value == 0


@pytest.mark.gpu
def test_fused_weight_step_for_every_argument(gpu):
    """Bound: with u = 2^-24, 12 + x is off by 4.8e-7, the next two Horner steps by
    3.57 times that of the one before and half an ulp of their own: 1.0e-5 on a
    numerator of 13.3 at the cutoff (7.5e-7), 5.0e-5 on a denominator of 532 (0.9e-7);
    the approximate reciprocal adds one ulp (1.2e-7) and the product u: 1.03e-6."""
    worst = C.c_double(-1)
    _lib.check(_lib.load().inlm_debug_fused_weight_error(C.byref(worst)), "fused_weight_error")
    assert 0 < worst.value <= 1.1e-6


@pytest.mark.parametrize("pr", [(1, 1, 1), (1, 1, 2), (2, 2, 1), (2, 2, 2), (3, 3, 2), (3, 3, 3)])
@pytest.mark.parametrize("sr,nslices", [((3, 4, 2), 11), ((5, 5, 5), 7), ((10, 10, 10), 11), ((2, 7, 9), 15)])
def test_offsets_come_in_mirrored_pairs(lib, pr, sr, nslices):
    """What the paired form rests on: offset S-1-j is the negative of offset j,
    z never descends, and a tap's weight depends on |x|, |y|, |z| alone."""
    cp = DenoiseParameters(radius_patchspace=pr, radius_searchspace=sr, nslices=nslices, z_anisotropy=1.7,
                           weight_table="distweight").to_c()
    ns, npatch = C.c_int(0), C.c_int(0)
    _lib.check(lib.inlm_geometry(C.byref(cp), 40, None, C.byref(ns), None, None, C.byref(npatch), None), "geometry")
    s, t = np.zeros((ns.value, 3), np.int32), np.zeros((npatch.value, 3), np.int32)
    w = np.zeros(npatch.value, np.float32)
    _lib.check(lib.inlm_geometry(C.byref(cp), 40, s.ctypes.data, C.byref(ns), t.ctypes.data, w.ctypes.data,
                                 C.byref(npatch), None), "geometry")
    assert np.array_equal(s, -s[::-1]) and (np.diff(s[:, 2]) >= 0).all()
    by_size = {}
    for tap, weight in zip(np.abs(t), w):
        assert by_size.setdefault(tuple(tap), weight) == weight


@pytest.mark.gpu
@pytest.mark.parametrize("shape,paired", [((17, 40, 64), True), ((65, 72, 127), False)])
def test_fused_patch_radius_1_runs_the_column_form_on_volumes_that_fill_the_gpu(gpu, shape, paired):
    raw = synth.small_case(shape, seed=9)
    dp = DenoiseParameters(radius_patchspace=(1, 1, 1), radius_searchspace=(2, 2, 2), precision="f32_fma")
    outs = []
    for form in (None, "column"):
        g = IterativeNLM_GPU()
        g.configure_device(shape, dp)
        if form:
            g.select_tile_form(form)
        else:
            assert ("paired" in g.describe()) == paired, g.describe()
        g.set_sigma(_sigmas(shape[0])[1])
        g.Run_GaussianNoise(1, raw)
        outs.append(g.get_result())
        g.free_device()
    assert np.array_equal(outs[0], outs[1])
