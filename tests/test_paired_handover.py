"""The hand-over of distance stages and raw tiles in the weight kernel of the
paired form, walked on the CPU with the library's own offset tables: one producer,
four consumers, three stages of two offsets, two raw buffers, barriers by phase
parity as mbarrier waits see them. Every search shape has to end with every
consumer reading the tile it asked for."""
import ctypes as C

import numpy as np
import pytest

from microtomodenoise_b200 import DenoiseParameters, _lib

STAGES, PER_STAGE, RAW, WARPS = 3, 2, 2, 4


class Barrier:
    def __init__(self, count):
        self.count, self.pending, self.done = count, count, 0

    def arrive(self):
        self.pending -= 1
        if self.pending == 0:
            self.pending, self.done = self.count, self.done + 1

    def passes(self, parity):  # the phase of that parity is not the running one
        return (self.done & 1) != parity


class Cta:
    def __init__(self, z):
        self.S, planes = len(z), sorted(set(range(min(z), -min(z) + 1)))
        # first offset of every plane, then S (an empty plane starts where the next does)
        self.z_start = [next((s for s in range(self.S) if z[s] >= p), self.S) for p in planes] + [self.S]
        self.z = z
        self.full = [Barrier(1) for _ in range(STAGES)]
        self.empty = [Barrier(WARPS) for _ in range(STAGES)]
        self.raw_full = [Barrier(1) for _ in range(RAW)]
        self.raw_empty = [Barrier(WARPS) for _ in range(RAW)]
        self.stage_of, self.plane_of = [None] * STAGES, [None] * RAW

    def producer(self, by_plane):
        """by_plane: the hand-over this one replaced (raw tiles waited for before
        their stage is armed, buffer and use taken from the plane's index)."""
        g, nxt, u = -1, 0, 0
        for s in range(0, self.S, PER_STAGE):
            k = s // PER_STAGE
            slot, parity = k % STAGES, (k // STAGES & 1) ^ 1
            yield self.empty[slot], parity

            def arm():
                self.stage_of[slot] = s
                self.full[slot].arrive()

            if not by_plane:
                arm()
            for i in range(PER_STAGE):
                if s + i != nxt:
                    continue
                while s + i == nxt:
                    g += 1
                    nxt = self.z_start[g + 1]
                n = g if by_plane else u
                yield self.raw_empty[n % RAW], (n // RAW & 1) ^ 1
                self.plane_of[n % RAW] = g
                self.raw_full[n % RAW].arrive()
                u += 1
            if by_plane:
                arm()

    def consumer(self, by_plane):
        g, nxt, u, cur = -1, 0, 0, None
        for s in range(0, self.S, PER_STAGE):
            k = s // PER_STAGE
            yield self.full[k % STAGES], k // STAGES & 1
            assert self.stage_of[k % STAGES] == s
            for i in range(PER_STAGE):
                if s + i == nxt:
                    if cur is not None:
                        self.raw_empty[cur].arrive()
                    while s + i == nxt:
                        g += 1
                        nxt = self.z_start[g + 1]
                    n = g if by_plane else u
                    cur = n % RAW
                    yield self.raw_full[cur], n // RAW & 1
                    u += 1
                # the tile in the buffer is that of the offset's plane
                assert self.plane_of[cur] + min(self.z) == self.z[s + i]
            self.empty[k % STAGES].arrive()

    def ends(self, by_plane=False):
        running = [self.producer(by_plane)] + [self.consumer(by_plane) for _ in range(WARPS)]
        waits = {r: next(r, None) for r in running}
        while any(waits.values()):
            moved = False
            for r in running:
                while waits[r] and waits[r][0].passes(waits[r][1]):
                    waits[r] = next(r, None)
                    moved = True
            if not moved:
                return False
        return True


def offsets_z(lib, sr, nslices):
    cp = DenoiseParameters(radius_patchspace=(1, 1, 1), radius_searchspace=sr, nslices=nslices).to_c()
    ns, npatch = C.c_int(0), C.c_int(0)
    _lib.check(lib.inlm_geometry(C.byref(cp), 40, None, C.byref(ns), None, None, C.byref(npatch), None), "geometry")
    s, t = np.zeros((ns.value, 3), np.int32), np.zeros((npatch.value, 3), np.int32)
    w = np.zeros(npatch.value, np.float32)
    _lib.check(lib.inlm_geometry(C.byref(cp), 40, s.ctypes.data, C.byref(ns), t.ctypes.data, w.ctypes.data,
                                 C.byref(npatch), None), "geometry")
    return s[:, 2].tolist()


@pytest.mark.parametrize("rx", range(5))
def test_every_search_shape_ends(lib, rx):
    for ry in range(5):
        for rz in range(11):
            z = offsets_z(lib, (rx, ry, rz), 21)
            if len(z) >= 2 and len(z) % 2 == 0:  # what the form takes
                assert Cta(z).ends(), (rx, ry, rz)


@pytest.mark.parametrize("sr,nslices", [((2, 2, 8), 21), ((5, 5, 5), 11), ((10, 10, 10), 11), ((3, 4, 2), 11),
                                        ((7, 1, 9), 15), ((11, 11, 11), 23)])
def test_larger_search_shapes_end(lib, sr, nslices):
    assert Cta(offsets_z(lib, sr, nslices)).ends()


@pytest.mark.parametrize("sr,nslices", [((1, 1, 2), 11), ((0, 0, 1), 11), ((0, 0, 2), 11), ((1, 0, 3), 11), ((2, 2, 8), 21)])
def test_the_model_sees_a_blocked_hand_over(lib, sr, nslices):
    """With raw tiles waited for before their stage is armed these shapes block,
    or read a tile that is not theirs."""
    try:
        ended = Cta(offsets_z(lib, sr, nslices)).ends(by_plane=True)
    except AssertionError:
        ended = False
    assert not ended
