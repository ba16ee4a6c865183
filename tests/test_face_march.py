"""The march length that the face kernels take (grhd_face_march, host only;
the launches call the same function with the device's resident blocks)
against an independent list-scheduling simulation: every block of the launch,
in launch order (the full z blocks of every 16 x 16-cell tile, then the short
last z row), starts on the resident slot that frees first and costs its
planes plus 0.7 of one; the chosen length is the candidate whose launch
finishes first (ties keep the longer march).  And the accretion partials, one
per block, of every box that the static right-hand side takes fit its
scratch."""
import ctypes as C
import heapq

import numpy as np
import pytest

TILE = 16
CANDIDATES = (48, 40, 32, 24, 20, 16, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2,
              1)
# limits of grhd_compute_rhs_static
STATIC_GHOSTED, STATIC_INTERIOR, STATIC_PARTIALS = 65536, 32768, 4096


def tiles_of(nx, ny):
    return -(-nx // TILE) * -(-ny // TILE)


def makespan(nx, ny, nz, z, slots):
    tiles = tiles_of(nx, ny)
    costs = [10 * z + 7] * (tiles * (nz // z))
    if nz % z:
        costs += [10 * (nz % z) + 7] * tiles
    free = [0] * min(slots, max(len(costs), 1))
    heapq.heapify(free)
    end = 0
    for c in costs:
        t = heapq.heappop(free) + c
        end = max(end, t)
        heapq.heappush(free, t)
    return end


def choice(nx, ny, nz, slots):
    best, cost = None, None
    for z in CANDIDATES:
        m = makespan(nx, ny, nz, z, slots)
        if cost is None or m < cost:
            best, cost = z, m
    return best


@pytest.fixture(scope="module")
def march():
    from grdzhadzha_b200 import _lib as L
    lib = L.load()

    def call(nx, ny, nz, slots):
        out = C.c_int(0)
        assert lib.grhd_face_march(nx, ny, nz, slots, C.byref(out)) == 0
        return out.value
    call.lib = lib
    return call


def test_matches_list_scheduling(march):
    rng = np.random.default_rng(20261206)
    sides = [1, 15, 16, 17, 31, 32, 33]
    for it in range(200):
        nx, ny, nz = (int(v) for v in
                      (rng.choice(sides, 3) if it < 60 else
                       rng.integers(1, 200, 3)))
        slots = int(rng.choice([1, 7, 148, 296, 444]))
        assert march(nx, ny, nz, slots) == choice(nx, ny, nz, slots), \
            (nx, ny, nz, slots)


@pytest.mark.parametrize("slots", [296, 444])
def test_static_boxes_fit_their_accretion_partials(march, slots):
    """The boxes with the most face blocks: every shape at the limits."""
    most = 0
    for ghost in (2, 3):
        for nx in range(1, 400):
            for ny in range(1, 400):
                plane = (nx + 2 * ghost) * (ny + 2 * ghost)
                nz = min(STATIC_GHOSTED // plane - 2 * ghost,
                         STATIC_INTERIOR // (nx * ny))
                # (more tiles of one column count only at their widths' ends)
                if nz < 1 or (nx % TILE not in (0, 1)) or \
                        (ny % TILE not in (0, 1)):
                    continue
                for n in {nz, max(1, nz // 2), 1}:
                    blocks = tiles_of(nx, ny) * \
                        -(-n // march(nx, ny, n, slots))
                    most = max(most, blocks)
    assert 0 < most <= STATIC_PARTIALS, most


def test_rejects_empty_boxes_and_no_slots(march):
    out = C.c_int(0)
    for args in ((0, 8, 8, 296), (8, 8, 0, 296), (8, 8, 8, 0)):
        assert march.lib.grhd_face_march(*args, C.byref(out)) != 0
    assert march.lib.grhd_face_march(8, 8, 8, 296, None) != 0
