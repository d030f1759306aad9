"""The tile widths that a batch chooses for its jobs (qcb_debug_batch_widths, on
the host), judged by the times of its tiles placed longest first on the SMs."""
import ctypes
import heapq

import numpy as np
import pytest

import qcb200
from qcb200._lib import check, lib, ptr

SMS = 148
# widest tile of a surface-code memory of distance d
TMAX = {3: 256, 5: 256, 7: 256, 9: 168, 11: 114, 13: 80, 15: 58, 17: 44, 19: 34, 21: 28, 23: 22, 25: 18}


def widths(jobs):
    L, a, b = (np.array([j[i] for j in jobs], float) for i in range(3))
    nc = np.array([j[3] for j in jobs], np.uint64)
    tm = np.array([j[4] for j in jobs], np.uint32)
    w = np.array([j[5] if len(j) > 5 else 0 for j in jobs], np.uint32)
    check(lib().qcb_debug_batch_widths(ptr(L), ptr(a), ptr(b), ptr(nc), ptr(tm), len(jobs), SMS, ptr(w)))
    return w.tolist()


def job(d, shots, *given):
    """(words, time of a tile apart from and per column, columns, widest tile) of d rounds"""
    return (40.0 * d**3, 4.5 * d + 0.01 * d**3, 0.0012 * d**3, (shots + 31) // 32, TMAX[d], *given)


def tile_time(j, t):
    odd = 1 if t & (t - 1) == 0 else 1.05 if t % 16 == 0 else 1.15 if t % 8 == 0 or t > 48 else 1.25
    return (j[1] + j[2] * t) * odd


def longest_sm(jobs, ts):
    tiles = sorted(((tile_time(j, t), -(-j[3] // t)) for j, t in zip(jobs, ts)), reverse=True)
    free, end = [0.0] * SMS, 0.0
    for time, count in tiles:
        for _ in range(count):
            e = free[0] + time
            heapq.heapreplace(free, e)
            end = max(end, e)
    return end


@pytest.mark.parametrize("d", [3, 9, 13, 15, 17, 19, 21, 23, 25])
@pytest.mark.parametrize("jobs,shots", [(1, 3000), (8, 30_000), (4, 200_000), (16, 150_000)])
def test_equal_jobs_lose_little_to_any_single_width(d, jobs, shots):
    """Equal jobs are within 6 % of the best of the multiples of 16, their powers
    of two and the widest tile, one width for all (the choice leaves powers of
    two for a gain of 3 %, and its cost model for them is another one)."""
    js = [job(d, shots)] * jobs
    got = widths(js)
    assert len(set(got)) == 1 and 16 <= got[0] <= TMAX[d] and got[0] % 2 == 0
    best = min(longest_sm(js, [t] * jobs) for t in [*range(16, TMAX[d], 16), TMAX[d]])
    assert longest_sm(js, got) <= 1.06 * best


def test_many_tiles_of_a_program_between_powers_of_two():
    """d = 15: tiles of 32 columns are not the only choice below the 58 that fit."""
    assert set(widths([job(15, 200_000)] * 16)) - {32}


@pytest.mark.parametrize("seed", range(8))
def test_uneven_jobs(seed):
    """Uneven batches keep within each job's widest tile, and gain on 16 columns
    for all where there are tiles enough."""
    rng = np.random.default_rng(seed)
    js = [job(int(rng.choice(list(TMAX))), int(10 ** rng.uniform(4, 5.3))) for _ in range(int(rng.integers(8, 25)))]
    got = widths(js)
    assert all(16 <= t <= j[4] and t % 2 == 0 for t, j in zip(got, js))
    assert longest_sm(js, got) <= longest_sm(js, [16] * len(js))


def test_given_widths_stay():
    js = [job(21, 50_000, 20), job(15, 50_000), job(3, 100, 64)]
    got = widths(js)
    assert got[0] == 20 and got[2] == 64


def test_frames_without_shots():
    got = widths([job(15, 0), job(15, 200_000), job(3, 0)])
    assert all(16 <= t <= 256 for t in got)
    assert widths([job(7, 0)])[0] >= 16


def test_bad_arguments():
    with pytest.raises(qcb200.ArgumentError):
        widths([(1.0, 1.0, 1.0, 10, 8)])
    with pytest.raises(qcb200.ArgumentError):
        widths([(1.0, 1.0, 1.0, 10, 32, 64)])
    assert lib().qcb_debug_batch_widths(None, None, None, None, None, 1, SMS, ctypes.c_void_p()) == 4  # QCB_EARG
