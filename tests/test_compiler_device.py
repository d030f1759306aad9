"""CPU tests of the program that is uploaded: qcb_debug_program_device gives it
as qcb_program_compile does (x of an odd slot in plane 2s + 1, the entries of
two-qubit records ordered by their planes' parities).  With the planes renamed
to the interpreter's numbering it must reproduce the oracle bit for bit."""
import ctypes

import numpy as np
import pytest

import stream_emu
import test_compiler
from qcb200 import circuits, ops as O
from qcb200._lib import check, lib, ptr, qcb_program_info
from test_gpu_frames import random_circuit, xor_chain_circuit

E = stream_emu
# words of an entry, and which of them hold two 16-bit plane numbers
ENTRY = {E.SEG_CNOT: (2, (0, 1)), E.SEG_CZ: (2, (0, 1)), E.SEG_S: (2, (0,)), E.SEG_G1: (2, (0,)), E.SEG_G2: (4, (0, 1)),
         E.SEG_MZ: (2, (0,)), E.SEG_FLUSH: (4, (2, 3))}


def dump_device(arr):
    a = O.to_array(arr)
    sl, ns, nsl, info = ctypes.c_size_t(), ctypes.c_size_t(), ctypes.c_size_t(), qcb_program_info()
    aptr = ptr(a) if len(a) else None
    f = lib().qcb_debug_program_device
    check(f(aptr, len(a), None, 0, ctypes.byref(sl), None, 0, ctypes.byref(ns), None, None, 0, ctypes.byref(nsl),
            ctypes.byref(info)))
    stream = np.zeros(max(sl.value, 1), np.uint32)
    sites = np.zeros(max(ns.value, 1), E.SITE_DTYPE)
    sq, sw = np.zeros(max(nsl.value, 1), np.uint32), np.zeros(max(nsl.value, 1), np.uint32)
    check(f(aptr, len(a), ptr(stream), len(stream), ctypes.byref(sl), ptr(sites.view(np.uint8)), sites.nbytes,
            ctypes.byref(ns), ptr(sq), ptr(sw), len(sq), ctypes.byref(nsl), ctypes.byref(info)))
    return stream[: sl.value], sites[: ns.value], sq[: nsl.value], sw[: nsl.value], {k: getattr(info, k) for k, _ in info._fields_}


def entries(stream):
    """(kind, entries, planes' word columns) of every record, views into the stream."""
    pc = 0
    while True:
        kind, cnt = int(stream[pc]) >> 24, int(stream[pc]) & 0xFFFFFF
        if kind == E.SEG_END:
            return
        if kind == E.SEG_WIN:
            pc = pc // cnt * cnt + cnt
            continue
        pc += 4
        if kind == E.SEG_MRZ:  # groups of four entries (plane word, bit, reset, -)
            e = stream[pc: pc + 16 * cnt].reshape(-1, 4)
            yield kind, e, (0,)
            pc += 16 * cnt
        elif kind == E.SEG_XOR:
            pc += 32 * cnt
        else:
            n, cols = ENTRY[kind]
            yield kind, stream[pc: pc + n * cnt].reshape(cnt, n), cols
            pc += (n * cnt + 3) // 4 * 4


def x_first(stream, swap):
    """The stream and the slots' final planes with x of every slot in its even plane."""
    stream, swap = stream.copy(), swap ^ (np.arange(len(swap), dtype=np.uint32) & 1)
    for _, e, cols in entries(stream):
        for c in cols:
            lo, hi = e[:, c] & 0xFFFF, e[:, c] >> 16
            e[:, c] = (lo ^ ((lo >> 1) & 1)) | ((hi ^ ((hi >> 1) & 1)) << 16)
    return stream, swap


@pytest.fixture
def uploaded(monkeypatch):
    def dump(arr):
        stream, sites, sq, sw, info = dump_device(arr)
        stream, sw = x_first(stream, sw)
        return stream, sites, sq, sw, info

    monkeypatch.setattr(stream_emu, "dump", dump)


CIRCUITS = [("rep", lambda: circuits.repetition_code_memory(7, 7, 0.1)),
            ("surface3", lambda: circuits.rotated_surface_code_memory(3, 3, 0.05)),
            ("surface5", lambda: circuits.rotated_surface_code_memory(5, 5, 0.02)),
            ("xor", lambda: xor_chain_circuit(np.random.default_rng(21)))]
CIRCUITS += [(f"random{s}", lambda s=s: random_circuit(3 + 4 * s, 300, np.random.default_rng(s), p=0.1)) for s in range(8)]


@pytest.mark.parametrize("name,circ", CIRCUITS, ids=[n for n, _ in CIRCUITS])
def test_uploaded_program_reproduces_the_oracle(uploaded, name, circ):
    test_compiler.check_circuit(circ(), 170, 5)


def test_uploaded_program_across_windows(uploaded):
    test_compiler.check_circuit(circuits.rotated_surface_code_memory(13, 3, 0.01), 70, 8)


def test_odd_slots_start_in_their_second_plane():
    """The planes of an odd slot are exchanged, nothing else differs but the
    order within two-qubit records, whose neighbours differ in parity as far as
    the record's planes allow."""
    circ = circuits.rotated_surface_code_memory(5, 2, 0.01)
    plain, _, sq0, sw0, _ = stream_emu.dump(circ)
    dev, _, sq1, sw1, _ = dump_device(circ)
    odd = np.arange(len(sw1), dtype=np.uint32) & 1
    assert np.array_equal(sq0, sq1) and np.array_equal(sw0 ^ odd, sw1) and odd.any()
    back, _ = x_first(dev, sw1)
    paired = 0
    for (kind, a, cols), (kind1, b, _), (_, raw, _) in zip(entries(plain.copy()), entries(back), entries(dev.copy())):
        assert kind == kind1 and len(a) == len(b)
        if kind in (E.SEG_CNOT, E.SEG_CZ, E.SEG_G2):
            assert sorted(map(tuple, a)) == sorted(map(tuple, b))
            cls = (raw[:, 0] & 1) | ((raw[:, 1] & 1) << 1)
            n = np.bincount(cls, minlength=4)
            pairs = min(n[0], n[3]) + min(n[1], n[2])
            assert all(cls[2 * i] ^ cls[2 * i + 1] == 3 for i in range(pairs))
            paired += pairs
        else:
            assert np.array_equal(a, b)
    assert paired
