"""The rules by which persistent phases are admitted to a device together (csrc/phase_slots.hpp, host
code): as many CTAs as it holds, of which those not yet placed at most one an SM."""
import ctypes
import os
import random
import subprocess
import threading

import pytest

from gkr_gb300 import build as libbuild

SOURCE = """
#include "phase_slots.hpp"
using gkrgpu::PhaseSlots;
extern "C" {
void* new_state() { return new std::atomic<uint64_t>(0); }
uint64_t value(void* s) { return static_cast<std::atomic<uint64_t>*>(s)->load(); }
void* new_slots(void* s, int sms, int per_sm) { return new PhaseSlots(*static_cast<std::atomic<uint64_t>*>(s), sms, per_sm); }
int acquire(void* p, unsigned n, int own_share) { return static_cast<PhaseSlots*>(p)->acquire(n, own_share != 0); }
void placed(void* p) { static_cast<PhaseSlots*>(p)->placed(); }
void drop(void* p) { delete static_cast<PhaseSlots*>(p); }
}
"""
SMS = 152


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("slots")
    (d / "slots.cpp").write_text(SOURCE)
    subprocess.check_call([os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-Wall", "-fPIC", "-shared", "-I", libbuild.CSRC,
                           str(d / "slots.cpp"), "-o", str(d / "slots.so")])
    lib = ctypes.CDLL(str(d / "slots.so"))
    for f in (lib.new_state, lib.new_slots):
        f.restype = ctypes.c_void_p
    lib.value.restype = ctypes.c_uint64
    return lib


class Device:
    def __init__(self, lib, per_sm=2):
        self.lib, self.state, self.per_sm = lib, ctypes.c_void_p(lib.new_state()), per_sm

    def phase(self, n, own_share=True):
        """A phase of n CTAs, or None where it is kept out."""
        p = ctypes.c_void_p(self.lib.new_slots(self.state, SMS, self.per_sm))
        if self.lib.acquire(p, n, int(own_share)):
            return p
        self.lib.drop(p)

    def counts(self):
        v = self.lib.value(self.state)
        return v & 0xFFFFFFFF, v >> 32


def test_what_is_not_placed_stays_within_one_cta_an_sm(lib):
    d = Device(lib)
    a = d.phase(100)
    assert a and d.phase(53) is None and d.counts() == (100, 100)
    b = d.phase(52)
    assert b and d.phase(1) is None
    lib.placed(a)
    assert d.counts() == (152, 52)
    c = d.phase(100)
    assert c and d.counts() == (252, 152) and d.phase(1) is None
    lib.placed(b)
    lib.placed(c)
    e = d.phase(52)
    assert e and d.phase(1) is None  # all that the device holds
    for p in (a, b, c, e):
        lib.drop(p)
    assert d.counts() == (0, 0)


def test_more_ctas_than_sms_wait_for_no_other(lib):
    d = Device(lib)
    a = d.phase(1)
    assert d.phase(153) is None
    lib.placed(a)
    b = d.phase(303)
    assert b and d.phase(1) is None
    lib.placed(b)
    lib.drop(a)
    c = d.phase(1)
    assert c
    lib.drop(b)
    lib.drop(c)
    assert d.phase(305) is None and d.counts() == (0, 0)


def test_beyond_its_share_a_phase_leaves_half_of_the_device(lib):
    d = Device(lib)
    a = d.phase(100, own_share=False)
    lib.placed(a)
    assert a and d.phase(53, own_share=False) is None
    b = d.phase(52, own_share=False)
    lib.placed(b)
    assert b and d.phase(1, own_share=False) is None and d.phase(152)
    assert Device(lib, per_sm=0).phase(1) is None  # a device that holds no phase kernel


def test_phases_of_many_threads(lib):
    d = Device(lib)
    over = []

    def lane(seed):
        rng = random.Random(seed)
        for _ in range(3000):
            p = d.phase(rng.choice([1, 4, 28, 67, 128]), rng.random() < 0.5)
            held, waiting = d.counts()
            if held > 2 * SMS or waiting > SMS or waiting > held:
                over.append((held, waiting))
            if p:
                if rng.random() < 0.8:  # (a phase that fails is dropped before it is placed)
                    lib.placed(p)
                lib.drop(p)

    threads = [threading.Thread(target=lane, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not over and d.counts() == (0, 0)
