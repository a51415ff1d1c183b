"""Host-side rules of the engine (csrc/sj_host.h), compiled alone: g++, no device."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "self-join-hpbdc2019_b200", "csrc")


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text('#include "sj_host.h"\n'
                                 'extern "C" int expand_team(uint64_t n, uint64_t cnt, int threads)\n'
                                 '{ return sj_expand_team(n, cnt, threads); }\n')
    lib = str(d / "rules.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(d / "rules.cpp"), "-o", lib])
    return C.CDLL(lib)


@pytest.mark.parametrize("n,cnt,threads,team", [
    (1000, 5000, 64, 1),                    # a small batch of a small set: no team
    (100_000, 3_200_000, 64, 7),
    (10_000_000, 65_536, 64, 20),           # few pairs, but ten million run offsets to pass over
    (2_000_000_000, 65_536, 64, 64),
    (1000, 2_000_000_000, 64, 64),
    (2**31 - 1, 2**32 - 1, 1, 1), (1, 1, 0, 1)])
def test_key_expansion_team(rules, n, cnt, threads, team):
    assert rules.expand_team(C.c_uint64(n), C.c_uint64(cnt), threads) == team
