"""The indexer's score order and value bins, compiled for the host: no GPU needed."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BINS = 4096


@pytest.fixture(scope="module")
def bins(tmp_path_factory):
    d = tmp_path_factory.mktemp("dsa_bins")
    src = d / "bins.cc"
    src.write_text('#include "dsa_bins.h"\n'
                   'extern "C" int bin(float s, float lowest, float scale) { return syfi::score_bin(s, lowest, scale); }\n'
                   'extern "C" unsigned key(float s) { return syfi::score_key(s); }\n'
                   'extern "C" float back(unsigned k) { return syfi::key_score(k); }\n'
                   'extern "C" int count() { return syfi::kBins; }\n')
    csrc = os.path.join(ROOT, "mlsys-contest-syfi-agent-assisted_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + csrc, str(src), "-o", str(d / "bins.so")], check=True)
    lib = ctypes.CDLL(str(d / "bins.so"))
    lib.bin.argtypes = [ctypes.c_float] * 3
    lib.key.argtypes, lib.key.restype = [ctypes.c_float], ctypes.c_uint32
    lib.back.argtypes, lib.back.restype = [ctypes.c_uint32], ctypes.c_float
    assert lib.count() == BINS
    return lib


@pytest.mark.parametrize("lowest,highest", [(-3.5, 8.25), (0.0, 1e-30), (-1e30, 1e30), (5.0, 5.0001)])
def test_every_score_has_a_bin_inside_the_table(lowest, highest, bins):
    """Also a score outside the range the bins were laid over: it indexes a table in shared memory."""
    lowest, highest = np.float32(lowest), np.float32(highest)
    scale = np.float32(BINS - 1) / (highest - lowest)
    span = highest - lowest
    outside = [lowest - span, np.nextafter(lowest, np.float32(-np.inf)), np.float32(-3e38), -np.inf,
               highest + span, np.float32(3e38), np.inf]
    inside = np.sort(np.concatenate([np.linspace(lowest, highest, 2001, dtype=np.float32), [lowest, highest]]))
    with np.errstate(over="ignore"):
        scores = np.sort(np.concatenate([inside, np.array(outside, dtype=np.float32)]))
    got = [bins.bin(float(s), float(lowest), float(scale)) for s in scores]
    assert min(got) >= 0 and max(got) <= BINS - 1
    assert got == sorted(got)
    assert bins.bin(float(lowest), float(lowest), float(scale)) == 0
    assert bins.bin(-np.inf, float(lowest), float(scale)) == 0 and bins.bin(np.inf, float(lowest), float(scale)) == BINS - 1
    assert bins.bin(float("nan"), float(lowest), float(scale)) == 0


def test_keys_order_scores_and_come_back(bins):
    s = np.array([-np.inf, -3e38, -1.0, -1e-40, -0.0, 0.0, 1e-40, 1.0, 3e38, np.inf], dtype=np.float32)
    keys = [bins.key(float(x)) for x in s]
    assert keys == sorted(set(keys)) and keys[0] > 0
    assert [np.float32(bins.back(k)) for k in keys] == list(s)
