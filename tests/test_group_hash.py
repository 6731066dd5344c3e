"""The hash that instances are grouped by (tc_group_key.h), compiled for the host: whatever the keys differ in, the
grouping's table needs few probes, and next to no record is read of an instance of another key."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

KEY = np.dtype([(n, np.uint64) for n in ("positions", "normals", "texcoords", "clusters", "localTriangles")]
               + [(n, np.uint32) for n in ("map", "numClusters", "scale", "offset")])
SOURCE = """
#include "tc_group_key.h"
extern "C" void hashes(const tc::GroupKey* k, int n, uint64_t* hash, uint32_t* slot, uint16_t* print) {
  static_assert(sizeof(tc::GroupKey) == 56, "");
  for(int i = 0; i < n; i++)
    hash[i] = tc::group_hash(k[i]), slot[i] = tc::group_slot(hash[i]), print[i] = tc::group_print(hash[i]);
}
"""
N = 4096  # the most instances that are grouped


@pytest.fixture(scope="module")
def hashes(tmp_path_factory):
    d = tmp_path_factory.mktemp("hash")
    (d / "h.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "vk_tessellated_clusters_gb300", "csrc"),
                           str(d / "h.cpp"), "-o", str(d / "h.so")])
    lib = ctypes.CDLL(str(d / "h.so"))

    def run(keys):
        out = [np.zeros(len(keys), t) for t in (np.uint64, np.uint32, np.uint16)]
        lib.hashes(*[ctypes.c_void_p(keys.ctypes.data), len(keys)], *[ctypes.c_void_p(o.ctypes.data) for o in out])
        return out
    return run


def _bits(x):
    return np.asarray(x, np.float32).view(np.uint32)


def _keys(case):
    k, i = np.zeros(N, KEY), np.arange(N)
    for n in KEY.names[:5]:
        k[n] = 0x7F2A00000000 + 0x40000 * KEY.names.index(n)
    k["numClusters"], k["scale"] = 200, _bits(0.03)
    if case in KEY.names[:5]:
        k[case] += np.uint64(256) * i.astype(np.uint64)  # allocations next to one another
    elif case == "pages":
        k["normals"] += (i.astype(np.uint64) << np.uint64(21))
    elif case in ("map", "numClusters"):
        k[case] = i
    elif case in ("scale", "offset"):
        k[case] = _bits(0.001 * (i + 1))
    elif case == "powers":
        k["offset"], k["scale"] = _bits(2.0 ** (i % 64 - 32)), _bits(2.0 ** (i // 64 - 32))
    elif case == "seeded":
        rng = np.random.default_rng(5)
        k["offset"], k["scale"] = _bits(rng.random(N)), _bits(rng.random(N))
        k["positions"] += np.uint64(0x100000) * (i % 4).astype(np.uint64)
    elif case == "groups":  # 8 to a group
        k["offset"] = _bits(0.001 * (i // 8))
    return k


@pytest.mark.parametrize("case", ["positions", "normals", "texcoords", "clusters", "localTriangles", "pages", "map",
                                  "numClusters", "scale", "offset", "powers", "seeded", "groups"])
def test_few_probes(hashes, case):
    keys = _keys(case)
    hash_, slot, fingerprint = hashes(keys)
    distinct = len(np.unique(keys))
    assert distinct == (N // 8 if case == "groups" else N) and len(np.unique(hash_)) == distinct
    assert slot.max() < 2 * N
    table, probes, foreign, longest = {}, 0, 0, 0
    for i in range(N):
        s, chain = int(slot[i]), 0
        while True:
            chain += 1
            found = table.get(s)
            if found is None:
                table[s] = i
                break
            if fingerprint[found] == fingerprint[i]:
                if keys[found] == keys[i]:
                    break
                foreign += 1
            s = (s + 1) % (2 * N)
        probes += chain
        longest = max(longest, chain)
    # linear probing in a half full table takes 1.5 probes in the mean and has chains of a few dozen
    assert probes <= 2 * N and longest <= 64 and foreign <= N // 256, (probes / N, longest, foreign)
