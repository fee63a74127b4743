"""The table that keeps tensor-map descriptors (csrc/map_table.h), compiled on its own: the descriptors that a decode loop
cycles through must stay in it."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "ezops_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "map_table.h"

struct Key {
    unsigned long long base;
    int box;
    bool operator==(const Key& o) const { return base == o.base && box == o.box; }
    uint64_t hash() const { return ezb::hash_mix(ezb::hash_mix(base, 0), (uint64_t)box); }
};
using Table = ezb::MapTable<Key, long long, 256>;

// Keys asked for `rounds` times in a fixed order; misses of the last round, -1 on a wrong value.
static long long cycle(Table& t, const std::vector<Key>& keys, int rounds) {
    long long misses = 0;
    for (int r = 0; r < rounds; ++r) {
        misses = 0;
        for (size_t i = 0; i < keys.size(); ++i) {
            const long long want = (long long)(keys[i].base * 64 + keys[i].box);
            if (const long long* v = t.find(keys[i])) {
                if (*v != want) return -1;
            } else {
                ++misses;
                t.put(keys[i], want);
            }
        }
    }
    return misses;
}

int main() {
    auto model = [](int layers, int batches, unsigned long long step) {
        std::vector<Key> keys;
        for (int b = 0; b < batches; ++b)
            for (int l = 0; l < layers; ++l)
                for (int m = 0; m < 5; ++m) keys.push_back({0x7f0000000000ull + (unsigned long long)(l * 5 + m) * step, 8 + 3 * b + m});
        return keys;
    };
    Table* t = new Table;
    for (unsigned long long step : {2097152ull, 512ull, 33554432ull, 104857600ull})
        for (int layers : {28, 64})
            for (int batches : {1, 2, 4}) printf("%lld\n", cycle(*t, model(layers, batches, step), 3));
    // far more keys than entries: values stay right, every key is found directly after it was put
    std::vector<Key> many = model(6000, 2, 4096);
    printf("%d\n", cycle(*t, many, 1) >= 0);
    for (const Key& k : many) {
        t->put(k, 7);
        if (!t->find(k) || *t->find(k) != 7) printf("lost\n");
    }
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_decode_loops_fit_the_table(tmp_path):
    """A loop over 28 or 64 layers at one, two or four batch sizes misses nothing from its second round on, whatever the
    distance of the weights in memory (a table of 256 entries replaced in turn missed every look-up of most of these)."""
    (tmp_path / "t.cc").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), str(tmp_path / "t.cc"), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0"] * 24 + ["1"]
