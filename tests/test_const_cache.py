"""The constant cache's rule alone (const_cache.h), stepped on the CPU: no two
places that one call holds overlap, and a place keeps its bytes until the call
that holds it is over, through several fillings of the buffer."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <cstdio>
#include <string>
#include <utility>
#include "const_cache.h"

struct Held { size_t off, bytes; std::string want; };

int main(int argc, char** argv) {
    const size_t cap = 1 << 16;
    vta::ConstCache cc;
    cc.init(cap);
    std::string dev(cap, '\0');  // the device buffer: uploads land in order
    unsigned rng = 1;
    auto next = [&] { return rng = rng * 1664525u + 1013904223u, rng >> 8; };
    auto bytes_of = [](unsigned key, size_t n) {
        std::string s(n, '\0');
        for (size_t i = 0; i < n; ++i) s[i] = (char)((key + 1) * 2654435761u >> (i % 24));
        return s;
    };
    long hits = 0, places = 0, none = 0;
    for (int call = 0; call < 20000; ++call) {
        cc.begin_call();
        std::vector<Held> held;
        const int uploads = 1 + next() % 6;
        for (int u = 0; u < uploads; ++u) {
            // one list in two is an old one, as a sweep's periods are
            const unsigned key = next() % 2 ? next() % 8 : 1000 + next();
            const size_t n = key < 8 ? 100 + 700 * key : 1 + next() % 5000;
            const std::string s = bytes_of(key, n);
            size_t off = 0;
            if (cc.find(s.data(), n, &off)) ++hits;
            else if (cc.place(s.data(), n, &off)) {
                ++places;
                dev.replace(off, n, s);
                cc.keep(off, n);
            } else { ++none; continue; }  // the caller's own slot
            if (off % 256 || off + n > cap) return std::printf("bad place %zu\n", off), 1;
            for (const Held& h : held)
                if (h.off < off + n && off < h.off + h.bytes && !(h.off == off && h.bytes == n && h.want == s))
                    return std::printf("call %d: two places overlap\n", call), 1;
            held.push_back({off, n, s});
        }
        for (const Held& h : held)  // what the call's kernels read
            if (dev.compare(h.off, h.bytes, h.want)) return std::printf("call %d: bytes changed\n", call), 1;
    }
    size_t off = 0;
    const std::string big(cap + 1, 'x');
    if (cc.place(big.data(), big.size(), &off)) return std::printf("too large\n"), 1;
    std::printf("%ld %ld %ld\n", hits, places, none);
    return hits > 1000 && places > 1000 && none > 0 ? 0 : 1;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_places_of_a_call_stay_its_own(tmp_path):
    src = tmp_path / "cc.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "cc"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "vectorta_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
