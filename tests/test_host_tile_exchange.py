"""Shared-memory exchange of the tile FFT (csrc/fft_tile_layout.h, compiled for the host): every value has its place, banks.

8-byte accesses are served per half-warp from 16 bank pairs.  Both strides of the exchange are odd, so a half-warp whose 16 lanes
run along one index meets 16 pairs; one that spans two lines or columns of 8 lanes each at most twice each.
"""
import json
import subprocess

import pytest

SRC = r"""
#include <cstdio>
#include "%s"
using namespace fftso3::ffast;
template <int R, bool C2T, bool REAL>
void one(bool& first)
{
    constexpr int A = rad_a<R, C2T>(), B = rad_b<R, C2T>(), ROWS = REAL ? TL / 2 : TL;
    std::printf("%%s{\"R\":%%d,\"c2t\":%%d,\"real\":%%d,\"A\":%%d,\"B\":%%d,\"rows\":%%d,\"size\":%%d,\"s1\":[", first ? "" : ",", R, C2T, REAL, A, B,
                ROWS, ROWS * tile_ls<R, C2T>());
    first = false;
    for (int u = 0; u < ROWS * B; ++u) {
        const TilePlace p = step1_place<R, C2T, REAL>(u);
        std::printf("%%s[%%d,%%d", u ? "," : "", p.l, p.x);
        for (int k = 0; k < A; ++k) std::printf(",%%d", step1_slot<R, C2T>(p, k));
        std::printf("]");
    }
    std::printf("],\"s2\":[");
    for (int u = 0; u < ROWS * A; ++u) {
        const TilePlace p = step2_place<R, C2T, REAL>(u);
        std::printf("%%s[%%d,%%d", u ? "," : "", p.l, p.x);
        for (int j = 0; j < B; ++j) std::printf(",%%d", step2_slot<R, C2T>(p, j));
        std::printf("]");
    }
    std::printf("]}");
}
template <int R>
void all(bool& f)
{
    one<R, true, false>(f);
    one<R, true, true>(f);
    one<R, false, false>(f);
    one<R, false, true>(f);
}
int main()
{
    bool f = true;
    std::printf("[");
    all<2>(f), all<4>(f), all<8>(f), all<16>(f), all<32>(f);
    std::printf("]");
}
"""


@pytest.fixture(scope="module")
def tiles(tmp_path_factory):
    import os
    from conftest import ROOT
    d = tmp_path_factory.mktemp("tile")
    src, exe = d / "t.cpp", d / "t"
    src.write_text(SRC % os.path.join(ROOT, "fftso3_gb300", "csrc", "fft_tile_layout.h"))
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", str(exe), str(src)], check=True)
    return json.loads(subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout)


def test_every_value_has_its_place(tiles):
    assert len(tiles) == 20
    for t in tiles:
        assert t["A"] * t["B"] == 32 * t["R"]
        put, got = {}, {}
        for l, x, *slots in t["s1"]:
            put.update({s: (l, k1, x) for k1, s in enumerate(slots)})
        for l, x, *slots in t["s2"]:
            got.update({s: (l, x, j2) for j2, s in enumerate(slots)})
        assert put == got and len(put) == t["rows"] * 32 * t["R"]
        assert set(v[0] for v in put.values()) == set(range(t["rows"])) and max(put) < t["size"]


def test_banks(tiles):
    for t in tiles:
        for step in ("s1", "s2"):
            for h in range(0, len(t[step]), 16):
                lanes = t[step][h:h + 16]
                along_one = len({p[0] for p in lanes}) == 1 or len({p[1] for p in lanes}) == 1
                for i in range(2, len(lanes[0])):
                    pairs = [p[i] % 16 for p in lanes]
                    ways = max(pairs.count(b) for b in set(pairs))
                    assert ways <= (1 if along_one else 2), (t["R"], t["c2t"], t["real"], step, h)
