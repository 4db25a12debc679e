"""The byte arithmetic of the tag search (imagestack_b200/csrc/lattice_compact.cuh), compiled
for the host and compared with a loop over the bytes."""
import os
import subprocess

import pytest

from imagestack_b200 import build

PROGRAM = r"""
#include <cstdio>
#include "lattice_compact.cuh"
static uint64_t state = 88172645463325252ull;
static uint64_t next() { state ^= state << 13; state ^= state >> 7; return state ^= state << 17; }
int main() {
    const uint8_t few[] = {0, 1, 2, 3, 5, 0x81, 0xFF, 0x02};
    for (int n = 0; n < 4000000; ++n) {
        uint64_t word = 0;
        for (int b = 0; b < 8; ++b) {
            const uint8_t t = n % 3 ? few[next() % (n % 2 ? 8 : 5)] : (uint8_t)next();
            word |= (uint64_t)(t ? t | 1 : 0) << (8 * b);
        }
        const uint8_t tag = (n % 3 ? few[next() % 8] : (uint8_t)next()) | 1;
        const uint32_t first = next() % 8;
        bool end, is_end = false;
        const uint64_t got = pgpu::tag_matches(word, first, tag, &end);
        uint64_t must = 0, may = 0;
        for (uint32_t s = first; s < 8; ++s) {
            const uint8_t t = (uint8_t)(word >> (8 * s));
            if (!t) { is_end = true; break; }
            may |= 0x80ull << (8 * (s - first));
            if (t == tag) must |= 0x80ull << (8 * (s - first));
        }
        if (end != is_end || (must & ~got) || (got & ~may)) {
            printf("word %016llx first %u tag %02x: %016llx, end %d\n", (unsigned long long)word, first, tag,
                   (unsigned long long)got, end);
            return 1;
        }
    }
    return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(build.NVCC), reason="no nvcc")
def test_tag_matches_stay_in_their_word(tmp_path):
    src = tmp_path / "tags.cu"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "tags")
    subprocess.run([build.NVCC] + build.ARCH + ["-std=c++17", "-O2", "-ccbin", build.HOSTCXX, "-I", build.CSRC,
                                                "-I", build.INCLUDE, str(src), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
