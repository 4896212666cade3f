"""How the sort cuts its input (csrc/chunks.cuh), compiled for the host: every entry is in one place, up to the
largest number of entries that the library takes (2^31 - 1); the chunk of a CTA that gets nothing is empty."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include <cstdio>
#include "chunks.cuh"

int main() {
  const uint32_t top = 0x7fffffffu;
  const uint32_t counts[] = {0, 1, 1023, 1024, 65537, 282624, 2000000, top - 200000, top - 151552, top - 150000,
                             top - 1024, top - 31, top};
  const int ctas_list[] = {1, 32, 33, 132, 148, 160};
  const int items_list[] = {2, 4, 8, 16};
  for (uint32_t n : counts)
    for (int ctas : ctas_list)
      for (int items : items_list) {
        const uint32_t tile = 1024u * items;
        const hb::SortChunks c(n, ctas, 1024);
        if (c.chunk % 1024 || (uint64_t)c.chunk * ctas < n) return std::printf("chunk n=%u ctas=%d\n", n, ctas), 1;
        uint32_t next = 0;
        for (int r = 0; r < ctas; ++r) {
          if (c.begin(r) != next || c.end(r) < next || c.end(r) > n) return std::printf("cut n=%u ctas=%d r=%d\n", n, ctas, r), 1;
          next = c.end(r);
          // the last tiles of the chunk, whose entries lie around its end: taken below the end, in 64 bits too
          const uint32_t tiles = (c.chunk + tile - 1) / tile;
          for (uint32_t t = tiles > 2 ? tiles - 2 : 0; t < tiles; ++t)
            for (uint32_t at = 0; at < tile; at += (at % 1024 < 33 || at % 1024 > 990) ? 1 : 31) {
              const uint64_t exact = (uint64_t)r * c.chunk + (uint64_t)t * tile + at;
              const bool taken = c.entry(r, t, tile, at) < c.end(r), mine = exact < c.end(r);
              if (taken != mine || (taken && c.entry(r, t, tile, at) != exact))
                return std::printf("entry n=%u ctas=%d r=%d t=%u at=%u\n", n, ctas, r, t, at), 1;
              // what a warp has left from its first entry on, as the ranking counts it
              if ((int64_t)(int32_t)(c.end(r) - c.entry(r, t, tile, at)) != (int64_t)c.end(r) - (int64_t)exact)
                return std::printf("left n=%u ctas=%d r=%d t=%u at=%u\n", n, ctas, r, t, at), 1;
            }
        }
        if (next != n) return std::printf("end n=%u ctas=%d\n", n, ctas), 1;
      }
  // a cluster: chunks of one size, of which the last CTAs may get nothing
  for (uint32_t chunk = 512; chunk <= 4096; chunk *= 2)
    for (int ctas = 1; ctas <= 16; ++ctas)
      for (uint32_t n = 0; n <= chunk * ctas; n += (n % 512 < 3 || n % 512 > 509) ? 1 : 101) {
        const hb::SortChunks c(n, chunk);
        uint32_t next = 0;
        for (int r = 0; r < ctas; ++r) {
          if (c.begin(r) != next || c.end(r) < next || c.end(r) - c.begin(r) > chunk)
            return std::printf("cluster n=%u chunk=%u ctas=%d r=%d\n", n, chunk, ctas, r), 1;
          next = c.end(r);
        }
        if (next != n) return std::printf("cluster end n=%u chunk=%u ctas=%d\n", n, chunk, ctas), 1;
      }
  return 0;
}
"""


def test_every_entry_is_in_one_chunk(tmp_path):
    (tmp_path / "chunks.cpp").write_text(PROGRAM)
    exe = tmp_path / "chunks"
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=signed-integer-overflow", "-fno-sanitize-recover", "-I",
                    str(ROOT / "hades_b200" / "csrc"), str(tmp_path / "chunks.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
