"""The page touching of copies into a caller's memory (host_copy.hpp), compiled
against a stand-in for the CUDA call it asks about the pointer: memory that has
its pages is left alone, fresh memory gets all of them and nothing beyond.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <sys/mman.h>
#include "host_copy.hpp"
static cudaMemoryType g_type = cudaMemoryTypeUnregistered;
extern "C" cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  a->type = g_type;
  return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError(void) { return cudaSuccess; }
int main(int argc, char** argv) {
  const size_t page = sysconf(_SC_PAGESIZE), bytes = strtoull(argv[1], 0, 10), piece = strtoull(argv[2], 0, 10);
  const size_t there = strtoull(argv[3], 0, 10);  // bytes from the start that have pages, filled with 0xa5
  if (argv[4][0] == 'p') g_type = cudaMemoryTypeHost;
  const size_t pages = bytes / page + 8;
  char* m = (char*)mmap(0, pages * page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  madvise(m, pages * page, MADV_NOHUGEPAGE);
  char* p = m + 3 * page + 20;  // not the start of a page
  if (there) memset(p, 0xa5, there);
  {
    umwm::PageTouch t(p, bytes, piece);
    for (size_t c = 0; c * piece < bytes; ++c) t.wait(c);
  }
  unsigned char* v = (unsigned char*)malloc(pages);
  if (mincore(m, pages * page, v)) return 2;
  size_t in = 0, out = 0, changed = 0;
  for (size_t i = 0; i < pages; ++i) {  // whole pages of the range, and pages outside it
    char *a = m + i * page, *b = a + page;
    if (a >= p && b <= p + bytes) in += !(v[i] & 1);
    if (b <= p || a >= p + bytes) out += v[i] & 1;
  }
  for (size_t i = 0; i < there; ++i) changed += p[i] != (char)0xa5;
  printf("%zu %zu %zu\n", in, out, changed);
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp("host_copy")
    (d / "t.cpp").write_text(SRC)
    exe = str(d / "t")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + CUDA, "-I" + os.path.join(ROOT, "umwm_gb300", "csrc"), str(d / "t.cpp"),
                    "-o", exe, "-lpthread"], check=True)

    def run(nbytes, piece, there, kind="u"):
        out = subprocess.run([exe, str(nbytes), str(piece), str(there), kind], check=True, capture_output=True, text=True)
        return [int(x) for x in out.stdout.split()]

    return run


MB = 1 << 20


@pytest.mark.parametrize("nbytes,piece", [(24 * MB, 32 * MB), (70 * MB + 12, 32 * MB), (5 * MB, 4 * MB)])
def test_memory_with_pages_is_left_alone(probe, nbytes, piece):
    missing, beyond, changed = probe(nbytes, piece, nbytes)
    assert (missing, beyond, changed) == (0, 0, 0)


@pytest.mark.parametrize("nbytes,piece", [(24 * MB, 32 * MB), (70 * MB + 12, 32 * MB), (5 * MB, 4 * MB)])
@pytest.mark.parametrize("there", [0, 100, 1 * MB])
def test_fresh_memory_gets_its_pages(probe, nbytes, piece, there):
    missing, beyond, _ = probe(nbytes, piece, there)
    assert (missing, beyond) == (0, 0)


def test_pinned_and_small_memory_is_left_alone(probe):
    missing, beyond, _ = probe(24 * MB, 32 * MB, 0, "p")
    assert missing > 0 and beyond == 0
    missing, beyond, _ = probe(1 * MB, 32 * MB, 0)
    assert missing > 0 and beyond == 0
