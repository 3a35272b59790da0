"""The pages of a caller's buffer are all touched, whether or not there is a thread, or memory for
one, to share them: nothing is thrown out of a C entry point.  A small program around host.cpp,
whose allocations fail when told to."""
import os
import subprocess

from conftest import ROOT

SOURCE = r"""
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>
#include <new>
#include "epi_internal.h"
static int left = -1;  // allocations that still succeed (-1: all)
static void* take(size_t n) {
    if (left == 0) throw std::bad_alloc();
    if (left > 0) --left;
    return malloc(n ? n : 1);
}
void* operator new(size_t n) { return take(n); }
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }
int main() {
    const size_t sizes[] = {0, 1, 4096, 4097, (3u << 20) + 1, (6u << 20) + 5, (64u << 20) + 123};
    for (size_t n : sizes)
        for (int k = -1; k < 4; ++k) {
            char* p = (char*)mmap(nullptr, n + 8192, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
            if (p == MAP_FAILED) return 2;
            memset(p, 7, n + 8192);
            char* q = p + 24;  // (not on a page boundary)
            left = k;
            epi::touch_pages(q, n);
            left = -1;
            // a write to every page that the buffer has a byte in, none outside it
            for (size_t page = 0; page < n + 8192; page += 4096) {
                bool touched = false, inside = false;
                for (size_t b = page; b < page + 4096 && b < n + 8192; ++b) {
                    const bool in = b >= 24 && b < 24 + n;
                    inside |= in;
                    if (p[b] == 0) {
                        if (!in) return 3;
                        touched = true;
                    }
                }
                if (inside != touched) return 4;
            }
            munmap(p, n + 8192);
        }
    return 0;
}
"""


def test_every_page_is_touched(tmp_path):
    csrc = os.path.join(ROOT, "epirust_gb300", "csrc")
    main = str(tmp_path / "main.cpp")
    with open(main, "w") as f:
        f.write(SOURCE)
    exe = str(tmp_path / "touch")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", csrc, main, os.path.join(csrc, "host.cpp"), "-o", exe, "-lpthread"],
                   check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])
