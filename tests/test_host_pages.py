"""First touch of a caller's pages (CPU: the host code is compiled and run): no thread or no memory for one is
no error, and the caller's own thread takes the rest; no value changes, in the array or beside it."""
import os
import shutil
import subprocess

import pytest
from conftest import PKG_NAME, ROOT

HEAD = r'''
#include <sys/mman.h>
#include <cstdlib>
#include <new>
#include <vector>
#include "pic_host_pages.h"
static long fresh(size_t bytes) {  // pages of a fresh mapping that are there after the touch, -1: not all
    char* p = (char*)mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    pic::touch_pages(p, bytes);
    const size_t page = sysconf(_SC_PAGESIZE), n = (bytes + page - 1) / page;
    unsigned char* in = (unsigned char*)malloc(n);
    mincore(p, bytes, in);
    long have = 0;
    for (size_t k = 0; k < n; k++) have += in[k] & 1;
    free(in);
    munmap(p, bytes);
    return have == (long)n ? have : -1;
}
'''


def run(tmp_path, src):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    f, exe = tmp_path / "t.cpp", tmp_path / "t"
    f.write_text(HEAD + src)
    subprocess.run([gxx, "-O1", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, PKG_NAME, "csrc"), str(f), "-o",
                    str(exe)], check=True)
    return subprocess.run([str(exe)]).returncode


@pytest.mark.parametrize("threads", [0, 1, 3])
def test_no_memory_for_a_thread(tmp_path, threads):
    assert run(tmp_path, r'''
static int left = 1 << 30;
void* operator new(size_t n) {  // a thread's state takes one allocation
    if (left-- <= 0) throw std::bad_alloc();
    return malloc(n);
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }
int main() {
    left = %d;
    return fresh(64u << 20) > 0 ? 0 : 1;
}
''' % threads) == 0


def test_values_stay(tmp_path):
    assert run(tmp_path, r'''
int main() {
    const size_t page = sysconf(_SC_PAGESIZE);
    const size_t sizes[] = {0, 1, 8, page - 1, page, page + 1, 3 * page + 8, (8u << 20) - 1, (16u << 20) + 3 * page + 8, 41u << 20};
    for (size_t bytes : sizes)
        for (size_t at : {(size_t)0, (size_t)8, page - 8, page + 1}) {
            std::vector<unsigned char> v(bytes + at + 2 * page);
            for (size_t k = 0; k < v.size(); k++) v[k] = (unsigned char)(k * 7 + 1);
            pic::touch_pages(v.data() + at, bytes);
            for (size_t k = 0; k < v.size(); k++)
                if (v[k] != (unsigned char)(k * 7 + 1)) return 1;
        }
    // pages that cannot be written are left to the copy's own error
    void* ro = mmap(nullptr, 4 * page, PROT_READ, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    pic::touch_pages(ro, 4 * page);
    return 0;
}
''') == 0


@pytest.mark.parametrize("bytes_", [1, 70_000, 8 << 20, 64 << 20])
def test_fresh_pages_are_there(tmp_path, bytes_):
    assert run(tmp_path, "int main() { return fresh(%d) > 0 ? 0 : 1; }" % bytes_) == 0
