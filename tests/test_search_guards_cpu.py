"""Guards of the selection and of the resident search that need no GPU: the register sort
refuses more keys per thread than it can order, and an entry of the survivor list is taken
for a survivor only if it names a parent and a place in its list, and applied only inside
the parent's present list."""
import os
import subprocess

import pytest

from beamsearch_jssp_gpu_gb300 import build as B

SORT = '#define BSJ_SELECT_THREADS {threads}\n#include "bsj_select.cuh"\n'
ENTRY = """
#include <cstdio>
#include "bsj_kernels.h"
int main()
{
    unsigned e;
    int P, n;
    while (std::scanf("%u %d %d", &e, &P, &n) == 3)
        std::printf("%d\\n", (n > 0 ? bsj::search_entry_ok(e, P, n) : bsj::search_position_ok(P, e)) ? 1 : 0);
}
"""


def _nvcc(tmp_path, source, *flags):
    src = tmp_path / "t.cu"
    src.write_text(source)
    return subprocess.run([B.nvcc(), *B.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", B.CSRC, *flags, str(src)],
                          capture_output=True, text=True, cwd=tmp_path)


@pytest.mark.parametrize("threads,ok", [(1024, True), (512, True), (256, False)])
def test_register_sort_keys_per_thread(tmp_path, threads, ok):
    r = _nvcc(tmp_path, SORT.format(threads=threads), "-cuda", "-o", os.devnull)
    assert (r.returncode == 0) == ok, r.stderr
    assert ok or "at most 32 keys per thread" in r.stderr


def test_survivor_entries(tmp_path):
    r = _nvcc(tmp_path, ENTRY, "-o", str(tmp_path / "t"))
    assert r.returncode == 0, r.stderr
    filler = 1 << 31
    cases = [(0, 1, 1, 1), (127, 1, 128, 1), (127, 1, 127, 0), (128, 1, 128, 0), (4095 << 7 | 49, 4096, 50, 1),
             (4095 << 7 | 50, 4096, 50, 0), (4096 << 7, 4096, 50, 0), (filler | 16383 << 7 | 3, 16384, 4, 1),
             (filler | 16384 << 7, 16384, 4, 0), (0xFFFFFFFF, 16384, 128, 0), (0x7FFFFFFF, 16384, 128, 0), (0, 0, 5, 0)]
    # a list's header, a position in it (told apart by the last number)
    cases += [(3, 2, 0, 1), (3, 3, 0, 0), (3, -1, 0, 0), (7 << 16, 0, 0, 0), (7 << 16 | 1, 0, 0, 1)]
    text = "\n".join(f"{e} {P} {n}" for e, P, n, _ in cases)
    got = subprocess.run([str(tmp_path / "t")], input=text, capture_output=True, text=True).stdout.split()
    assert [int(x) for x in got] == [c[3] for c in cases]
