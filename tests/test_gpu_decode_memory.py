"""Staging a decoded stream and running a batch take no memory from operator
new in proportion to the frame or the batch: a failure there is an exception,
which must not cross the C interface (a failed malloc or cudaMallocHost is a
status).  A child process runs with an operator new that refuses large
blocks while the calls run."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

REFUSE = """
#include <cstdlib>
#include <new>
static size_t limit = (size_t)-1;
extern "C" void refuse_above(size_t n) { limit = n; }
void* operator new(size_t n) {
  void* p = n > limit ? nullptr : std::malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void* operator new[](size_t n) { return operator new(n); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete[](void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
void operator delete[](void* p, size_t) noexcept { std::free(p); }
"""

CHILD = """
import ctypes as C, sys
from pathlib import Path
import numpy as np
import jpxl_gb300 as jg
golden = Path("tests/golden/codestream")
large = (golden / "64_vardct_lfgroupseam_rgb_128x2176_nofilters_d6.jxl").read_bytes()
small = (golden / "63_vardct_outofgamut_rgb_64x64_nofilters_d4.jxl").read_bytes()
refuse = C.CDLL(sys.argv[1]).refuse_above
refuse.argtypes = [C.c_size_t]
off = 2 ** 64 - 1
ctx = jg.Context(0)
cs = jg.Codestream(large)
want = cs.render(ctx, "srgb8")
refuse(1 << 20)  # the coefficient image of the frame is 3.3 MB
got = cs.render(ctx, "srgb8")
refuse(off)
assert np.array_equal(got, want)
streams = [jg.Codestream(small) for _ in range(400)]
batch = jg.DecodeBatch(ctx, streams, "srgb8", lanes=4)
refuse(2000)  # a word per stream is 3200 bytes
outs = batch.run()
refuse(off)
want = streams[0].render(ctx, "srgb8")
assert all(np.array_equal(o, want) for o in outs)
batch.close()
print("done")
"""


def test_large_blocks_refused(ctx, tmp_path):
    src, lib = tmp_path / "refuse.cpp", tmp_path / "librefuse.so"
    src.write_text(REFUSE)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
    res = subprocess.run([sys.executable, "-c", CHILD, str(lib)], cwd=ROOT, text=True,
                         capture_output=True, timeout=300,
                         env={**os.environ, "LD_PRELOAD": str(lib)})
    assert res.returncode == 0 and "done" in res.stdout, (res.returncode, res.stderr[-2000:])
