"""Growing buffers on a fake allocator (CPU): new memory is reported as new.

An allocator may hand out the address it was just given back, for a larger
block whose contents are not the old ones.
"""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "artefact_b200" / "csrc"

SOURCE = r"""
#include "growbuf.h"
#include <cstdio>
static char arena[16];
static int fails, live;
struct Same {  // every block at the same address
    static int alloc(void **p, size_t) { if (fails) return 7; live++; *p = arena; return 0; }
    static void free(void *) { live--; }
};
#define CHECK(c) if (!(c)) { std::printf("line %d: " #c "\n", __LINE__); return 1; }
int main()
{
    art::GrowBuf<Same> b;
    CHECK(!b.fresh && !b.ensure(1) && b.fresh && b.n == 2u << 20);
    b.fresh = false;
    CHECK(!b.ensure(b.n) && !b.fresh);                         // large enough: the same memory
    CHECK(!b.ensure(b.n + 1) && b.fresh && b.n == 4u << 20 && b.p == arena && live == 1);
    b.fresh = false;
    fails = 1;
    CHECK(b.ensure(b.n + 1) == 7 && !b.p && !b.n && live == 0);
    fails = 0;
    CHECK(!b.ensure(4u << 20) && b.fresh && b.n == 4u << 20);  // the old size again, other memory
    b.fresh = false;
    b.release();
    CHECK(!b.p && !b.n && live == 0 && !b.ensure(1) && b.fresh);
    return 0;
}
"""


def test_new_memory_is_fresh_whatever_its_address(tmp_path):
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), "-o", str(tmp_path / "t"),
                    str(tmp_path / "t.cpp")], check=True)
    res = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
