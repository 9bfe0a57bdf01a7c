"""Growth of the plaquette-loop buffer with a fake allocator, on the host: which size a request aims at,
what is tried when memory is short, and when a buffer is kept."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "ecmc-qncb_b200" / "csrc"

PROGRAM = r"""
#include "loop_buf.h"
#include <cstdio>
#include <vector>
using namespace qcb;
static size_t room;                  // the fake device's largest free block
static std::vector<size_t> asked;
static int freed;
static bool grow(LoopBuf* b, size_t want, size_t least) {
  asked.clear();
  return loops_grow(b, want, least,
                    [](size_t n) { asked.push_back(n); return n <= room ? (void*)0x1000 : nullptr; },
                    [](void*) { ++freed; });
}
#define CHECK(x) if (!(x)) return std::printf("line %d: %s\n", __LINE__, #x), 1
int main() {
  const size_t M = 1 << 20, G = 1 << 30;
  {
    LoopBuf b;
    room = 100 * G;
    CHECK(grow(&b, 5 * G, 3 * M) && b.bytes == G && asked.size() == 1);  // capped at 1 GiB
    CHECK(grow(&b, 5 * G, 3 * M) && asked.empty() && b.gen == 1);        // and then kept
    CHECK(grow(&b, 5 * G, 2 * G) && b.bytes == 2 * G && freed == 1 && b.gen > 1);  // two slices need more
  }
  {
    LoopBuf b;
    room = 300 * M;
    CHECK(grow(&b, 4 * G, 100 * M));  // halves until it fits
    CHECK((asked == std::vector<size_t>{G, G / 2, G / 4}) && b.bytes == G / 4);
    room = 100 * G;
    CHECK(grow(&b, 4 * G, 100 * M) && asked.empty());  // the same request is not tried again
    room = 150 * M;
    CHECK(grow(&b, 4 * G, 140 * M) && asked.empty());  // nor one that the buffer answers
    CHECK(!grow(&b, 4 * G, 400 * M) && b.p == nullptr && b.bytes == 0);
    CHECK(asked.back() == 400 * M && asked.size() == 3);  // 1 GiB, 512 MiB, then exactly the least
    room = 100 * G;
    CHECK(grow(&b, 4 * G, 400 * M) && b.bytes == G);  // memory is there again
  }
  {
    LoopBuf b;
    b.limit = 10 * M;
    room = 100 * G;
    CHECK(grow(&b, 4 * G, 4 * M) && b.bytes == 10 * M);
    CHECK(!grow(&b, 4 * G, 11 * M));  // two slices do not fit into the user's limit
    CHECK(b.bytes == 10 * M && asked.empty());  // other lattices go on using what there is
    b.limit = 0;
    loops_drop(&b, [](void*) {});
    CHECK(!grow(&b, 4 * G, 4 * M) && asked.empty());
  }
  return 0;
}
"""


def test_growth(tmp_path):
    src, exe = tmp_path / "grow.cpp", tmp_path / "grow"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_limit_needs_a_context():
    import qcb

    lib = qcb._lib.lib()
    assert lib.qcb_ctx_set_loop_bytes(None, 0) == 1
    assert b"null" in lib.qcb_last_error()
