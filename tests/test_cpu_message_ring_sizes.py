"""Messages of both kinds in a context's ring (csrc/cuda/message_ring.h): short ones that one block takes and long ones that are for several,
mixed, around operations of the stream.  The model of tests/test_cpu_message_ring.py with sizes, and blocks that know which they are."""
import shutil
import subprocess

import pytest

from tests.test_cpu_message_ring import CUDA, MODEL

CHANGES = [
    # the block's kind, and what it finds in a message's size
    ("static void block(Ring* r, uint32_t next, uint32_t generation) {", "static std::atomic<int> unfit{0};\nstatic uint32_t size_of(uint32_t id);\n"
     "static void block(Ring* r, uint32_t next, uint32_t generation, bool wide) {"),
    ("        done[id].batch = b;", "        const uint32_t n = (uint32_t)v[i][2] & kRingSizeMask;\n        unfit += n != size_of(id) || (n > kRingNarrowMax && !wide);\n"
     "        done[id].batch = b;"),
    ("struct Context {", """static int long_every = 1;
static uint32_t size_of(uint32_t id) { return id % long_every == long_every - 1 ? kRingMessageMax - id % 7 : 1 + id % kRingNarrowMax; }
struct Context {"""),
    ("return writer.message((uint64_t)id, (uint64_t)id + (1ull << 40), 1,", "const uint32_t n = size_of(id);\n    "
     "return writer.message((uint64_t)id << 24, (uint64_t)id + (1ull << 47), n,"),
    ("const uint64_t id = v[i][0] & ((1ull << 48) - 1);", "const uint64_t id = (v[i][0] & ((1ull << 48) - 1)) >> 24;"),
    ("stream.enqueue([=, this] { block(&ring, from, g); });", "stream.enqueue([=, this] { block(&ring, from, g, n > kRingNarrowMax); });"),
    ("  if (n == 1) return full();\n  if (n == 2) return shared(atoi(a[1]));\n", "  long_every = atoi(a[5]);\n"),
    ('printf("early %d left %d unordered %d repeated %d\\n", early.load(), left, unordered, repeated);',
     'printf("early %d left %d unordered %d repeated %d unfit %d\\n", early.load(), left, unordered, repeated, unfit.load());'),
]


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs a C++ compiler")
    text = MODEL
    for a, b in CHANGES:
        assert text.count(a) == 1, a
        text = text.replace(a, b)
    d = tmp_path_factory.mktemp("ring")
    (d / "model.cc").write_text(text)
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-I", str(CUDA), "-o", str(d / "model"), str(d / "model.cc"), "-lpthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return lambda *a: subprocess.run([str(d / "model")] + [str(x) for x in a], capture_output=True, text=True, timeout=120)


@pytest.mark.parametrize("before,behind,length,rounds,long_every", [(3, 40, 50, 300, 1), (40, 40, 50, 200, 2), (64, 64, 20, 200, 17), (0, 700, 100, 40, 300)])
def test_short_and_long_messages(model, before, behind, length, rounds, long_every):
    r = model(before, behind, length, rounds, long_every)
    assert r.returncode == 0 and r.stdout == "early 0 left 0 unordered 0 repeated 0 unfit 0\n", r.stdout + r.stderr
