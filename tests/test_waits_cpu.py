"""Bounded waits inside warps (csrc/waits.cuh), by reading the kernels' sources.
Around an expiry the lanes of a warp can come to different verdicts on one wait,
and a barrier, vote or shuffle of the whole warp then waits for a lane that has
left the loop.  So a wait by a thread (tc_wait) is called only
  - by one thread of a warp;
  - or where a lane without what it waited for exits, which takes it out of the
    barriers that follow;
  - or in a loop without anything that waits for the other lanes."""
import glob
import os
import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "idash2019_2_gb300", "csrc")
WARP_WIDE = r"_sync\(|__syncwarp|__syncthreads|tc_warp_wait|tc_team_|load_rows\(|load_rotated<"


def _code(path):
    return re.sub(r"//[^\n]*|\"(\\.|[^\"\\\n])*\"", "", open(path).read())


def _close(text, at, opening, closing):
    """Position after the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == opening) - (text[i] == closing)
        if depth == 0:
            return i + 1
    raise AssertionError("unbalanced")


def _blocks_around(text, at):
    """(header, body) of the braces open at position `at`, outermost first."""
    stack = []
    for i, ch in enumerate(text[:at]):
        if ch == "{":
            stack.append(i)
        elif ch == "}":
            stack.pop()
    headers = []
    for i in stack:
        j = i - 1  # back to the end of the statement before the header; `for (;;)` has some inside
        depth = 0
        while j >= 0 and not (depth == 0 and text[j] in ";{}"):
            depth += (text[j] == ")") - (text[j] == "(")
            j -= 1
        headers.append((text[j + 1:i].strip(), text[i:_close(text, i, "{", "}")]))
    return headers


def _exits(text, at):
    """Whether the `if` whose condition holds position `at` ends the thread."""
    start = max(text.rfind(c, 0, at) for c in ";{}") + 1
    head = re.match(r"\s*(?:else\s+)?if \(", text[start:])
    if not head:
        return False
    after = text[_close(text, start + head.end() - 1, "(", ")"):].lstrip()
    return bool(re.match(r"return;|\{[^{}]*\breturn;\s*\}", after))


def _alone(text, at):
    blocks = _blocks_around(text, at)
    if any(re.search(r"if \(lane == 0\)$", h) for h, _ in blocks) or _exits(text, at):
        return True
    loops = [body for h, body in blocks if re.search(r"\bfor \(", h)]
    return bool(loops) and not re.search(WARP_WIDE, loops[0])


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_no_lane_is_waited_for_after_it_gave_up(path):
    text = _code(path)
    for m in re.finditer(r"\btc_wait\(", text):
        assert _alone(text, m.start()), (path, text[max(0, m.start() - 80):m.end() + 80])


@pytest.mark.parametrize("name", ["score_tc.cu", "key_product.cu", "intpoly.cu"])
def test_copies_in_flight_land_on_every_way_out(name):
    """A role's wait for its own copies (the one that reports no error) does not
    depend on its verdict: other roles may give up after it has issued all."""
    text = _code(os.path.join(CSRC, name))
    for m in re.finditer(r"\bmbar_wait_bounded\([^;]*nullptr\);", text):
        for header, _ in _blocks_around(text, m.start()):
            assert not re.search(r"if \(.*!\s*ok\b", header), (name, header)


LIMITS = """#include <cstdint>
#define __device__
#define __forceinline__ inline
static long long now, done;  // the clock, and when the phase completes
inline long long clock64() { return now; }
inline uint32_t __shfl_sync(uint32_t, uint32_t v, int) { return v; }
namespace idash {
constexpr long long kWaitLimitCycles = 2000000000ll;
constexpr uint32_t kDevTimeout = 2;
inline void report_error(uint32_t *err, uint32_t code) { *err = code; }
inline bool mbar_try_wait(uint64_t *, uint32_t) { return now >= done; }
inline bool mbar_try_wait_sleep(uint64_t *, uint32_t, uint32_t) { now += 40000; return now >= done; }
}
#include "waits.cuh"
using namespace idash;
int main() {
    // a phase after three seconds: late for a hand-off, in time for 2^20 steps
    for (int grown = 0; grown < 2; ++grown) {
        uint32_t abort = 0, err = 0;
        uint64_t bar = 0;
        now = 0;
        done = 6000000000ll;
        const long long limit = kWaitLimitCycles + (grown ? (1ll << 20) * (1 << 14) : 0);
        if (tc_wait(&abort, &bar, 0, &err, limit) != (grown == 1) || err != (grown ? 0u : kDevTimeout)) return 1;
    }
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_a_groups_sums_are_waited_for_as_long_as_the_group(tmp_path):
    """The wait for an integer-polynomial group's sums lasts as long as its row
    steps (up to 2^20): its limit grows with them."""
    shutil.copy(os.path.join(CSRC, "waits.cuh"), tmp_path / "waits.cuh")
    (tmp_path / "common.cuh").write_text("#pragma once\n")
    (tmp_path / "main.cpp").write_text(LIMITS)
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-o", str(tmp_path / "limits"), str(tmp_path / "main.cpp")],
                   check=True)
    assert subprocess.run([str(tmp_path / "limits")], timeout=60).returncode == 0
    text = _code(os.path.join(CSRC, "intpoly.cu"))
    assert re.search(r"limit\s*=\s*kWaitLimitCycles \+ \(polls \? [^;]*kStepLimitCycles", text)
    assert re.search(r"sh\.sums_full, turn & 1u, a\.err, limit\)", text)
