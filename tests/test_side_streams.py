"""Side streams of a launch (csrc/side_streams.hpp) against a fake of the stream
calls: a launch that fails between fork and join leaves no side stream that
neither the main stream nor the host waits for."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "bf-new_b200" / "csrc"
PROGRAM = r"""
#include "side_streams.hpp"
#include <cstdio>
#include <cstdlib>
#include <stdexcept>
#include <string>

static int calls_left;  // the call that fails, counted down
static std::string log_;

struct Fake {
  using Stream = int;
  using Event = int;
  static void call(const char* what, int a, int b) {
    if (calls_left-- == 0) throw std::runtime_error(what);
    log_ += std::string(what) + std::to_string(a) + "," + std::to_string(b) + " ";
  }
  static void record(Event e, Stream s) { call("r", e, s); }
  static void wait(Stream s, Event e) { call("w", s, e); }
  static void synchronize(Stream s) noexcept { log_ += "s" + std::to_string(s) + " "; }
};

int main(int, char** argv) {
  calls_left = std::atoi(argv[1]);
  const bool launch_fails = std::atoi(argv[2]) != 0;
  const std::size_t count = std::atoi(argv[3]);
  const bfx::SideStreams<Fake>::Side sides[] = {{1, 11}, {2, 12}, {3, 13}};
  try {
    bfx::SideStreams<Fake> s(0, 10, sides, count);
    log_ += "| ";
    if (launch_fails) throw std::runtime_error("launch");
    s.join();
  } catch (const std::runtime_error& e) {
    log_ += std::string("!") + e.what();
  }
  std::puts(log_.c_str());
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("side_streams")
    (d / "p.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-I", str(CSRC), "-o", str(d / "p"), str(d / "p.cpp")],
                   check=True)
    return d / "p"


@pytest.mark.parametrize("fails_at,launch_fails,count,expect", [
    (99, 0, 3, "r10,0 w1,10 w2,10 w3,10 | r11,1 w0,11 r12,2 w0,12 r13,3 w0,13"),
    (99, 0, 0, "|"),
    (99, 1, 3, "r10,0 w1,10 w2,10 w3,10 | s1 s2 s3 !launch"),
    (99, 1, 0, "| !launch"),
    (2, 0, 3, "r10,0 w1,10 !w"),  # no launch was made yet
    (4, 0, 3, "r10,0 w1,10 w2,10 w3,10 | s1 s2 s3 !r"),
    (7, 0, 3, "r10,0 w1,10 w2,10 w3,10 | r11,1 w0,11 r12,2 s2 s3 !w"),
])
def test_every_side_is_waited_for(program, fails_at, launch_fails, count, expect):
    out = subprocess.run([program, str(fails_at), str(launch_fails), str(count)], capture_output=True, text=True,
                         check=True).stdout
    assert out.strip() == expect
