"""Helper threads of a download (run_together, csrc/bfx_internal.hpp): where a
thread cannot be started, the parts that run take all of the work, and no
started thread is left unjoined (which would end the process)."""
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parent.parent
PROGRAM = r"""
#include "bfx_internal.hpp"
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <system_error>

static int starts_left;
static std::string failure;

struct Fake {
  std::thread thread;
  template <typename F>
  explicit Fake(F f) {
    if (starts_left-- == 0) {
      if (failure == "bad_alloc") throw std::bad_alloc();
      throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
    }
    thread = std::thread(f);
  }
  Fake(Fake&&) = default;
  void join() { thread.join(); }
};

int main(int, char** argv) {
  starts_left = std::atoi(argv[1]);
  failure = argv[2];
  const bool caller_throws = std::atoi(argv[3]) != 0;
  std::atomic<int> next{0}, done{0}, parts{0};
  const auto work = [&](unsigned t) {
    ++parts;
    if (t == 0U && caller_throws) throw std::runtime_error("caller");
    while (next++ < 1000) ++done;
  };
  const char* caught = "";
  try {
    bfx::run_together<Fake>(4U, work);
  } catch (const std::runtime_error&) {
    caught = " caught";
  }
  std::printf("%d %d%s\n", done.load(), parts.load(), caught);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("run_together")
    (d / "p.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++20", "-Wall", "-Wextra", "-pthread", "-I", str(REPO / "include"),
                    "-I", str(REPO / "bf-new_b200" / "csrc"), "-o", str(d / "p"), str(d / "p.cpp")], check=True)
    return d / "p"


@pytest.mark.parametrize("starts,failure,caller_throws,expect", [
    (99, "", 0, "1000 4"), (0, "bad_alloc", 0, "1000 1"), (2, "bad_alloc", 0, "1000 3"),
    (1, "system_error", 0, "1000 2"), (99, "", 1, "1000 4 caught"), (1, "bad_alloc", 1, "1000 2 caught")])
def test_all_work_is_done_and_all_threads_joined(program, starts, failure, caller_throws, expect):
    out = subprocess.run([program, str(starts), failure, str(caller_throws)], capture_output=True, text=True)
    assert (out.returncode, out.stdout.strip()) == (0, expect)
