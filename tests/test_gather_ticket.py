"""The host's record of the gather's work counter (gp_ticket.h), compiled for the host: the
counter, which a gather uses up and its integrate takes back to zero, is zero at the start of
every gather, also of one that follows a gather whose integrate an error kept away."""
from __future__ import annotations

import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gazpart_b200", "csrc")

# g: gather; i: integrate; x: an error, nothing enqueued; r: a graph captured earlier (one
# gather and its integrate), for which the host only looks before the launch
PROGRAM = r"""
#include <cstdio>
#include "gp_ticket.h"
int main(int, char **argv) {
  gp::GatherTicket t;
  int counter = 0, gathers = 0;
  for (const char *p = argv[1]; *p; ++p) {
    if (*p == 'g') {
      if (t.take()) counter = 0;
      if (counter != 0) return 1;
      counter = 1;
      ++gathers;
    } else if (*p == 'i') {
      counter = 0;
      t.paired();
    } else if (*p == 'r') {
      if (t.stale()) { counter = 0; t.paired(); }
      if (counter != 0) return 1;
      ++gathers;
    }
  }
  std::printf("%d\n", gathers);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("ticket")
    src, exe = d / "ticket.cpp", d / "ticket"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    return str(exe)


@pytest.mark.parametrize("calls", ["gigigi", "gxgi", "gxgxgigi", "gxr", "rrgir", "gigxrgi", "gxrgxgir"])
def test_every_gather_finds_the_counter_clear(program, calls):
    run = subprocess.run([program, calls], capture_output=True, text=True)
    assert run.returncode == 0, calls
    assert int(run.stdout) == calls.count("g") + calls.count("r")
