"""The tables of the streaming kernels hold an entry per device; a thread keeps a
reference to its own while another thread adds one for a new device."""

from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "per_device.cuh"
#include <atomic>
#include <cstdio>
#include <thread>
struct Entry { int id = 0; std::atomic<int> n{0}; };
int main() {
  topo::PerDevice<Entry> t;
  Entry& a = t.at(0);
  a.id = 7;
  std::thread grow([&] { for (int d = 1; d < 256; ++d) t.at(d).id = d; });
  for (int i = 0; i < 100000; ++i) a.n += a.id;
  grow.join();
  if (&t.at(0) != &a || t.at(0).n != 700000) return 1;
  for (int d = 1; d < 256; ++d)
    if (t.at(d).id != d) return 2;
  std::puts("ok");
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_entries_stay_in_place_while_the_table_grows(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-pthread",
                    "-I", str(ROOT / "topogpu_b200" / "csrc"), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "ok\n"


def test_every_kernel_table_is_of_that_kind():
    for name in ("kmatvec_pt.cu", "kmatvec_xs.cu", "kmatvec_cc.cu"):
        text = (ROOT / "topogpu_b200" / "csrc" / name).read_text()
        assert "PerDevice<" in text, name
        assert ".resize(dev + 1)" not in text, name
