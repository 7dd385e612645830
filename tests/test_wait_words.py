"""The host's book of waits that ran out (csrc/waits.cuh), with the devices played by the host: every device's lost wait is told, once."""
import pathlib
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "nano-qwen3tts-vllm_b200" / "csrc"
MAIN = r"""
#include <cstdio>
#include "waits.cuh"
using namespace b2;
int main() {
  static int words[WAIT_DEVICES * WAITS_KINDS], counter[100][WAITS_KINDS], told[WAITS_KINDS];
  auto lose = [&](int device, int kind) { words[wait_slot(device, kind)] = ++counter[device][kind]; };     // as a kernel does
  auto ask = [&](int kind) { std::printf("%d", wait_moved(words, kind, &told[kind])); };
  ask(0); ask(1);
  lose(0, 1); ask(0); ask(1); ask(1);
  lose(1, 1); ask(1); ask(1);                         // another device's first
  lose(1, 0); lose(0, 0); ask(0); ask(0); ask(1);
  lose(63, 1); ask(1); lose(0, 1); ask(1); ask(1);
  std::printf(" %d %d %d\n", wait_total(words, 0), wait_total(words, 1), wait_slot(99, 1) == wait_slot(63, 1));
}
"""


def test_every_device_is_heard(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run([cxx, "-std=c++17", "-I", str(CSRC), str(tmp_path / "main.cpp"), "-o", str(tmp_path / "main")], check=True)
    assert subprocess.run([str(tmp_path / "main")], check=True, capture_output=True, text=True).stdout.split() == ["00" "010" "10" "100" "110", "2", "4", "1"]
