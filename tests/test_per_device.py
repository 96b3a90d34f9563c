"""Kernel attributes are set on every device that a process uses (``csrc/dqb_per_device.cuh``,
compiled by the host compiler), and nowhere once per process."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, 'dynamiqs_b200', 'csrc')

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "dqb_per_device.cuh"

int main() {
  dqb::PerDevice once;
  int runs[3] = {0, 0, 0};
  bool ok = true;
  for (int pass = 0; pass < 2; ++pass)
    for (int dev = 0; dev < 2; ++dev) ok = once.run(dev, [&] { return ++runs[dev] > 0; }) && ok;
  ok = ok && runs[0] == 1 && runs[1] == 1;                        // each device, once
  ok = ok && !once.run(2, [&] { return ++runs[2] > 1; });         // a failure is told
  ok = ok && once.run(2, [&] { return ++runs[2] > 1; }) && runs[2] == 2;  // and tried again
  ok = ok && !once.run(-1, [] { return true; }) && !once.run(dqb::PerDevice::kMax, [] { return true; });
  dqb::PerDevice shared;
  int count = 0;
  std::vector<std::thread> threads;
  for (int i = 0; i < 8; ++i) threads.emplace_back([&] { shared.run(5, [&] { return ++count > 0; }); });
  for (auto& t : threads) t.join();
  ok = ok && count == 1;
  std::puts(ok ? "ok" : "failed");
}
"""


def test_set_up_runs_once_on_each_device(tmp_path):
    (tmp_path / 'main.cpp').write_text(PROGRAM)
    subprocess.run(['g++', '-O1', '-std=c++17', '-pthread', '-I', CSRC, 'main.cpp', '-o', 'main'], cwd=tmp_path,
                   check=True)
    out = subprocess.run([str(tmp_path / 'main')], check=True, capture_output=True, text=True, timeout=60)
    assert out.stdout.strip() == 'ok'


def test_no_set_up_once_per_process():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(('.cu', '.cuh')):
            with open(os.path.join(CSRC, name)) as f:
                assert 'call_once' not in f.read(), name
