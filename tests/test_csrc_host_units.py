"""Parts of the CUDA sources that are plain C++, compiled and run on the host."""
import glob
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'twinkle_b200', 'ops', 'csrc')
pytestmark = pytest.mark.skipif(shutil.which('g++') is None, reason='needs g++')


def run_cpp(tmp_path, source):
    (tmp_path / 'unit.cpp').write_text(source)
    subprocess.run(['g++', '-std=c++17', '-O1', '-Wall', '-Werror', '-pthread', '-I', CSRC, 'unit.cpp', '-o', 'unit'], cwd=tmp_path, check=True, capture_output=True, text=True, timeout=120)
    return subprocess.run(['./unit'], cwd=tmp_path, check=True, capture_output=True, text=True, timeout=60).stdout


def test_a_producer_that_gives_up_waits_for_every_fill_under_way_and_for_no_other(tmp_path):
    """Barriers as hardware has them: a wait on a parity passes unless the phase in progress has it.  For every number of fills issued and landed (in
    order), the waits of the give-up path pass exactly when the last fill of each stage has landed."""
    out = run_cpp(tmp_path, r'''
#include <cstdio>
#include <vector>
#include "ring.h"
int main() {
  int bad = 0, checked = 0;
  for (int stages = 1; stages <= 5; ++stages)
    for (int issued = 0; issued <= 4 * stages; ++issued)
      for (int landed = tk::ring_first_open(issued, stages); landed <= issued; ++landed) {
        std::vector<int> phases(stages, 0);              // completed phases of each stage's barrier
        for (int i = 0; i < landed; ++i) ++phases[i % stages];
        bool done = true;
        for (int i = tk::ring_first_open(issued, stages); i < issued; ++i) {
          const tk::RingFill f = tk::ring_fill(i, stages);
          const bool passes = (phases[f.stage] & 1u) != f.parity;
          if (passes != (i < landed)) ++bad;
          done = done && passes;
        }
        if (done != (landed == issued)) ++bad;
        ++checked;
      }
  std::printf("%d %d", bad, checked);
}
''')
    bad, checked = map(int, out.split())
    assert bad == 0 and checked > 100


def test_set_up_of_a_device_runs_on_each_device_once_and_again_after_a_failure(tmp_path):
    out = run_cpp(tmp_path, r'''
#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>
#include "once_per_device.h"
int main() {
  tk::OncePerDevice once;
  std::atomic<int> calls[70] = {};
  for (int round = 0; round < 3; ++round)
    for (int d : {0, 1, 5, 63}) once(d, [&] { ++calls[d]; });
  try { once(2, [] { throw std::runtime_error("x"); }); } catch (const std::exception&) {}
  once(2, [&] { ++calls[2]; });
  once(69, [&] { ++calls[69]; });
  once(69, [&] { ++calls[69]; });
  std::vector<std::thread> ts;
  std::atomic<int> ready{0}, late{0};
  for (int t = 0; t < 8; ++t) ts.emplace_back([&] {
    once(7, [&] { ++ready; });
    if (ready == 0) ++late;          // nobody goes on before the device is set up
  });
  for (auto& t : ts) t.join();
  std::printf("%d %d %d %d %d %d %d", calls[0].load(), calls[1].load(), calls[5].load(), calls[63].load(), calls[2].load(), calls[69].load(), late.load());
}
''')
    assert out.split() == ['1', '1', '1', '1', '1', '2', '0']


def test_no_kernel_attribute_is_set_once_per_process():
    """The limit belongs to a device: behind a flag of the process the kernel fails to launch on the second one."""
    flag = re.compile(r'static\s+(?:bool|int|size_t)\s+\w+(?:\[\d+\])?\s*(?:=[^;]*)?;(?:(?!\n}).){0,600}?cudaFuncSetAttribute', re.S)
    for f in sorted(glob.glob(os.path.join(CSRC, '*.cu'))):
        with open(f) as fh:
            found = flag.search(fh.read())
        assert found is None, (os.path.basename(f), found.group(0)[:120])
