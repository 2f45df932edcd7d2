"""What the launchers of the torch extension remember between calls is atomic and kept per device (csrc/torch/device_state.h)."""
import re
import subprocess
from pathlib import Path

import pytest

TORCH = Path(__file__).resolve().parent.parent / "csrc" / "torch"


@pytest.mark.parametrize("path", sorted(p for p in TORCH.iterdir() if p.suffix in (".cu", ".cuh", ".cpp", ".h")), ids=lambda p: p.name)
def test_no_plain_static_variable_inside_a_function(path):
    """Allowed: constants (initialised once, by the language's rules), atomics, OncePerDevice.  Not allowed: a flag or count that
    two threads may write, nor one per thread (a thread that changes devices would skip the second one's set-up); the one
    exception is the context binding, which is a matter of the thread."""
    text = path.read_text()
    bad = [line.strip() for line in re.findall(r"^[ \t]+static [^()\n]*[;=][^\n]*$", text, re.M)
           if not re.match(r"\s*static (const |constexpr |std::atomic<|fcxhost::OncePerDevice |thread_local bool bound)", line)]
    assert not bad, bad


def test_kernels_share_no_memory_of_the_library_image():
    """A __device__ array is one for all launches on a device: two streams that use it at a time take each other's values.  The
    one exception is the scratch of the entry point whose contract says so (train_ops_noalloc.h)."""
    bad = []
    for path in TORCH.glob("*.cu*"):
        bad += [(path.name, line) for line in re.findall(r"^(?:static )?__device__ (?:__align__\(\d+\) )?[^()\n]*;.*$", path.read_text(), re.M)]
    assert [b for b in bad if "gNoAllocScratch" not in b[1]] == []


PROGRAM = r"""
#include "device_state.h"
#include <cstdio>
#include <thread>
#include <vector>
static thread_local int current = 0;
static std::atomic<int> lookups{0};
extern "C" cudaError_t cudaGetDevice(int *d) { *d = current; return current < 0 ? cudaErrorNoDevice : cudaSuccess; }
extern "C" cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int d) { lookups++; *v = 100 + d; return cudaSuccess; }
int main() {
  static fcxhost::OncePerDevice once, failing;
  std::atomic<int> runs[70] = {}, wrong{0};
  std::vector<std::thread> ts;
  for (int t = 0; t < 8; t++)
    ts.emplace_back([&, t] {
      for (int i = 0; i < 2000; i++) {
        current = (i + t) % 70;  // every thread goes through all devices
        if (fcxhost::smCount() != 100 + current) wrong++;
        if (once([&] { runs[current]++; return cudaSuccess; }) != cudaSuccess) wrong++;
        if (failing([] { return cudaErrorInvalidValue; }) != cudaErrorInvalidValue) wrong++;  // tried again, reported again
      }
    });
  for (auto &t : ts) t.join();
  for (int d = 0; d < 70; d++) {
    if (runs[d] < 1) wrong++;
    if (d < fcxhost::MAX_DEVICES && runs[d] > 8) wrong++;  // at most once per thread that came first at the same time
  }
  std::printf("%d\n", wrong.load());
  return wrong != 0;
}
"""


def test_device_state_with_many_threads_and_devices(tmp_path):
    src, exe = tmp_path / "state.cc", tmp_path / "state"
    src.write_text(PROGRAM)
    cmd = ["g++", "-O1", "-g", "-std=c++17", "-fsanitize=thread", f"-I{TORCH}", "-I/usr/local/cuda/include", str(src), "-o", str(exe), "-pthread"]
    subprocess.run(cmd, check=True, capture_output=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    if "unexpected memory mapping" in run.stderr:
        pytest.skip("the thread sanitizer does not run under this kernel's address layout")
    assert run.returncode == 0 and "WARNING: ThreadSanitizer" not in run.stderr, run.stdout + run.stderr[-2000:]
