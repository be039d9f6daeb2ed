"""What the launchers set once per GPU: against a fake of the CUDA runtime's calls, on the CPU (a second GPU gets its kernel attributes,
failures are not remembered, threads go on only behind a success); no launcher keeps such a thing once per process; and, where there
are two GPUs, a layer on each of them in one process."""
import glob
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gfx1151_engine_b200", "csrc")

PROGRAM = r"""
#include "per_device.h"
#include <cassert>
#include <thread>
#include <vector>
static thread_local int current = 0;
static int lookups = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = current; return current < 0 ? cudaErrorNoDevice : cudaSuccess; }
extern "C" cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr, int dev) { lookups++; *v = 100 + dev; return cudaSuccess; }
int main() {
  using namespace b200moe;
  OncePerDevice once;
  int calls[70] = {};
  auto set = [&] { calls[current]++; return cudaSuccess; };
  for (int round = 0; round < 3; round++)
    for (current = 0; current < 70; current++) assert(once(set) == cudaSuccess);
  for (int d = 0; d < 70; d++) assert(calls[d] == (d < kPerDeviceMax ? 1 : 3));
  OncePerDevice fails;
  current = 5;
  int tries = 0;
  assert(fails([&] { return ++tries, cudaErrorInvalidValue; }) == cudaErrorInvalidValue);
  assert(fails([&] { return ++tries, cudaSuccess; }) == cudaSuccess);
  assert(fails([&] { return ++tries, cudaSuccess; }) == cudaSuccess && tries == 2);
  current = -1;
  assert(fails([&] { return ++tries, cudaSuccess; }) == cudaErrorNoDevice && tries == 2);
  OncePerDevice shared;
  std::atomic<int> done{0}, early{0};
  std::vector<std::thread> threads;
  for (int i = 0; i < 8; i++)
    threads.emplace_back([&] {
      current = 3;
      assert(shared([&] { std::this_thread::yield(); done++; return cudaSuccess; }) == cudaSuccess);
      if (done.load() == 0) early++;
    });
  for (auto& t : threads) t.join();
  assert(early == 0 && done >= 1);
  int sms = 0;
  for (int round = 0; round < 2; round++)
    for (current = 0; current < 4; current++) assert(sm_count(&sms) == cudaSuccess && sms == 100 + current);
  assert(lookups == 4);
  return 0;
}
"""


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-pthread", "-I" + CSRC, "-I" + cuda + "/include", str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)


def test_launchers_keep_nothing_per_process():
    """Every attribute is set through OncePerDevice, or per handle (router_plan_create); no static flags or SM counts."""
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = open(path).read()
        assert not re.search(r"static (bool|int|size_t) \w+ = (false|0);", text), path
        for m in re.finditer("cudaFuncSetAttribute", text):
            before = text[max(0, m.start() - 900):m.start()]
            assert "once([]" in before[-120:] or "cudaError_t router_plan_create" in before, (path, text[m.start() - 80:m.start() + 60])


@pytest.mark.gpu
def test_two_gpus_in_one_process(cuda):
    torch = cuda
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    from gfx1151_engine_b200 import synth
    from test_gpu_parity import make_op
    d, T = 512, 200
    spec = synth.LayerSpec(experts=16, topk=4, d=d, mid=256)
    layer = synth.make_layer(spec, seed=71)
    xs, lg = torch.randn(T, d).bfloat16(), torch.from_numpy(synth.make_logits(synth.rng_for(71, 1), T, 16))
    got = []
    for dev in (0, 1):
        with torch.cuda.device(dev):
            op = make_op(torch, spec, T, layer=layer, device=dev)
            outs = []
            for n in (5, 40, T):  # decode GEMV, tiles of few rows, all forms
                out = torch.empty(n, d, dtype=torch.bfloat16, device="cuda")
                op.moe_b(0, xs[:n].cuda(), lg[:n].contiguous().cuda(), out)
                op.synchronize()
                outs.append(out.cpu())
            op.close()
        got.append(outs)
    assert all(torch.equal(a, b) for a, b in zip(*got))
