"""A call that fails leaves none of its work on the device: its arena belongs to
the next call, which writes it from two streams."""
import os
import shutil
import subprocess

import pytest

import oracle_py as O
import subgraphmatchgpu_b200 as sme
from conftest import ROOT

# the guard of engine.h against a runtime that only notes what is waited for
GUARD_SRC = r"""
#include <cstdio>
#include <cstdint>
#include "engine.h"
extern "C" cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::printf("%d ", (int)(uintptr_t)s);
  return cudaSuccess;
}
namespace sme { DeviceContext::~DeviceContext() {} }
int main() {
  sme::DeviceContext c;
  c.stream = (cudaStream_t)(uintptr_t)1;
  c.copy_stream = (cudaStream_t)(uintptr_t)2;
  try {
    sme::QuiesceOnError q(c);
    throw 1;
  } catch (int) {
    std::printf("caught ");
  }
  { sme::QuiesceOnError q(c); q.done = true; }
  std::printf("end\n");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_both_streams_are_waited_for_before_the_handler_runs(tmp_path):
    src, exe = tmp_path / "guard.cpp", tmp_path / "guard"
    src.write_text(GUARD_SRC)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    csrc = os.path.join(ROOT, "subgraphmatchgpu_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-I", csrc, "-I", f"{cuda}/include", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60, check=True)
    assert r.stdout.split() == ["1", "2", "caught", "end"]


@pytest.mark.gpu
@pytest.mark.parametrize("query", [1, 3])
def test_a_packed_upload_after_a_call_that_ran_out_of_memory(query):
    # both in one arena (a budget of its own would be another context)
    budget = 1 << 20
    big, small = sme.Graph.rmat(14, 8, seed=2), sme.Graph.rmat(8, 4, seed=3)
    small.pack()
    big.to_device(0)
    rp, cl = small.csr()
    want = O.count(rp, cl, query)
    for _ in range(8):
        with pytest.raises(sme.SmeError) as e:
            big.count(query, mem_limit_bytes=budget)
        assert e.value.status == 3  # no room for a level's batch, the ones before it are running
        assert small.count(query, mem_limit_bytes=budget) == want


@pytest.mark.gpu
def test_failed_external_calls_leave_the_arena_as_it_was():
    # each of them asks for a list cache that the budget cannot hold, after
    # taking 32 KB for the offsets
    budget = 1 << 20
    big, small = sme.Graph.rmat(12, 8, seed=2), sme.Graph.rmat(8, 4, seed=3)
    rp, cl = small.csr()
    want = O.count(rp, cl, 3)
    for _ in range(40):
        with pytest.raises(sme.SmeError) as e:
            big.count(3, mode=sme.EXTERNAL_GPU, mem_limit_bytes=budget)
        assert e.value.status == 3
    assert small.count(3, mem_limit_bytes=budget) == want
