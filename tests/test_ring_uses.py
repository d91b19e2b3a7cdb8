"""The phase of a barrier's last commit, for which a tensor-core kernel's block waits
before it exits: commits go round the barriers one after another."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-orb_b200", "csrc")
SOURCE = r"""
#define __host__
#define __device__
#include "orbx_match_plan.cuh"
#include <initializer_list>
#include <cstdio>
using namespace orbx;
int main() {
  for (unsigned k : {1u, 2u, 3u, 4u, 8u}) {
    unsigned uses[8] = {};
    for (unsigned n = 0; n < 100; n++) {
      for (unsigned i = 0; i < k; i++)
        if (m_ring_uses(n, k, i) != uses[i]) { printf("n %u k %u i %u\n", n, k, i); return 1; }
      uses[n % k]++;
    }
  }
  return 0;
}
"""


def test_uses_of_each_entry(tmp_path):
    src, exe = tmp_path / "ring.cpp", tmp_path / "ring"
    src.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-x", "c++", "-I", CSRC, str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_every_commit_is_waited_for():
    """Each barrier that a kernel commits MMAs to is drained by it before its block
    exits: the ring's "empty" barriers by the producer, the others by the MMA thread."""
    def kernel(name, text):
        at = text.index(name)
        return text[at:text.index("tcgen05.dealloc", at)]

    imma = open(os.path.join(CSRC, "orbx_match_imma.cu")).read()
    gemm = open(os.path.join(CSRC, "orbx_gemm.cu")).read()
    for src, commit, barriers in (
            (kernel("k_match_imma(const __grid", imma), "umma_commit(", ("BAR_BEMPTY", "BAR_ACCFULL", "BAR_AEMPTY")),
            (kernel("k_rerank_imma(RerankImmaArgs", imma), "umma_commit(", ("RR_XEMPTY", "RR_ACCFULL", "RR_AEMPTY")),
            (kernel("k_gemm_bf16(const __grid", gemm), "g_umma_commit(", ("GBAR_EMPTY", "GBAR_ACCFULL"))):
        assert {c.split("(")[0] for c in src.split(commit)[1:]} == set(barriers)
        for b in barriers:
            assert "mbar_drain(" + b + "(" in src or "mbar_try(" + b + "(" in src, b
