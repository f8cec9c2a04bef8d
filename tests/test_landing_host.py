"""The pinned chunks that logits land in, over stand-ins for the CUDA calls."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = next((d for d in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if d and os.path.exists(os.path.join(d, "include", "cuda_runtime.h"))), None)

PROGRAM = r"""
#include "landing.hpp"
#include <cstdio>
#include <cstdlib>
#include <cstring>
static int left = 0, live = 0;  // calls that still work; events and chunks that exist
static cudaError_t one() { return left-- > 0 ? cudaSuccess : cudaErrorMemoryAllocation; }
extern "C" {
cudaError_t cudaMallocHost(void** p, size_t n) { *p = (void*)1; if (auto e = one()) return e; *p = std::malloc(n); live++; return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); live--; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; if (auto x = one()) return x; *e = (cudaEvent_t)std::malloc(1); live++; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); live--; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { if (!e) std::abort(); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { if (!e) std::abort(); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
}
int main() {
    const size_t sizes[] = {1, oxrt::Landing::kBytes, oxrt::Landing::kBytes + 1, 3 * oxrt::Landing::kBytes - 2};
    for (int works = 0; works <= 3; works++) {
        {
            oxrt::Landing l;
            left = works;
            if ((l.open() == cudaSuccess) != (works == 3)) return 1;
            left = 100;
            for (size_t n : sizes) {  // whatever failed is made now
                uint8_t *from = (uint8_t*)std::malloc(n), *to = (uint8_t*)std::calloc(n, 1);
                for (size_t i = 0; i < n; i++) from[i] = (uint8_t)(i * 7 + i / 1000 + 1);
                if (l.land(from, n, 0, [&](size_t at, const uint8_t* p, size_t m) { std::memcpy(to + at, p, m); })) return 2;
                if (std::memcmp(from, to, n)) return 3;
                std::free(from);
                std::free(to);
            }
        }
        if (live) return 4;
    }
    return 0;
}
"""


@pytest.mark.skipif(CUDA is None or shutil.which("g++") is None, reason="needs g++ and CUDA's headers")
def test_chunks_and_events_that_could_not_be_made_are_made_the_next_time(tmp_path):
    source, program = tmp_path / "landing.cpp", tmp_path / "landing"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "onyxia_b200", "csrc", "backend"), "-I", os.path.join(CUDA, "include"), str(source), "-o", str(program)], check=True)
    assert subprocess.run([str(program)]).returncode == 0
