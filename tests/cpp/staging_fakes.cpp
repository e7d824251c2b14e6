// The staging of small results (scx_b200/csrc/staging.h) on the CPU, over
// fakes of the CUDA calls it makes: copies land when they are enqueued, and
// page-locked memory is refused after the first requests.  Each size given is
// fetched through one buffer; the program prints whether every result came
// back, what was asked for and what is kept.
//
// Usage: staging_fakes <requests granted> <size> ...
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "staging.h"

static int granted = 0, asked = 0, freed = 0, waits = 0;
static cudaError_t last = cudaSuccess;

extern "C" {
cudaError_t CUDARTAPI cudaHostAlloc(void** p, size_t n, unsigned) {
  if (asked++ >= granted) return last = cudaErrorMemoryAllocation;
  *p = malloc(n);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaFreeHost(void* p) {
  ++freed;
  free(p);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t) {
  ++waits;
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaGetLastError(void) {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
}

int main(int argc, char** argv) {
  granted = std::stoi(argv[1]);
  bool same = true;
  for (int i = 2; i < argc; ++i) {
    const size_t n = std::stoul(argv[i]);
    std::vector<char> src(n);
    for (size_t b = 0; b < n; ++b) src[b] = (char)(b * 31 + i);
    scx::Staging h(n, nullptr);
    same &= h.fetch(0, src.data(), n) == cudaSuccess && h.wait() == cudaSuccess;
    same &= memcmp(h.at<char>(0), src.data(), n) == 0;
  }
  {  // a buffer given up before its copies were waited for
    const char c = 1;
    scx::Staging h(1, nullptr);
    (void)h.fetch(0, &c, 1);
  }
  printf("same=%d asked=%d freed=%d waits=%d held=%zu error=%d\n", same, asked, freed, waits, scx::stage_list().held,
         (int)last);
  return 0;
}
