// mod_once and fast_mod on the device, with make_div_magic's constants, for
// test_gpu_mod.py.  Standard input: divisors, each behind its number of
// dividends and followed by them (64-bit words); output: the two remainders
// of each.
#include <cstdio>
#include <vector>

#include "k2g_device.cuh"
#include "k2g_internal.h"

using namespace k2g;

__global__ void mods(const uint64_t *n, uint64_t *out, uint64_t count, DivMagic m) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= count) return;
  out[2 * i] = mod_once(n[i], m);
  out[2 * i + 1] = fast_mod(n[i], m);
}

int main() {
  uint64_t head[2];
  while (fread(head, 8, 2, stdin) == 2) {
    std::vector<uint64_t> n(head[0]), out(2 * head[0]);
    if (fread(n.data(), 8, n.size(), stdin) != n.size()) return 1;
    uint64_t *d_n = nullptr, *d_out = nullptr;
    if (cudaMalloc(&d_n, n.size() * 8) != cudaSuccess || cudaMalloc(&d_out, out.size() * 8) != cudaSuccess) return 2;
    cudaMemcpy(d_n, n.data(), n.size() * 8, cudaMemcpyHostToDevice);
    mods<<<(unsigned)((n.size() + 255) / 256), 256>>>(d_n, d_out, n.size(), make_div_magic(head[1]));
    if (cudaMemcpy(out.data(), d_out, out.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    cudaFree(d_n);
    cudaFree(d_out);
    fwrite(out.data(), 8, out.size(), stdout);
  }
  return 0;
}
