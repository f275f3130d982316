// Kernels' limits of dynamic shared memory (prepare_smem): a call that needs
// less leaves a launch that needs more its room, as two threads' calls
// interleave, and static shared memory counts against the 48 KB that need no
// limit set.
#include <cstdio>

#include "bbs_launch.cuh"

namespace {

__device__ void touch(int *out, int words) {
  extern __shared__ int dynamic[];
  __shared__ int fixed[40];
  fixed[threadIdx.x & 31] = (int)threadIdx.x;
  for (int i = threadIdx.x; i < words; i += blockDim.x) dynamic[i] = i;
  __syncthreads();
  if (threadIdx.x == 0) *out = dynamic[words - 1] + fixed[0];
}

__global__ void first(int *out, int words) { touch(out, words); }
__global__ void second(int *out, int words) { touch(out, words); }

template <typename K>
bool runs(K kernel, int *d, int bytes) {
  kernel<<<1, 32, bytes>>>(d, bytes / 4);
  if (cudaGetLastError() != cudaSuccess) return false;
  int got = 0;
  return cudaMemcpy(&got, d, sizeof(int), cudaMemcpyDeviceToHost) ==
             cudaSuccess && got == bytes / 4 - 1;
}

}  // namespace

int main() {
  int *d;
  if (cudaMalloc(&d, sizeof(int)) != cudaSuccess) return 2;
  bool ok = true;
  for (int bytes = 48 * 1024 - 512; bytes <= 48 * 1024 + 64; bytes += 16)
    if (bbs::prepare_smem(first, bytes) != cudaSuccess || !runs(first, d, bytes)) {
      std::printf("FAIL %d bytes and static ones\n", bytes);
      ok = false;
    }
  if (bbs::prepare_smem(second, 59136) != cudaSuccess ||
      bbs::prepare_smem(second, 56544) != cudaSuccess ||
      !runs(second, d, 59136)) {
    std::printf("FAIL 59136 bytes after another call's 56544\n");
    ok = false;
  }
  if (bbs::prepare_smem(second, 240 * 1024) == cudaSuccess) {
    std::printf("FAIL 240 KB accepted\n");
    ok = false;
  }
  if (ok) std::printf("limits ok\n");
  return ok ? 0 : 1;
}
