// One bounded wait of a warp (mbar_wait_bounded) whose lanes have different limits, on an mbarrier that the other
// warp completes after `arrive_ns` (0: never).  ok[lane]: what each lane got.  Every loop ends by itself.
#include "common.cuh"

__global__ void k_wait_probe(unsigned long long limit, unsigned long long step, unsigned long long arrive_ns, int *ok) {
  __shared__ __align__(8) uint64_t bar;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) cube::mbar_init(&bar, 1);
  __syncthreads();
  if (threadIdx.x < 32) {
    ok[lane] = cube::mbar_wait_bounded(&bar, 0u, limit + step * lane) ? 1 : 0;
  } else if (lane == 0 && arrive_ns) {
    const unsigned long long t0 = cube::ns_now();
    for (int i = 0; i < 100000 && cube::ns_now() - t0 < arrive_ns; i++) __nanosleep(200);
    cube::mbar_arrive(&bar);
  }
  __syncthreads();
}

extern "C" int wait_probe(unsigned long long limit, unsigned long long step, unsigned long long arrive_ns, int ok[32]) {
  int *d = nullptr;
  if (cudaMalloc(&d, 32 * sizeof(int)) != cudaSuccess) return 1;
  k_wait_probe<<<1, 64>>>(limit, step, arrive_ns, d);
  const bool good = cudaMemcpy(ok, d, 32 * sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(d);
  return good ? 0 : 1;
}
